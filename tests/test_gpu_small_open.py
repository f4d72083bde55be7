"""FP64 runs of few particles (four lanes a particle) with open boundaries:
what becomes of the particles that have left."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
tp = pytest.importorskip("test_particle_gb300")


def test_departed_particle_reports_nothing():
    """The box reaches beyond the last grid plane in z.  The particle leaves
    through x before it gets there, and a push from where it stopped would
    sample past the plane: the run has to end without a status bit."""
    g = tp.Grids()
    g.nx = g.ny = g.nz = 4
    g.nt = 1
    g.dx = g.dy = g.dz = 1.0
    dom = tp.Domain()
    dom.xmax, dom.ymax, dom.zmax = 3.0, 3.0, 10.0
    dt, steps = 1.0, 150
    dom.tmax = (steps + 0.5) * dt
    b = np.zeros((64, 3), np.float32)
    b[:, 2] = 1e-6  # straight orbits
    tp.configure(system_type=tp.SYS_PIC, dom=dom, grd=g, bgrid=b, egrid=np.zeros_like(b), bc_flag=1)
    tp.set_spectrum(10, 1e-3, 1e2)
    p = np.zeros(3, dtype=tp.PARTICLE_DTYPE)
    p["qm"] = 1.0
    gam = 1.0 / np.sqrt(1.0 - 0.5 ** 2 - 0.5 ** 2)
    p["x"], p["y"], p["z"] = 2.6, 1.5, 2.3
    p["ux"], p["uz"] = 0.5 * gam, 0.5 * gam
    r = tp.track(p, dt, 1, 10, precision=tp.PREC_FP64)
    assert tp.device_status() == 0
    assert (r["ptl"]["x"] > 3.0).all() and (r["ptl"]["z"] < 3.0).all() and (r["nsteps"] == 2).all()


import make_golden as mg  # noqa: E402
import test_particle_gb300.workloads as wl  # noqa: E402

SC = mg.scenarios()
LARGE = 4 * 152 * 32 + 1  # more particles than any small run takes


def _open_box(name):
    if name == "modesum":
        dom = tp.Domain()
        dom.xmax = dom.ymax = dom.zmax = 1.0
        tp.configure(system_type=tp.SYS_MODESUM, dom=dom, bc_flag=1, modes=wl.kolmogorov_modes(37, 1.0, 16.0, 0.5, 3, va=0.1))
        return dom, 0.02
    s = SC[name]
    tp.configure(bc_flag=1, dom=s["dom"], grd=s["grd"], **{k: v for k, v in s.items() if k not in ("dom", "grd")})
    return s["dom"], 2e-5 if name in ("wlcs", "loop") else 0.02


@pytest.mark.parametrize("name", ["test", "abc111", "ff_vel", "mhd", "pic", "pic_mt", "pic_off", "wlcs", "loop", "modesum"])
@pytest.mark.parametrize("outside", ["third", "first", "all but last"])
def test_departed_among_others(name, outside):
    """Groups, warps and blocks in which some, none or all particles have left,
    at the start and on the way: bit for bit the one-lane kernel's run."""
    dom, dt = _open_box(name)
    tp.Domain.in_dll(tp.lib(), "simul_domain").tmax = 400.5 * dt
    nbins, nt_out = 30, 4
    tp.set_spectrum(nbins, 1e-3, 1e2)
    lo = np.array([dom.xmin, dom.ymin, dom.zmin])
    L = np.array([dom.xmax, dom.ymax, dom.zmax]) - lo
    p = wl.shell_particles(LARGE, 0.6, lo + 0.02 * L, lo + 0.98 * L, 5)
    k = np.arange(LARGE)
    p["x"][{"third": k % 3 == 0, "first": k < 100, "all but last": (k % 67 != 66)}[outside]] += 1.01 * L[0]
    one = tp.track(p, dt, nt_out, nbins)
    for n in (1, 9, 67, 300):
        few = tp.track(p[:n], dt, nt_out, nbins)
        assert few["info"].grid == (n + 31) // 32
        assert one["ptl"][:n].tobytes() == few["ptl"].tobytes()
        assert np.array_equal(one["nsteps"][:n], few["nsteps"])
        parts = [tp.track(p[i:i + 1], dt, nt_out, nbins) for i in range(min(n, 9))]
        if n <= 9:
            for key in ("espect", "espect_escape"):
                assert np.array_equal(few[key], sum(r[key] for r in parts)), key
            assert np.array_equal(few["remain"] - n, sum(r["remain"] - 1 for r in parts))
    assert tp.device_status() == 0
