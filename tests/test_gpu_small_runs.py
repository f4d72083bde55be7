"""FP64 runs of few particles (four lanes a particle, csrc/track_small.cuh)
against the same particles inside a run large enough for the one-lane kernel:
bit for bit in the parity precision."""
import numpy as np
import pytest

import make_golden as mg

pytestmark = pytest.mark.gpu
tp = pytest.importorskip("test_particle_gb300")
import test_particle_gb300.workloads as wl  # noqa: E402

SC = mg.scenarios()
LARGE = 4 * 152 * 32 + 1  # more particles than any small run takes


def _configure(name, bc):
    if name == "modesum":
        dom = tp.Domain()
        dom.xmax = dom.ymax = dom.zmax = 1.0
        tp.configure(system_type=tp.SYS_MODESUM, dom=dom, bc_flag=bc, mode_B0=1.0,
                     modes=wl.kolmogorov_modes(37, 1.0, 16.0, 0.5, 3, va=0.1))
        return dom, 0.02
    s = SC[name]
    kw = {k: v for k, v in s.items() if k not in ("dom", "grd")}
    tp.configure(bc_flag=bc, dom=s["dom"], grd=s["grd"], **kw)
    return s["dom"], 2e-5 if name in ("wlcs", "loop") else 0.02


@pytest.mark.parametrize("name,bc", [("test", 0), ("abc111", 0), ("abc111", 1), ("ff_vel", 0), ("mhd", 1), ("pic", 0),
                                     ("wlcs", 2), ("loop", 1), ("modesum", 0), ("modesum", 1)])
@pytest.mark.parametrize("n", [1, 33])
def test_small_matches_large(name, bc, n):
    dom, dt = _configure(name, bc)
    d = tp.Domain.in_dll(tp.lib(), "simul_domain")
    d.tmax = 203.5 * dt
    nbins, nt_out = 40, 3
    tp.set_spectrum(nbins, 1e-3, 1e2)
    lo = np.array([dom.xmin, dom.ymin, dom.zmin])
    L = np.array([dom.xmax, dom.ymax, dom.zmax]) - lo
    p = wl.shell_particles(LARGE, 0.6, lo + 0.02 * L, lo + 0.98 * L, 5)
    one = tp.track(p, dt, nt_out, nbins, precision=tp.PREC_FP64)
    few = tp.track(p[:n], dt, nt_out, nbins, precision=tp.PREC_FP64)
    assert one["ptl"][:n].tobytes() == few["ptl"].tobytes()
    assert np.array_equal(one["nsteps"][:n], few["nsteps"])
    # the counts and sums of n particles against the oracle of one particle at a time
    parts = [tp.track(p[i:i + 1], dt, nt_out, nbins, precision=tp.PREC_FP64) for i in range(n)]
    for k in ("espect", "espect_escape"):
        assert np.array_equal(few[k], sum(r[k] for r in parts)), k
    assert np.array_equal(few["remain"] - n, sum(r["remain"] - 1 for r in parts))
    total = sum(r["dsum"] for r in parts)
    assert np.all(np.abs(few["dsum"] - total) <= n * 2.0 ** -52 * np.abs(total))


@pytest.mark.parametrize("n,off", [(1, 0.0), (9, 0.0), (257, -0.75)])
def test_few_field_lines_match_many(n, off):
    """Field lines of few seeds (four lanes a seed) against the same seeds in a
    map of more than 16,384, and seeds outside the box as the reference wraps them."""
    g = tp.Grids()
    g.nx, g.ny, g.nz, g.nt = 17, 13, 15, 1
    g.dx, g.dy, g.dz = 0.25, 0.3, 0.2
    dom = tp.Domain()
    dom.xmin, dom.ymin, dom.zmin = off, 0.0, 0.0
    dom.xmax, dom.ymax, dom.zmax = off + 16 * 0.25, 12 * 0.3, 14 * 0.2
    rng = np.random.default_rng(11)
    b = (rng.normal(0, 0.4, (17 * 13 * 15, 3)) + [0.0, 0.0, 1.0]).astype(np.float32)
    tp.configure(system_type=tp.SYS_PIC, dom=dom, grd=g, bgrid=b, egrid=np.zeros_like(b))
    seeds = [off, 0.0, 0.0] + rng.random((16385, 3)) * [4.0, 3.6, 2.8]
    seeds[:, 2] = 1.4
    seeds[0] = [off + 5.0, 1.0, 1.4]
    many = tp.poincare_trace(seeds, 2, 0.05, 20.0, 3)
    few = tp.poincare_trace(seeds[:n], 2, 0.05, 20.0, 3)
    for m, w in zip(many, few):
        assert m[:n].tobytes() == w.tobytes()
