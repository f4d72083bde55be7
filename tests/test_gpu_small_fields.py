"""FP64 runs of few particles against the same particles in a run of many, over
the forms of the fields: two time frames, a grid off the origin, values so
small that the filtered sums never hold, particles outside the box, Bessel
wires; bit for bit in the parity precision, to rounding with contraction."""
import numpy as np
import pytest

import make_golden as mg

pytestmark = pytest.mark.gpu
tp = pytest.importorskip("test_particle_gb300")
import test_particle_gb300.workloads as wl  # noqa: E402

SC = mg.scenarios()
LARGE = 4 * 152 * 32 + 1  # more particles than any small run takes


def _case(name):
    """(scenario, bc): the scenarios of the golden files, changed where named so."""
    base, _, form = name.partition(" ")
    if base == "modesum":
        dom = tp.Domain()
        dom.xmax = dom.ymax = dom.zmax = 1.0
        return dict(system_type=tp.SYS_MODESUM, dom=dom, grd=None, modes=wl.kolmogorov_modes(37, 1.0, 16.0, 0.5, 3, va=0.1)), 0
    s = dict(SC["mhd" if base == "mhd_mt" else base])
    if base == "mhd_mt":
        rng = np.random.default_rng(3)
        v, b = s.pop("vgrid_f"), s.pop("bgrid")
        s["vgrid_f_ab"] = (v, (v + rng.normal(0, 0.02, v.shape)).astype(np.float32))
        s["bgrid_ab"] = (b, (b + rng.normal(0, 0.1, b.shape)).astype(np.float32))
        s["mt"] = 1
        s["grd"] = mg.grid_for(s["dom"], (9, 7, 5), nt=3, tmax=4.0)
    if form == "tiny":  # the same orbits: q/m B as before
        for k in ("bgrid", "egrid", "vgrid_f"):
            if k in s and (k != "vgrid_f"):
                s[k] = s[k] * np.float32(2.0 ** -70)
        s["charge_mass"] *= 2.0 ** 70
    if form == "bessel":
        s["ibessel"] = 1
        s["wl"] = [mg.wlcs_rec(0.3, (0.4, 0.5, 0.45), 0.3, 0.7, 0.5, 1.0, 0.25, (0.5, 0.45, 0.5), 0.4, 1.1, 0.001)]
    return s, 2 if form == "outside" else 0


def _configure(name, steps):
    s, bc = _case(name)
    dt = 2e-5 if s["system_type"] == tp.SYS_WLCS else 0.02
    tp.configure(bc_flag=bc, **s)
    dom = s["dom"]
    tp.Domain.in_dll(tp.lib(), "simul_domain").tmax = (steps + 0.5) * dt
    tp.set_spectrum(40, 1e-3, 1e2)
    lo = np.array([dom.xmin, dom.ymin, dom.zmin])
    L = np.array([dom.xmax, dom.ymax, dom.zmax]) - lo
    return wl.shell_particles(LARGE, 0.6, lo + 0.02 * L, lo + 0.98 * L, 5), dt


@pytest.mark.parametrize("name", ["pic_mt", "mhd_mt", "pic_off", "pic tiny", "mhd tiny", "pic outside", "mhd outside",
                                  "pic_mt outside", "wlcs bessel"])
@pytest.mark.parametrize("n", [1, 33])
def test_small_matches_large_bit_for_bit(name, n):
    p, dt = _configure(name, 203)
    one = tp.track(p, dt, 3, 40)
    few = tp.track(p[:n], dt, 3, 40)
    assert few["info"].grid == (n + 31) // 32
    assert np.isfinite(one["ptl"]["ux"]).all()
    assert one["ptl"][:n].tobytes() == few["ptl"].tobytes()
    assert np.array_equal(one["nsteps"][:n], few["nsteps"])
    parts = [tp.track(p[i:i + 1], dt, 3, 40) for i in range(n)]
    assert np.array_equal(few["espect"], sum(r["espect"] for r in parts))
    total = sum(r["dsum"] for r in parts)
    assert np.all(np.abs(few["dsum"] - total) <= n * 2.0 ** -52 * np.abs(total))
    assert tp.device_status() == 0


@pytest.mark.parametrize("name", ["abc111", "mhd", "pic", "pic_mt", "wlcs", "wlcs bessel", "modesum"])
def test_small_matches_large_with_contraction(name):
    """The two kernels contract differently.  A step rounds a coordinate some
    thirty times; over 50 steps of orbits that spread by less than a factor of
    ten in this time the states differ by less than 50 x 30 x 10 units of 2^-53."""
    p, dt = _configure(name, 50)
    one = tp.track(p, dt, 1, 40, precision=tp.PREC_FP64_FAST)
    few = tp.track(p[:300], dt, 1, 40, precision=tp.PREC_FP64_FAST)
    assert few["info"].grid == 10
    for k in ("x", "y", "z", "ux", "uy", "uz"):
        a, b = one["ptl"][k][:300], few["ptl"][k]
        scale = np.abs(one["ptl"][k]).max()
        # (the float grids round a sample to 2^-24: one that falls the other way moves a momentum by that)
        tol = 2.0 ** -24 * 50 * dt if name in ("mhd", "pic", "pic_mt") else 15000 * 2.0 ** -53
        assert np.abs(a - b).max() <= tol * scale, k
    assert np.array_equal(one["nsteps"][:300], few["nsteps"])
