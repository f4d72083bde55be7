"""Open-boundary runs shorter than a diffusion interval (100 steps): the
remaining counts have one entry, and particles that start outside the box are
counted nowhere else.  In the no-allocation call the entry behind it is the
caller's."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
tp = pytest.importorskip("test_particle_gb300")
import test_particle_gb300.workloads as wl  # noqa: E402

STEPS, DT = 40, 0.02


def _setup(system, n, steps=STEPS):
    dom = tp.Domain()
    dom.xmax = dom.ymax = dom.zmax = 1.0
    dom.tmax = (steps + 0.5) * DT
    modes = wl.kolmogorov_modes(8, 1.0, 4.0, 0.3, 3, va=0.1)
    tp.configure(system_type=system, dom=dom, bc_flag=1, abc=(1.0, 1.0, 1.0), lambda0=2 * np.pi, modes=modes)
    tp.set_spectrum(50, 1e-3, 1e2)
    p = wl.shell_particles(n, 0.3, (0.1,) * 3, (0.9,) * 3, 4)
    p["x"][::3] += 1.5  # every third outside
    return p, modes


@pytest.mark.parametrize("system,prec,n", [
    (tp.SYS_FORCEFREE, tp.PREC_FP64, 100),            # four lanes a particle
    (tp.SYS_FORCEFREE, tp.PREC_FP64, 3 * 152 * 32 + 1),
    (tp.SYS_FORCEFREE, tp.PREC_FP64_FAST, 100),
    (tp.SYS_FORCEFREE, tp.PREC_MIXED, 300),
    (tp.SYS_MODESUM, tp.PREC_MIXED, 3 * 152 * 128 + 1),  # two particles a thread
    (tp.SYS_MODESUM, tp.PREC_SURROGATE, 300)])
@pytest.mark.parametrize("steps,rows", [(STEPS, 1), (100, 2)])
def test_particles_outside_at_the_start(system, prec, n, steps, rows):
    p, modes = _setup(system, n, steps)
    if prec == tp.PREC_SURROGATE:
        tp.mlp_init(wl.surrogate_features(modes), seed=3)
    r = tp.track(p, DT, 2, 50, precision=prec)
    out = np.zeros(n, bool)
    out[::3] = True
    assert r["remain"].tolist() == [n, n - out.sum()][:rows]
    assert (r["nsteps"][out] == 1).all() and (r["nsteps"][~out] > 1).all()
    assert np.array_equal(r["ptl"]["ux"][out], p["ux"][out].astype(np.float32 if prec > 1 else np.float64))
    assert r["espect"].sum(axis=1).max() <= n - out.sum()


@pytest.mark.parametrize("steps", [1, STEPS, 99, 100])
def test_noalloc_leaves_the_word_behind_the_counts(steps):
    torch = pytest.importorskip("torch")
    import test_zz_no_alloc as na

    n = 300
    p, _ = _setup(tp.SYS_FORCEFREE, n)
    a = na.NoallocArgs()
    a.system_type, a.bc_flag, a.B0, a.lambda0 = tp.SYS_FORCEFREE, 1, 1.0, 2 * np.pi
    a.abc[:], a.lo[:], a.hi[:] = (1.0,) * 3, (0.0,) * 3, (1.0,) * 3
    a.n, a.estep, a.nt_out, a.nbins, a.dt, a.charge_mass = n, steps, 1, 50, DT, 1.0
    a.emin, a.emax = 1e-3, 1e2
    rows = steps // 100 + 1
    state0 = torch.from_numpy(np.stack([np.ascontiguousarray(p[c]) for c in na.COLS])).cuda()
    state = state0.clone()
    nst = torch.zeros(n, dtype=torch.int32, device="cuda")
    esp = torch.zeros((2, 50), dtype=torch.int32, device="cuda")
    dsum = torch.zeros(8 * rows, dtype=torch.float64, device="cuda")
    rem = torch.full((rows + 1,), 77, dtype=torch.int32, device="cuda")
    a.d_state, a.d_state0, a.d_nsteps = state.data_ptr(), state0.data_ptr(), nst.data_ptr()
    a.d_espect, a.d_espect_escape = esp[0].data_ptr(), esp[1].data_ptr()
    a.d_dsum, a.d_remain = dsum.data_ptr(), rem.data_ptr()
    a.stream = torch.cuda.current_stream().cuda_stream
    assert na._fn()(C.byref(a)) == 0
    torch.cuda.synchronize()
    assert rem.tolist() == [n, n - 100][:rows] + [77]
