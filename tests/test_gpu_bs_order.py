"""The batched Bulirsch-Stoer run takes particles in another order and spreads
them over warps by their number: a particle's result does not depend on it."""
import ctypes as C

import numpy as np
import pytest

import make_golden as mg

pytestmark = pytest.mark.gpu
tp = pytest.importorskip("test_particle_gb300")
import test_particle_gb300.workloads as wl  # noqa: E402

SC = mg.scenarios()
LANES = 152 * 128  # one warp a sub-partition


def _run(y0, t_end=2e-4, nt_out=2, nbins=40):
    n = len(y0)
    y, t = y0.copy(), np.zeros(n)
    steps, status = np.zeros(n, np.int32), np.zeros(n, np.int32)
    esp, dfr = np.zeros(nt_out * nbins), np.zeros(8 * (nt_out + 1))
    tp.check(tp.lib().tp_bs_run(C.c_int(n), tp._ptr(y), tp._ptr(t), C.c_double(t_end), C.c_int(nt_out), C.c_int(nbins),
                                C.c_double(1e-6), C.c_double(1e-10), C.c_double(1e-10), C.c_int(8), C.c_int(0),
                                C.c_int(1000000), tp._ptr(steps), tp._ptr(status), tp._ptr(esp), tp._ptr(dfr), None), "bs")
    return y, t, steps, status, esp, dfr


@pytest.mark.parametrize("n", [1, 609, LANES, LANES + 1, 4 * LANES + 1])
def test_order_and_spread(n):
    s = SC["loop"]
    tp.configure(system_type=tp.SYS_WLCS, charge_mass=s["charge_mass"], bc_flag=2, dom=s["dom"], wl=s["wl"], ibessel=0)
    tp.set_spectrum(40, 1e-3, 1e1)
    y0 = wl.torus_particles(n, 1.0, 0.05, 0.3, 0.1, 0.9, 9)
    y, t, steps, status, esp, dfr = _run(y0)
    assert (status == 0).all() and (t == 2e-4).all() and (steps > 0).all()
    assert esp.reshape(2, 40).sum(axis=1).tolist() == [n, n]
    pick = np.unique(np.concatenate([[0, n - 1], np.arange(0, n, max(1, n // 300))]))
    yp, _, sp, _, _, _ = _run(y0[pick])
    assert y[pick].tobytes() == yp.tobytes()
    assert np.array_equal(steps[pick], sp)
