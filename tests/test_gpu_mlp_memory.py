"""The learned field's workspaces after an allocation that failed."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
tp = pytest.importorskip("test_particle_gb300")
import test_particle_gb300.workloads as wl  # noqa: E402


def test_batches_after_one_too_large():
    """A batch whose first workspace alone is 512 GB is refused; smaller batches
    before and after it, below and above the earlier capacity, are the same."""
    modes = wl.kolmogorov_modes(16, 1.0, 4.0, 0.3, 3)
    dom = tp.Domain()
    dom.xmax = dom.ymax = dom.zmax = 1.0
    tp.configure(system_type=tp.SYS_MODESUM, dom=dom, modes=modes)
    tp.mlp_init(wl.surrogate_features(modes), seed=3)
    rng = np.random.default_rng(4)
    u = rng.integers(0, 2 ** 32, size=(3000, 3), dtype=np.uint64).astype(np.uint32)
    want = tp.mlp_eval(u)
    L = tp.lib()
    for n in (2_000_000_000, 2 ** 31 - 1):
        assert L.tp_mlp_eval(C.c_int(n), tp._ptr(u), tp._ptr(want)) == -1
        L.tp_clear_status()
        assert np.array_equal(tp.mlp_eval(u[:200]), want[:200])
        assert np.array_equal(tp.mlp_eval(u), want)
        t = rng.normal(size=(256, 6)).astype(np.float32)
        loss, y, grads = tp.mlp_grad(u[:256], t)
        assert np.isfinite(loss) and np.isfinite(grads).all()
    assert tp.device_status() == 0
