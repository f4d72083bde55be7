"""Batches of field points: a block stages 128 points; every size gives each
point the value it has alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
tp = pytest.importorskip("test_particle_gb300")


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 1000])
def test_batch_equals_single_points(n):
    dom = tp.Domain()
    dom.xmax = dom.ymax = dom.zmax = 2.0 * np.pi
    tp.configure(system_type=tp.SYS_FORCEFREE, dom=dom, abc=(1.0, 0.7, 0.4), B0=1.0)
    rng = np.random.default_rng(n)
    pts = rng.uniform(-7.0, 7.0, size=(n, 4))
    out = tp.get_emf(pts)
    assert out.shape == (n, 6) and np.all(np.isfinite(out))
    for i in {0, 1, 63, 126, 127, 128, n // 2, n - 1}:
        if i < n:
            assert np.array_equal(tp.get_emf(pts[i:i + 1])[0], out[i]), i
