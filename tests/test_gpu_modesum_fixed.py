"""The fixed-point mode sum of the FP64 path (csrc/modesum_fx.cuh) at the
edges of its range: mode counts around a chunk of 8, large and small
amplitudes, one component empty, lattice vectors past 32 bits of phase, and
the tables that stay in FP64."""
import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
tp = pytest.importorskip("test_particle_gb300")


def _modes(n, scale, seed, nmax=64):
    rng = np.random.default_rng(seed)
    m = np.zeros(n, dtype=tp.MODE_DTYPE)
    m["n"] = rng.integers(-nmax, nmax + 1, (n, 3))
    m["amp_b"] = scale * rng.normal(size=(n, 3))
    m["amp_e"] = scale * rng.normal(size=(n, 3)) * [1.0, 1e-6, 0.0]
    m["phase"] = rng.uniform(0, 2 * np.pi, n)
    return m


@pytest.mark.parametrize("n,scale,nmax", [(1, 1.0, 64), (7, 1.0, 64), (8, 1e-30, 64), (9, 1e20, 64), (129, 1.0, 2000000000),
                                          (5, 1e-290, 64), (16384, 1.0, 64), (16385, 1.0, 64)])
def test_modesum_fixed_matches_oracle(n, scale, nmax):
    m = _modes(n, scale, 5 * n, nmax)
    dom = tp.Domain()
    dom.xmin, dom.ymin, dom.zmin = -0.5, 0.0, 2.0
    dom.xmax, dom.ymax, dom.zmax = 1.5, 1.0, 2.25
    tp.configure(system_type=tp.SYS_MODESUM, dom=dom, modes=m, mode_B0=scale)
    f = po.make_field(system_type=tp.SYS_MODESUM, dom=po.Domain.from_buffer_copy(dom), modes=m, B0=scale)
    rng = np.random.default_rng(3)
    x = np.zeros((64, 4))
    x[:, :3] = [-0.5, 0.0, 2.0] + rng.random((64, 3)) * [2.0, 1.0, 0.25]
    x[:4, :3] = [[-0.5, 0.0, 2.0], [1.5, 1.0, 2.25], [0.0, 0.25, 2.125], [-0.5, 0.5, 2.0625]]
    got, ref = tp.get_emf(x), po.get_emf(f, x)
    # each term of either sum is within 2^-50 of |a| (cosine and products), and
    # an FP64 sum of n terms within n 2^-53 of the sum of |a|
    amp = np.concatenate([np.abs(m["amp_b"]).sum(0) + [0, 0, scale], np.abs(m["amp_e"]).sum(0)])
    tol = amp * (2.0 ** -49 + n * 2.0 ** -53)
    assert np.all(np.abs(got - ref) <= tol + 1e-320), np.max(np.abs(got - ref) / (tol + 1e-320))
    assert np.all(got[:, 5] == 0.0)
