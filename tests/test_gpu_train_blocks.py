"""The training GEMMs at the edges of their tiles: one 128-sample tile, an odd
number of tiles, and more tiles than blocks (each block takes several)."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo
from test_gpu_mlp import bf16_round, lattice_freq

pytestmark = pytest.mark.gpu
tp = pytest.importorskip("test_particle_gb300")


def draw(n, seed):
    rng = np.random.default_rng(seed)
    u = rng.integers(0, 2 ** 32, size=(n, 3), dtype=np.uint64).astype(np.uint32)
    return u, rng.normal(0, 1, size=(n, 6)).astype(np.float32)


def parts(g):
    off = 0
    for l, (i, o) in enumerate(mo.SIZES):
        for name, sz in (("W", i * o), ("b", o)):
            yield (l, name), g[off:off + sz].astype(np.float64)
            off += sz


@pytest.mark.parametrize("n", [128, 384])
def test_few_tiles_match_the_fp64_oracle(n):
    freq = lattice_freq()
    tp.mlp_init(freq, seed=5)
    tp.mlp_set_output_norm(np.zeros(6), np.ones(6))
    w = tp.mlp_weights()
    u, t = draw(n, n)
    _, _, g = tp.mlp_grad(u, t)
    wq = w.astype(np.float64)
    off = 0
    for i, o in mo.SIZES:
        wq[off:off + i * o] = bf16_round(w[off:off + i * o])
        off += i * o + o
    x = bf16_round(mo.features(u, freq)).astype(np.float64)
    _, _, rg = mo.loss_and_grads(wq, x, t.astype(np.float64))
    # BF16 activations and gradients (2^-9 each) through five layers
    for (key, a), (_, b) in zip(parts(g), parts(rg)):
        assert np.linalg.norm(a - b) < 0.05 * np.linalg.norm(b), key
    assert tp.device_status() == 0


@pytest.mark.parametrize("tiles", [64, 256, 512])
def test_many_tiles_add_up_to_single_ones(tiles):
    """The gradient of a batch is the mean of its tiles' gradients: the scale
    2 / (6 n) differs by a power of two, so every sample's BF16 values are the
    same and only the order of the FP32 sums differs.  Chains of at most 600
    FP32 additions of terms that cancel to a 1/sqrt(n) part: below 1e-3 of the
    norm; a tile left out or taken twice moves it by 1/sqrt(tiles) or more."""
    tp.mlp_init(lattice_freq(), seed=5)
    tp.mlp_set_output_norm(np.zeros(6), np.ones(6))
    n = 128 * tiles
    u, t = draw(n, tiles)
    loss, y, g = tp.mlp_grad(u, t)
    gs, ls = 0.0, 0.0
    for k in range(tiles):
        s = slice(128 * k, 128 * (k + 1))
        lk, yk, gk = tp.mlp_grad(u[s], t[s])
        assert np.array_equal(yk, y[s]), k
        gs, ls = gs + gk.astype(np.float64) / tiles, ls + lk / tiles
    assert abs(loss - ls) < 1e-6 * ls
    for (key, a), (_, b) in zip(parts(g), parts(gs)):
        assert np.linalg.norm(a - b) < 1e-3 * np.linalg.norm(b), key
    assert tp.device_status() == 0
