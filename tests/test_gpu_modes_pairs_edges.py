"""The mixed mode-sum run with two particles a thread (above three 128-particle
blocks an SM, up to 1,024 modes): sizes at the edges of its 256-particle tiles
and of its range, and open-boundary runs in segments, whose later ones have
few enough particles for the one-particle kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
tp = pytest.importorskip("test_particle_gb300")
import test_particle_gb300.workloads as wl  # noqa: E402

FROM = 3 * 128 * 152


def _run(n, nmodes, bc, seg, steps=205, nbins=200):
    modes = wl.kolmogorov_modes(nmodes, 1.0, 32.0, 0.5, 3, va=0.1)
    dom = tp.Domain()
    dom.xmax = dom.ymax = dom.zmax = 1.0
    dt = 0.01
    dom.tmax = (steps + 0.5) * dt
    tp.configure(system_type=tp.SYS_MODESUM, dom=dom, modes=modes, mode_B0=1.0, bc_flag=bc)
    tp.set_spectrum(nbins, 1e-3, 1e2)
    p = wl.shell_particles(n, 0.7, (0, 0, 0), (1, 1, 1), 9)
    tp.set_compaction(seg)
    try:
        return p, tp.track(p, dt, 4, nbins, precision=tp.PREC_MIXED), lambda q: tp.track(q, dt, 4, nbins, precision=tp.PREC_MIXED)
    finally:
        tp.set_compaction(-1)


@pytest.mark.parametrize("n", [FROM, FROM + 1, FROM + 127, FROM + 128, FROM + 129, FROM + 255, FROM + 257])
@pytest.mark.parametrize("nmodes,bc", [(2, 0), (33, 1), (1024, 0)])
def test_tile_edges(n, nmodes, bc):
    p, whole, track = _run(n, nmodes, bc, 0)
    parts = [track(p[a:a + 32768]) for a in range(0, n, 32768)]
    assert whole["ptl"].tobytes() == b"".join(r["ptl"].tobytes() for r in parts)
    assert np.array_equal(whole["nsteps"], np.concatenate([r["nsteps"] for r in parts]))
    for k in ("espect", "espect_escape", "remain"):
        assert np.array_equal(whole[k], sum(r[k] for r in parts)), k
    total = sum(r["dsum"] for r in parts)  # n terms in another order
    assert np.all(np.abs(whole["dsum"] - total) <= n * 2.0 ** -52 * np.abs(total))


def test_segments_that_end_below_the_range():
    n = FROM + 301
    _, one, _ = _run(n, 24, 1, 0, steps=900)
    _, cut, _ = _run(n, 24, 1, 100, steps=900)
    left = one["espect_escape"].sum()
    assert left > 0.3 * n  # later segments are below the range
    assert cut["info"].launches > one["info"].launches
    assert cut["ptl"].tobytes() == one["ptl"].tobytes()
    for k in ("nsteps", "espect", "espect_escape", "remain"):
        assert np.array_equal(cut[k], one[k]), k
    np.testing.assert_allclose(cut["dsum"], one["dsum"], rtol=1e-12, atol=1e-300)
