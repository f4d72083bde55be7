"""The mixed mode-sum run with two particles a thread (above 58,368 particles)
against the one-particle kernel: the same particles in small runs, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
tp = pytest.importorskip("test_particle_gb300")
import test_particle_gb300.workloads as wl  # noqa: E402


@pytest.mark.parametrize("n,nmodes,bc,nbins", [(38912, 33, 0, 200), (38913, 32, 1, 200), (39000 + 255, 1, 0, 5000),
                                               (40001, 1024, 0, 200), (38912, 1025, 0, 3),
                                               (58368, 33, 0, 200), (58369, 32, 1, 200), (58369 + 255, 1, 0, 5000),
                                               (60001, 1024, 0, 200), (58369, 1025, 0, 3)])
def test_pairs_match_single(n, nmodes, bc, nbins):
    modes = wl.kolmogorov_modes(nmodes, 1.0, 32.0, 0.5, 3, va=0.1)
    dom = tp.Domain()
    dom.xmax = dom.ymax = dom.zmax = 1.0
    dt, steps, nt_out = 0.01, 205, 4
    dom.tmax = (steps + 0.5) * dt
    tp.configure(system_type=tp.SYS_MODESUM, dom=dom, modes=modes, mode_B0=1.0, bc_flag=bc)
    tp.set_spectrum(nbins, 1e-3, 1e2)
    p = wl.shell_particles(n, 0.7, (0, 0, 0), (1, 1, 1), 9)
    whole = tp.track(p, dt, nt_out, nbins, precision=tp.PREC_MIXED)
    parts = [tp.track(p[a:a + 16384], dt, nt_out, nbins, precision=tp.PREC_MIXED) for a in range(0, n, 16384)]
    assert whole["ptl"].tobytes() == b"".join(r["ptl"].tobytes() for r in parts)
    assert np.array_equal(whole["nsteps"], np.concatenate([r["nsteps"] for r in parts]))
    for k in ("espect", "espect_escape", "remain"):
        assert np.array_equal(whole[k], sum(r[k] for r in parts)), k
    # sums of n terms in another order: n 2^-53 of the sum of their magnitudes
    total = sum(r["dsum"] for r in parts)
    assert np.all(np.abs(whole["dsum"] - total) <= n * 2.0 ** -52 * np.abs(total))
