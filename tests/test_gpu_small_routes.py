"""FP64 runs of few particles: which kernel they take, seen in the number of
blocks of the launch (32 particles a block of the four-lane kernel, 128 of the
one-lane kernel)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
tp = pytest.importorskip("test_particle_gb300")
import test_particle_gb300.workloads as wl  # noqa: E402


@pytest.mark.parametrize("amp,nmodes,blocks", [(1.0, 40, 4), (np.inf, 40, 1), (1.0, 16385, 1)])
def test_mode_tables_outside_the_fixed_point_range(amp, nmodes, blocks):
    """A table that stays in FP64 (too many modes, values that are not finite)
    takes the one-lane kernel: nothing of its sum would be split."""
    dom = tp.Domain()
    dom.xmax = dom.ymax = dom.zmax = 1.0
    dom.tmax = 2.5 * 0.01
    modes = wl.kolmogorov_modes(nmodes, 1.0, 8.0, 0.1, 3)
    modes["amp_b"][0, 0] *= amp
    tp.configure(system_type=tp.SYS_MODESUM, dom=dom, modes=modes)
    tp.set_spectrum(20, 1e-3, 1e2)
    p = wl.shell_particles(100, 0.5, (0, 0, 0), (1, 1, 1), 1)
    assert tp.track(p, 0.01, 1, 20)["info"].grid == blocks
    tp.device_status()
