"""FP64 runs of few particles (four lanes a particle) with open boundaries:
what becomes of the particles that have left."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
tp = pytest.importorskip("test_particle_gb300")


def test_departed_particle_reports_nothing():
    """The box reaches beyond the last grid plane in z.  The particle leaves
    through x before it gets there, and a push from where it stopped would
    sample past the plane: the run has to end without a status bit."""
    g = tp.Grids()
    g.nx = g.ny = g.nz = 4
    g.nt = 1
    g.dx = g.dy = g.dz = 1.0
    dom = tp.Domain()
    dom.xmax, dom.ymax, dom.zmax = 3.0, 3.0, 10.0
    dt, steps = 1.0, 150
    dom.tmax = (steps + 0.5) * dt
    b = np.zeros((64, 3), np.float32)
    b[:, 2] = 1e-6  # straight orbits
    tp.configure(system_type=tp.SYS_PIC, dom=dom, grd=g, bgrid=b, egrid=np.zeros_like(b), bc_flag=1)
    tp.set_spectrum(10, 1e-3, 1e2)
    p = np.zeros(3, dtype=tp.PARTICLE_DTYPE)
    p["qm"] = 1.0
    gam = 1.0 / np.sqrt(1.0 - 0.5 ** 2 - 0.5 ** 2)
    p["x"], p["y"], p["z"] = 2.6, 1.5, 2.3
    p["ux"], p["uz"] = 0.5 * gam, 0.5 * gam
    r = tp.track(p, dt, 1, 10, precision=tp.PREC_FP64)
    assert tp.device_status() == 0
    assert (r["ptl"]["x"] > 3.0).all() and (r["ptl"]["z"] < 3.0).all() and (r["nsteps"] == 2).all()
