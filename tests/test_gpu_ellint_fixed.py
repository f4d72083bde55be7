"""The loop's field with the fixed-point elliptic integrals (csrc/ellint_fx.cuh)
at the edges of their intervals, near the wire, near the axis and on it."""
import numpy as np
import pytest

import make_golden as mg
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
tp = pytest.importorskip("test_particle_gb300")

SC = mg.scenarios()


@pytest.mark.parametrize("corrected", [0, 1])
def test_loop_field_at_interval_edges(corrected):
    s = SC["loop"]
    tp.configure(system_type=tp.SYS_WLCS, charge_mass=s["charge_mass"], bc_flag=2, dom=s["dom"], wl=s["wl"], ibessel=0,
                 ellint_corrected=corrected)
    f = mg.field_from(s, bc_flag=2, ellint_corrected=corrected)
    # m = 4 a rho / ((a + rho)^2 + z^2) at and next to every edge, for points
    # outside and inside the loop's radius
    edges = np.concatenate([np.arange(1, 9) / 10, [0.85, 0.9, 0.95, 0.999, 1 - 1e-6, 1 - 1e-10, 1e-4, 0.05]])
    m = np.concatenate([edges, np.nextafter(edges, 0), np.nextafter(edges, 1), edges - 1e-9, edges + 1e-11])
    m = m[(m > 0) & (m < 1)]
    pts = []
    for z in (0.0, 1e-3):
        for sgn in (1.0, -1.0):
            # rho of the plane z = 0: (rho + 1)^2 m = 4 rho, then a little off it
            b = 2.0 / m - 1.0
            rho = b + sgn * np.sqrt(b * b - 1.0)
            pts += [[r * 0.6, r * 0.8, z, 0.0] for r in rho if 1e-3 < r < 3.0]
    x = np.array(pts)
    got, ref = tp.get_emf(x), po.get_emf(f, x)
    rho = np.hypot(x[:, 0], x[:, 1])
    # a few 2^-53 of K and E, whose difference the field takes: of order m ~
    # rho / a near the axis, and divided by rho once more
    tol = 1e-14 * (1.0 + 1.0 / rho ** 2) * np.abs(ref[:, :3]).max(axis=1)
    assert np.all(np.abs(got[:, :3] - ref[:, :3]).max(axis=1) <= tol)
    assert np.all(got[:, 3:] == 0.0)
    # on the axis: the reference's not-a-numbers, or zero when corrected
    on = np.array([[0.0, 0.0, 0.4, 0.0]])
    a, b = tp.get_emf(on), po.get_emf(f, on)
    assert np.array_equal(np.isnan(a), np.isnan(b))
    assert np.allclose(a[~np.isnan(a)], b[~np.isnan(b)], rtol=1e-13, atol=0)
