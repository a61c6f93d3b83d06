"""The 1D core's CFL numbers at states that are not physical, against the
reference's formula (Euler1DCore.cpp:70-94)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_cfl_of_a_negative_density():
    """sqrt(m * m) / rho has the density's sign: at points of negative density
    whose pressure is negative too the number is -|m| / |rho| dt / 2 / dx, and
    NaN where the pressure is not.  The first half step, which does not change
    the even points, gives the same numbers.  Tolerance: x is a rounding of
    equal spacing (1e-14 of it), the rest some ten roundings."""
    from solvcon_gb300.onedim import Euler1DCore
    n, dt = 201, 1e-3
    rng = np.random.default_rng(7)
    x = np.linspace(-1.0, 1.0, n)
    so0 = rng.uniform(0.9, 1.1, (n, 3)) * [1.0, 0.4, 2.5]
    so0[40:60, 0] *= -1.0
    so0[40:50, 2] = -3.0  # E - m^2 / 2 rho < 0: no pressure
    so0[50:60, 2] = 2.0   # E - m^2 / 2 rho > 0: NaN
    so0[100:104, 1] *= -1.0
    gamma = rng.uniform(1.2, 1.6, n)
    core = Euler1DCore(n, dt)
    core.coord[...], core.gamma[...] = x, gamma
    core.so0[...], core.so1[...] = so0, 0.0
    core.setup_march()
    rho, m, e = so0.T
    with np.errstate(invalid="ignore"):
        pr = (gamma - 1.0) * (e - m * m / (2.0 * rho))
        pr = (pr + np.abs(pr)) / 2.0
        speed = np.sqrt(gamma * pr / rho) + np.sqrt(m * m) / rho
    want = dt / 2.0 * speed / (2.0 / (n - 1))
    even = np.arange(2, n - 3, 2)
    got = np.array(core.cfl[...])
    assert (want[even] < 0).sum() == 5 and np.isnan(want[even]).sum() == 5
    np.testing.assert_allclose(got[even], want[even], rtol=3e-14)
    core.march_half1_alpha2()
    got = np.array(core.cfl[...])
    np.testing.assert_allclose(got[even], want[even], rtol=3e-14)
