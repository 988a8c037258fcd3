"""Helium steps far above the rate table (its last row is log T = 9): the
row is the table's last however high the temperature is, also where the
temperature itself overflows a double, so the species come out the same."""
import numpy as np
import pytest

from psphray_b200 import api
from psphray_b200.units import Units

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("on_the_spot", [True, False])
def test_overflowing_temperature_reads_the_last_row(on_the_spot):
    units = Units(hmf=0.76)
    ctx = api.Context(0)
    ctx.set_physics(api.Physics(units, isothermal=False, h_only=False, on_the_spot=on_the_spot))
    n = 64
    rng = np.random.default_rng(3)
    s = np.zeros(n, api.STEP_DTYPE)
    s["lambdaH"], s["lambdaHeI"], s["lambdaHeII"] = rng.uniform(0.2, 0.8, n), rng.uniform(0.2, 0.5, n), 0.3
    s["time"] = 0.01 * units.MYR
    s["nH"] = 1e-3 / units.CM ** 3
    s["T"] = 1e4
    T_per_ie = units.MPROTON_OVER_BOLTZMANN      # (times a number of order one)
    finite, over = s.copy(), s.copy()
    finite["ie"] = 1e250 / T_per_ie
    over["ie"] = 1e308
    with np.errstate(over="ignore"):
        assert np.all(np.isfinite(finite["ie"] * T_per_ie)) and not np.any(np.isfinite(over["ie"] * T_per_ie))
    a, b = ctx.step_evolve(finite), ctx.step_evolve(over)
    ctx.close()
    for k in ("lambdaH", "lambdaHeI", "lambdaHeII"):
        np.testing.assert_array_equal(a[k], b[k])
    assert np.all(a["lambdaH"] < s["lambdaH"])      # ionised: no recombining row
