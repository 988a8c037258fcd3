"""The ticks' integrators, whose lanes share particles and take new ones as
they finish, against psg_step_evolve (one thread per step, itself held to the
oracle elsewhere): the same arithmetic on the same inputs, so the same bits.

Rays without photons hit particles but deposit nothing, so each hit particle
is updated with known inputs: nothing absorbed, no heat, the time since the
start. Temperatures and densities spread over decades, so that some particles
take one explicit step, some many, and some go stiff and finish implicitly.
"""
import numpy as np
import pytest

from psphray_b200 import api, fields
from psphray_b200.units import Units

pytestmark = pytest.mark.gpu


def _field(side, units, seed):
    rng = np.random.default_rng(seed)
    f = fields.uniform_field(side, seed, units=units, nngb=min(32, side ** 3 - 1))
    n = f.n
    f.rho *= (10 ** rng.uniform(-1, 4, n)).astype(np.float32)
    f.ie *= (10 ** rng.uniform(-1, 2.5, n)).astype(np.float32)
    f.xHI = (10 ** rng.uniform(-5, -0.01, n)).astype(np.float32)
    f.ye = np.float32(1) - f.xHI + (rng.uniform(0, 0.15, n).astype(np.float32) if units.hemf > 0 else np.float32(0))
    return f


def _dark_rays(f, n, seed):
    rng = np.random.default_rng(seed)
    r = np.zeros(n, fields.RAY_DTYPE)
    r["s"] = rng.random((n, 3)) * f.boxsize
    d = rng.normal(size=(n, 3))
    r["dir"] = d / np.linalg.norm(d, axis=1)[:, None]
    r["freq"] = 13.6 * f.units.EV
    r["length"] = 2 * f.boxsize
    return r


@pytest.mark.parametrize("helium,on_the_spot", [(False, True), (False, False), (True, True), (True, False)])
@pytest.mark.parametrize("side,nray", [(2, 3), (5, 40), (11, 300), (30, 3000)])
def test_ticks_match_step_evolve(helium, on_the_spot, side, nray):
    units = Units(hmf=0.76 if helium else 1.0)
    f = _field(side, units, 7 + side)
    phys = api.Physics(units, isothermal=False, h_only=not helium, on_the_spot=on_the_spot)
    ctx = api.Context(0)
    ctx.set_physics(phys)
    ctx.load(f)
    ctx.build_tree(8)
    if not on_the_spot:
        ctx.set_recombination(nrec=0)
    before = ctx.state()
    he0 = ctx.he_state()
    tick_time = 0.5 * units.MYR
    ctx.run_ticks(_dark_rays(f, nray, side), nray, 1, 1, tick_time)
    after = ctx.state()
    hit = after["lasthit"] == 1
    assert hit.sum() > 0.3 * f.n or side == 2
    s = np.zeros(int(hit.sum()), api.STEP_DTYPE)
    s["lambdaH"], s["ie"] = before["lambdaH"][hit], before["ie"][hit]
    s["yeMET"] = he0["yeMET"][hit]
    s["lambdaHeI"], s["lambdaHeII"] = he0["lambdaHeI"][hit], he0["lambdaHeII"][hit]
    s["time"] = tick_time
    s["nH"] = phys.unit("H_PER_MASS") * f.rho[hit].astype(np.float64)
    s["T"] = 1e4      # (read by isothermal steps only)
    out = ctx.step_evolve(s)
    np.testing.assert_array_equal(after["lambdaH"][hit], out["lambdaH"])
    np.testing.assert_array_equal(after["ie"][hit], out["ie"].astype(np.float32))
    if helium:
        he = ctx.he_state()
        np.testing.assert_array_equal(he["lambdaHeI"][hit], out["lambdaHeI"])
        np.testing.assert_array_equal(he["lambdaHeII"][hit], out["lambdaHeII"])
        if not on_the_spot:
            np.testing.assert_array_equal(he["yGrecHeII"][hit], out["yGrecHeII"].astype(np.float32))
            np.testing.assert_array_equal(he["yGrecHeIII"][hit], out["yGrecHeIII"].astype(np.float32))
    if not on_the_spot:
        np.testing.assert_array_equal(ctx.rec_state()[0][hit], out["yGrecHII"].astype(np.float32))
    # the untouched ones stayed as they were
    np.testing.assert_array_equal(after["lambdaH"][~hit], before["lambdaH"][~hit])
    ctx.close()
