"""The ticks' integrators over the whole range of temperatures, from below
the rate rows that they keep in shared memory (from log T = 3; up to 8 for
hydrogen, 6.9 with helium) to above the table's end (log T = 9), against
psg_step_evolve, which reads device memory throughout: the same bits. With
helium a tick of up to 524,288 active particles takes the integrator without
these rows, so the field has more, hit by many rays, by few (a particle or
less to each of its threads) or by some (several)."""
import numpy as np
import pytest

from psphray_b200 import api
from psphray_b200.units import Units
from test_gpu_update_lanes import _dark_rays, _field

pytestmark = pytest.mark.gpu

HE_FEW = 1 << 19


@pytest.mark.parametrize("helium,on_the_spot,side,nray", [
    (False, True, 30, 3000), (False, False, 30, 3000),
    (True, True, 90, 6000), (True, False, 90, 6000), (True, True, 90, 60), (True, False, 90, 60),
    (True, True, 90, 400), (True, False, 90, 400)])
def test_all_temperatures(helium, on_the_spot, side, nray):
    units = Units(hmf=0.76 if helium else 1.0)
    f = _field(side, units, 11)
    logT = np.random.default_rng(12).uniform(2.0, 10.0, f.n)
    f.ie[:] = units.Tye2ie(1e4, 0.5) * 10 ** (logT - 4.0)      # (ye moves log T by 0.2 at most)
    phys = api.Physics(units, isothermal=False, h_only=not helium, on_the_spot=on_the_spot)
    ctx = api.Context(0)
    ctx.set_physics(phys)
    ctx.load(f)
    ctx.build_tree(8)
    if not on_the_spot:
        ctx.set_recombination(nrec=0)
    before, he0 = ctx.state(), ctx.he_state()
    tick_time = 0.02 * units.MYR
    ctx.run_ticks(_dark_rays(f, nray, side), nray, 1, 1, tick_time)
    after, he = ctx.state(), ctx.he_state()
    hit = after["lasthit"] == 1
    if helium:
        assert f.n > HE_FEW and (hit.sum() > HE_FEW) == (nray > 1000)
    for lo, hi in ((2.0, 2.7), (3.3, 6.6), (7.1, 7.7), (8.3, 8.7), (9.3, 10.0)):
        assert (hit & (logT > lo) & (logT < hi)).sum() > 100
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
        for k in ("lambdaHeI", "lambdaHeII"):
            np.testing.assert_array_equal(he[k][hit], out[k], err_msg=k)
    if not on_the_spot:
        np.testing.assert_array_equal(ctx.rec_state()[0][hit], out["yGrecHII"].astype(np.float32))
        if helium:
            for k in ("yGrecHeII", "yGrecHeIII"):
                np.testing.assert_array_equal(he[k][hit], out[k].astype(np.float32), err_msg=k)
    np.testing.assert_array_equal(after["lambdaH"][~hit], before["lambdaH"][~hit])
    ctx.close()
