"""The integrators' bounded wait for their copy of the rate rows: given up at
once (a limit of none), the rows come from device memory. The call reports
it by name, the ticks' results are those of a call that waited, and the
context goes on."""
import numpy as np
import pytest

from psphray_b200 import api
from psphray_b200.units import Units
from test_gpu_update_lanes import _dark_rays, _field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("helium,on_the_spot", [(False, True), (False, False), (True, True), (True, False)])
def test_rows_not_waited_for(helium, on_the_spot):
    units = Units(hmf=0.76 if helium else 1.0)
    side, nray = (90, 6000) if helium else (11, 300)      # (helium: more than 524,288 active particles use the rows)
    f = _field(side, units, 5)
    phys = api.Physics(units, isothermal=False, h_only=not helium, on_the_spot=on_the_spot)
    rays, tick_time = _dark_rays(f, nray, 4), 0.5 * units.MYR
    got = []
    for limit in (None, 0):
        ctx = api.Context(0)
        ctx.set_physics(phys)
        ctx.load(f)
        ctx.build_tree(8)
        if not on_the_spot:
            ctx.set_recombination(nrec=0)
        if limit is None:
            ctx.run_ticks(rays, nray, 1, 1, tick_time)
        else:
            ctx.set_copy_limit(limit)
            with pytest.raises(api.PsgError, match="0x40: rate rows not copied in time") as e:
                ctx.run_ticks(rays, nray, 1, 1, tick_time)
            assert e.value.code == -6
        got.append({**ctx.state(), **ctx.he_state()})
        if limit is not None:      # the next call waits again, and succeeds
            ctx.set_copy_limit(40_000_000)
            ctx.run_ticks(rays, nray, 1, 2, tick_time)
            assert (ctx.state()["lasthit"] == 2).any()
        ctx.close()
    assert (got[0]["lasthit"] == 1).any()
    for k in got[0]:
        np.testing.assert_array_equal(got[0][k], got[1][k], err_msg=k)
    with pytest.raises(api.PsgError):
        c = api.Context(0)
        c.set_copy_limit(-1)
