"""A tick with so many hits that its slots are placed part by part (80 MB of
them, 21M hits, to a part): every particle's run is complete whichever part
it falls in -- against the sequential restatement, one part, two and more;
the particle number is no multiple of the parts."""
import numpy as np
import pytest

from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nray,least", [(2500, 0), (5000, 1), (12000, 2)])
def test_slots_in_parts(phys, nray, least):
    from psphray_b200 import api, fields
    w = fields.make_workload("iliev32", n_side=19, nray=nray, seed=5)
    f = w.field
    f.sml[:] = np.float32(0.9 * f.boxsize)
    rays = w.schedule.rays_for_tick(1)
    orc = Oracle(f, phys)
    orc.build_tree(8)
    nhit = orc.tick(rays, 1, w.tick_time)["hits"]
    assert nhit * 4 > least * (80 << 20)
    ctx = api.Context(0)
    try:
        ctx.set_physics(phys)
        ctx.load(f)
        ctx.build_tree(8)
        st = ctx.run_ticks(rays, nray, 1, 1, w.tick_time)
        s = ctx.state()
    finally:
        ctx.close()
    assert st["hits"] == nhit
    assert np.array_equal(s["hits"], orc.hits) and np.array_equal(s["lasthit"], orc.lasthit)
    assert np.max(np.abs(s["lambdaH"] - orc.lambdaH)) < 1e-9
