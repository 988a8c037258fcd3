"""A context that loads field after field keeps its arrays: what it computes
must be what a fresh context computes, also where ticks were captured before
(other contents, another box, another leaf order behind the same addresses),
and the state calls must follow the caller's order before and after a tree."""
import dataclasses

import numpy as np
import pytest

from psphray_b200 import api, fields

pytestmark = pytest.mark.gpu


def _state(ctx):
    return dict(ctx.state(), **ctx.he_state(), ygrec=ctx.rec_state()[0], mark=ctx.rec_state()[1])


def _run(ctx, w, calls, T=3, nray=48):
    t = 1
    for _ in range(calls):
        ctx.run_ticks(w.schedule.rays_for_ticks(t, T), nray, T, t, w.tick_time)
        t += T
    return _state(ctx)


def _same(a, b):
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("on_the_spot", [True, False])
@pytest.mark.parametrize("n_side", [12, 13])
def test_reloaded_context_equals_fresh(on_the_spot, n_side):
    def work(seed, scale):
        w = fields.make_workload("lognormal128", seed=seed, n_side=n_side, nray=48)
        f = dataclasses.replace(w.field, pos=(w.field.pos * np.float32(scale)), sml=w.field.sml * np.float32(scale),
                                boxsize=float(np.float32(w.field.boxsize * scale)))
        return dataclasses.replace(w, field=f)

    phys = api.Physics(work(1, 1.0).field.units, isothermal=False, on_the_spot=on_the_spot)

    def context():
        c = api.Context(0)
        c.set_physics(phys)
        if not on_the_spot:
            c.set_recombination(nrec=20, seed=5)
        return c

    kept = context()
    for seed, scale, side in ((1, 1.0, n_side), (2, 0.5, n_side), (3, 2.0, n_side)):
        a, b = work(seed, scale), work(seed, scale)
        kept.load(a.field)
        s0 = kept.state()
        np.testing.assert_array_equal(s0["ie"], a.field.ie)      # before the tree: the caller's order
        assert not s0["hits"].any() and not s0["lasthit"].any()
        kept.build_tree(8)
        np.testing.assert_array_equal(kept.state()["ie"], a.field.ie)
        fresh = context()
        if seed > 1:
            # not on the spot a context's very first call runs tick by tick
            # (it sizes the buffers) and picks the deposit's settle form per
            # tick instead of per call: made here on a field of another size,
            # so that the fresh arrays' calls replay captured ticks as well
            other = fields.make_workload("lognormal128", seed=1, n_side=n_side + 1, nray=48)
            fresh.load(other.field)
            fresh.build_tree(8)
            _run(fresh, other, 3)
        fresh.load(b.field)
        fresh.build_tree(8)
        _same(kept.tree(), fresh.tree())
        _same(_run(kept, a, 3), _run(fresh, b, 3))
        fresh.close()
    # a rebuild of the tree on the loaded field, then a smaller field
    kept.build_tree(4)
    kept.build_tree(8)
    small = fields.make_workload("lognormal128", seed=9, n_side=7, nray=48)
    fresh = context()
    for c in (kept, fresh):
        c.load(small.field)
        c.build_tree(8)
    _same(kept.tree(), fresh.tree())
    kept.close()
    fresh.close()
