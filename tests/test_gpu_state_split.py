"""Reading the state of a field just under and just over the size from which
each array has a kernel of its own and overlaps the others' copies, and of
one whose arrays are scattered in two parts: every value in its caller's
place, twice in a row and on a stream of the caller's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [111, 112, 205])
def test_state_comes_back_in_place(phys_noniso, side):
    import torch
    from psphray_b200 import api, fields
    f = fields.uniform_field(side, 3)
    rng = np.random.default_rng(side)
    lam, ie = rng.random(f.n), rng.random(f.n).astype(np.float32) + 1
    last = rng.integers(0, 1 << 40, f.n)
    ctx = api.Context(0)
    try:
        ctx.set_physics(phys_noniso)
        ctx.load(f)
        ctx.build_tree(8)
        ctx.set_state(lam, ie, last)
        stream = torch.cuda.Stream()
        for s in (0, 0, stream.cuda_stream):
            ctx.set_stream(s)
            st = ctx.state()
            assert np.array_equal(st["lambdaH"], lam) and np.array_equal(st["ie"], ie)
            assert np.array_equal(st["lasthit"], last) and not st["hits"].any()
        ctx.set_stream(0)
    finally:
        ctx.close()
