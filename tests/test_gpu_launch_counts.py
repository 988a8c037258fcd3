"""The launches a call reports are the library's kernels it launched, and a
batch's launches follow its own hits: the slots of a tick past L2's size are
placed in parts (80 MB of slots, 21M hits, to a part), which a small batch on
the same context does not inherit."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from psphray_b200 import api, fields
from psphray_b200.units import Units

pytestmark = pytest.mark.gpu


def _kernels(call):
    """(what call returns, the kernels it launched)"""
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        r = call()
        torch.cuda.synchronize()
    names = [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    if not names:
        pytest.skip("the profiler traces no kernels here")
    return r, [n for n in names if not n.startswith(("Memcpy", "Memset"))]


def test_parts_follow_the_batch(phys):
    w = fields.make_workload("iliev32", n_side=19, nray=12000, seed=5)
    f = w.field
    f.sml[:] = np.float32(0.9 * f.boxsize)      # every ray hits every particle
    rays = w.schedule.rays_for_tick(1)
    ctx = api.Context(0)
    ctx.set_physics(phys)
    ctx.load(f)
    ctx.build_tree(8)
    for tick, (n, parts) in enumerate(((2500, 1), (12000, 3), (2500, 1), (5000, 2)), 1):
        st, names = _kernels(lambda: ctx.run_ticks(rays[:n], n, 1, tick, w.tick_time))
        assert int(4 * st["hits"]) // (80 << 20) + 1 == parts
        assert sum("k_slot_place" in k for k in names) == parts
        assert st["launches"] == len(names)
    ctx.close()


@pytest.mark.parametrize("helium,on_the_spot,iso,nray,nticks,nrec", [
    (False, True, True, 300, 3, 0), (False, True, False, 300, 3, 0), (True, True, False, 2000, 2, 0),
    (False, False, True, 300, 3, 50), (True, False, False, 100, 2, 50), (False, False, False, 300, 2, -1)])
@pytest.mark.parametrize("side", [14, 82])
def test_launches_are_the_kernels(helium, on_the_spot, iso, nray, nticks, nrec, side):
    units = Units(hmf=0.76 if helium else 1.0)
    f = fields.uniform_field(side, 3, units=units)
    ctx = api.Context(0)
    ctx.set_physics(api.Physics(units, isothermal=iso, h_only=not helium, on_the_spot=on_the_spot))
    ctx.load(f)
    ctx.build_tree(8)
    tick_time = 0.05 * units.MYR
    ctx.set_sources([fields.Source(pos=(0.0, 0.0, 0.0), ngamma_dot=5e48 / units.SEC)],
                    [(np.array([13.6 * units.EV]), np.array([1.0]))], seed=4)
    if not on_the_spot:
        ctx.set_recombination(nrec=nrec, threshold=0.1, seed=5)
    for call in range(3):      # the first sizes the buffers, the next capture or replay the ticks
        st, names = _kernels(lambda: ctx.run_ticks_emit(nray, nticks, 1 + call * nticks, tick_time))
        assert st["launches"] == len(names), (call, sorted(set(names)))
    ctx.close()
