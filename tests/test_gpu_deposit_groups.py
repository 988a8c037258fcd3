"""Which group of threads deposits a ray does not change its deposits: the
same bright rays in a tick of their own (few hits: groups as wide as the
rays' steps) and in a tick that a crowd of rays without photons fills up (the
load rule hands them to narrower groups) leave the same bits on every
particle that the crowd does not touch. (On one that it touches the deposits
are the same too, but a run of more than 32 hits is summed by a warp, in
another order than a shorter one by a thread.) A first tick, the same for
both, has the second settle its capped runs by the affine maps where it
capped enough of its hits (hydrogen)."""
import numpy as np
import pytest

from psphray_b200 import api, fields
from psphray_b200.units import Units

pytestmark = pytest.mark.gpu


def _rays(f, n, nph, seed):
    rng = np.random.default_rng(seed)
    r = np.zeros(n, fields.RAY_DTYPE)
    r["s"] = rng.random((n, 3)) * f.boxsize * 0.2 + 0.4 * f.boxsize
    d = rng.normal(size=(n, 3))
    r["dir"] = d / np.linalg.norm(d, axis=1)[:, None]
    r["freq"] = rng.choice([13.7, 20.0, 60.0], n) * f.units.EV
    r["length"] = 2 * f.boxsize
    r["Nph"] = nph * 10 ** rng.uniform(-3, 0, n)
    return r


def _crowd(f, n):
    """Dark rays along one edge of the box: many hits on few particles."""
    rng = np.random.default_rng(9)
    r = np.zeros(n, fields.RAY_DTYPE)
    r["s"] = rng.random((n, 3)) * f.boxsize * [0.0, 0.05, 0.05]
    r["dir"][:, 0] = 1.0
    r["freq"] = 13.7 * f.units.EV
    r["length"] = 2 * f.boxsize
    return r


def _run(f, phys, batches, long, mid):
    ctx = api.Context(0)
    ctx.set_physics(phys)
    ctx.load(f)
    ctx.build_tree(8)
    ctx.set_tune(deposit_long=long, deposit_mid=mid)
    sat = []
    for t, rays in enumerate(batches):
        sat.append(ctx.run_ticks(rays, len(rays), 1, t + 1, 0.05 * f.units.MYR)["saturated"])
    st = ctx.state()
    he = ctx.he_state()
    ctx.close()
    return st, he, sat


@pytest.mark.parametrize("physics", ["iso", "noniso", "helium"])
@pytest.mark.parametrize("long,mid", [(32, 32), (40, 150), (96, 384)])
@pytest.mark.parametrize("boost", [1e-2, 1e3])
def test_groups_do_not_change_deposits(physics, long, mid, boost):
    helium = physics == "helium"
    units = Units(hmf=0.76 if helium else 1.0)
    f = fields.uniform_field(40, 5, units=units)
    phys = api.Physics(units, isothermal=physics == "iso", h_only=not helium, secondary_ionization=helium)
    nph = boost * float(f.mass[0]) * phys.unit("H_PER_MASS")      # a particle's atoms
    first, bright, crowd = _rays(f, 37, nph, 1), _rays(f, 37, nph, 2), _crowd(f, 60000)
    a, he_a, sat_a = _run(f, phys, [first, bright], long, mid)
    b, he_b, sat_b = _run(f, phys, [first, np.concatenate([bright, crowd])], long, mid)
    c, _, _ = _run(f, phys, [crowd], long, mid)
    free = c["lasthit"] == 0
    assert (free & (a["lasthit"] == 2)).sum() > 2000
    assert sat_a == sat_b
    if boost > 1:
        assert min(sat_a) > 50
    for k in ("lambdaH", "ie", "hits", "lasthit"):
        np.testing.assert_array_equal(a[k][free], b[k][free])
    if helium:
        for k in ("lambdaHeI", "lambdaHeII"):
            np.testing.assert_array_equal(he_a[k][free], he_b[k][free])


@pytest.mark.parametrize("physics", ["iso", "helium"])
@pytest.mark.parametrize("n", [1100, 1200, 2500])
def test_more_rays_than_quarters(physics, n):
    """As above, the bright rays behind a crowd that 128-thread quarters take,
    just fewer and more of them than the chip holds."""
    helium = physics == "helium"
    units = Units(hmf=0.76 if helium else 1.0)
    f = fields.uniform_field(40, 5, units=units)
    phys = api.Physics(units, isothermal=physics == "iso", h_only=not helium, secondary_ionization=helium)
    nph = float(f.mass[0]) * phys.unit("H_PER_MASS")
    bright, crowd = _rays(f, 37, nph, 2), _crowd(f, n)
    a, he_a, sat_a = _run(f, phys, [bright], 32, 32)
    b, he_b, sat_b = _run(f, phys, [np.concatenate([crowd, bright])], 32, 32)
    c, _, _ = _run(f, phys, [crowd], 32, 32)
    free = c["lasthit"] == 0
    assert (free & (a["lasthit"] == 1)).sum() > 2000
    assert sat_a == sat_b
    for k in ("lambdaH", "ie", "hits", "lasthit"):
        np.testing.assert_array_equal(a[k][free], b[k][free])
    if helium:
        for k in ("lambdaHeI", "lambdaHeII"):
            np.testing.assert_array_equal(he_a[k][free], he_b[k][free])
