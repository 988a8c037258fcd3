"""The traversal's line test is decided in single precision except near the
boundary: rays made to pass particles at their smoothing length, give or take
a few roundings and a few margins, along directions that are unit vectors or
not and from near and far, against the restatement's exact test."""
import numpy as np
import pytest

from oracle import Oracle
from psphray_b200 import api, fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 0.25, 6.0])
@pytest.mark.parametrize("far", [0.01, 1.0])
def test_grazing_rays_bit_exact(gpu_ctx, phys, scale, far):
    f = fields.uniform_field(12, 3, units=phys.units)
    flag = np.zeros(f.n, np.int8)
    flag[::37] = 1
    rng = np.random.default_rng(11)
    n = 600
    p = rng.integers(0, f.n, n)
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    v = np.cross(u, rng.normal(size=(n, 3)))
    v /= np.linalg.norm(v, axis=1)[:, None]
    eps = rng.choice([0.0, 1e-7, -1e-7, 1e-6, -1e-6, 1e-5, -1e-5, 1e-4, -1e-4], n)
    back = far * f.boxsize * rng.random(n)
    rays = np.zeros(n, fields.RAY_DTYPE)
    rays["s"] = f.pos[p] + v * (f.sml[p] * (1 + eps))[:, None] - u * back[:, None]
    rays["dir"] = u * scale
    rays["length"] = 2 * f.boxsize
    gpu_ctx.set_physics(phys)
    gpu_ctx.load(f, flag=flag)
    gpu_ctx.build_tree(8)
    orc = Oracle(f, phys, flag=flag)
    orc.build_tree(8)
    off, hits = gpu_ctx.trace(rays)
    o_off, o = orc.trace_all(rays)
    np.testing.assert_array_equal(off, o_off)
    for k in ("ipar", "d", "b"):
        np.testing.assert_array_equal(hits[k], o[k])
    assert off[-1] > 5 * n


@pytest.mark.parametrize("n_side,nrays", [(2, (1, 3)), (4, (1, 37)), (9, (1, 23, 24)), (20, (1, 22, 23, 185, 186, 1480, 1481, 3000))])
def test_few_rays_divided_among_warps(gpu_ctx, phys, n_side, nrays):
    """Few rays are walked by several warps each, from an upper level of the
    tree on: the same lists as the restatement's, around the sizes where the
    level changes, on trees that have these levels in full and that do not."""
    f = fields.uniform_field(n_side, 21 + n_side, units=phys.units, nngb=min(32, n_side ** 3 - 1))
    rng = np.random.default_rng(4)
    n = max(nrays)
    rays = np.zeros(n, fields.RAY_DTYPE)
    rays["s"] = (rng.random((n, 3)) * 1.2 - 0.1) * f.boxsize
    d = rng.normal(size=(n, 3))
    d[::7, 0] = 0.0
    d[::11] = [0.0, 0.0, 1.0]
    rays["dir"] = d / np.linalg.norm(d, axis=1)[:, None]
    rays["length"] = rng.choice([0.3, 2.0], n) * f.boxsize
    gpu_ctx.set_physics(phys)
    gpu_ctx.load(f)
    gpu_ctx.build_tree(8)
    orc = Oracle(f, phys)
    orc.build_tree(8)
    o_off, o = orc.trace_all(rays)
    for m in nrays:
        off, hits = gpu_ctx.trace(rays[:m])
        np.testing.assert_array_equal(off, o_off[:m + 1])
        for k in ("ipar", "d", "b"):
            np.testing.assert_array_equal(hits[k], o[k][:off[-1]])
