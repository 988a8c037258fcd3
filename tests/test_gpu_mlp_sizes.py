"""The network's gradient and forward kernels at the edges of their 64-sample
tiles and past one tile per block: the gradient's grid of 296 blocks covers
18,944 samples, the forward's 37,888, so 18,945 gives a block a second tile
of one sample and 40,001 loops both kernels with a ragged end."""
import ctypes as C

import numpy as np
import pytest
import torch

from mlp import NPARAM, forward, init_params, loss_and_grad
from test_gpu_surrogate import _p, _rows, _t

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 18944, 18945, 37889, 40001])
def test_grad_and_forward(gpu_ctx, n):
    from psphray_b200 import api
    rng = np.random.default_rng(n)
    p = (init_params(2) + rng.normal(0, 0.05, NPARAM)).astype(np.float32)
    x = _rows(rng, n)
    t = rng.normal(size=(n, 2)).astype(np.float32)
    dp, dx, dt = _t(p), _t(x), _t(t)
    L = api.lib()
    sse, g = loss_and_grad(p.astype(np.float64), x.astype(np.float64), t.astype(np.float64))
    got = []
    for _ in range(2):
        grad, y = _t(np.zeros(NPARAM + 1)), _t(np.zeros((n + 1, 2)))
        torch.cuda.synchronize()      # (the context has a stream of its own)
        gpu_ctx._check(L.psg_mlp_grad(gpu_ctx.h, _p(dp), _p(dx), _p(dt), C.c_size_t(n), _p(grad), None), "grad")
        gpu_ctx._check(L.psg_mlp_forward(gpu_ctx.h, _p(dp), _p(dx), C.c_size_t(n), _p(y)), "forward")
        torch.cuda.synchronize()
        got.append((grad.cpu().numpy(), y.cpu().numpy()))
    gg = got[0][0].astype(np.float64)
    # FP32 terms (1e-6 of themselves) in sums of up to 128 samples' outputs a
    # tile, a few tiles and 296 blocks: a random walk's error, with room
    assert np.linalg.norm(gg[:NPARAM] - g) <= 1e-4 * np.linalg.norm(g)
    # ... of positive terms, at worst one rounding an addition
    assert abs(gg[NPARAM] - sse) <= 430 * 2.0 ** -23 * sse
    assert np.max(np.abs(got[0][1][:n] - forward(p.astype(np.float64), x.astype(np.float64)))) < 1e-4
    assert not got[0][1][n].any()      # nothing past the rows asked for
    for a, b in zip(got[0], got[1]):      # deterministic
        np.testing.assert_array_equal(a, b)
