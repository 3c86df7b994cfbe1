"""Backward passes of four pairs in flight, again and again: every sweep ends.

The lanes of a warp wait for words of their own, so that they leave a wait at different
times; with the warps not brought together again before a block barrier, about one pass in a
thousand ended in a timeout.  A few hundred passes find that now and then only, and must never
time out.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_many_backward_passes():
    from deedsbcv_gb300 import api
    m, n, o, g = 112, 112, 128, 4
    rng = np.random.default_rng(0)
    fixed = torch.from_numpy(rng.normal(0, 100, (4, m * n * o)).astype(np.float32)).cuda()
    fixed = torch.nn.functional.avg_pool3d(fixed.view(4, 1, o, n, m), 5, 1, 2).view(4, -1).contiguous()
    moving = fixed.roll(2, 1) + 1.0
    ctx = api.Context(0)
    trees = [[api.soft_tree(f, m, n, o, g, ctx)] for f in fixed]
    first = None
    for k in range(60):
        F, M = fixed.detach().requires_grad_(), moving.detach().requires_grad_()
        d = api.soft_register_levels_batch(F, M, torch.tensor(1.6), (m, n, o), ((g, 3, 1, 1),), tau=0.5, trees=trees,
                                           ctx=ctx, keep_state=k % 2 == 0)
        (d ** 2).mean().backward()
        first = (d.detach(), F.grad) if first is None else first
        assert (d - first[0]).abs().max().item() < 1e-3
        assert ((F.grad - first[1]).norm() / first[1].norm()).item() < 1e-4
    del d
    ctx.close()
