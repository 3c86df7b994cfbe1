"""Device memory that the first backward of a soft level takes beyond its forward.

Row arrays are (nodes x labels) floats.  A label width of 11 needs two of them (the adjoint
messages and the cost gradient), widths up to 9 a third.  The other buffers are the two
descriptor gradients (12 volumes each), six more volumes and the returned gradients; blocks
of the allocators round up to 2 MB, and tens of MB are left for that."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius,rows", [(5, 2), (4, 3), (3, 3)])
def test_backward_scratch(radius, rows):
    from deedsbcv_gb300 import api
    m, n, o = 88, 80, 96
    g, sz = 4, 88 * 80 * 96
    row = (m // g) * (n // g) * (o // g) * (2 * radius + 1) ** 3 * 4
    rng = np.random.default_rng(0)
    F = torch.from_numpy(rng.normal(0, 100, sz).astype(np.float32)).cuda().requires_grad_()
    M = torch.from_numpy(rng.normal(0, 100, sz).astype(np.float32)).cuda().requires_grad_()
    tree = api.soft_tree(F, m, n, o, g)
    params = api.soft_params(g, radius, 1, 1.6, 0.5, 0.01, 1)
    ctx = api.Context(0)
    d = api.SoftDeedsLevel.apply(F, M, torch.tensor(1.6), None, (m, n, o), params, tree, ctx)
    loss = (d ** 2).mean()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    loss.backward()
    torch.cuda.synchronize()
    taken = before - torch.cuda.mem_get_info()[0]
    others = (24 + 6 + 4) * sz * 4
    assert rows * row <= taken <= (rows + 0.2) * row + others + 40e6, (taken / row, others / row)
    del d, loss
    ctx.close()
