"""Tree sweeps at every label width that has a kernel of its own (3, 5, 7 and 9) and at
one that takes the general form (11), with and without a prior's offsets, against the
float64 definition: displacements, and the gradients of the fixed image and the prior.

Tolerances: messages and marginals carry a few float roundings per node and tau = 0.5,
which the definition's own tests bound by 2e-3 (absolute for displacements of a few
voxels, relative in the 2-norm for gradients); wider label sets add no roundings per
node, only terms of the same sums.
"""
import numpy as np
import pytest
import torch

import softmin_ref as sref

pytestmark = pytest.mark.gpu

DIMS = (16, 12, 20)


@pytest.mark.parametrize("with_prior", [False, True])
@pytest.mark.parametrize("hw", [1, 2, 3, 4, 5])
def test_sweeps_match_float64(hw, with_prior):
    from deedsbcv_gb300 import api, phantom
    m, n, o = DIMS
    g, q, tau = 4, 1, 0.5
    nodes = (m // g) * (n // g) * (o // g)
    pr = phantom.make_pair(DIMS, seed=7, max_disp=2.0, spacing=8)
    f, mv = (np.asarray(pr[k], np.float32).ravel(order="F") for k in ("fixed", "moving"))
    rng = np.random.default_rng(hw)
    prior = rng.normal(0, 1.0, (3, nodes)).astype(np.float32)
    gt = rng.normal(0, 1, (3, nodes))
    F = torch.from_numpy(f).cuda().requires_grad_()
    M = torch.from_numpy(mv).cuda()
    P = torch.from_numpy(prior).cuda().requires_grad_() if with_prior else None
    tree = api.soft_tree(F, m, n, o, g)
    params = api.soft_params(g, hw, q, 1.6, tau, 0.01, 1)
    d = api.SoftDeedsLevel.apply(F, M, torch.tensor(1.6), P, DIMS, params, tree, api.context(0))
    ((d - torch.from_numpy(gt).float().cuda()) ** 2).mean().backward()

    F64, M64 = (torch.from_numpy(x.astype(np.float64).reshape(o, n, m)) for x in (f, mv))
    F64.requires_grad_()
    P64 = torch.from_numpy(prior.astype(np.float64)).requires_grad_() if with_prior else None
    cost = sref.soft_cost(sref.soft_mind(F64, 1), sref.soft_mind(M64, 1), g, hw, q,
                          torch.tensor(1.6, dtype=torch.float64), 0.01)
    ref = sref.soft_tree(cost, *tree, hw, q, tau, prior=P64)
    ((ref - torch.from_numpy(gt)) ** 2).mean().backward()
    assert (d.detach().cpu().double() - ref.detach()).abs().max().item() < 2e-3
    pairs = [(F.grad.cpu().double(), F64.grad.reshape(-1))]
    if with_prior:
        pairs.append((P.grad.cpu().double(), P64.grad))
    for got, want in pairs:
        assert ((got - want).norm() / want.norm()).item() < 2e-3
