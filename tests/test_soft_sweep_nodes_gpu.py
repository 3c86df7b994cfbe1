"""Tree sweeps over thousands of nodes, ten and more for every block of the persistent
launches: the reuse of a block's shared arrays from node to node, long chains, and nodes of
more children than are polled together (six), at every label width with a kernel of its
own.  Two contexts run at once, three times each, on streams of their
own; nothing on the displacements' way depends on the order of blocks, so that all six
agree bit for bit.  They are compared with the float64 definition, oracle/softmin_ref.py's
with the label transforms axis by axis and a depth's nodes together (checked against it on a
small tree).

Tolerances are those of the sweeps' other tests, 2e-3: displacements on both trees, and the
gradients of the fixed image and the prior on the image's own tree.  Along a chain of 500
nodes with random weights the float method's own gradients are 1 to 3e-3 off (the sweeps'
earlier form's to the same four digits); there the prior's have to agree from run to run, to
the rounding of the atomic sums of a node's edges (six and more terms: 1e-5 of the norm).
"""
import threading

import numpy as np
import pytest
import torch

import softmin_ref as sref

pytestmark = pytest.mark.gpu

DIMS, GRID, TAU = (24, 24, 44), 2, 0.5


def _lse_axis(r, off, axis, sign):
    """r (K, z, x, y): log sum over a of exp(r(a) - (sign (b - a) + off)^2 / tau) along one axis."""
    n = r.shape[axis]
    k = torch.arange(n, dtype=r.dtype, device=r.device)
    d2 = (sign * (k[:, None] - k[None, :])[None] + off[:, None, None]) ** 2 / TAU  # (K, b, a)
    r = r.movedim(axis, -1)
    return torch.logsumexp(r.unsqueeze(-2) - d2[:, None, None], -1).movedim(-1, axis)


def _transform(r, off, length, sign):
    shape = r.shape
    r = r.view(shape[0], length, length, length)
    for axis, o in ((3, 1), (2, 0), (1, 2)):  # y, x, z; offsets are (x, y, z)
        r = _lse_axis(r, off[:, o], axis, sign)
    return r.reshape(shape)


def tree64(cost, ordered, parents, edgemst, hw, q, prior):
    sz1, len3 = cost.shape
    length, dev = 2 * hw + 1, cost.device
    par = torch.as_tensor(np.asarray(parents, np.int64), device=dev)
    depth = np.zeros(sz1, np.int64)
    for c in ordered[1:]:
        depth[c] = depth[parents[c]] + 1
    levels = [torch.as_tensor(np.flatnonzero(depth == k), device=dev) for k in range(int(depth.max()) + 1)]
    e = torch.as_tensor(np.asarray(edgemst, np.float64), device=dev)[:, None]
    off = sref.edge_offsets(prior, parents, int(ordered[0]), q).to(dev) if prior is not None else \
        torch.zeros(sz1, 3, dtype=cost.dtype, device=dev)
    below, B, M = None, {}, {}
    for k in range(len(levels) - 1, -1, -1):
        at = levels[k]
        b = cost[at]
        if below is not None:
            slot = torch.zeros(sz1, dtype=torch.int64, device=dev)
            slot[at] = torch.arange(len(at), device=dev)
            b = b.index_add(0, slot[par[levels[k + 1]]], below - below.min(1, keepdim=True).values.detach())
        B[k] = b
        if k > 0:
            below = M[k] = -TAU * _transform(-e[at] * b / TAU, off[at], length, 1.0)
    lp = {0: torch.log_softmax(-B[0] / TAU, 1)}
    disp = (sref.label_grid(hw).to(dev) - hw) * q
    out = torch.zeros(sz1, 3, dtype=cost.dtype, device=dev)
    out = out.index_add(0, levels[0], lp[0].exp() @ disp)
    for k in range(1, len(levels)):
        at = levels[k]
        slot = torch.zeros(sz1, dtype=torch.int64, device=dev)
        slot[levels[k - 1]] = torch.arange(len(levels[k - 1]), device=dev)
        r = lp[k - 1][slot[par[at]]] + M[k] / TAU
        lp[k] = -e[at] * B[k] / TAU + _transform(r, off[at], length, -1.0)
        out = out.index_add(0, at, lp[k].exp() @ disp)
    return out.T


def _spine_tree(nodes, rng):
    """A chain of 500 nodes, every other node hung on one of them at random."""
    ids = rng.permutation(nodes)
    spine, rest = ids[:500], ids[500:]
    parents = np.zeros(nodes, np.int32)
    parents[spine[0]] = -1
    parents[spine[1:]] = spine[:-1]
    hang = rng.integers(0, 500, rest.size)
    parents[rest] = spine[hang]
    depth = np.zeros(nodes, np.int64)
    depth[spine] = np.arange(500)
    depth[rest] = hang + 1
    ordered = np.argsort(depth, kind="stable").astype(np.int32)
    assert np.bincount(hang, minlength=500).max() > 6
    return ordered, parents, rng.uniform(0.3, 0.9, nodes).astype(np.float32)


def test_definition_by_depth():
    rng = np.random.default_rng(0)
    nodes, hw = 30, 1
    parents = np.array([-1] + [rng.integers(0, c) for c in range(1, nodes)], np.int32)
    tree = (np.arange(nodes, dtype=np.int32), parents, rng.uniform(0.3, 0.9, nodes).astype(np.float32))
    cost = torch.from_numpy(rng.uniform(0, 5, (nodes, 27)))
    prior = torch.from_numpy(rng.normal(0, 1, (3, nodes)))
    ref = sref.soft_tree(cost, *tree, hw, 1, TAU, prior=prior)
    assert (tree64(cost, *tree, hw, 1, prior) - ref).abs().max() < 1e-10


@pytest.mark.parametrize("shape", ["image", "spine"])
@pytest.mark.parametrize("hw", [1, 2, 3, 4])
def test_many_nodes(hw, shape):
    from deedsbcv_gb300 import api, phantom
    m, n, o = DIMS
    nodes = (m // GRID) * (n // GRID) * (o // GRID)
    pr = phantom.make_pair(DIMS, seed=5, max_disp=2.0, spacing=8)
    f, mv = (np.asarray(pr[k], np.float32).ravel(order="F") for k in ("fixed", "moving"))
    rng = np.random.default_rng(hw)
    prior = rng.normal(0, 1.0, (3, nodes)).astype(np.float32)
    gt = torch.from_numpy(rng.normal(0, 1, (3, nodes)))
    if shape == "image":
        ordered, parents, edge = api.soft_tree(torch.from_numpy(f).cuda(), m, n, o, GRID)
        tree = ordered, parents, np.minimum(edge, np.float32(0.9))
    else:
        tree = _spine_tree(nodes, rng)
    params = api.soft_params(GRID, hw, 1, 1.6, TAU, 0.01, 1)

    image = shape == "image"
    F64, M64 = (torch.from_numpy(x.astype(np.float64).reshape(o, n, m)) for x in (f, mv))
    P64 = torch.from_numpy(prior.astype(np.float64)).requires_grad_(image)
    F64.requires_grad_(image)
    cost = sref.soft_cost(sref.soft_mind(F64, 1), sref.soft_mind(M64, 1), GRID, hw, 1,
                          torch.tensor(1.6, dtype=torch.float64), 0.01)
    ref = tree64(cost, *tree, hw, 1, P64)
    if image:
        ((ref - gt) ** 2).mean().backward()

    results, errors = [], []

    def work(ctx):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(3):
                    F = torch.from_numpy(f).cuda().requires_grad_()
                    P = torch.from_numpy(prior).cuda().requires_grad_()
                    d = api.SoftDeedsLevel.apply(F, torch.from_numpy(mv).cuda(), torch.tensor(1.6), P, DIMS, params, tree,
                                                 ctx)
                    ((d - gt.float().cuda()) ** 2).mean().backward()
                    torch.cuda.current_stream().synchronize()
                    results.append([t.cpu().double() for t in (d.detach(), F.grad, P.grad)])
        except Exception as e:  # reported by the main thread
            errors.append(e)

    contexts = [api.Context(0), api.Context(0)]
    threads = [threading.Thread(target=work, args=(c,)) for c in contexts]
    [t.start() for t in threads]
    [t.join() for t in threads]
    for c in contexts:
        c.close()
    assert not errors and len(results) == 6, errors
    def off(got, want):
        return ((got - want).norm() / want.norm()).item()

    for disp, gf, gp in results:
        assert torch.equal(disp, results[0][0]) and off(gp, results[0][2]) < 1e-5
        assert (disp - ref.detach()).abs().max().item() < 2e-3
        if image:
            assert off(gf, F64.grad.reshape(-1)) < 2e-3 and off(gp, P64.grad) < 2e-3
