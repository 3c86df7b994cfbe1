"""Warps and upsampling from control grids, bit for bit against the oracle, where the
row-staged field and the integer evaluation of dyadic blends can go wrong: line
lengths around a block, grids whose voxels share no, two or more nodes, one-node
grids, dyadic and other fractions, corners that are all zero, zeros of either sign,
mixed magnitudes, and values whose blends land between two floats.
"""
import numpy as np
import pytest
import torch

import pyoracle as orc

pytestmark = pytest.mark.gpu


def _grid(kind, n, rng):
    if kind == "smooth":
        return [(rng.normal(0, 4, n)).astype(np.float32) for _ in range(3)]
    if kind == "zero":
        return [np.zeros(n, np.float32), np.full(n, -0.0, np.float32),
                np.where(rng.random(n) < 0.5, 0.0, -0.0).astype(np.float32)]
    if kind == "ties":   # odd multiples of the last bit: dyadic sums end between two floats
        return [(1.0 + rng.integers(0, 2 ** 23, n) * 2.0 ** -23).astype(np.float32) * np.float32(s) for s in (1, -1, 4)]
    # magnitudes over 2^40, with zeros
    return [np.where(rng.random(n) < 0.2, 0.0, rng.normal(0, 1, n) * 2.0 ** rng.integers(-35, 5, n)).astype(np.float32)
            for _ in range(3)]


def _bits(t):
    return t.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("kind", ["smooth", "zero", "ties", "mixed"])
@pytest.mark.parametrize("dims,grid", [((33, 17, 20), (8, 4, 5)), ((64, 12, 24), (16, 3, 6)), ((257, 9, 8), (32, 1, 1)),
                                       ((40, 24, 16), (5, 3, 2)), ((31, 10, 14), (6, 2, 2)), ((48, 16, 16), (41, 13, 13)),
                                       ((37, 11, 12), (1, 1, 1)), ((300, 5, 6), (42, 2, 2))])
def test_upsample_from_grid(dims, grid, kind):
    from deedsbcv_gb300 import api
    m, n, o = dims
    f = _grid(kind, int(np.prod(grid)), np.random.default_rng(m + grid[0]))
    out = api.upsampleDeformationsCL(*[torch.from_numpy(a).cuda() for a in f], *grid, m, n, o)
    ref = orc.upsample(*f, m, n, o, *grid)
    for a, b in zip(out, ref):
        assert np.array_equal(_bits(a), np.asarray(b).view(np.uint32))


@pytest.mark.parametrize("kind", ["smooth", "zero", "ties"])
@pytest.mark.parametrize("dims,g", [((61, 24, 28), 4), ((80, 17, 24), 8), ((35, 20, 25), 5)])
def test_apply_flow_from_grid(dims, g, kind):
    from deedsbcv_gb300 import api
    m, n, o = dims
    rng = np.random.default_rng(g)
    grid = tuple(d // g for d in dims)
    f = _grid(kind, int(np.prod(grid)), rng)
    X = np.array([1.01, .02, 0, -1, 0, .98, .01, 1, .01, 0, 1, .5, 0, 0, 0, 1], np.float32)
    full = orc.upsample(*f, m, n, o, *grid)
    im = np.where(rng.random(m * n * o) < 0.3, 0, rng.integers(-200, 300, m * n * o)).astype(np.float32)
    out = api.apply_flow(np.concatenate(f), im, dims=dims, X=X, grid_step=g)
    assert np.array_equal(out.view(np.uint32), np.asarray(orc.warp_affine(im, X, *full, m, n, o)).view(np.uint32))
    seg = rng.integers(0, 14, m * n * o).astype(np.int16)
    assert np.array_equal(api.apply_flow(np.concatenate(f), seg, dims=dims, X=X, grid_step=g),
                          orc.warp_affine_s(seg, X, *full, m, n, o))


@pytest.mark.parametrize("dims,g", [((12, 9, 10), 4), ((33, 5, 7), 8)])
@pytest.mark.parametrize("scale", [3.0, 1e-34])
def test_consistent_mapping(dims, g, scale):
    from deedsbcv_gb300 import api
    m, n, o = dims
    rng = np.random.default_rng(g)
    f = [(np.round(rng.normal(0, 2, m * n * o) * 4) / 4 * scale).astype(np.float32) for _ in range(6)]
    dev = [torch.from_numpy(a).cuda() for a in f]
    api.consistentMappingCL(*dev, m, n, o, g)
    ref = orc.consistent_mapping(*f, m, n, o, g)
    for a, b in zip(dev, ref):
        assert np.array_equal(_bits(a), np.asarray(b).view(np.uint32))
