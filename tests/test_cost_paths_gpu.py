"""The cost volume's three kernels at the edges of their ranges, bit for bit against the
oracle.  Codes are random 64-bit words.

- the integer kernel: every grid spacing with each label width that is known to the compiler
  (3, 5 and 7) at compiled label steps (1 and 2) and others, tiles of one node and of a whole
  line, lines that leave a remainder, wider labels at grid 2, and the largest steps whose box
  still fits with the first ones beyond, which the generic kernel takes;
- the tensor cores at sizes that they take: every grid spacing, label steps that share ring
  columns and ones that do not, label counts that leave a remainder in the z groups, tiles
  cut short by the volume, and label reaches beyond 128 rows (several chunks of y labels).
"""
import numpy as np
import pytest
import torch

import pyoracle as orc

pytestmark = pytest.mark.gpu


def _check(dims, g, hw, q):
    from deedsbcv_gb300 import api
    m, n, o = dims
    rng = np.random.default_rng(g * 1000 + hw * 10 + q)
    F, M = (rng.integers(0, 2 ** 64, m * n * o, dtype=np.uint64) for _ in range(2))
    dev = [torch.from_numpy(a.view(np.int64)).cuda() for a in (F, M)]
    cost = api.dataCostCL(dev[0], dev[1], m, n, o, g, hw, q, 1.6).cpu().numpy()
    ref = orc.data_cost(F, M, m, n, o, g, hw, q, 1.6)
    assert np.array_equal(cost.view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("g", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("hw,q", [(1, 1), (1, 4), (2, 2), (3, 1), (3, 9)])
def test_widths(g, hw, q):
    _check((g * 13 + g - 1, 2 * g + 1, 3 * g), g, hw, q)


@pytest.mark.parametrize("rows", [1, 2, 11, 12, 13, 24, 25, 31])
def test_lines(rows):
    _check((rows * 8, 9, 8), 8, 2, 1)
    _check((rows * 3 + 2, 7, 6), 3, 1, 2)


@pytest.mark.parametrize("g,hw,q", [
    (2, 1, 32), (2, 1, 36), (2, 2, 40), (2, 2, 44), (2, 5, 24), (2, 5, 26), (3, 3, 40), (3, 3, 44), (4, 3, 22),
    (4, 3, 24), (5, 2, 24), (5, 2, 26), (8, 3, 21), (8, 3, 22), (8, 1, 9), (8, 1, 120)])
def test_wide_steps(g, hw, q):
    _check((50, 100, 100), g, hw, q)


@pytest.mark.parametrize("dims,g,hw,q", [
    ((60, 48, 52), 2, 4, 1), ((60, 47, 52), 3, 4, 5), ((66, 48, 48), 3, 6, 1), ((41, 33, 42), 3, 4, 2),
    ((41, 30, 42), 4, 4, 1), ((129, 30, 30), 4, 4, 3), ((41, 33, 42), 4, 3, 4), ((70, 42, 47), 5, 5, 2),
    ((87, 41, 46), 5, 4, 3), ((75, 38, 40), 6, 6, 3), ((75, 38, 40), 6, 4, 1), ((93, 36, 44), 7, 7, 4),
    ((93, 36, 44), 7, 4, 3), ((60, 42, 35), 7, 3, 5), ((95, 44, 57), 8, 8, 5), ((131, 40, 41), 8, 4, 3),
    ((61, 33, 41), 8, 10, 6), ((95, 33, 41), 8, 10, 8), ((60, 42, 48), 8, 3, 8)])
def test_tensor_cores(dims, g, hw, q):
    _check(dims, g, hw, q)


@pytest.mark.parametrize("dims,g,hw,q", [
    ((9, 4, 4), 4, 62, 1), ((17, 8, 5), 4, 70, 1), ((11, 5, 5), 5, 64, 2), ((9, 8, 8), 8, 66, 1)])
def test_label_reach_beyond_a_tile(dims, g, hw, q):
    _check(dims, g, hw, q)
