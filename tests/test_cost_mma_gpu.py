"""The tensor-core cost volume at the edges of its tiling, bit for bit against the oracle.

Codes are random 64-bit words (all 64 bits count).  The cases cover every grid
spacing with its compiled label step and with a run-time one, label steps that
share ring columns and ones that do not, label counts that leave a remainder in
the z groups, volumes narrower than a tile, and label reaches beyond 128 rows.
"""
import numpy as np
import pytest
import torch

import pyoracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,g,hw,q", [
    ((17, 9, 11), 2, 1, 1), ((23, 16, 13), 2, 3, 2), ((31, 20, 17), 3, 2, 1), ((20, 13, 16), 3, 4, 5),
    ((41, 17, 22), 4, 4, 1), ((70, 9, 13), 4, 2, 1), ((129, 12, 9), 4, 3, 3), ((9, 12, 41), 4, 6, 1),
    ((38, 16, 23), 5, 5, 2), ((63, 11, 12), 5, 3, 2), ((27, 21, 16), 5, 4, 3), ((11, 16, 21), 5, 1, 1),
    ((50, 19, 13), 6, 6, 3), ((37, 13, 25), 6, 2, 2), ((25, 20, 19), 7, 7, 4), ((93, 15, 22), 7, 5, 4),
    ((30, 22, 16), 7, 3, 1), ((67, 17, 18), 8, 8, 5), ((131, 8, 9), 8, 3, 5), ((24, 25, 17), 8, 2, 3),
    ((40, 9, 17), 8, 10, 6), ((35, 17, 9), 8, 10, 8), ((33, 8, 16), 4, 2, 70), ((26, 13, 14), 3, 1, 200),
])
def test_cost_volume_matches_oracle(dims, g, hw, q):
    from deedsbcv_gb300 import api
    m, n, o = dims
    rng = np.random.default_rng(g * 1000 + hw * 10 + q)
    F, M = (rng.integers(0, 2 ** 64, m * n * o, dtype=np.uint64) for _ in range(2))
    dev = [torch.from_numpy(a.view(np.int64)).cuda() for a in (F, M)]
    cost = api.dataCostCL(dev[0], dev[1], m, n, o, g, hw, q, 1.6).cpu().numpy()
    ref = orc.data_cost(F, M, m, n, o, g, hw, q, 1.6)
    assert np.array_equal(cost.view(np.uint32), ref.view(np.uint32))
