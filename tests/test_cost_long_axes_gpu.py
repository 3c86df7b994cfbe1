"""Cost volumes of volumes with more than 65535 lines along an axis (a launch grid's limit in
its second and third direction), bit for bit against the oracle: label widths and steps of
each kernel."""
import numpy as np
import pytest
import torch

import pyoracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hw,q", [(4, 2), (4, 1), (2, 2), (4, 30)])
@pytest.mark.parametrize("dims", [(9, 65540, 8), (9, 8, 65540)])
def test_long_axes(dims, hw, q):
    from deedsbcv_gb300 import api
    m, n, o = dims
    rng = np.random.default_rng(hw + q)
    F, M = (rng.integers(0, 2 ** 64, m * n * o, dtype=np.uint64) for _ in range(2))
    dev = [torch.from_numpy(a.view(np.int64)).cuda() for a in (F, M)]
    cost = api.dataCostCL(dev[0], dev[1], m, n, o, 8, hw, q, 1.6).cpu().numpy()
    ref = orc.data_cost(F, M, m, n, o, 8, hw, q, 1.6)
    assert np.array_equal(cost.view(np.uint32), ref.view(np.uint32))
