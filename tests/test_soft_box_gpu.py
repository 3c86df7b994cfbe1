"""The soft descriptor's windowed sums at every radius with a fused kernel (1 to 3) and at
one without (4): extents around the 32 x 8 tiles and the 32-plane marches, against the
float64 descriptor.  Tolerance: the descriptor's own test's (2e-4 of values up to 6): the
sums have at most 729 terms whatever the extents."""
import numpy as np
import pytest
import torch

import softmin_ref as sref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qs", [1, 2, 3, 4])
@pytest.mark.parametrize("dims", [(9, 9, 9), (31, 9, 32), (32, 8 + 2, 33), (33, 17, 31), (65, 11, 34), (12, 24, 65)])
def test_descriptor_matches_float64(qs, dims):
    from deedsbcv_gb300 import api
    m, n, o = dims
    rng = np.random.default_rng(sum(dims) + qs)
    f = rng.normal(0, 40.0, (o, n, m)).cumsum(2).astype(np.float32)
    s = api.soft_descriptor(torch.from_numpy(f.ravel()).cuda(), m, n, o, qs).cpu().numpy()
    ref = sref.soft_mind(torch.from_numpy(f.astype(np.float64)), qs).reshape(12, -1).numpy()
    assert np.abs(s - ref).max() < 2e-4
