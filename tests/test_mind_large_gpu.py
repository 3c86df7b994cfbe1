"""MIND codes of images so bright that the distances come near the largest float: a sum of
twelve that is still finite leaves a noise below 2^125, whose reciprocal the quantiser's fast
path forms without leaving the normal range.  Codes are whole numbers: every bit is the
oracle's.  (One bright voxel and a few dim ones: a box sum's prefix holds at most 54 times the
bright voxel's square, 2^127.8 at 2^61.)"""
import numpy as np
import pytest
import torch

import pyoracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [50, 56, 59, 60, 61])
def test_bright_voxel(power):
    from deedsbcv_gb300 import api
    shape = (20, 17, 12)
    rng = np.random.default_rng(power)
    im = np.zeros(shape, np.float32)
    im[9, 8, 6] = 2.0 ** power
    for _ in range(6):
        im[tuple(rng.integers(0, s) for s in shape)] += np.float32(2.0 ** (power - 3) * rng.random())
    im = im.ravel(order="F")
    got = api.descriptor(torch.from_numpy(im).cuda(), *shape, 1).cpu().numpy().view(np.uint64)
    ref = orc.descriptor(im, *shape, 1).view(np.uint64)
    assert np.array_equal(got, ref), int(np.count_nonzero(got != ref))
