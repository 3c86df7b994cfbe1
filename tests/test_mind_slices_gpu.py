"""MIND codes at the edges of the slice passes: extents around the 32-sample strips and
the 16-step columns, the smallest volume each radius takes, the largest slice of one
line per thread (512 lines) and the first beyond it, and an image of constants and
steps.  Codes are whole numbers: every bit is the oracle's."""
import numpy as np
import pytest
import torch

import pyoracle as orc

pytestmark = pytest.mark.gpu


def _codes(im, shape, qs):
    from deedsbcv_gb300 import api
    got = api.descriptor(torch.from_numpy(im).cuda(), *shape, qs).cpu().numpy().view(np.uint64)
    return got, orc.descriptor(im, *shape, qs).view(np.uint64)


@pytest.mark.parametrize("shape,qs", [
    ((3, 3, 3), 1), ((5, 5, 5), 2), ((7, 7, 7), 3), ((9, 9, 9), 4), ((11, 11, 11), 5), ((13, 13, 13), 6),
    ((15, 15, 15), 7), ((31, 16, 9), 1), ((32, 17, 9), 2), ((33, 15, 9), 3), ((35, 32, 8), 3), ((34, 33, 17), 2),
    ((64, 47, 16), 1), ((65, 48, 15), 5), ((70, 49, 18), 7), ((36, 512, 7), 3), ((33, 513, 7), 3), ((20, 600, 5), 2)])
def test_edges(shape, qs):
    rng = np.random.default_rng(sum(shape) + qs)
    im = (rng.normal(0, 1, shape).cumsum(0) * 100).astype(np.float32).ravel(order="F")
    got, ref = _codes(im, shape, qs)
    assert np.array_equal(got, ref), int(np.count_nonzero(got != ref))


@pytest.mark.parametrize("qs", [1, 2, 3])
def test_steps_and_constants(qs):
    shape = (45, 38, 21)
    rng = np.random.default_rng(qs)
    im = np.zeros(shape, np.float32)
    im[10:30, 8:30, 5:15] = 1000.0                       # exact quotients at the thresholds' far sides
    im[:, 30:, :] += rng.integers(0, 3, (45, 8, 21)).astype(np.float32)
    got, ref = _codes(im.ravel(order="F"), shape, qs)
    assert np.array_equal(got, ref), int(np.count_nonzero(got != ref))
