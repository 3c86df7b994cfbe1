"""Blends at coordinates far outside the volume, bit for bit against the oracle.

Below -2^31 a coordinate's integer part saturates, so its fraction is a large negative
number in place of one in [0, 1).  Both corners along that axis are then the edge voxel
and the reference's double expression is evaluated as it stands.  (Only the negative
side: above 2^31 the reference's own x + 1 overflows.)

- ties: image values of 24 bits whose mean over four corners lies half way between two
  floats, where the blend is decided in integers or in double.
"""
import numpy as np
import pytest
import torch

import pyoracle as orc

pytestmark = pytest.mark.gpu

DIMS = (33, 10, 9)


def _image(rng, n):
    return rng.integers(2 ** 23, 2 ** 24, n).astype(np.float32)


def _check(out, ref):
    assert np.array_equal(out.cpu().numpy().view(np.uint32), np.asarray(ref).view(np.uint32))


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("beyond", [2 ** 9, 2 ** 18])
def test_ties(axis, beyond):
    from deedsbcv_gb300 import api
    n = int(np.prod(DIMS))
    rng = np.random.default_rng(axis)
    im = _image(rng, n)
    f = [rng.choice(np.array([0.5, -0.5, 1.5, 0.25], np.float32), n) for _ in range(3)]
    far = rng.random(n) < 0.5
    f[axis][far] = np.float32(-2.0 ** 31 - beyond)
    dev = [torch.from_numpy(a).cuda() for a in f]
    _check(api.warpImageCL(torch.from_numpy(im).cuda(), *dev, *DIMS), orc.warp_image(im, *f, *DIMS))
