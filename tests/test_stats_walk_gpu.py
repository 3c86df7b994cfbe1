"""Image statistics at the edges of the walk over chunks: one chunk of 512 elements, one
warp's 32 of them, one tile's 1024, each with one element more and less, with sums that
change binade inside a group, or sign.  Every bit is the sequential oracle's."""
import numpy as np
import pytest
import torch

import pyoracle as orc

pytestmark = pytest.mark.gpu

CHUNK = 512


def _image(kind, n):
    rng = np.random.default_rng(n)
    if kind == "ties":
        return rng.integers(0, 1500, n)
    if kind == "binades":  # the sum doubles many times inside one group of chunks
        return np.exp2(np.linspace(0.0, 12.0, n)) * rng.integers(1, 3, n)
    x = rng.integers(-700, 701, n).astype(np.float64)  # sums that pass through zero
    x[n // 2:] *= -1.0
    return x


@pytest.mark.parametrize("kind", ["ties", "binades", "signs"])
@pytest.mark.parametrize("n", [CHUNK - 1, CHUNK, CHUNK + 1, 32 * CHUNK - 1, 32 * CHUNK, 32 * CHUNK + 1, 33 * CHUNK,
                               1024 * CHUNK - 1, 1024 * CHUNK, 1024 * CHUNK + 1, 1057 * CHUNK + 3])
def test_walk_edges(kind, n):
    from deedsbcv_gb300 import api
    im = np.ascontiguousarray(_image(kind, n), np.float32)
    got = np.asarray(api.image_stats_device(torch.from_numpy(im).cuda()), np.float32)
    ref = np.asarray(orc.image_stats(im), np.float32)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32)), (got, ref)
