"""The affine fit's blocked sums at the edges of a block (64 points) and where a fused
multiply-add could round otherwise than a double sum rounded to float: whole-number points
(sums exactly half way between floats), points so small that their squares are subnormal
floats, and mixed magnitudes.  Bit for bit the oracle's.  Run on the GPU's host too: its
processor takes the fused form, others the chain of doubles."""
import numpy as np
import pytest

import pyoracle as orc


def _points(kind, n):
    rng = np.random.default_rng(n + len(kind))
    p1 = np.ones((4, n), np.float32)
    if kind == "whole":
        p1[:3] = rng.integers(0, 256, (3, n))
        d = rng.integers(-5, 6, (3, n))
    else:
        p1[:3] = rng.uniform(0, 200, (3, n)) if kind != "mixed" else np.exp(rng.uniform(-12, 12, (3, n)))
        d = rng.normal(0, 1, (3, n))
    p2 = p1.copy()
    p2[:3] += d.astype(np.float32)
    if kind == "tiny":
        p1[:3] *= np.float32(3e-21)
        p2[:3] *= np.float32(3e-21)
    return p1.ravel(), p2.ravel()


def _check(kind, n):
    from deedsbcv_gb300 import api
    p1, p2 = _points(kind, n)
    for rigid in (0, 1):
        got = np.asarray(api.affineRobust(p1, p2, n, rigid), np.float32)
        ref = np.asarray(orc.affine_robust(p1, p2, n, rigid), np.float32)
        same = (got.view(np.uint32) == ref.view(np.uint32)) | (np.isnan(got) & np.isnan(ref))
        assert same.all(), (rigid, got, ref)


KINDS = ["whole", "real", "tiny", "mixed"]
SIZES = [8, 63, 64, 65, 127, 128, 129, 130, 5000]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", KINDS)
def test_fit_matches_oracle(kind, n):
    _check(kind, n)


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", KINDS)
def test_fit_matches_oracle_on_the_gpu_host(kind, n):
    _check(kind, n)
