"""The tensor-core cost volume ends and reports when a wait of its warps expires.

The production launch runs with epilogue warps that give up after one try of a few
microseconds, shorter than a step: they leave while producers and MMAs are at work, an MMA
warp waits for their accumulator until the production limit (a second), and then the CTA has
to end without further waits, its MMAs drained, and later CTAs have to do nothing.  A CTA
of this launch has 420 classes to wait for, minutes if every wait ran into the limit; the
bound of a launch is three limits, here 4 s.  With the production limit the same launch, and the
next cost volume, are as ever.
"""
import ctypes as C

import numpy as np
import pytest
import torch

import pyoracle as orc

pytestmark = pytest.mark.gpu


def _run(ctx, tries):
    err, secs = C.c_int(-1), C.c_double(0.0)
    ctx.check(ctx._L.deeds_selftest_cost_volume(ctx.handle, tries, C.byref(err), C.byref(secs)))
    return err.value, secs.value


def test_expired_waits_end_the_launch():
    from deedsbcv_gb300 import api
    ctx = api.context(0)
    assert _run(ctx, 0)[0] == 0
    for _ in range(2):
        err, secs = _run(ctx, 1)
        assert err == 3 and secs < 4.0, (err, secs)
    assert _run(ctx, 0)[0] == 0
    m, n, o = 70, 42, 47
    rng = np.random.default_rng(0)
    F, M = (rng.integers(0, 2 ** 64, m * n * o, dtype=np.uint64) for _ in range(2))
    cost = api.dataCostCL(*(torch.from_numpy(a.view(np.int64)).cuda() for a in (F, M)), m, n, o, 5, 5, 2, 1.6)
    ref = orc.data_cost(F, M, m, n, o, 5, 5, 2, 1.6)
    assert np.array_equal(cost.cpu().numpy().view(np.uint32), ref.view(np.uint32))
