"""Cost smoothing of the affine estimate where its sums end exactly half way between two
floats, carry more bits than a double holds, or mix magnitudes: bit for bit the recurrence
c'[t] = c[t] + (0.5 c[t+1] + 0.5 c'[t-1]) in double, each result rounded to float."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(c, m1, n1, o1, labels):
    c = c.reshape(o1, n1, m1, labels).copy()
    for axis in (2, 1, 0):
        v = np.moveaxis(c, axis, 0)
        old, prev = v.copy(), v[0].copy()
        for t in range(v.shape[0]):
            up = old[min(t + 1, v.shape[0] - 1)].astype(np.float64)
            prev = (old[t].astype(np.float64) + (0.5 * up + 0.5 * prev.astype(np.float64))).astype(np.float32)
            v[t] = prev
    return c.reshape(-1)


@pytest.mark.parametrize("dims", [(9, 7, 5), (1, 8, 17), (16, 1, 1), (3, 33, 2)])
@pytest.mark.parametrize("kind", ["halves", "random", "wide", "sparse", "tiny"])
def test_smoothing_matches_double(dims, kind):
    from deedsbcv_gb300 import api
    m1, n1, o1 = dims
    labels = 27
    n = m1 * n1 * o1 * labels
    rng = np.random.default_rng(sum(dims) + len(kind))
    c = {"halves": lambda: rng.integers(0, 2 ** 24, n) * 2.0 ** -20,
         "random": lambda: rng.random(n) * 300.0,
         "wide": lambda: np.exp(rng.uniform(-40.0, 40.0, n)),
         "sparse": lambda: np.where(rng.random(n) < 0.7, 0.0, rng.integers(1, 2 ** 24, n)),
         "tiny": lambda: rng.random(n) * 2.0 ** -70}[kind]().astype(np.float32)
    d = torch.from_numpy(c).cuda()
    api.smoothCosts(d, m1, n1, o1, labels)
    got = d.cpu().numpy()
    assert np.array_equal(got.view(np.uint32), _reference(c, m1, n1, o1, labels).view(np.uint32))
