"""Label fusion at the edges of its tiles and register sizes, bit for bit against the
float32 restatement: columns around the 32 x 16 tile, slices around a block's share,
radii of the fused and of the separate passes, atlas counts around the vote's sizes.
"""
import numpy as np
import pytest
import torch

import fusion_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,n_atlas,radius,power", [((33, 16, 9), 2, 1, 2), ((32, 17, 70), 4, 2, 1), ((31, 15, 40), 8, 3, 2),
                                                          ((65, 33, 6), 9, 2, 2), ((3, 2, 5), 5, 3, 0), ((40, 20, 24), 16, 1, 3),
                                                          ((34, 18, 12), 17, 2, 2), ((20, 20, 20), 3, 4, 1), ((1, 1, 1), 1, 2, 1)])
def test_fusion_tiles(shape, n_atlas, radius, power):
    from deedsbcv_gb300 import api
    m, n, o = shape
    rng = np.random.default_rng(m + n_atlas)
    target = np.asfortranarray(rng.normal(0, 100, shape).astype(np.float32))
    images = [np.asfortranarray((target + rng.normal(0, 40, shape)).astype(np.float32)) for _ in range(n_atlas)]
    labels = [np.asfortranarray(rng.integers(-2, 5, shape).astype(np.int16)) for _ in range(n_atlas)]
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a.ravel(order="F"))).cuda()  # noqa: E731
    got = api.fuse_labels_device(cu(target), [cu(a) for a in images], [cu(a) for a in labels], m, n, o, radius=radius,
                                 eps=1.0, power=power).cpu().numpy()
    ref = fusion_ref.fuse_labels(target, images, labels, radius=radius, eps=1.0, power=power)
    assert np.array_equal(got, ref.ravel(order="F"))
