"""Displacements and affines that are NaN or infinite, over images with and without air
(zero voxels): a value that the reference makes NaN is NaN, also where all eight corners
are zero, and every other voxel is the reference's bit for bit.  So are coordinates so far
beyond the integers that their fractions are far outside [0, 1].

The expected values are the reference's expressions (interp3, warpAffine and
consistentMappingCL, src/transformations.h:5-26, src/dataCostD.h:278-295,
src/transformations.h:189-242) in numpy: converting a coordinate beyond the integers, and
adding to the largest of them, has no defined result in C++.  On finite fields the same
functions are checked against the oracle.  NaN payloads are not compared.
"""
import numpy as np
import pytest
import torch

import pyoracle as orc

pytestmark = [pytest.mark.gpu, pytest.mark.filterwarnings("ignore::RuntimeWarning")]

DIMS = (35, 12, 10)
BAD = {"nan": np.nan, "inf": np.inf, "-inf": -np.inf}
AFFINE = np.array([1.01, .02, 0, -1, 0, .98, .01, 1, .01, 0, 1, .5, 0, 0, 0, 1], np.float32)
F32 = np.float32


def _split(c):
    """Integer part (saturating, 0 for NaN) and fraction of float32 coordinates."""
    fl = np.nan_to_num(np.floor(c).astype(np.float64), nan=0.0, posinf=2.0 ** 31 - 1, neginf=-2.0 ** 31)
    i = np.clip(fl, -2.0 ** 31, 2.0 ** 31 - 1).astype(np.int64)
    return i, c - i.astype(F32)


def _blend(vol, dims, yc, xc, zc, base=(0, 0, 0)):
    m, n, o = dims
    vol = np.asarray(vol, F32).reshape(o, n, m)
    (y, dy), (x, dx), (z, dz) = _split(yc), _split(xc), _split(zc)
    y0, y1 = (np.clip(y + base[0] + d, 0, m - 1) for d in (0, 1))
    x0, x1 = (np.clip(x + base[1] + d, 0, n - 1) for d in (0, 1))
    z0, z1 = (np.clip(z + base[2] + d, 0, o - 1) for d in (0, 1))
    ex, ey, ez = (d.astype(np.float64) for d in (dx, dy, dz))
    ax, ay, az = 1.0 - ex, 1.0 - ey, 1.0 - ez
    acc = ax * ay * az * vol[z0, x0, y0]
    acc = acc + ax * ey * az * vol[z0, x0, y1]
    acc = acc + ex * ay * az * vol[z0, x1, y0]
    acc = acc + ax * ay * ez * vol[z1, x0, y0]
    acc = acc + (dx * dy).astype(np.float64) * az * vol[z0, x1, y1]
    acc = acc + ax * ey * ez * vol[z1, x0, y1]
    acc = acc + ex * ay * ez * vol[z1, x1, y0]
    acc = acc + (dx * dy * dz * vol[z1, x1, y1]).astype(np.float64)
    return acc.astype(F32).ravel()


def _voxels(dims):
    k, j, i = np.meshgrid(*(np.arange(d) for d in dims[::-1]), indexing="ij")
    return i.ravel(), j.ravel(), k.ravel()


def warp_image(im, u, v, w, dims):
    return _blend(im, dims, v, u, w, _voxels(dims))


def warp_affine(im, X, u, v, w, dims):
    i, j, k = (a.astype(F32) for a in _voxels(dims))
    row = [i * X[4 * r] + j * X[4 * r + 1] + k * X[4 * r + 2] + X[4 * r + 3] + d for r, d in ((0, v), (1, u), (2, w))]
    return _blend(im, dims, *row)


def consistent(f, dims, g):
    a = [x * F32(1.0 / g) for x in f]
    for _ in range(10):
        def step(s, t):
            return [(0.5 * p.astype(np.float64) - 0.5 * warp_image(q, *s, dims).astype(np.float64)).astype(F32)
                    for p, q in zip(s, t)]
        a = step(a[:3], a[3:]) + step(a[3:], a[:3])
    return [x * F32(g) for x in a]


def _image(kind, n, rng):
    if kind == "zero":
        return np.zeros(n, F32)
    im = rng.normal(0, 300, n).astype(F32)
    return np.where(rng.random(n) < 0.5, 0.0, im).astype(F32) if kind == "air" else im


def _field(bad, n, rng, share):
    f = [rng.normal(0, 3, n).astype(F32) for _ in range(3)]
    for a in f:
        a[rng.random(n) < share] = bad
    return f


def _check(out, ref):
    out = out.cpu().numpy() if isinstance(out, torch.Tensor) else np.asarray(out).ravel(order="F")
    nan = np.isnan(ref)
    assert np.array_equal(np.isnan(out), nan)
    assert np.array_equal(out.view(np.uint32)[~nan], ref.view(np.uint32)[~nan])


def _cuda(f):
    return [torch.from_numpy(a).cuda() for a in f]


def test_expected_values_on_finite_fields():
    n = int(np.prod(DIMS))
    rng = np.random.default_rng(0)
    im, f, b = _image("air", n, rng), _field(0.0, n, rng, 0.1), _field(0.0, n, rng, 0.1)
    for got, ref in [(warp_image(im, *f, DIMS), orc.warp_image(im, *f, *DIMS)),
                     (warp_affine(im, AFFINE, *f, DIMS), orc.warp_affine(im, AFFINE, *f, *DIMS)),
                     *zip(consistent(f + b, DIMS, 4), orc.consistent_mapping(*f, *b, *DIMS, 4))]:
        assert np.array_equal(got.view(np.uint32), np.asarray(ref).view(np.uint32))


@pytest.mark.parametrize("kind", ["zero", "air", "dense"])
@pytest.mark.parametrize("bad", list(BAD))
def test_full_fields(bad, kind):
    from deedsbcv_gb300 import api
    n = int(np.prod(DIMS))
    rng = np.random.default_rng(len(bad) * 7 + len(kind))
    im, f = _image(kind, n, rng), _field(BAD[bad], n, rng, 0.1)
    dev = torch.from_numpy(im).cuda()
    ref = warp_image(im, *f, DIMS)
    assert np.isnan(ref).any() and not np.isnan(ref).all()
    _check(api.warpImageCL(dev, *_cuda(f), *DIMS), ref)
    _check(api.warpAffine(dev, AFFINE, *_cuda(f), *DIMS), warp_affine(im, AFFINE, *f, DIMS))


@pytest.mark.parametrize("kind", ["zero", "air", "dense"])
@pytest.mark.parametrize("bad", list(BAD))
def test_apply_flow(bad, kind):
    from deedsbcv_gb300 import api
    grid = tuple(d // 4 for d in DIMS)
    n = int(np.prod(DIMS))
    rng = np.random.default_rng(len(bad) * 11 + len(kind))
    im, f = _image(kind, n, rng), _field(BAD[bad], int(np.prod(grid)), rng, 0.05)
    ref = warp_affine(im, AFFINE, *orc.upsample(*f, *DIMS, *grid), DIMS)
    assert np.isnan(ref).any() and not np.isnan(ref).all()
    _check(api.apply_flow(np.concatenate(f), im, dims=DIMS, X=AFFINE, grid_step=4), ref)


@pytest.mark.parametrize("kind", ["zero", "dense"])
@pytest.mark.parametrize("bad", list(BAD))
@pytest.mark.parametrize("entry", [0, 3, 6, 11])
def test_affine(entry, bad, kind):
    from deedsbcv_gb300 import api
    n = int(np.prod(DIMS))
    im = _image(kind, n, np.random.default_rng(entry))
    X = np.eye(4, dtype=F32).ravel()
    X[entry] = BAD[bad]
    zero = np.zeros(n, F32)
    ref = warp_affine(im, X, zero, zero, zero, DIMS)
    assert np.isnan(ref).any()
    _check(api.warpAffine(torch.from_numpy(im).cuda(), X, None, None, None, *DIMS), ref)
    flow = np.zeros(3 * int(np.prod([d // 4 for d in DIMS])), F32)
    _check(api.apply_flow(flow, im, dims=DIMS, X=X, grid_step=4), ref)


@pytest.mark.parametrize("kind", ["zero", "dense"])
def test_linear_warp_of_a_degenerate_fit(kind):
    from deedsbcv_gb300 import api
    im = _image(kind, int(np.prod(DIMS)), np.random.default_rng(3))
    X = np.full(16, np.nan, F32)
    assert torch.isnan(api.warpAffineLinear(torch.from_numpy(im).cuda(), X, *DIMS)).all()


@pytest.mark.parametrize("other", ["zero", "smooth"])
@pytest.mark.parametrize("bad", list(BAD))
def test_consistent_mapping(bad, other):
    from deedsbcv_gb300 import api
    dims = (43, 31, 29)  # the ten steps' spread of a NaN leaves voxels without one
    sz = int(np.prod(dims))
    rng = np.random.default_rng(len(bad))
    f = [np.zeros(sz, F32) if other == "zero" else rng.normal(0, 1, sz).astype(F32) for _ in range(6)]
    f[1][sz // 2] = BAD[bad]
    f[5][7] = BAD[bad]
    dev = _cuda(f)
    api.consistentMappingCL(*dev, *dims, 4)
    ref = consistent(f, dims, 4)
    assert np.isnan(ref[0]).any() and not np.isnan(ref[0]).all()
    for a, b in zip(dev, ref):
        _check(a, b)


@pytest.mark.parametrize("bad", list(BAD))
def test_soft_warp(bad):
    from deedsbcv_gb300 import api
    grid = (8, 3, 2)
    n, nodes = int(np.prod(DIMS)), int(np.prod(grid))
    rng = np.random.default_rng(5)
    im = torch.from_numpy(_image("dense", n, rng)).cuda().requires_grad_()
    f = rng.normal(0, 2, (3, nodes)).astype(F32)
    f[:, 0] = BAD[bad]
    field = torch.from_numpy(f).cuda().requires_grad_()
    ctx = api.context(0)
    hit = ~torch.isfinite(api.SoftUpsample.apply(field, grid, DIMS, ctx)).all(0)
    out = api.SoftWarp.apply(im, field, DIMS, grid, ctx)
    assert torch.equal(torch.isnan(out), hit) and hit.any() and not hit.all()
    clean = torch.nan_to_num(field.detach(), nan=0.0, posinf=0.0, neginf=0.0)
    assert torch.equal(out[~hit], api.SoftWarp.apply(im.detach(), clean, DIMS, grid, ctx)[~hit])
    out.backward(torch.ones_like(out))
    assert not torch.isnan(im.grad).all() and torch.isnan(im.grad).any()
    assert not torch.isnan(field.grad).all() and torch.isnan(field.grad).any()


@pytest.mark.parametrize("sign", [-1, 1])
@pytest.mark.parametrize("beyond", [2.0 ** 21, 2.0 ** 26, 2.0 ** 35, 2.0 ** 90])
def test_fractions_far_outside(beyond, sign):
    from deedsbcv_gb300 import api
    n = int(np.prod(DIMS))
    rng = np.random.default_rng(int(np.log2(beyond)))
    im, f = _image("air", n, rng), _field(F32(sign * (2.0 ** 31 + beyond)), n, rng, 0.2)
    _check(api.warpImageCL(torch.from_numpy(im).cuda(), *_cuda(f), *DIMS), warp_image(im, *f, DIMS))
