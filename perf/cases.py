"""The work that users of this package have it do, as timed cases.

Each case is one call (or one training step) through the public entry points of
``deedsbcv_gb300.api`` on seeded synthetic CT-like volumes.  The kinds:

* ``register``    one deeds registration of device-resident volumes;
* ``batch``       several pairs of uneven sizes from host memory;
* ``linear``      the affine / rigid pre-registration;
* ``descriptor``  MIND-SSC codes of one volume;
* ``cost``        the cost volume of one level between two code volumes;
* ``apply``       a stored displacement field applied to a host volume;
* ``soft``        forward and backward of one differentiable level;
* ``soft_batch``  a batch of pairs in the differentiable form: forward and backward of
                  one level, or the forward pass of several;
* ``fuse``        multi-atlas label fusion of already warped atlases.

Volumes are m x n x o with i (size m) fastest; inside this file they are tensors
of shape (o, n, m).
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.utils.checkpoint

from deedsbcv_gb300 import api

# (grid, radius, quant) per level, coarse to fine
DEFAULT = "8x7x6x5x4/8x7x6x5x4/5x4x3x2x1"      # deedsBCV's default schedule
THREE = "6x5x4/5x4x3/3x2x1"                    # a quicker three-level schedule
TWO = "6x4/3x2/2x1"                            # two levels, small displacements
LINEAR = "7x6x5x4/5x4x3x2/4x3x2x1"             # linearBCV's default schedule
SOFT = "6x5x4/3x3x3/3x2x1"                     # differentiable form, 7^3 labels
SOFT_FINEST = "4/3/1"


def listed():
    return [
        # smallest call: a cropped organ region, three levels; launches and host latency
        {"name": "register_crop", "kind": "register", "m": 56, "n": 48, "o": 64, "levels": THREE, "affine": False,
         "warped": False, "whole": True},
        # an ordinary odd-sized scan after affine pre-registration, warped image wanted
        {"name": "register_odd", "kind": "register", "m": 113, "n": 97, "o": 131, "levels": DEFAULT, "affine": True,
         "warped": True, "whole": True},
        # the benchmark's full-size pair
        {"name": "register_full", "kind": "register", "m": 192, "n": 160, "o": 256, "levels": DEFAULT,
         "affine": False, "warped": False, "whole": False},
        # a cohort of uneven scans from host memory, several pairs in flight
        {"name": "batch_uneven", "kind": "batch", "sizes": "128x112x144,181x151x243,224x192x288,163x140x199",
         "levels": DEFAULT, "whole": False},
        # affine pre-registration of a full-size pair
        {"name": "linear_full", "kind": "linear", "m": 192, "n": 160, "o": 256, "levels": LINEAR, "rigid": False},
        # descriptors of one full-size volume
        {"name": "descriptor_full", "kind": "descriptor", "m": 192, "n": 160, "o": 256, "radius": 2},
        # the finest default level's cost volume at full size
        {"name": "cost_finest", "kind": "cost", "m": 192, "n": 160, "o": 256, "grid": 4, "radius": 4, "quant": 1},
        # a level of a user's own schedule on an odd volume
        {"name": "cost_custom", "kind": "cost", "m": 131, "n": 118, "o": 141, "grid": 5, "radius": 4, "quant": 3},
        # applyBCVfloat: a stored field applied to a host volume
        {"name": "apply_image", "kind": "apply", "m": 192, "n": 160, "o": 256, "grid": 4, "labels": False},
        # training step through one differentiable level on a patch
        {"name": "soft_patch", "kind": "soft", "m": 96, "n": 80, "o": 112, "grid": 4, "radius": 3, "quant": 1,
         "tau": 0.5, "keep": True},
        # training step through the finest level, four full-size pairs at once
        {"name": "soft_batch", "kind": "soft_batch", "m": 160, "n": 160, "o": 192, "pairs": 4, "levels": SOFT_FINEST,
         "tau": 0.5, "backward": True, "keep": True},
        # multi-atlas segmentation's vote
        {"name": "fuse_eight", "kind": "fuse", "m": 192, "n": 160, "o": 256, "atlases": 8, "radius": 2, "power": 2},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo=(48, 40, 56), hi=(224, 192, 288)):
    """Three sizes drawn together, so that small and large volumes both come up."""
    t = rng.random()
    out = []
    for a, b in zip(lo, hi):
        s = math.exp(math.log(a) + t * (math.log(b) - math.log(a))) * rng.uniform(0.85, 1.15)
        out.append(int(min(max(round(s), a), b)))
    return {"m": out[0], "n": out[1], "o": out[2]}


def draw(rng):
    kind = rng.choice(["register", "register", "batch", "linear", "descriptor", "cost", "cost", "apply", "soft",
                       "soft_batch", "fuse"])
    if kind == "register":
        return {"kind": kind, **_dims(rng), "levels": rng.choice([DEFAULT, DEFAULT, THREE, TWO]),
                "affine": rng.random() < 0.5, "warped": rng.random() < 0.5, "whole": rng.random() < 0.5}
    if kind == "batch":
        pairs = [_dims(rng, (64, 56, 72), (200, 176, 256)) for _ in range(rng.randint(2, 4))]
        return {"kind": kind, "sizes": ",".join(f"{p['m']}x{p['n']}x{p['o']}" for p in pairs),
                "levels": rng.choice([DEFAULT, THREE]), "whole": rng.random() < 0.5}
    if kind == "linear":
        return {"kind": kind, **_dims(rng, (64, 56, 72)), "levels": LINEAR, "rigid": rng.random() < 0.5}
    if kind == "descriptor":
        return {"kind": kind, **_dims(rng), "radius": rng.randint(1, 3)}
    if kind == "cost":
        if rng.random() < 0.5:
            g, r, q = rng.choice(_levels(DEFAULT) + _levels(LINEAR))
        else:
            g, r, q = rng.randint(3, 8), rng.randint(2, 6), rng.randint(1, 4)
        return {"kind": kind, **_dims(rng, hi=(192, 160, 256)), "grid": g, "radius": r, "quant": q}
    if kind == "apply":
        return {"kind": kind, **_dims(rng), "grid": rng.randint(3, 6), "labels": rng.random() < 0.5}
    if kind == "soft":
        g, q = rng.choice([(4, 1), (5, 2), (6, 3)])
        return {"kind": kind, **_dims(rng, (32, 32, 36), (96, 80, 112)), "grid": g, "radius": rng.randint(2, 3),
                "quant": q, "tau": rng.choice([0.1, 0.5, 2.0]), "keep": rng.random() < 0.7}
    if kind == "soft_batch":
        # a training step stays at one level: over several, the backward passes of two
        # runs differ where a coarser field moves a finer sample across a voxel face
        backward = rng.random() < 0.6
        return {"kind": kind, **_dims(rng, (40, 40, 48), (160, 160, 192)), "pairs": rng.randint(1, 3),
                "levels": rng.choice([SOFT_FINEST, "5/3/2", "6/3/3"]) if backward else SOFT,
                "tau": rng.choice([0.5, 2.0]), "backward": backward, "keep": backward and rng.random() < 0.7}
    return {"kind": kind, **_dims(rng), "atlases": _size(rng, 2, 12), "radius": rng.randint(1, 3),
            "power": rng.randint(0, 2)}


# ------------------------------------------------------------------ inputs

def _levels(text):
    g, r, q = ([int(v) for v in part.split("x")] for part in text.split("/"))
    return list(zip(g, r, q))


def _params(text):
    lv = _levels(text)
    return api.default_params(grid=[l[0] for l in lv], radius=[l[1] for l in lv], quant=[l[2] for l in lv])


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(gen, *shape):
    return torch.rand(*shape, generator=gen, device="cuda")


def _noise(gen, *shape):
    return torch.randn(*shape, generator=gen, device="cuda")


def _bspline(size, spacing):
    """(size, control points) uniform cubic B-spline weights."""
    t = torch.arange(size, device="cuda", dtype=torch.float64) / spacing + 1.0
    f = t.floor()
    u = t - f
    w = torch.stack([(1 - u) ** 3, 3 * u ** 3 - 6 * u ** 2 + 4, -3 * u ** 3 + 3 * u ** 2 + 3 * u + 1, u ** 3], 1) / 6
    ctrl = int(math.ceil(size / spacing)) + 3
    idx = (f.long()[:, None] - 1 + torch.arange(4, device="cuda")[None]).clamp(0, ctrl - 1)
    return torch.zeros(size, ctrl, device="cuda", dtype=torch.float64).scatter_add(1, idx, w).float()


def _field(gen, dims, peak, spacing=16):
    """Smooth displacement (3, o, n, m), components x, y, z, of the given peak."""
    m, n, o = dims
    B = [_bspline(s, spacing) for s in (o, n, m)]
    c = _rand(gen, 3, B[0].shape[1], B[1].shape[1], B[2].shape[1]) * 2 - 1
    f = torch.einsum("za,xb,yc,dabc->dzxy", B[0], B[1], B[2], c)
    return f * (peak / f.abs().max().clamp(min=1e-6))


def _coords(dims):
    m, n, o = dims
    r = [torch.arange(s, device="cuda", dtype=torch.float32) for s in (n, m, o)]
    return r[0][None, :, None], r[1][None, None, :], r[2][:, None, None]   # x, y, z


def _labels(gen, dims, organs=12):
    """Body mask and organ labels: random ellipsoids inside an ellipsoidal body."""
    m, n, o = dims
    x, y, z = _coords(dims)
    body = ((x - n / 2) / (0.45 * n)) ** 2 + ((y - m / 2) / (0.45 * m)) ** 2 + ((z - o / 2) / (0.45 * o)) ** 2 <= 1
    lab = torch.zeros(o, n, m, dtype=torch.int16, device="cuda")
    par = _rand(gen, organs, 6).cpu().tolist()
    for i, (a, b, c, ra, rb, rc) in enumerate(par):
        e = (((x - n * (0.5 + 0.4 * (a - 0.5))) / (n * (0.08 + 0.14 * ra))) ** 2
             + ((y - m * (0.5 + 0.4 * (b - 0.5))) / (m * (0.08 + 0.14 * rb))) ** 2
             + ((z - o * (0.5 + 0.4 * (c - 0.5))) / (o * (0.08 + 0.14 * rc))) ** 2) <= 1
        lab[e & body] = i + 1
    return body, lab


def _pull(vol, disp, dims, mode):
    """vol (o, n, m) sampled at p + disp(p)."""
    m, n, o = dims
    x, y, z = _coords(dims)
    gx, gy, gz = ((x + disp[0]) * 2 / (n - 1) - 1, (y + disp[1]) * 2 / (m - 1) - 1, (z + disp[2]) * 2 / (o - 1) - 1)
    grid = torch.stack([gy, gx, gz], -1)[None]
    return torch.nn.functional.grid_sample(vol.float()[None, None], grid, mode=mode, padding_mode="border",
                                           align_corners=True)[0, 0]


def _anatomy(gen, dims, organs=12):
    body, lab = _labels(gen, dims, organs)
    hu = torch.cat([torch.zeros(1, device="cuda"), _rand(gen, organs) * 400 - 100])
    img = hu[lab.long()]
    img[~body] = -1000.0
    return img, lab


def _pair(gen, dims, peak=10.0, whole=False, affine=None):
    """Fixed and moving CT-like volumes (o, n, m) in Hounsfield units, noise of 20 units."""
    img, _ = _anatomy(gen, dims)
    disp = _field(gen, dims, peak)
    if affine is not None:
        x, y, z = _coords(dims)
        p = torch.stack([t.expand(dims[2], dims[1], dims[0]) for t in (y, x, z)])
        A = affine.view(4, 4)
        q = torch.einsum("ab,bzxy->azxy", A[:3, :3], p) + A[:3, 3][:, None, None, None]
        disp = disp + torch.stack([q[1] - p[1], q[0] - p[0], q[2] - p[2]])
    moving = _pull(img, disp, dims, "bilinear")
    fixed, moving = (v + 20.0 * _noise(gen, *v.shape) for v in (img, moving))
    if whole:   # scanners store whole Hounsfield units
        fixed, moving = fixed.round(), moving.round()
    return fixed.contiguous(), moving.contiguous()


def _affine(gen, dims, size=1.0):
    """A small affine map about the centre: 16 floats, rows y, x, z."""
    A = torch.eye(4, device="cuda")
    A[:3, :3] += size * 0.05 * (_rand(gen, 3, 3) * 2 - 1)
    c = torch.tensor([(s - 1) / 2 for s in dims], device="cuda")
    A[:3, 3] = c - A[:3, :3] @ c + size * 4.0 * (_rand(gen, 3) * 2 - 1)
    return A.reshape(16)


def _codes(gen, dims):
    """Spatially smooth 12-channel descriptor codes: five-bit thermometer levels."""
    m, n, o = dims
    code = torch.zeros(o, n, m, dtype=torch.int64, device="cuda")
    for c in range(12):
        v = _noise(gen, 1, 1, o, n, m)
        v = torch.nn.functional.avg_pool3d(v, 3, 1, 1)[0, 0] * 12 + 2.5
        lev = v.clamp(0, 5.99).long()
        code |= ((1 << lev) - 1) << (5 * c)
    return code


def _node_field(gen, dims, g, peak):
    """A control-grid field [u, v, w] of 3 * nodes values as a .dat file holds it."""
    m, n, o = (s // g for s in dims)
    return _field(gen, (m, n, o), peak, spacing=max(16 / g, 2)).reshape(-1).contiguous()


def _host(t):
    return t.reshape(-1).cpu().numpy()


def prepare(case, seed):
    gen = _gen(seed)
    kind = case["kind"]
    st = {"case": case}
    if kind == "batch":
        st["pairs"] = []
        for text in case["sizes"].split(","):
            dims = tuple(int(v) for v in text.split("x"))
            f, mv = _pair(gen, dims, whole=case["whole"])
            st["pairs"].append(tuple(t.permute(2, 1, 0).cpu().numpy() for t in (f, mv)))   # (m, n, o), i fastest
        st["params"] = _params(case["levels"])
        return st
    dims = (case["m"], case["n"], case["o"])
    if kind == "register":
        X = _affine(gen, dims) if case["affine"] else None
        f, mv = _pair(gen, dims, peak=min(10.0, min(dims) / 12), whole=case["whole"])
        st.update(fixed=f.reshape(-1), moving=mv.reshape(-1), X=_host(X) if X is not None else None,
                  params=_params(case["levels"]))
        if case["warped"]:
            st["warped"] = torch.empty(f.numel(), device="cuda")
    elif kind == "linear":
        f, mv = _pair(gen, dims, peak=2.0, affine=_affine(gen, dims, 0.8 if not case["rigid"] else 0.3))
        lv = _levels(case["levels"])
        st.update(fixed=f.reshape(-1), moving=mv.reshape(-1),
                  params=api.linear_params([l[0] for l in lv], [l[1] for l in lv], [l[2] for l in lv],
                                           rigid=case["rigid"]))
    elif kind == "descriptor":
        f, _ = _pair(gen, dims, whole=True)
        st["image"] = f.reshape(-1)
    elif kind == "cost":
        st.update(F=_codes(gen, dims).reshape(-1), M=_codes(gen, dims).reshape(-1))
    elif kind == "apply":
        img, lab = _anatomy(gen, dims)
        vol = lab if case["labels"] else img + 20.0 * _noise(gen, *img.shape)
        st.update(volume=_host(vol), flow=_host(_node_field(gen, dims, case["grid"], 10.0)),
                  X=_host(_affine(gen, dims)))
    elif kind == "soft":
        f, mv = _pair(gen, dims, peak=3.0)
        nodes = math.prod(s // case["grid"] for s in dims)
        st.update(fixed=f.reshape(-1).requires_grad_(), moving=mv.reshape(-1).requires_grad_(),
                  alpha=torch.tensor(1.6, requires_grad=True), target=_noise(gen, 3, nodes) * 2)
        st["tree"] = api.soft_tree(st["fixed"], *dims, case["grid"])
    elif kind == "soft_batch":
        lv = _levels(case["levels"])
        pairs = [_pair(gen, dims, peak=6.0) for _ in range(case["pairs"])]
        nodes = math.prod(s // lv[-1][0] for s in dims)
        st.update(fixed=torch.stack([p[0].reshape(-1) for p in pairs]).requires_grad_(),
                  moving=torch.stack([p[1].reshape(-1) for p in pairs]).requires_grad_(),
                  alpha=torch.tensor(1.6, requires_grad=True), target=_noise(gen, case["pairs"], 3, nodes) * 2,
                  levels=[(g, r, q, int(0.5 * q + 1)) for g, r, q in lv])
        st["trees"] = [[api.soft_tree(f, *dims, l[0]) for l in lv] for f in st["fixed"].detach()]
        if not case["backward"]:
            st.update({k: st[k].detach() for k in ("fixed", "moving", "alpha")})
    elif kind == "fuse":
        img, lab = _anatomy(gen, dims)
        st["target"] = (img + 20.0 * _noise(gen, *img.shape)).reshape(-1)
        st["images"], st["labels"] = [], []
        for _ in range(case["atlases"]):   # atlases after registration: two voxels of error left
            d = _field(gen, dims, 2.0)
            st["images"].append((_pull(img, d, dims, "bilinear") + 20.0 * _noise(gen, *img.shape)).reshape(-1))
            st["labels"].append(_pull(lab, d, dims, "nearest").to(torch.int16).reshape(-1))
    else:
        raise ValueError(kind)
    st["dims"] = dims
    return st


# ------------------------------------------------------------------ one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        return [flow for flow, _ in api.register_batch(state["pairs"], params=state["params"])]
    m, n, o = state["dims"]
    if kind == "register":
        flow = api.register_device(state["fixed"], state["moving"], m, n, o, X=state["X"], params=state["params"],
                                   warped_out=state.get("warped"))
        return [flow, state["warped"]] if case["warped"] else flow
    if kind == "linear":
        return api.linear_register(state["fixed"], state["moving"], (m, n, o), state["params"])
    if kind == "descriptor":
        return api.descriptor(state["image"], m, n, o, case["radius"])
    if kind == "cost":
        return api.dataCostCL(state["F"], state["M"], m, n, o, case["grid"], case["radius"], case["quant"], 1.6)
    if kind == "apply":
        return api.apply_flow(state["flow"], state["volume"], dims=(m, n, o), X=state["X"], grid_step=case["grid"])
    if kind == "soft":
        d = api.soft_level(state["fixed"], state["moving"], state["alpha"], (m, n, o), grid=case["grid"],
                           radius=case["radius"], quant=case["quant"], tau=case["tau"], tree=state["tree"],
                           keep_state=case["keep"])
    elif kind == "soft_batch":
        d = api.soft_register_levels_batch(state["fixed"], state["moving"], state["alpha"], (m, n, o),
                                           state["levels"], tau=case["tau"], trees=state["trees"],
                                           keep_state=case["keep"])
    else:
        return api.fuse_labels_device(state["target"], state["images"], state["labels"], m, n, o,
                                      radius=case["radius"], power=case["power"])
    if kind == "soft_batch" and not case["backward"]:
        return d
    loss = ((d - state["target"]) ** 2).mean()
    grads = torch.autograd.grad(loss, (state["fixed"], state["moving"], state["alpha"]))
    return [d.detach(), *grads]


# ------------------------------------------------------------------ work

def _samples(g):
    s = 2 if g > 4 else 1
    return g * math.ceil(g / s) ** 2


def _level_work(m, n, o, g, r, q):
    """(cost-volume operations, message operations) of one direction of one level:
    a code difference and a 64-bit count per sample and label; two operations per
    candidate of the separable minimum, upward and downward pass."""
    nodes = (m // g) * (n // g) * (o // g)
    length = 2 * r + 1
    return 2 * nodes * length ** 3 * _samples(g), 6 * nodes * length ** 4


def _register_work(m, n, o, levels, messages=True):
    sz = m * n * o
    ops = 0
    for g, r, q in levels:
        c, msg = _level_work(m, n, o, g, r, q)
        ops += 2 * (c + (msg if messages else 0))
        ops += 4 * 150 * sz   # two descriptors, two warps
    return ops


def _soft_work(m, n, o, g, r):
    """Forward and backward of one differentiable level: five operations a term of
    the cost and eight of its adjoint, messages and marginals and their adjoints."""
    nodes = (m // g) * (n // g) * (o // g)
    length = 2 * r + 1
    return nodes * length ** 3 * _samples(g) * 12 * 13 + 4 * 3 * 5 * nodes * length ** 4 + 600 * m * n * o


def work(case):
    kind = case["kind"]
    if kind == "batch":
        lv = _levels(case["levels"])
        b = f = 0
        for text in case["sizes"].split(","):
            m, n, o = (int(v) for v in text.split("x"))
            g = lv[-1][0]
            b += 8 * m * n * o + 12 * (m // g) * (n // g) * (o // g)
            f += _register_work(m, n, o, lv)
        return {"bytes": b, "flops": f}
    m, n, o = case["m"], case["n"], case["o"]
    sz = m * n * o
    if kind == "register":
        lv = _levels(case["levels"])
        g = lv[-1][0]
        out = 12 * (m // g) * (n // g) * (o // g) + (4 * sz if case["warped"] else 0)
        return {"bytes": 8 * sz + out, "flops": _register_work(m, n, o, lv)}
    if kind == "linear":
        return {"bytes": 8 * sz + 64, "flops": _register_work(m, n, o, _levels(case["levels"]), messages=False)}
    if kind == "descriptor":   # shifted squares, three running sums, normalisation, five thresholds a channel
        return {"bytes": 12 * sz, "flops": (6 * (2 + 3 * 3) + 12 * 8) * sz}
    if kind == "cost":
        g, r, q = case["grid"], case["radius"], case["quant"]
        nodes = (m // g) * (n // g) * (o // g)
        return {"bytes": 16 * sz + 4 * nodes * (2 * r + 1) ** 3, "flops": _level_work(m, n, o, g, r, q)[0]}
    if kind == "apply":
        g = case["grid"]
        each = 2 if case["labels"] else 4
        return {"bytes": 2 * each * sz + 12 * (m // g) * (n // g) * (o // g), "flops": 60 * sz}
    if kind == "soft":
        g = case["grid"]
        nodes = (m // g) * (n // g) * (o // g)
        return {"bytes": 16 * sz + 24 * nodes, "flops": _soft_work(m, n, o, g, case["radius"])}
    if kind == "soft_batch":
        lv = _levels(case["levels"])
        g = lv[-1][0]
        nodes = (m // g) * (n // g) * (o // g)
        part = 1.0 if case["backward"] else 0.35   # the forward's share of the operations
        return {"bytes": int(case["pairs"] * ((16 if case["backward"] else 8) * sz + 24 * nodes)),
                "flops": int(case["pairs"] * part * sum(_soft_work(m, n, o, g, r) for g, r, q in lv))}
    a = case["atlases"]
    return {"bytes": sz * (4 + 6 * a + 2), "flops": sz * a * (2 + 3 * (2 * case["radius"] + 1) + 3)}


# ------------------------------------------------------------------ 64-bit values

def exact(case, seed):
    kind = case["kind"]
    if kind == "cost":
        return _exact_cost(case, prepare(case, seed))
    if kind == "apply":
        return None if case["labels"] else _exact_apply(case, prepare(case, seed))
    if kind == "soft":
        return _exact_soft(case, prepare(case, seed))
    # registrations end in labels chosen among costs, linear fits in points selected by
    # them, codes and votes are whole numbers; the batch takes too long
    return None


def _popcount(v):
    m1, m2, m4 = 0x5555555555555555, 0x3333333333333333, 0x0F0F0F0F0F0F0F0F
    v = v - ((v >> 1) & m1)
    v = (v & m2) + ((v >> 2) & m2)
    v = (v + (v >> 4)) & m4
    v = v + (v >> 8)
    v = v + (v >> 16)
    return (v + (v >> 32)) & 0x7F


def _block_sums(case, dims, diff):
    """Sum over each node's sampled block of diff(label shift) for every label:
    (nodes, labels); diff returns an (o, n, m) volume for one shift."""
    m, n, o = dims
    g, r, q = case["grid"], case["radius"], case["quant"]
    m1, n1, o1 = m // g, n // g, o // g
    s = 2 if g > 4 else 1
    out = []
    for lz in range(-r, r + 1):
        for lx in range(-r, r + 1):
            for ly in range(-r, r + 1):
                v = diff(lz * q, lx * q, ly * q)[:o1 * g, :n1 * g, :m1 * g].view(o1, g, n1, g, m1, g)
                out.append(v[:, ::s, :, ::s].sum((1, 3, 5)).reshape(-1))
    return torch.stack(out, 1)


def _shifter(dims):
    m, n, o = dims
    ar = [torch.arange(s, device="cuda") for s in (o, n, m)]

    def shift(vol, dz, dx, dy):   # vol[..., clamp(k + dz), clamp(j + dx), clamp(i + dy)]
        for dim, d, a, s in zip((-3, -2, -1), (dz, dx, dy), ar, (o, n, m)):
            vol = vol.index_select(vol.dim() + dim, (a + d).clamp(0, s - 1))
        return vol
    return shift


def _scale(case, alpha):
    g, q = case["grid"], case["quant"]
    return 0.5 * (g / (alpha * q)) / _samples(g)


def _exact_cost(case, st):
    dims = st["dims"]
    m, n, o = dims
    F, M = (st[k].view(o, n, m) for k in ("F", "M"))
    shift = _shifter(dims)
    sums = _block_sums(case, dims, lambda dz, dx, dy: _popcount(F ^ shift(M, dz, dx, dy)))
    return (sums.double() * _scale(case, 1.6)).reshape(-1)


def _trilinear(vol, x, y, z):
    o, n, m = vol.shape
    x0, y0, z0 = x.floor(), y.floor(), z.floor()
    dx, dy, dz = x - x0, y - y0, z - z0
    acc = 0
    for cz in (0, 1):
        for cx in (0, 1):
            for cy in (0, 1):
                idx = (((z0 + cz).clamp(0, o - 1) * n + (x0 + cx).clamp(0, n - 1)) * m
                       + (y0 + cy).clamp(0, m - 1)).long()
                w = (dz if cz else 1 - dz) * (dx if cx else 1 - dx) * (dy if cy else 1 - dy)
                acc = acc + w * vol.reshape(-1)[idx]
    return acc


def _exact_apply(case, st):
    m, n, o = dims = st["dims"]
    g = case["grid"]
    g1 = (o // g, n // g, m // g)
    flow = torch.from_numpy(st["flow"]).cuda().double().view(3, *g1)
    X = torch.from_numpy(st["X"]).cuda().double()
    x, y, z = (t.double() for t in _coords(dims))
    gx, gy, gz = torch.broadcast_tensors(x * (g1[1] / n), y * (g1[2] / m), z * (g1[0] / o))
    u, v, w = (_trilinear(f, gx, gy, gz) for f in flow)
    py = y * X[0] + x * X[1] + z * X[2] + X[3] + v
    px = y * X[4] + x * X[5] + z * X[6] + X[7] + u
    pz = y * X[8] + x * X[9] + z * X[10] + X[11] + w
    vol = torch.from_numpy(st["volume"]).cuda().double().view(o, n, m)
    return _trilinear(vol, px, py, pz).reshape(-1)


def _box(x, r):
    for dim in (-1, -2, -3):
        size = x.shape[dim]
        p = torch.nn.functional.pad(x.cumsum(dim).movedim(dim, -1), (1, 0))
        a = torch.arange(size, device=x.device)
        x = (p[..., (a + r + 1).clamp(max=size)] - p[..., (a - r).clamp(min=0)]).movedim(-1, dim)
    return x


def _soft_descriptor(vol, r):
    """(12, o, n, m) levels 6 exp(-d / mean d) of the self-similarity distances."""
    def at(v, dz, dx, dy):   # the neighbour, or the voxel itself outside the volume
        for dim, d in ((-3, dz), (-2, dx), (-1, dy)):
            if d:
                assert abs(d) < v.shape[dim]
        o, n, m = v.shape
        k, j, i = (torch.arange(s, device=v.device) for s in (o, n, m))
        ok = (((k + dz >= 0) & (k + dz < o))[:, None, None] & ((j + dx >= 0) & (j + dx < n))[None, :, None]
              & ((i + dy >= 0) & (i + dy < m))[None, None, :])
        return torch.where(ok, v.roll((-dz, -dx, -dy), (0, 1, 2)), v)
    dx, dy, dz = (1, 1, -1, 0, 1, 0), (1, -1, 0, -1, 0, 1), (0, 0, 1, 1, 1, 1)
    sx, sy = (-1, 0, -1, 0, 0, 1, 0, 0, 0, -1, 0, 0), (0, -1, 0, 1, 0, 0, 0, 1, 0, 0, 0, -1)
    sz = (0, 0, 0, 0, -1, 0, -1, 0, -1, 0, -1, 0)
    d = [_box((at(vol, dz[c] * r, dx[c] * r, dy[c] * r) - vol) ** 2, r) for c in range(6)]
    v = torch.stack([at(d[c // 2], sz[c] * r, sx[c] * r, sy[c] * r) for c in range(12)])
    v = v - v.min(0, keepdim=True).values
    return 6 * torch.exp(-v / (v.sum(0, keepdim=True) / 12).clamp(min=1e-6))


def _lse(x, tau, length):
    """logsumexp over a of x[..., a] - |a - b|^2 / tau along the three label axes of x
    (nodes, z, x, y)."""
    a = torch.arange(length, device=x.device, dtype=x.dtype)
    pen = -((a[:, None] - a[None, :]) ** 2) / tau
    for dim in (1, 2, 3):
        x = torch.logsumexp(x.movedim(dim, -1)[..., :, None] + pen, -2).movedim(-1, dim)
    return x


def _exact_soft(case, st):
    """The level in 64-bit floats: descriptor, robust cost, soft-min messages up the
    tree, marginals down, expected displacement; gradients by autograd."""
    m, n, o = dims = st["dims"]
    g, r, q, tau = case["grid"], case["radius"], case["quant"], case["tau"]
    length, eps = 2 * r + 1, 0.01
    qs = int(0.5 * q + 1)
    fixed, moving = (st[k].detach().double().view(o, n, m).requires_grad_() for k in ("fixed", "moving"))
    alpha = torch.tensor(1.6, dtype=torch.float64, device="cuda", requires_grad=True)
    sF, sM = _soft_descriptor(fixed, qs), _soft_descriptor(moving, qs)
    shift = _shifter(dims)

    def term(a, b, dz, dx, dy):
        return torch.sqrt((a - shift(b, dz, dx, dy)) ** 2 + eps * eps).sum(0) - 12 * eps

    def diff(dz, dx, dy):
        return torch.utils.checkpoint.checkpoint(term, sF, sM, dz, dx, dy, use_reentrant=False)

    # the 32-bit entry point takes alpha as a float
    cost = _block_sums(case, dims, diff) * (0.5 * (g / (alpha.float().double() * q)) / _samples(g))
    ordered, parents, weight = (np.asarray(a) for a in st["tree"])
    nodes = len(ordered)
    depth = np.zeros(nodes, np.int64)
    for t in ordered[1:]:
        depth[t] = depth[parents[t]] + 1
    order = np.argsort(depth, kind="stable")
    starts = np.searchsorted(depth[order], np.arange(depth.max() + 2))
    groups = [torch.from_numpy(order[starts[d]:starts[d + 1]]).cuda() for d in range(len(starts) - 1)]
    slot = np.zeros(nodes, np.int64)
    for d in range(len(starts) - 1):
        slot[order[starts[d]:starts[d + 1]]] = np.arange(starts[d + 1] - starts[d])
    parent = torch.from_numpy(slot[np.where(depth > 0, parents, ordered[0])]).cuda()
    edge = torch.from_numpy(weight.astype(np.float64)).cuda()
    shape = (-1, length, length, length)
    belief, message = [None] * len(groups), [None] * len(groups)
    for d in range(len(groups) - 1, -1, -1):
        b = cost[groups[d]]
        if d + 1 < len(groups):
            b = b.index_add(0, parent[groups[d + 1]], message[d + 1] - message[d + 1].detach().amin(1, keepdim=True))
        belief[d] = b * edge[groups[d]][:, None] if d else b
        if d:
            message[d] = -tau * _lse((-belief[d] / tau).view(shape), tau, length).reshape(len(b), -1)
    logp = torch.log_softmax(-belief[0] / tau, 1)
    marg = [logp]
    for d in range(1, len(groups)):
        up = logp[parent[groups[d]]] + message[d] / tau
        logp = -belief[d] / tau + _lse(up.view(shape), tau, length).reshape(len(up), -1)
        marg.append(logp)
    prob = torch.zeros(nodes, length ** 3, dtype=torch.float64, device="cuda")
    prob = prob.index_copy(0, torch.cat(groups), torch.cat(marg).exp())
    lab = torch.arange(length ** 3, device="cuda")
    steps = torch.stack([lab // length % length, lab % length, lab // length ** 2], 1).double()   # x, y, z
    disp = (prob @ ((steps - r) * q)).T
    loss = ((disp - st["target"].double()) ** 2).mean()
    gf, gm, ga = torch.autograd.grad(loss, (fixed, moving, alpha))
    return [disp.detach(), gf.reshape(-1), gm.reshape(-1), ga.cpu()]
