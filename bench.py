"""Benchmark: deeds registrations per second at 192x160x256, 5 default levels.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl gb300|reference]

One step = one full 5-level deeds registration (forward + backward per level,
inverse-consistent mapping) of one seeded synthetic CT-like pair, through the
library's C ABI.  ``value`` is measured with inputs already in HBM
(deeds_register_dev) with CUDA events on the launching stream; ``e2e`` through
deeds_register with host buffers (H2D of both images and D2H of the
displacement field inside the timed region).  The per-step working set
(cost volume 289-358 MB, three code volumes 189 MB, MIND scratch 189 MB) is
larger than the 129 MB L2, so every step runs cold.

--impl reference times the unmodified reference deedsBCV (built on this host by
oracle/Makefile from the reference's sources staged in oracle/_ref/src) on all
host cores, one full registration of the same pair per step, by the binary's
own timer; the oracle restatement stands in only where the binary was not
built.

Multi-GPU: registrations are independent, so N GPUs run N replicas (one process
per GPU, no collective on the data path); value = all ranks' pairs / max time.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

SHAPE = (192, 160, 256)
G, L, Q = (8, 7, 6, 5, 4), (8, 7, 6, 5, 4), (5, 4, 3, 2, 1)
METRIC = "pairs/s at 192x160x256 (5 levels)"
# DRAM bytes (read + write) of one finest-level launch at 192x160x256, from
# `ncu --metrics dram__bytes_read.sum,dram__bytes_write.sum` captures of the
# bench workload (under profiles/; mean of two launches),
# beside the algorithmic bytes of the same launch as `achieved` counts them
# (k_bp_up: the 122,880 x 729 float cost volume read and its message rows
# written; k_data_cost_mma: both code volumes read once, the cost volume written).
TRAFFIC = {"k_bp_up": 1029424768, "k_data_cost_mma": 422125440}
TRAFFIC_ALGORITHMIC = {"k_bp_up": 2 * 122880 * 729 * 4, "k_data_cost_mma": 2 * 192 * 160 * 256 * 8 + 122880 * 729 * 4}
TRAFFIC_NOTE = ("finest-level launch (grid 4) at 192x160x256, ncu dram__bytes_read.sum + dram__bytes_write.sum; "
                "k_bp_up also writes each node's scaled input row, which the downward pass reads to evaluate "
                "the node's label")
SEED = 2


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--small", action="store_true", help="96x80x128 workload (profiling runs)")
    ap.add_argument("--no-batched", action="store_true", help="skip the 16-pair batched measurement")
    ap.add_argument("--lanes", type=int, default=3, help="pairs in flight for the batched form")
    ap.add_argument("--no-soft", action="store_true", help="skip the soft-min (differentiable) measurement")
    ap.add_argument("--soft-only", action="store_true",
                    help="only the soft-min measurement (one JSON object; for profiling runs)")
    ap.add_argument("--soft-pairs", type=int, default=4)
    ap.add_argument("--soft-taus", default="0.1,0.5,2.0")
    ap.add_argument("--soft-shape", default="160x160x192", help="soft-min pair shape (profiling runs use smaller)")
    ap.add_argument("--soft-single", action="store_true", help="--soft-only: the finest soft level alone")
    ap.add_argument("--no-linear", action="store_true", help="skip the linearBCV measurement")
    ap.add_argument("--linear-only", action="store_true", help="only the linearBCV measurement (one JSON object)")
    ap.add_argument("--profile-once", action="store_true",
                    help="one warm-up registration of the workload, then one inside an NVTX range 'deeds_pair' "
                         "(for ncu --nvtx --nvtx-include deeds_pair/), and exit")
    return ap.parse_args()


def dist_env():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return ws, rank, local


def replica_rate(local_s, steps, device=None):
    """Pairs/s of the whole job: every rank (one replica per GPU, no collective on
    the data path) registers `steps` pairs; the job's time is the slowest rank's
    (max over ranks), so value = ranks * steps / max time.  Returns (value, time)."""
    import torch
    import torch.distributed as dist
    ws = dist.get_world_size() if dist.is_available() and dist.is_initialized() else 1
    t = float(local_s)
    if ws > 1:
        x = torch.tensor([t], dtype=torch.float64, device=device)
        dist.all_reduce(x, op=dist.ReduceOp.MAX)
        t = float(x.item())
    return ws * steps / t, t


def popc64_per_pair(shape):
    """Algorithmic 64-bit Hamming operations of one pair (both directions)."""
    m, n, o = shape
    total = 0
    for g, hw in zip(G, L):
        skip = 2 if g > 4 else 1
        samples = -(-g // skip) * -(-g // skip) * g
        total += 2 * (m // g) * (n // g) * (o // g) * (2 * hw + 1) ** 3 * samples
    return total


def isolated_data_cost(api, ctx, pair, shape, reps=3):
    """Each level's cost-volume launch timed alone (CUDA events on the launching
    stream, after a warm-up), on the workload's own descriptor codes: the two
    direction streams of a registration share the GPU, so per-stage times inside
    the pipeline overstate a single launch.  Returns (popc64, seconds, per-level)."""
    import torch
    m, n, o = shape
    fx = torch.from_numpy(np.ascontiguousarray(pair["fixed"].ravel(order="F") + np.float32(1024))).cuda()
    mv = torch.from_numpy(np.ascontiguousarray(pair["moving"].ravel(order="F") + np.float32(1024))).cuda()
    total_pop, total_s, per = 0, 0.0, []
    for g, hw, q in zip(G, L, Q):
        qs = int(np.floor(0.5 * q + 1.0))
        F = api.descriptor(fx, m, n, o, qs, ctx)
        M = api.descriptor(mv, m, n, o, qs, ctx)
        api.dataCostCL(F, M, m, n, o, g, hw, q, 1.6, ctx)  # warm-up (and tile choice)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        e0.record()
        for _ in range(reps):
            api.dataCostCL(F, M, m, n, o, g, hw, q, 1.6, ctx)
        e1.record()
        torch.cuda.synchronize()
        sec = e0.elapsed_time(e1) / 1000.0 / reps
        skip = 2 if g > 4 else 1
        pop = (m // g) * (n // g) * (o // g) * (2 * hw + 1) ** 3 * (-(-g // skip)) ** 2 * g
        per.append({"grid": g, "ms": round(sec * 1000, 3), "Tpopc64_s": round(pop / sec / 1e12, 3)})
        total_pop += pop
        total_s += sec
    return total_pop, total_s, per


def tree_depth(ordered, parents):
    """Breadth levels of a tree given in breadth-level order (root first)."""
    depth = np.zeros(len(ordered), np.int64)
    for v in ordered[1:]:
        depth[v] = depth[parents[v]] + 1
    return int(depth.max()) + 1


def isolated_bp(api, ctx, pair, shape, reps=3):
    """Each level's tree belief propagation timed alone on the workload's own
    cost volume and MST (forward direction, zero prior field), as the registration
    runs it (no argmin tables: the downward pass evaluates each node's entry from
    its stored row): the upward sweep (k_bp_up) and the downward pass (k_bp_down)
    from the library's per-stage CUDA events.  Returns per-level rows and the sums
    over the 5 levels of one direction."""
    import torch
    m, n, o = shape
    fx = torch.from_numpy(np.ascontiguousarray(pair["fixed"].ravel(order="F") + np.float32(1024))).cuda()
    mv = torch.from_numpy(np.ascontiguousarray(pair["moving"].ravel(order="F") + np.float32(1024))).cuda()
    per, tot = [], {"up_ms": 0.0, "argmin_ms": 0.0, "down_ms": 0.0, "cost_bytes": 0}
    for g, hw, q in zip(G, L, Q):
        qs = int(np.floor(0.5 * q + 1.0))
        F = api.descriptor(fx, m, n, o, qs, ctx)
        M = api.descriptor(mv, m, n, o, qs, ctx)
        cost0 = api.dataCostCL(F, M, m, n, o, g, hw, q, 1.6, ctx)
        ordered, parents, edgemst = api.primsGraph(fx, m, n, o, g, ctx)
        m1, n1, o1 = m // g, n // g, o // g
        sz1 = m1 * n1 * o1
        z = torch.zeros(sz1, dtype=torch.float32, device=fx.device)
        c = cost0.clone()
        api.regularisationCL(c, z, z, z, m1, n1, o1, hw, q, ordered, parents, edgemst, ctx=ctx)
        torch.cuda.synchronize()
        ctx.reset_stage_times()
        ctx.set_profiling(True)
        for _ in range(reps):
            c.copy_(cost0)
            api.regularisationCL(c, z, z, z, m1, n1, o1, hw, q, ordered, parents, edgemst, ctx=ctx)
        torch.cuda.synchronize()
        ctx.set_profiling(False)
        st = ctx.stage_times()
        up, arg, down = (st[k][0] / reps for k in ("bp_up", "bp_argmin", "bp_down"))
        depth = tree_depth(ordered, parents)
        cost_bytes = sz1 * (2 * hw + 1) ** 3 * 4
        per.append({"grid": g, "label_width": 2 * hw + 1, "nodes": sz1, "tree_depth": depth,
                    "up_ms": round(up, 3), "argmin_ms": round(arg, 3), "down_ms": round(down, 3),
                    "up_us_per_depth_step": round(up * 1000.0 / depth, 2),
                    "up_GBs_on_cost_volume": round(2 * cost_bytes / (up / 1000.0) / 1e9, 1)})
        tot["up_ms"] += up
        tot["argmin_ms"] += arg
        tot["down_ms"] += down
        tot["cost_bytes"] += cost_bytes
    return per, tot


def isolated_mind(api, ctx, pair, shape, reps=5):
    """One MIND-SSC descriptor call (i pass, j pass, k pass, quantise) of the
    fixed image timed alone per distinct radius of the schedule; returns
    (seconds per call averaged over the radii, voxels)."""
    import torch
    m, n, o = shape
    fx = torch.from_numpy(np.ascontiguousarray(pair["fixed"].ravel(order="F") + np.float32(1024))).cuda()
    total, calls = 0.0, 0
    for qs in sorted({int(np.floor(0.5 * q + 1.0)) for q in Q}):
        api.descriptor(fx, m, n, o, qs, ctx)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        e0.record()
        for _ in range(reps):
            api.descriptor(fx, m, n, o, qs, ctx)
        e1.record()
        torch.cuda.synchronize()
        total += e0.elapsed_time(e1) / 1000.0 / reps
        calls += 1
    return total / calls, m * n * o


def mind_calls():
    steps = [int(np.floor(0.5 * q + 1.0)) for q in Q]
    extra = sum(1 for i, s in enumerate(steps) if i == 0 or s != steps[i - 1])
    return 2 * len(G) + 2 * extra


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled every 200 ms."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.path = None

    def __enter__(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None
        time.sleep(0.3)
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        rows = []
        try:
            with open(self.path) as f:
                for line in f:
                    parts = [p.strip() for p in line.split(",")]
                    if len(parts) >= 9:
                        rows.append(parts)
            os.unlink(self.path)
        except OSError:
            pass
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"], "samples": 0}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in rows for i in range(4) if r[5 + i].lower().startswith("active")})
        load = [s for s in sm if mx and s > 0.5 * max(mx)] or sm
        return {"sm_mhz": float(np.median(load)) if load else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(rows)}


def make_workload(shape):
    from deedsbcv_gb300 import phantom
    return phantom.make_pair(shape, seed=SEED, n_organs=13, max_disp=10.0)


def pinned(vol):
    """A Fortran-ordered (m, n, o) view of a pinned host copy of `vol`."""
    import torch
    flat = torch.from_numpy(np.ascontiguousarray(np.asarray(vol, np.float32).ravel(order="F"))).pin_memory()
    return flat.numpy().reshape(vol.shape, order="F")


def batched_pairs(n=16, seed=100):
    """16 pairs with dims drawn uniformly from 128x112x144 .. 224x192x288 (max
    10-voxel deformation), the uneven-size batch workload, in pinned host memory."""
    from deedsbcv_gb300 import phantom
    out = []
    for shape, s in phantom.batch_workload(n, seed):
        p = phantom.make_pair(shape, seed=s, max_disp=10.0)
        out.append((pinned(p["fixed"]), pinned(p["moving"])))
    return out


def measure_batched(api, ctx, lanes):
    """Plain (one pair per call) vs batched (deeds_register_batch) on the same
    16 uneven pairs; both after one untimed pass that sizes buffers and tiles."""
    pairs = batched_pairs()
    params = api.default_params()
    api.register_batch(pairs, params=params, lanes=lanes, ctx=ctx)  # warm: buffers, tiles, lanes
    for f, mv in pairs[:2]:
        api.register(f, mv, params=params, want_warped=False, ctx=ctx)
    t0 = time.perf_counter()
    plain = [api.register(f, mv, params=params, want_warped=False, ctx=ctx)[0] for f, mv in pairs]
    t_plain = time.perf_counter() - t0
    t0 = time.perf_counter()
    batched = api.register_batch(pairs, params=params, lanes=lanes, ctx=ctx)
    t_batch = time.perf_counter() - t0
    same = all(np.array_equal(a, b[0]) for a, b in zip(plain, batched))
    voxels = sum(int(np.prod(f.shape)) for f, _ in pairs)
    return {"pairs": len(pairs), "lanes": lanes, "mean_voxels": voxels // len(pairs),
            "plain_pairs_per_s": len(pairs) / t_plain, "batched_pairs_per_s": len(pairs) / t_batch,
            "speedup": t_plain / t_batch, "flows_identical": bool(same),
            "workload": "16 pairs, dims uniform in 128x112x144..224x192x288, pinned host buffers end to end"}


SOFT_SHAPE = (160, 160, 192)
SOFT_TAUS = (0.1, 0.5, 2.0)
# (grid, radius, quant, MIND radius) per level, coarse to fine: label set 7^3 at
# every level, displacement range +-9, +-6 and +-3 voxels
SOFT_LEVELS = ((6, 3, 3, 2), (5, 3, 2, 2), (4, 3, 1, 1))


def measure_soft(api, ctx, n_pairs=4, levels=SOFT_LEVELS, taus=SOFT_TAUS, shape=SOFT_SHAPE):
    """Differentiable soft-min registration on 4 pairs at 160x160x192, label set 7^3
    at the finest level, tau in {0.1, 0.5, 2.0}: forward (expected displacement
    after the last level) + backward (hand-written adjoints: gradients w.r.t. both
    images and alpha) of loss = MSE between that field and the seeded ground-truth
    field at the finest control points.  With several levels each level's prior is
    the previous field upsampled, the moving image is warped by it and the
    pairwise term is taken relative to it.  Each pair's MSTs are built once from
    its fixed image (constants of the levels) before timing; device time with CUDA
    events over all pairs per tau."""
    import torch
    from deedsbcv_gb300 import phantom
    m, n, o = shape
    g = levels[-1][0]
    m1, n1, o1 = m // g, n // g, o // g
    data = []
    for i in range(n_pairs):
        pr = phantom.make_pair(shape, seed=200 + i, max_disp=10.0)
        fx = torch.from_numpy(pr["fixed"].ravel(order="F").astype(np.float32)).cuda()
        mv = torch.from_numpy(pr["moving"].ravel(order="F").astype(np.float32)).cuda()
        c = g // 2
        d = pr["disp"][:, c::g, c::g, c::g][:, :m1, :n1, :o1]  # (y, x, z) components at node voxels
        gt = -np.stack([d[1], d[0], d[2]]).reshape(3, -1, order="F")  # u (x), v (y), w (z), node order y fastest
        trees = [api.soft_tree(fx, m, n, o, lv[0], ctx) for lv in levels]
        data.append((fx, mv, torch.from_numpy(gt.astype(np.float32)).cuda(), trees))

    FX = torch.stack([d[0] for d in data])
    MV = torch.stack([d[1] for d in data])
    GT = torch.stack([d[2] for d in data])
    TREES = [d[3] for d in data]

    def step_one(fx, mv, gt, trees, tau, keep=True):
        F, M = fx.detach().requires_grad_(), mv.detach().requires_grad_()
        a = torch.tensor(1.6, requires_grad=True)
        disp = api.soft_register_levels(F, M, a, shape, levels, tau=tau, trees=trees, ctx=ctx, keep_state=keep)
        loss = ((disp - gt) ** 2).mean()
        loss.backward()
        return loss.detach()

    def step_batch(tau, backward=True, keep=True):
        # loss = sum over pairs of each pair's MSE: pair i's gradients are those
        # of its own MSE
        F, M = FX.detach().requires_grad_(backward), MV.detach().requires_grad_(backward)
        a = torch.tensor(1.6, requires_grad=backward)
        disp = api.soft_register_levels_batch(F, M, a, shape, levels, tau=tau, trees=TREES, ctx=ctx,
                                              keep_state=keep)
        per_pair = ((disp - GT) ** 2).mean(dim=(1, 2))
        if backward:
            per_pair.sum().backward()
            return per_pair.detach(), F.grad[-1], M.grad[-1], a.grad
        return per_pair.detach(), None, None, None

    out = {}
    launches0 = api.kernel_launches()
    for tau in taus:
        step_batch(tau)  # warm-up: buffers of every lane
        step_batch(tau, keep=False)
        step_one(*data[0], tau)
        res = {}
        # forward_backward: the pairs of each level run concurrently on lane
        # streams and each level's forward state stays on the device for its
        # backward; _recompute: the backward recomputes that state instead;
        # _one_by_one: the pairs one after another through soft_register_levels
        for mode in ("forward", "forward_backward", "forward_backward_recompute", "forward_backward_one_by_one"):
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            if mode == "forward_backward_one_by_one":
                losses = torch.stack([step_one(fx, mv, gt, tr, tau) for fx, mv, gt, tr in data])
            else:
                losses, gf, gm, ga = step_batch(tau, backward=(mode != "forward"),
                                                keep=(mode != "forward_backward_recompute"))
            e1.record()
            torch.cuda.synchronize()
            ms = e0.elapsed_time(e1)
            res[mode + "_ms_per_pair"] = ms / len(data)
            if mode == "forward_backward_recompute":
                # the form that recomputes each level's forward state in the backward
                # instead of keeping it on the device
                res["pairs_per_s_recompute"] = 1000.0 * len(data) / ms
            if mode == "forward_backward":
                res["pairs_per_s"] = 1000.0 * len(data) / ms
                res["grad_norms_last_pair"] = {"fixed": float(gf.norm()), "moving": float(gm.norm()),
                                               "alpha_all_pairs": float(ga)}
                res["mean_loss"] = float(losses.mean())
        out[str(tau)] = res
    lv = " ".join(f"G{a}L{b}Q{c}" for a, b, c, _ in levels)
    return {"workload": f"{n_pairs} pairs {m}x{n}x{o} (seeds 200..{199 + n_pairs}), soft levels {lv}, label set "
                        f"{2 * levels[-1][1] + 1}^3 at the finest, alpha 1.6, eps 0.01; loss = MSE(expected "
                        f"displacement, ground-truth field at control points); MSTs per pair built before timing",
            "per_tau": out, "gpu_launches": api.kernel_launches() - launches0}


def measure_linear(api, ctx, shape, steps=5, warmup=3, cpu=True):
    """linearBCV (4 default levels, affine fit) on one 192x160x256 pair with a seeded
    affine misalignment (up to 6 degrees, 6% scaling, 5 voxels) plus a 2-voxel
    B-spline field.  e2e: through the public host-buffer call (copies in, matrix
    out; the call returns after the work), wall clock.  value: the device-pointer
    call on resident inputs, CUDA events on its stream.  The oracle restatement of
    the same registration gives the CPU baseline and the bit-parity check."""
    import torch
    from deedsbcv_gb300 import phantom
    pair = phantom.make_pair(shape, seed=21, max_disp=2.0, affine=(6.0, 0.06, 5.0))
    f = np.ascontiguousarray(pair["fixed"].ravel(order="F"), np.float32)
    mv = np.ascontiguousarray(pair["moving"].ravel(order="F"), np.float32)
    params = api.linear_params()
    for _ in range(warmup):
        X = api.linear_register(f, mv, shape, params, ctx)
    t0 = time.perf_counter()
    for _ in range(steps):
        X = api.linear_register(f, mv, shape, params, ctx)
    e2e_s = (time.perf_counter() - t0) / steps
    df, dm = torch.from_numpy(f).cuda(), torch.from_numpy(mv).cuda()
    launches0 = api.kernel_launches()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(steps):
        Xd = api.linear_register(df, dm, shape, params, ctx)
    e1.record()
    torch.cuda.synchronize()
    dev_s = e0.elapsed_time(e1) / 1000.0 / steps
    launches = (api.kernel_launches() - launches0) // steps
    # one more registration with per-stage CUDA events: the GPU stages; the rest of
    # the pair time is cost smoothing, node statistics and the host fit
    ctx.reset_stage_times()
    ctx.set_profiling(True)
    t0 = time.perf_counter()
    api.linear_register(df, dm, shape, params, ctx)
    prof_s = time.perf_counter() - t0
    ctx.set_profiling(False)
    st = ctx.stage_times()
    ctx.reset_stage_times()
    gpu_stages = {k: round(v[0], 3) for k, v in st.items() if v[1] > 0}
    A = pair["affine"].reshape(4, 4).astype(np.float64)
    Xm = np.array([[X[i * 4 + j] for j in range(4)] for i in range(3)] + [[0, 0, 0, 1]], np.float64)
    corners = np.array([[a, b, c, 1.0] for a in (0, shape[0] - 1) for b in (0, shape[1] - 1) for c in (0, shape[2] - 1)])
    out = {"workload": f"linearBCV affine, 4 levels G7x6x5x4 L5x4x3x2 Q4x3x2x1, one {shape[0]}x{shape[1]}x{shape[2]} "
                       "pair (seed 21, affine up to 6 deg / 6% / 5 voxels + 2-voxel B-spline field)",
           "pairs_per_s": 1.0 / dev_s, "ms_per_pair": dev_s * 1000.0,
           "e2e": {"value": 1.0 / e2e_s, "unit": "pairs/s", "h2d_bytes_per_step": 2 * f.nbytes,
                   "d2h_bytes_per_step": 64},
           "gpu_launches_per_pair": int(launches),
           "stages_ms": {"gpu (both direction streams summed)": gpu_stages,
                         "profiled pair wall ms": round(prof_s * 1000.0, 3)},
           "device_and_host_calls_agree": bool(np.array_equal(X.view(np.uint32), Xd.view(np.uint32))),
           "max_corner_error_vs_truth_voxels": float(np.abs((A @ Xm) @ corners.T - corners.T)[:3].max())}
    if cpu:
        sys.path.insert(0, os.path.join(ROOT, "oracle"))
        import pyoracle as orc
        t0 = time.perf_counter()
        ref = orc.linear_register(f + np.float32(1024), mv + np.float32(1024), *shape)
        secs = time.perf_counter() - t0
        out["cpu_baseline"] = {"value": 1.0 / secs, "unit": "pairs/s",
                               "cores": int(os.environ.get("OMP_NUM_THREADS", os.cpu_count())), "kind": "port",
                               "sample": f"one full linear registration of the same pair ({secs:.1f} s), oracle/ "
                                         "restatement with OpenMP"}
        out["matrix_identical_to_oracle"] = bool(np.array_equal(X.view(np.uint32), ref.view(np.uint32)))
    return out


def measure_gzio(pair, shape):
    """NIfTI-gz IO of one volume of the workload (the fixed image, 352-byte header +
    float32 data) through the library's parallel gzip writer/reader: one thread
    (the reference's single-threaded zlib rate) against all host threads."""
    import ctypes as C
    import tempfile
    from deedsbcv_gb300 import _lib
    L = _lib.load()
    data = np.ascontiguousarray(pair["fixed"].ravel(order="F"), np.float32)
    head = np.zeros(352, np.uint8)
    out = np.zeros(352 + data.nbytes, np.uint8)
    res = {"volume": f"{shape[0]}x{shape[1]}x{shape[2]} float32 ({data.nbytes / 1e6:.1f} MB)", "level": 6}
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "v.nii.gz").encode()
        for label, th in (("1_thread", 1), ("all_threads", 0)):
            t0 = time.perf_counter()
            st = L.deeds_gz_write(path, head.ctypes.data_as(C.c_void_p), 352, data.ctypes.data_as(C.c_void_p),
                                  data.nbytes, -1, th)
            w = time.perf_counter() - t0
            tot = C.c_size_t(0)
            t0 = time.perf_counter()
            st2 = L.deeds_gz_read(path, out.ctypes.data_as(C.c_void_p), out.size, C.byref(tot), th)
            r = time.perf_counter() - t0
            ok = st == 0 and st2 == 0 and bool(np.array_equal(out[352:].view(np.float32), data))
            res[label] = {"write_s": round(w, 4), "read_s": round(r, 4), "roundtrip_identical": ok,
                          "compressed_MB": round(os.path.getsize(path) / 1e6, 2)}
    res["threads"] = os.cpu_count()
    return res


def cpu_reference_pair(pair, shape):
    """The oracle registration of one pair on all host cores: (seconds, flow, ux, vx, wx)."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import pyoracle as orc
    f = pair["fixed"].ravel(order="F") + np.float32(1024)
    mv = pair["moving"].ravel(order="F") + np.float32(1024)
    t0 = time.perf_counter()
    flow, ux, vx, wx, _ = orc.register(f, mv, *shape, G=G, L=L, Q=Q, want_full=True)
    return time.perf_counter() - t0, flow, ux, vx, wx


# The unmodified reference deedsBCV, built from its own sources by oracle/Makefile
# (ref-deeds) on this host; absent when the reference sources were not staged.
REF_BIN = os.path.join(ROOT, "oracle", "_ref", "deedsBCV")


def host_cores():
    try:
        return len(os.sched_getaffinity(0))
    except AttributeError:
        return os.cpu_count() or 1


def config_dict(shape, ws):
    m, n, o = shape
    return {"workload": f"deeds 5-level registration, {m}x{n}x{o} CT-like phantom pair "
                        f"(13 organs, max 10-voxel B-spline deformation, seed {SEED})",
            "levels": "G8x7x6x5x4 L8x7x6x5x4 Q5x4x3x2x1", "alpha": 1.6,
            "l2": "per-step working set ~1 GB > 129 MB L2 (no extra flush)",
            "parallelism": f"replicas x{ws}"}


class ReferenceBinary:
    """Runs the reference deedsBCV binary on the workload's pair written as NIfTI-gz
    files, with OMP_NUM_THREADS = all host cores, and reads its own timer: the
    "Finished. Total time: T sec." line, which covers the level loop
    (src/deedsBCV0.cpp:222-337) and excludes reading and writing the files."""

    def __init__(self, pair):
        from deedsbcv_gb300 import nifti
        self.tmp = tempfile.TemporaryDirectory()
        d = self.tmp.name
        self.fixed, self.moving = os.path.join(d, "fixed.nii.gz"), os.path.join(d, "moving.nii.gz")
        nifti.write(self.fixed, pair["fixed"])
        nifti.write(self.moving, pair["moving"])
        self.stem = os.path.join(d, "out")
        self.cores = host_cores()
        self.env = dict(os.environ, OMP_NUM_THREADS=str(self.cores))

    @staticmethod
    def available():
        return os.access(REF_BIN, os.X_OK)

    def run(self):
        """One registration: (internal timer seconds, process wall seconds)."""
        t0 = time.perf_counter()
        p = subprocess.run([REF_BIN, "-F", self.fixed, "-M", self.moving, "-O", self.stem], env=self.env,
                           capture_output=True, text=True)
        wall = time.perf_counter() - t0
        if p.returncode != 0 or "Total time:" not in p.stdout:
            raise RuntimeError(f"reference deedsBCV failed ({p.returncode}): {p.stdout[-400:]} {p.stderr[-400:]}")
        return float(p.stdout.split("Total time:")[1].split()[0]), wall

    def close(self):
        self.tmp.cleanup()


def run_reference(args, shape):
    """--impl reference: the unmodified reference deedsBCV (oracle/_ref, built on this
    host from the reference's sources) registers the workload's pair once per step,
    all host cores, W untimed runs then K timed ones; each step's time is the
    binary's own timer.  Where the binary was not built (no staged sources), the
    oracle restatement registers the pair instead (kind "port")."""
    ws, rank, _ = dist_env()
    if rank != 0:
        return
    pair = make_workload(shape)
    cores = host_cores()
    walls = []
    if ReferenceBinary.available():
        kind = "reference"
        ref = ReferenceBinary(pair)
        try:
            for _ in range(args.warmup):
                ref.run()
            times = []
            for _ in range(args.steps):
                t, w = ref.run()
                times.append(t)
                walls.append(w)
        finally:
            ref.close()
        sample = (f"one full 5-level registration of the same {shape[0]}x{shape[1]}x{shape[2]} pair per step by the "
                  f"unmodified reference deedsBCV built from its sources on this host (its Makefile flags; the x86 "
                  f"SIMD flags dropped on Arm), OMP_NUM_THREADS={cores}; step time = the binary's own timer "
                  f"(src/deedsBCV0.cpp:336-337, NIfTI IO outside); mean process wall "
                  f"{np.mean(walls):.2f} s")
    else:
        kind = "port"
        os.environ.setdefault("OMP_NUM_THREADS", str(cores))
        for _ in range(args.warmup):
            cpu_reference_pair(pair, shape)
        times = [cpu_reference_pair(pair, shape)[0] for _ in range(args.steps)]
        sample = (f"one full 5-level registration of the same pair per step by the oracle/ restatement with "
                  f"OpenMP ({cores} threads): the reference binary was not built on this host")
    pair_s = float(np.mean(times))
    value = 1.0 / pair_s
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": "pairs/s", "n_gpus": ws,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1000.0 * pair_s,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32+u64", "data": "synthetic",
        "config": config_dict(shape, ws),
        "cpu_baseline": {"value": value, "unit": "pairs/s", "cores": cores, "kind": kind, "sample": sample},
        "e2e": {"value": value, "unit": "pairs/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "step_seconds": {"min": float(np.min(times)), "median": float(np.median(times)), "max": float(np.max(times))},
    }
    print(json.dumps(line), flush=True)


def main():
    args = parse()
    shape = (96, 80, 128) if args.small else SHAPE
    if args.impl == "reference":
        run_reference(args, shape)
        return
    import torch

    ws, rank, local = dist_env()
    if ws > 1:
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", init_method="env://")
    device = local if ws > 1 else 0
    torch.cuda.set_device(device)
    from deedsbcv_gb300 import api, phantom

    ctx = api.context(device)
    if args.linear_only:
        print(json.dumps(measure_linear(api, ctx, shape, cpu=not args.no_cpu_baseline)), flush=True)
        return
    if args.soft_only:
        taus = tuple(float(t) for t in args.soft_taus.split(","))
        shp = tuple(int(v) for v in args.soft_shape.split("x"))
        lv = SOFT_LEVELS[-1:] if args.soft_single else SOFT_LEVELS
        print(json.dumps(measure_soft(api, ctx, n_pairs=args.soft_pairs, levels=lv, taus=taus, shape=shp)),
              flush=True)
        return
    pair = make_workload(shape)
    m, n, o = shape
    sz = m * n * o
    params = api.default_params()
    if args.profile_once:
        d_fix = torch.from_numpy(np.ascontiguousarray(pair["fixed"].ravel(order="F"))).cuda()
        d_mov = torch.from_numpy(np.ascontiguousarray(pair["moving"].ravel(order="F"))).cuda()
        api.register_device(d_fix, d_mov, m, n, o, params=params, ctx=ctx)
        torch.cuda.synchronize()
        torch.cuda.nvtx.range_push("deeds_pair")
        api.register_device(d_fix, d_mov, m, n, o, params=params, ctx=ctx)
        torch.cuda.synchronize()
        torch.cuda.nvtx.range_pop()
        return
    g_last = G[-1]
    sz1 = (m // g_last) * (n // g_last) * (o // g_last)
    d_fix = torch.from_numpy(np.ascontiguousarray(pair["fixed"].ravel(order="F"))).to(f"cuda:{device}")
    d_mov = torch.from_numpy(np.ascontiguousarray(pair["moving"].ravel(order="F"))).to(f"cuda:{device}")
    d_flow = torch.empty(3 * sz1, dtype=torch.float32, device=f"cuda:{device}")
    stream = torch.cuda.current_stream()

    def barrier():
        if ws > 1:
            torch.distributed.barrier()

    # warm-up (allocates the context's scratch, spins up the host worker threads)
    for _ in range(args.warmup):
        api.register_device(d_fix, d_mov, m, n, o, params=params, flow_out=d_flow, ctx=ctx)
    torch.cuda.synchronize()

    # ---- device-resident throughput, with per-stage CUDA-event tracing
    ctx.reset_stage_times()
    ctx.set_profiling(True)
    launches0 = api.kernel_launches()
    with ClockSampler(device) as clocks:
        barrier()
        torch.cuda.synchronize()
        ev0 = torch.cuda.Event(enable_timing=True)
        ev1 = torch.cuda.Event(enable_timing=True)
        ev0.record(stream)
        for _ in range(args.steps):
            api.register_device(d_fix, d_mov, m, n, o, params=params, flow_out=d_flow, ctx=ctx)
        ev1.record(stream)
        torch.cuda.synchronize()
        barrier()
    launches = api.kernel_launches() - launches0
    ctx.set_profiling(False)
    value, secs = replica_rate(ev0.elapsed_time(ev1) / 1000.0, args.steps, f"cuda:{device}")
    ms = secs * 1000.0
    stages = ctx.stage_times()
    clk = clocks.summary()

    # ---- end to end through the host-buffer entry point, inputs in pinned host memory
    fixed_h, moving_h = pinned(pair["fixed"]), pinned(pair["moving"])
    barrier()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        flow_h, _ = api.register(fixed_h, moving_h, dims=shape, params=params, want_warped=False, ctx=ctx)
    e2e_value, _ = replica_rate(time.perf_counter() - t0, args.steps, f"cuda:{device}")
    e2e = {"value": e2e_value, "unit": "pairs/s", "h2d_bytes_per_step": 2 * sz * 4,
           "d2h_bytes_per_step": 3 * sz1 * 4, "host_inputs": "pinned"}

    # ---- roofline of the dominant stage
    dc_ms, dc_launches = stages["datacost"]
    mind_ms, mind_launches = stages["mind"]
    pop = popc64_per_pair(shape) * args.steps
    dc_achieved = pop * 2 * 64 / (dc_ms / 1000.0) / 1e12 if dc_ms > 0 else None
    mind_bytes = 108 * sz * mind_calls() * args.steps
    peaks = {}
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            peaks = json.load(f)
    except OSError:
        pass
    hbm_peak = peaks.get("hbm_gbs", 6800.0)
    gpu_stage_ms = sum(v[0] for k, v in stages.items() if k != "tree_wait")
    mind_s, vox = isolated_mind(api, ctx, pair, shape)
    mind_roof = {
        "bound": "hbm", "unit": "GB/s", "peak": hbm_peak, "peak_source": "MEASURED_PEAKS.json hbm_gbs (of measured)",
        "ms_per_call": round(mind_s * 1000, 3),
        # bytes the three kernels move per voxel: image 4 (+ shifted rows from L2) and six
        # distance channels 24 written (i and j pass); 48 read and written (k pass); 24 read
        # and 8 written (quantise)
        "achieved": 108 * vox / mind_s / 1e9, "frac": 108 * vox / mind_s / 1e9 / hbm_peak,
        "algorithmic_bytes_per_voxel": 12,
        "note": "one call timed alone; the fused minimum is 12 B/voxel (image in, code out): the sequential "
                "float prefix sums of the reference's box filter (needed for bit-exact codes) keep the k pass "
                "and the quantiser separate",
        "in_pipeline_achieved": (mind_bytes / (mind_ms / 1000.0) / 1e9) if mind_ms else None,
    }
    iso_pop, iso_s, iso_levels = isolated_data_cost(api, ctx, pair, shape)
    # a code pair is a dot product of 64 four-bit floats
    pair_tflop = 2 * 64 / 1e12
    fp4_peak = 6.0 * peaks.get("bf16_tflops", 1900.0)
    iso_achieved = iso_pop * pair_tflop / iso_s
    cost_roof = {
        "kernel": "k_data_cost_mma (Hamming cost volume, one direction, all 5 levels)",
        "bound": "tensor (issue of small 4-bit MMAs, most of whose columns pair rows that no label needs)",
        "achieved": iso_achieved,
        "peak": fp4_peak,
        "unit": "TFLOP/s (4-bit, of code pairs that a label needs)",
        "frac": iso_achieved / fp4_peak,
        "ms_per_pair": round(2 * iso_s * 1000, 3),
        "levels": iso_levels,
        "in_pipeline": {"achieved": dc_achieved, "frac": (dc_achieved / fp4_peak) if dc_achieved else None,
                        "note": "code pairs / summed stage time of both direction streams, which share the GPU"},
        "peak_source": "6 x MEASURED_PEAKS.json bf16_tflops (the ratio of the nominal dense 4-bit and bf16 rates)",
        "note": "an MMA of N <= 32 columns costs 15 to 33 clocks whatever its size: 25 to 47 needed code pairs a clock and "
                "SM at most in this form (12 on the integer pipe), 13 to 20 reached",
        "work_per_pair": popc64_per_pair(shape),
        "share_of_gpu_time": dc_ms / gpu_stage_ms if gpu_stage_ms else None,
    }
    bp_levels, bp_tot = isolated_bp(api, ctx, pair, shape)
    # algorithmic bytes of the upward sweep: one read and one write of the cost
    # volume (both directions: 2 x 2 x sum over levels of sz1 * len^3 * 4 B)
    up_bytes = 2 * bp_tot["cost_bytes"]
    up_gbs = up_bytes / (bp_tot["up_ms"] / 1000.0) / 1e9
    bp_roof = {
        "kernel": "k_bp_up<LEN> (tree BP upward sweep, one direction, all 5 levels)",
        "bound": "hbm",
        "achieved": up_gbs,
        "peak": hbm_peak,
        "unit": "GB/s",
        "frac": up_gbs / hbm_peak,
        "peak_source": "MEASURED_PEAKS.json hbm_gbs (of measured)",
        "algorithmic_bytes_per_launch_set": up_bytes,
        "ms_per_pair": round(2 * bp_tot["up_ms"], 3),
        "note": "dependency bound: a chain of nodes per tree-depth step, one CTA per chain; the HBM fraction on "
                "the cost-volume read + write is reported against the copy peak as the contract asks",
        "levels": bp_levels,
        "argmin_ms_per_pair": round(2 * bp_tot["argmin_ms"], 3),
        "down_ms_per_pair": round(2 * bp_tot["down_ms"], 3),
    }
    # the roofline line names the kernel that takes the most device time per pair
    # (each kernel timed alone); the other is kept beside it
    if bp_roof["ms_per_pair"] >= cost_roof["ms_per_pair"]:
        roofline = dict(bp_roof, cost_volume=cost_roof)
        top = "k_bp_up"
    else:
        roofline = dict(cost_roof, bp_up=bp_roof)
        top = "k_data_cost_mma"
    roofline["traffic"] = TRAFFIC.get(top) if shape == SHAPE else None
    roofline["traffic_algorithmic_same_launch"] = TRAFFIC_ALGORITHMIC.get(top) if shape == SHAPE else None
    roofline["traffic_note"] = TRAFFIC_NOTE
    roofline["mind_hbm"] = mind_roof

    # ---- batched form on 16 uneven pairs (rank 0)
    batched = None
    if rank == 0 and not args.no_batched and not args.small:
        batched = measure_batched(api, ctx, args.lanes)

    # ---- differentiable soft-min form (rank 0)
    soft = None
    if rank == 0 and not args.no_soft and not args.small:
        soft = measure_soft(api, ctx)
        soft["finest_level_alone"] = measure_soft(api, ctx, levels=SOFT_LEVELS[-1:])

    # ---- NIfTI-gz IO of one volume (rank 0)
    gzio = measure_gzio(pair, shape) if rank == 0 else None

    # ---- linearBCV affine pre-registration (rank 0)
    linear = None
    if rank == 0 and not args.no_linear:
        linear = measure_linear(api, ctx, shape, cpu=(ws == 1 and not args.no_cpu_baseline))

    # ---- CPU baseline and full-size parity (rank 0, N=1)
    cpu = None
    parity = None
    if rank == 0 and ws == 1 and not args.no_cpu_baseline:
        secs, rflow, ux, vx, wx = cpu_reference_pair(pair, shape)
        sys.path.insert(0, os.path.join(ROOT, "oracle"))
        import pyoracle as orc
        cores = int(os.environ.get("OMP_NUM_THREADS", host_cores()))
        cpu = {"value": 1.0 / secs, "unit": "pairs/s", "cores": cores,
               "kind": "port", "sample": f"one full registration of the same {shape[0]}x{shape[1]}x{shape[2]} pair "
                                         f"({secs:.1f} s), oracle/ restatement with OpenMP"}
        if ReferenceBinary.available():
            # the unmodified reference binary on the same pair, one registration (its own timer)
            ref = ReferenceBinary(pair)
            try:
                rsecs, rwall = ref.run()
            finally:
                ref.close()
            cpu = {"value": 1.0 / rsecs, "unit": "pairs/s", "cores": ref.cores, "kind": "reference",
                   "sample": f"one full registration of the same {shape[0]}x{shape[1]}x{shape[2]} pair by the "
                             f"unmodified reference deedsBCV built on this host, OMP_NUM_THREADS={ref.cores}: "
                             f"{rsecs:.2f} s by its own timer (level loop; process wall {rwall:.2f} s with NIfTI "
                             f"IO); the oracle restatement took {secs:.2f} s",
                   "port_value": 1.0 / secs}
        gflow = d_flow.cpu().numpy()
        seg_gpu = api.apply_flow(gflow, pair["moving_labels"].astype(np.int16), dims=shape, ctx=ctx)
        seg_ref = orc.warp_affine_s(pair["moving_labels"].astype(np.int16), np.eye(4, dtype=np.float32).ravel(), ux,
                                    vx, wx, *shape)
        lab = pair["fixed_labels"].ravel(order="F")
        parity = {"flow_identical_frac": float(np.mean(gflow == rflow)),
                  "dice_gpu": phantom.dice(lab, seg_gpu), "dice_cpu": phantom.dice(lab, seg_ref),
                  "dice_before": phantom.dice(lab, pair["moving_labels"].ravel(order="F"))}

    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": "pairs/s", "n_gpus": ws, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms / args.steps, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32+u64", "data": "synthetic",
            "config": config_dict(shape, ws),
            "clocks": clk,
            "e2e": e2e,
            "gpu_launches": launches,
            "roofline": roofline,
            "stages_ms_per_pair": {k: round(v[0] / args.steps, 3) for k, v in stages.items()},
            "stage_launches_per_pair": {k: v[1] // max(args.steps, 1) for k, v in stages.items()},
            "cpu_baseline": cpu,
            "parity": parity,
            "batched": batched,
            "soft": soft,
            "linear": linear,
            "gzip_io": gzio,
        }
        print(json.dumps(line), flush=True)
    if ws > 1:
        torch.distributed.destroy_process_group()


if __name__ == "__main__":
    main()
