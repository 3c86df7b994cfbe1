// Hamming cost volume on the integer pipe (replaces dataCostCL, src/dataCostD.h:108-210),
// for few labels an axis: see datacost.cu for the definition and popc_faster there for where
// this form is the faster one.
//
// The moving codes are copied into a clamp-to-edge padded volume (the reference's data2p,
// src/dataCostD.h:124-138) with an even row pitch, so that every row starts on 16 bytes for
// TMA.  One CTA owns a tile of control nodes along y (same x, z) and one z label offset,
// and walks the len x offsets.  For each, the halo is one 3-D box of the padded volume, all
// rows of the tile plus the label reach and the sampled x columns and z slices, which one
// cp.async.bulk.tensor.3d copies into shared memory (element strides of 2 skip the unsampled
// columns); two boxes are in flight.  A thread owns one (node, sample row), its fixed codes
// in registers, and its len labels' sums; the node's rows are summed through shared
// memory.  With the label width known to the compiler (3, 5, 7) all sums stay in registers
// and three samples' XORs go through a carry-save adder, so that they cost two 64-bit POPCs
// in place of three; wider sets (grid 2 only) take eight labels at a time.
//
// Bound by the integer pipe (16 32-bit POPCs a clock and SM: 12 code pairs with the adder).
// Reached, 192x160x256, pairs a clock and SM: 6.7 to 7.9 at 5 and 7 labels of grid 4, 4.4 at 3;
// 4 at 9 and more.  Grid 5, 7 labels, step 2: 437 us; grid 4, 5 labels, step 1: 466 us.
#include <algorithm>

#include <cuda.h>

#include "common.cuh"
#include "kernels.h"

namespace deeds {

namespace {

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}

// clamp-to-edge padded copy of the moving codes, row pitch mpp (even)
__global__ void k_pad_codes(const uint64_t* __restrict__ M, uint64_t* __restrict__ Mp, int m, int n, int o, int pad,
                            int mpp, int np, int op) {
    const int y = blockIdx.x * blockDim.x + threadIdx.x;
    const int x = blockIdx.y, z = blockIdx.z;
    if (y >= mpp) return;
    const int64_t src = clampi(y - pad, 0, m - 1) + (int64_t)clampi(x - pad, 0, n - 1) * m +
                        (int64_t)clampi(z - pad, 0, o - 1) * m * n;
    Mp[y + (int64_t)x * mpp + (int64_t)z * mpp * np] = __ldg(M + src);
}

// Sum of the G sample-row partials of tile node t at label ly into its cost entry.
template <int G>
__device__ __forceinline__ void reduce_rows(const int* red, int nthr, int t, int ly, float* cost_lx, int len3,
                                            float alpha1) {
    const int* r = red + ly * nthr + t * G;
    int sum = 0;
#pragma unroll
    for (int ii = 0; ii < G; ii++) sum += r[ii];
    cost_lx[(int64_t)t * len3 + ly] = __fmul_rn((float)sum, alpha1);
}

// LEN_T > 0: label width known to the compiler, every label loop exact and unrolled; 0:
// at run time, labels in chunks of 8 with guards.  Q_T > 0: the label step is known too, so
// that a thread's rows are immediate offsets (grid 4, 5 labels, step 1: 466 us, 519
// with a run-time step; grid 5, 7 labels, step 2: 437, 502).
template <int G, int LEN_T, int Q_T>
__global__ void __launch_bounds__(256) k_data_cost_popc(const __grid_constant__ CUtensorMap map,
                                                        const uint64_t* __restrict__ F, float* __restrict__ cost,
                                                        int m, int n, int o, int len_rt, int q_rt, int ny_tile,
                                                        int yb, float alpha1, int* __restrict__ err) {
    constexpr bool kFixed = LEN_T > 0;
    const int len = kFixed ? LEN_T : len_rt;
    const int q = Q_T > 0 ? Q_T : q_rt;
    constexpr int S = G > 4 ? 2 : 1;  // x and z sampling stride (RAND_SAMPLES=1, src/dataCostD.h:141-155)
    constexpr int NX = (G + S - 1) / S, NZ = (G + S - 1) / S;
    constexpr int NC = NX * NZ;       // sampled (x, z) columns per node
    constexpr int CHUNK = 8;          // labels accumulated per pass over the columns
    extern __shared__ __align__(128) uint64_t smem_raw[];
    // TMA destinations must start on 128-byte boundaries: align explicitly
    uint64_t* smem = reinterpret_cast<uint64_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ int s_ok;
    const int box = NC * yb;
    const int bstride = (box + 15) & ~15;
    uint64_t* buf0 = smem;
    uint64_t* buf1 = smem + bstride;
    int* red = reinterpret_cast<int*>(smem + 2 * bstride);  // [len][threads] partial sums
    const int m1 = m / G, n1 = n / G;
    const int tiles_y = (m1 + ny_tile - 1) / ny_tile;
    int b = blockIdx.x;
    const int ty = b % tiles_y;
    b /= tiles_y;
    const int nxn = b % n1, nzn = b / n1;
    const int lz = blockIdx.y;
    const int y_first = ty * ny_tile;
    const int ny_here = min(ny_tile, m1 - y_first);
    const int y0 = y_first * G;  // padded y of the tile's first row (the pad offset cancels)
    const int y_al = y0 & ~1;    // TMA: the innermost coordinate must be 16-byte aligned
    const int yoff = y0 - y_al;
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int len2 = len * len, len3 = len2 * len;
    const int64_t mn = (int64_t)m * n;
    const uint32_t box_bytes = (uint32_t)box * 8u;
    const int xbase = nxn * G, zbase = nzn * G + lz * q;
    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_ok = *(volatile int*)err == 0;  // a wait of an earlier CTA gave up: no further waits
    }
    __syncthreads();
    if (!s_ok) return;
    if (tid == 0) {
        mbar_expect_tx(&bars[0], box_bytes);
        tma_load_3d(buf0, &map, &bars[0], y_al, xbase, zbase);
        if (len > 1) {
            mbar_expect_tx(&bars[1], box_bytes);
            tma_load_3d(buf1, &map, &bars[1], y_al, xbase + q, zbase);
        }
    }
    // this thread's node (within the tile) and sample row i: thread = node * G + i over
    // the whole block, so a node's rows may straddle two warps and no lane idles
    // but the last warp's tail; its fixed codes stay in registers
    const int tn = tid / G, i = tid - (tid / G) * G;  // node index within the tile, sample row
    const bool active = tn < ny_here;
    uint64_t fr[NC];
#pragma unroll
    for (int c = 0; c < NC; c++) {
        const int j = c % NX, k = c / NX;
        fr[c] = active ? F[(y0 + tn * G + i) + (int64_t)(xbase + j * S) * m + (int64_t)(nzn * G + k * S) * mn] : 0ull;
    }
    const int pos = yoff + tn * G + i;  // this thread's row in the box (for label ly add ly*q)
    // partial sums: [warp][len][32] when g divides 32 (the warp reduces its own
    // nodes), else [len][threads] (nodes straddle warps: the block reduces)
    constexpr bool kWarpLocal = 32 % G == 0;
    int* wred = kWarpLocal ? red + (tid >> 5) * len * 32 + (tid & 31) : red + tid;
    const int wstride = kWarpLocal ? 32 : nthr;
    for (int lx = 0; lx < len; lx++) {
        const int slot = lx & 1;
        const uint64_t* sb = slot ? buf1 : buf0;
        if (tid == 0) {
            if (!mbar_wait_bounded(&bars[slot], (uint32_t)((lx >> 1) & 1))) s_ok = 0;
        }
        __syncwarp();  // the barrier wants the waiting lane's warp together
        __syncthreads();
        if (!s_ok) break;
        if (kFixed && active) {
            constexpr int LF = kFixed ? LEN_T : 1;
            int acc[LF];
#pragma unroll
            for (int u = 0; u < LF; u++) acc[u] = 0;
            // for the XORs a, b, c: popc(a) + popc(b) + popc(c) = popc(a ^ b ^ c) + 2 popc(maj(a, b, c))
#pragma unroll
            for (int c = 0; c + 3 <= NC; c += 3) {
                const uint64_t* ca = sb + c * yb + pos;
                const uint64_t* cb = ca + yb;
                const uint64_t* cc = cb + yb;
#pragma unroll
                for (int u = 0; u < LF; u++) {
                    const uint64_t a = fr[c] ^ ca[u * q], b = fr[c + 1] ^ cb[u * q], x = fr[c + 2] ^ cc[u * q];
                    const uint64_t sum = a ^ b ^ x, carry = (a & b) | (x & (a ^ b));
                    acc[u] += __popcll(sum) + 2 * __popcll(carry);
                }
            }
#pragma unroll
            for (int c = NC - NC % 3; c < NC; c++) {
                const uint64_t* col = sb + c * yb + pos;
#pragma unroll
                for (int u = 0; u < LF; u++) acc[u] += __popcll(fr[c] ^ col[u * q]);
            }
#pragma unroll
            for (int u = 0; u < LF; u++) wred[u * wstride] = acc[u];
        } else if (active) {
            for (int ly0 = 0; ly0 < len; ly0 += CHUNK) {
                int acc[CHUNK];
#pragma unroll
                for (int u = 0; u < CHUNK; u++) acc[u] = 0;
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    const uint64_t* col = sb + c * yb + pos + ly0 * q;
#pragma unroll
                    for (int u = 0; u < CHUNK; u++)
                        if (ly0 + u < len) acc[u] += __popcll(fr[c] ^ col[u * q]);
                }
#pragma unroll
                for (int u = 0; u < CHUNK; u++)
                    if (ly0 + u < len) wred[(ly0 + u) * wstride] = acc[u];
            }
        }
        // sum the G sample rows of each (node, ly): within the warp when g divides 32
        // (no node straddles two warps), else over the block
        // (cost row of tile node t, label ly): node (y_first + t) + nxn m1 + nzn m1 n1
        float* cost_lx = cost + (int64_t)(y_first + nxn * m1 + nzn * m1 * n1) * len3 + lx * len + lz * len2;
        if constexpr (kWarpLocal) {
            constexpr int WN = 32 / G;  // nodes per warp
            __syncwarp();
            const int warp = tid >> 5, lane = tid & 31;
            const int* wr = red + warp * len * 32;
            for (int e = lane; e < WN * len; e += 32) {
                const int en = e / len, node_t = warp * WN + en;
                if (node_t < ny_here) reduce_rows<G>(wr, 32, en, e - en * len, cost_lx + (int64_t)warp * WN * len3, len3,
                                                     alpha1);
            }
        } else {
            __syncthreads();
            for (int e = tid; e < ny_here * len; e += nthr)
                reduce_rows<G>(red, nthr, e / len, e - (e / len) * len, cost_lx, len3, alpha1);
        }
        __syncthreads();  // every thread is done with this buffer and with red
        if (tid == 0 && lx + 2 < len) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_expect_tx(&bars[slot], box_bytes);
            tma_load_3d(const_cast<uint64_t*>(sb), &map, &bars[slot], y_al, xbase + (lx + 2) * q, zbase);
        }
    }
    if (!s_ok && tid == 0) {
        atomicCAS(err, 0, 3);
        // wait (bounded) for the copies this CTA may still have in flight
        for (int sl = 0; sl < 2; sl++)
            for (int ph = 0; ph < 2; ph++) mbar_wait_bounded(&bars[sl], (uint32_t)ph);
    }
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static const EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        const cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q);
        cudaGetLastError();
        return e == cudaSuccess && q == cudaDriverEntryPointSuccess ? reinterpret_cast<EncodeTiledFn>(p) : nullptr;
    }();
    return fn;
}

constexpr int kMaxSmem = 200 * 1024;

struct PopcPlan {
    int tile, threads, yb;  // nodes along y, threads (one per node and sample row, whole warps), rows of a box
    size_t smem;
    int mpp, np, op;  // the padded copy
};

bool popc_tile(int g, int len, int q, int tile, PopcPlan& p) {
    const int S = g > 4 ? 2 : 1, NX = (g + S - 1) / S;
    p.tile = tile;
    p.threads = (tile * g + 31) / 32 * 32;
    p.yb = ((tile * g + (len - 1) * q + 1) + 1) & ~1;  // +1 for the alignment shift, rounded to even
    p.smem = (size_t)2 * ((NX * NX * p.yb + 15) & ~15) * 8 + (size_t)p.threads * len * 4 + 128;
    return p.threads <= 256 && p.yb <= 256 && p.smem <= kMaxSmem;
}

bool popc_plan(int m, int n, int o, int g, int hw, int q, PopcPlan& p) {
    const int len = 2 * hw + 1;
    if (g < 2 || g > 8 || hw < 1 || (len > 7 && g > 2)) return false;
    const int64_t pad = (int64_t)q * hw;
    if (n + 2 * pad > 65535 || o + 2 * pad > 65535 || m + 2 * pad > (1 << 30)) return false;
    p.mpp = (int)((m + 2 * pad + 1) & ~1);
    p.np = (int)(n + 2 * pad);
    p.op = (int)(o + 2 * pad);
    // the tile that wastes the fewest lanes, of at most 96 threads (more are no faster at any
    // grid; 96x80x112 and 192x160x256), with six warps or more to an SM; of equals the largest
    const int m1 = m / g;
    int best = 0;
    for (int tile = 1; tile <= m1 && tile * g <= 96; tile++) {
        PopcPlan c = p;
        if (!popc_tile(g, len, q, tile, c) || 227 * 1024 / (int)(c.smem + 1024) * (c.threads / 32) < 6) break;
        const int lanes = (m1 + tile - 1) / tile * c.threads;
        if (best == 0 || lanes <= best) {
            best = lanes;
            p = c;
        }
    }
    return best > 0;
}

template <int G, int LEN_T, int Q_T>
cudaError_t launch_popc(const uint64_t* d_F, const uint64_t* d_Mp, int m, int n, int o, int len, int q,
                        const PopcPlan& p, float alpha1, float* d_cost, int* d_err, cudaStream_t s) {
    constexpr int S = G > 4 ? 2 : 1, NX = (G + S - 1) / S;
    CUtensorMap map;
    const cuuint64_t dims[3] = {(cuuint64_t)p.mpp, (cuuint64_t)p.np, (cuuint64_t)p.op};
    const cuuint64_t strides[2] = {(cuuint64_t)p.mpp * 8, (cuuint64_t)p.mpp * p.np * 8};
    const cuuint32_t boxd[3] = {(cuuint32_t)p.yb, (cuuint32_t)(NX * S), (cuuint32_t)(NX * S)};
    const cuuint32_t estr[3] = {1, (cuuint32_t)S, (cuuint32_t)S};
    const EncodeTiledFn enc = encode_fn();
    if (!enc) return cudaErrorNotSupported;
    if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, const_cast<uint64_t*>(d_Mp), dims, strides, boxd, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorInvalidValue;
    // the same limit on every call: other threads launch the kernel for other sizes
    cudaError_t e =
        cudaFuncSetAttribute(k_data_cost_popc<G, LEN_T, Q_T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    if (e != cudaSuccess) return e;
    const dim3 grid((unsigned)((m / G + p.tile - 1) / p.tile * (n / G) * (o / G)), (unsigned)len);
    k_data_cost_popc<G, LEN_T, Q_T>
        <<<grid, p.threads, p.smem, s>>>(map, d_F, d_cost, m, n, o, len, q, p.tile, p.yb, alpha1, d_err);
    count_launches(1);
    return cudaGetLastError();
}

template <int G, int LEN_T, class... Args>
cudaError_t launch_step(int q, Args... a) {
    if (q == 1) return launch_popc<G, LEN_T, 1>(a...);
    if (q == 2) return launch_popc<G, LEN_T, 2>(a...);
    return launch_popc<G, LEN_T, 0>(a...);
}

template <int G, class... Args>
cudaError_t launch_width(int len, int q, Args... a) {
    if (len == 3) return launch_step<G, 3>(q, a...);
    if (len == 5) return launch_step<G, 5>(q, a...);
    if (len == 7) return launch_step<G, 7>(q, a...);
    if constexpr (G == 2) return launch_popc<G, 0, 0>(a...);
    return cudaErrorInvalidValue;  // not planned (popc_plan)
}

}  // namespace

size_t data_cost_popc_count(int m, int n, int o, int g, int hw, int q) {
    PopcPlan p;
    return popc_plan(m, n, o, g, hw, q, p) ? (size_t)p.mpp * p.np * p.op : 0;
}

cudaError_t launch_data_cost_popc(const uint64_t* d_F, const uint64_t* d_M, uint64_t* d_pad, int m, int n, int o,
                                  int g, int hw, int q, float alpha1, float* d_cost, int* d_err, cudaStream_t s) {
    PopcPlan p;
    const int len = 2 * hw + 1;
    if (!popc_plan(m, n, o, g, hw, q, p)) return cudaErrorInvalidValue;
    k_pad_codes<<<dim3((p.mpp + 127) / 128, p.np, p.op), 128, 0, s>>>(d_M, d_pad, m, n, o, q * hw, p.mpp, p.np, p.op);
    count_launches(1);
    if (const cudaError_t e = cudaGetLastError(); e != cudaSuccess) return e;
#define DEEDS_POPC_ARGS len, q, d_F, d_pad, m, n, o, len, q, p, alpha1, d_cost, d_err, s
    switch (g) {
        case 2: return launch_width<2>(DEEDS_POPC_ARGS);
        case 3: return launch_width<3>(DEEDS_POPC_ARGS);
        case 4: return launch_width<4>(DEEDS_POPC_ARGS);
        case 5: return launch_width<5>(DEEDS_POPC_ARGS);
        case 6: return launch_width<6>(DEEDS_POPC_ARGS);
        case 7: return launch_width<7>(DEEDS_POPC_ARGS);
        default: return launch_width<8>(DEEDS_POPC_ARGS);
    }
#undef DEEDS_POPC_ARGS
}

}  // namespace deeds
