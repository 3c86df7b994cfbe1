// Multi-atlas label fusion on sm_103a.  The reference names joint label fusion
// as future work for multi-atlas segmentation (README.md:8, README.md:201) and
// implements none; this is the voting step that follows registering several
// atlases to one target with deeds: every atlas' labels and image, warped onto
// the target, vote per voxel.
//
// Rule (locally weighted voting by inverse patch distance):
//   D_i(x) = sum over the (2r+1)^3 patch around x (clamp-to-edge) of
//            (T - A_i)^2, summed as three separable window passes (i, then j,
//            then k; each window sum in offset order -r..r from 0);
//   w_i(x) = (1 / (D_i(x) + eps))^p  (p integer >= 0; p = 0 is majority vote);
//   label(x) = the label L maximising sum_i w_i [L_i(x) == L], the sum taken in
//              atlas order; ties go to the smaller label.
// Every step is a float operation whose order is fixed above (built with
// --fmad=false), so the CPU restatement reproduces it bit for bit.
//
// Roofline: HBM.  Per voxel and atlas: image read, distance written, distance and
// labels read by the vote (14 B), the target once per atlas from L2, and the 2 B label
// written.  192x160x256, 8 atlases, radius 2: 1.61 -> 0.39 ms (windows 0.24,
// vote 0.15; the bytes alone take 0.13 ms at the copy rate of 6.78 TB/s).
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace deeds {

namespace {

// Window sum along one axis (stride, extent) with clamp-to-edge, for every atlas
// (gridDim.y); SQ: the input is (T - A_i)^2 formed on the fly.
template <bool SQ>
__global__ void __launch_bounds__(256) k_window(const float* __restrict__ target, FusionAtlases at,
                                                const float* __restrict__ in, float* __restrict__ out, int m, int n,
                                                int o, int axis, int r) {
    const int64_t sz = (int64_t)m * n * o;
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= sz) return;
    const int a = blockIdx.y;
    const int64_t base = (int64_t)a * sz;
    const int i = (int)(v % m), j = (int)((v / m) % n), k = (int)(v / ((int64_t)m * n));
    const int c = axis == 0 ? i : (axis == 1 ? j : k);
    const int ext = axis == 0 ? m : (axis == 1 ? n : o);
    const int64_t stride = axis == 0 ? 1 : (axis == 1 ? (int64_t)m : (int64_t)m * n);
    const int64_t row0 = v - (int64_t)c * stride;
    float s = 0.0f;
    for (int d = -r; d <= r; d++) {
        const int64_t p = row0 + (int64_t)clampi(c + d, 0, ext - 1) * stride;
        float x;
        if (SQ) {
            const float df = target[p] - at.image[a][p];
            x = df * df;
        } else {
            x = in[base + p];
        }
        s = s + x;
    }
    out[base + v] = s;
}

// The three passes for radius R at once: a block covers TI x TJ columns of one atlas and
// marches along k.  Per slice the squared differences of the tile and its halo go to
// shared memory, their i sums too, each thread adds its column's j sum, and the last
// 2R + 1 of those stay in registers for the k sum.  The next slice's samples are loaded
// meanwhile.  The sums' order is the separate passes'.  Bound: shared memory and issue
// (three passes of 8 B per voxel and atlas through memory before: 1.36 ms of the 1.6).
constexpr int TI = 32, TJ = 16;

template <int R>
__global__ void __launch_bounds__(TI * TJ) k_window3(const float* __restrict__ target, FusionAtlases at,
                                                     float* __restrict__ out, int n_atlas, int m, int n, int o,
                                                     int k_chunk) {
    constexpr int W = TI + 2 * R, H = TJ + 2 * R, N = W * H, PER = (N + TI * TJ - 1) / (TI * TJ);
    constexpr int IPER = (TI * H + TI * TJ - 1) / (TI * TJ);
    __shared__ float sq[2][N];
    __shared__ float is[2][TI * H];
    const int a = blockIdx.z % n_atlas, kc = blockIdx.z / n_atlas;
    const int i0 = blockIdx.x * TI, j0 = blockIdx.y * TJ;
    const int t = threadIdx.x, ti = t % TI, tj = t / TI;
    const int k0 = kc * k_chunk, k1 = min(o, k0 + k_chunk);
    const int64_t mn = (int64_t)m * n;
    const float* image = at.image[a];
    int at_plane[PER];  // this thread's samples within a slice
#pragma unroll
    for (int e = 0; e < PER; e++) {
        const int x = t + e * TI * TJ;
        at_plane[e] = clampi(i0 + x % W - R, 0, m - 1) + clampi(j0 + x / W - R, 0, n - 1) * m;
    }
    float tv[PER], av[PER];
    auto load = [&](int k) {
        const int64_t base = (int64_t)clampi(k, 0, o - 1) * mn;
#pragma unroll
        for (int e = 0; e < PER; e++)
            if (t + e * TI * TJ < N) {
                tv[e] = __ldg(target + base + at_plane[e]);
                av[e] = __ldg(image + base + at_plane[e]);
            }
    };
    load(k0 - R);
    float ring[2 * R + 1];
#pragma unroll
    for (int d = 0; d <= 2 * R; d++) ring[d] = 0.0f;
    const bool in = i0 + ti < m && j0 + tj < n;
    float* dst = out + (int64_t)a * mn * o + (i0 + ti) + (int64_t)(j0 + tj) * m;
    for (int k = k0 - R; k < k1 + R; k++) {
        const int b = (k - k0 + R) & 1;
#pragma unroll
        for (int e = 0; e < PER; e++)
            if (t + e * TI * TJ < N) {
                const float df = tv[e] - av[e];
                sq[b][t + e * TI * TJ] = df * df;
            }
        if (k + 1 < k1 + R) load(k + 1);
        __syncthreads();
#pragma unroll
        for (int e = 0; e < IPER; e++) {
            const int x = t + e * TI * TJ;
            if (x < TI * H) {
                const float* r = sq[b] + (x / TI) * W + x % TI;
                float s = 0.0f;
#pragma unroll
                for (int d = 0; d <= 2 * R; d++) s = s + r[d];
                is[b][x] = s;
            }
        }
        __syncthreads();
        float s = 0.0f;
#pragma unroll
        for (int d = 0; d <= 2 * R; d++) s = s + is[b][(tj + d) * TI + ti];
#pragma unroll
        for (int d = 0; d < 2 * R; d++) ring[d] = ring[d + 1];
        ring[2 * R] = s;
        if (in && k >= k0 + R) {
            float v = 0.0f;
#pragma unroll
            for (int d = 0; d <= 2 * R; d++) v = v + ring[d];
            dst[(int64_t)(k - R) * mn] = v;
        }
    }
}

// The vote of up to NA atlases with weights and labels in registers (k_vote indexes
// them in local memory: 0.30 ms for 8 atlases at 192x160x256).
template <int NA>
__global__ void __launch_bounds__(256) k_vote_n(FusionAtlases at, int n_atlas, const float* __restrict__ dist, int64_t sz,
                                                float eps, int power, int16_t* __restrict__ out) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= sz) return;
    float w[NA];
    int lab[NA];
#pragma unroll
    for (int a = 0; a < NA; a++)
        if (a < n_atlas) {
            w[a] = __ldg(dist + (int64_t)a * sz + v);
            lab[a] = __ldg(at.labels[a] + v);
        }
#pragma unroll
    for (int a = 0; a < NA; a++)
        if (a < n_atlas) {
            const float inv = 1.0f / (w[a] + eps);
            float x = 1.0f;
            for (int q = 0; q < power; q++) x = x * inv;
            w[a] = x;
        }
    int best = lab[0];
    float best_s = -1.0f;
#pragma unroll
    for (int a = 0; a < NA; a++)
        if (a < n_atlas) {
            const int L = lab[a];
            float s = 0.0f;
#pragma unroll
            for (int b = 0; b < NA; b++)
                if (b < n_atlas && lab[b] == L) s = s + w[b];
            if (s > best_s || (s == best_s && L < best)) {
                best_s = s;
                best = L;
            }
        }
    out[v] = (int16_t)best;
}

// The vote: weights from the window sums, labels of every atlas, the winner.
__global__ void __launch_bounds__(256) k_vote(FusionAtlases at, int n_atlas, const float* __restrict__ dist,
                                              int64_t sz, float eps, int power, int16_t* __restrict__ out) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= sz) return;
    float w[kFuseMaxAtlases];
    int16_t lab[kFuseMaxAtlases];
    for (int a = 0; a < n_atlas; a++) {
        const float inv = 1.0f / (dist[(int64_t)a * sz + v] + eps);
        float x = 1.0f;
        for (int q = 0; q < power; q++) x = x * inv;
        w[a] = x;
        lab[a] = at.labels[a][v];
    }
    int best = lab[0];
    float best_s = -1.0f;
    for (int a = 0; a < n_atlas; a++) {
        const int L = lab[a];
        float s = 0.0f;
        for (int b = 0; b < n_atlas; b++)
            if (lab[b] == L) s = s + w[b];
        if (s > best_s || (s == best_s && L < best)) {
            best_s = s;
            best = L;
        }
    }
    out[v] = (int16_t)best;
}

}  // namespace

size_t fuse_scratch_floats(int n_atlas, int m, int n, int o) { return 2 * (size_t)n_atlas * m * n * o; }

cudaError_t launch_fuse_labels(const float* d_target, const FusionAtlases& at, int n_atlas, int m, int n, int o,
                               int radius, float eps, int power, float* d_scratch, int16_t* d_out, cudaStream_t s) {
    if (n_atlas < 1 || n_atlas > kFuseMaxAtlases || radius < 0 || power < 0) return cudaErrorInvalidValue;
    const int64_t sz = (int64_t)m * n * o;
    float* a = d_scratch;
    // slices per block: enough blocks for eight a SM, and halos of at most a quarter
    const int tiles = ((m + TI - 1) / TI) * ((n + TJ - 1) / TJ) * n_atlas;
    int chunks = (8 * 152 + tiles - 1) / tiles;
    chunks = std::max(1, std::min(chunks, o / (8 * std::max(radius, 1))));
    const int k_chunk = (o + chunks - 1) / chunks;
    chunks = (o + k_chunk - 1) / k_chunk;
    const dim3 g3((m + TI - 1) / TI, (n + TJ - 1) / TJ, n_atlas * chunks);
    if (radius >= 1 && radius <= 3) {
        if (radius == 1) k_window3<1><<<g3, TI * TJ, 0, s>>>(d_target, at, a, n_atlas, m, n, o, k_chunk);
        else if (radius == 2) k_window3<2><<<g3, TI * TJ, 0, s>>>(d_target, at, a, n_atlas, m, n, o, k_chunk);
        else k_window3<3><<<g3, TI * TJ, 0, s>>>(d_target, at, a, n_atlas, m, n, o, k_chunk);
        count_launches(1);
    } else {  // no window, or one whose halo outweighs the tile: pass by pass
        float* b = d_scratch + (size_t)n_atlas * sz;
        const dim3 grid((unsigned)((sz + 255) / 256), n_atlas);
        k_window<true><<<grid, 256, 0, s>>>(d_target, at, nullptr, a, m, n, o, 0, radius);
        k_window<false><<<grid, 256, 0, s>>>(d_target, at, a, b, m, n, o, 1, radius);
        k_window<false><<<grid, 256, 0, s>>>(d_target, at, b, a, m, n, o, 2, radius);
        count_launches(3);
    }
    const unsigned nb = (unsigned)((sz + 255) / 256);
    if (n_atlas <= 4) k_vote_n<4><<<nb, 256, 0, s>>>(at, n_atlas, a, sz, eps, power, d_out);
    else if (n_atlas <= 8) k_vote_n<8><<<nb, 256, 0, s>>>(at, n_atlas, a, sz, eps, power, d_out);
    else if (n_atlas <= 16) k_vote_n<16><<<nb, 256, 0, s>>>(at, n_atlas, a, sz, eps, power, d_out);
    else k_vote<<<nb, 256, 0, s>>>(at, n_atlas, a, sz, eps, power, d_out);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace deeds
