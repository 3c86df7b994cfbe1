// MIND-SSC descriptor on sm_103a (replaces descriptor(), src/MINDSSCbox.h:127-232).
//
// Layout in HBM: six distance channels D[l][p] (6 x m*n*o float32, context
// scratch) and the output codes C[p] (uint64).  Three launches:
//   1. k_pass_ij: per slice and channel, the shifted squared difference (imshift +
//      distances, src/MINDSSCbox.h:79-124) and its box sums along i and j (volumes of
//      more than 512 lines a slice: k_pass_i and k_pass_jk, one axis each);
//   2. k_pass_jk (k): the k-axis box sums, in place;
//   3. k_quantise: the 12 SSC pairs -> min/mean normalisation -> 5 thresholds
//      -> thermometer code (src/MINDSSCbox.h:175-224).
// Box sums keep the reference's sequential float prefix sum along each line and
// its edge rules (src/MINDSSCbox.h:9-73): one thread owns one line and streams it
// with a lag of r, keeping the last 2r+2 prefix values in a ring; a parallel
// scan would change the rounding and with it codes near thresholds.
// Traffic per voxel: 4 B read + 24 B write (pass ij), 48 B (pass k, bound by it), 24 B
// read + 8 B write (quantise) = 108 B; at 192x160x256 336 us before passes i and j were
// one and the quantiser counted with integer units, 229 us now.
#include <cmath>

#include "common.cuh"
#include "kernels.h"

namespace deeds {

namespace {

constexpr int kRing = 16;  // supports box radius r <= 7 (2r+2 <= 16)

// Shift vectors of the six distance channels (src/MINDSSCbox.h:132-134).
__constant__ int c_dx[6] = {1, 1, -1, 0, 1, 0};
__constant__ int c_dy[6] = {1, -1, 0, -1, 0, 1};
__constant__ int c_dz[6] = {0, 0, 1, 1, 1, 1};

// i-axis pass: CTA = one k slice x TJ consecutive j lines x all 6 channels.
// The image neighbourhood of an i-chunk (rows j-q..j+TJ+q at k and k+q, i-q..i+CH+q)
// is staged in shared memory with coalesced loads; each thread streams one
// (channel, line) through the sequential box sum; outputs go through a shared
// tile so that the six channel planes are written with coalesced stores.
// The radius QS is a compile-time constant and chunks start at multiples of 16,
// so every index into the ring of prefix values is static after unrolling and the
// ring lives in registers (a runtime index would place it in local memory); the
// tail outputs are emitted at the line's last step for the same reason.
constexpr int TJ = 32;  // lines per CTA
constexpr int CH = 32;  // i samples per chunk (a multiple of kRing)
static_assert(CH == 32 && TJ == 32, "one lane per sample; warp l of a CTA is channel l");

template <int QS>
__global__ void __launch_bounds__(6 * TJ) k_pass_i(const float* __restrict__ im, float* __restrict__ D, int m, int n,
                                                   int o) {
    extern __shared__ float sm[];
    constexpr int W = CH + 2 * QS + 1;     // padded row length of the image tile
    constexpr int WL = CH + 2 * QS;        // loaded row length
    constexpr int R = TJ + 2 * QS;         // image rows per k slice
    float* Tbuf = sm;                      // two tiles [2][R][W]: the chunk's, and the next one's in flight
    float* O = sm + 4 * R * W;             // [6][TJ][CH+1]
    const int k = blockIdx.y, j0 = blockIdx.x * TJ;
    const int l = threadIdx.x / TJ, jj = threadIdx.x % TJ, j = j0 + jj;
    const int64_t mn = (int64_t)m * n, sz = mn * o;
    const int dx = c_dx[l] * QS, dy = c_dy[l] * QS, dz = c_dz[l] * QS;
    const bool line_ok = j < n;
    const bool other_ok = j + dx >= 0 && j + dx < n && k + dz < o;
    const int kk = dz ? 1 : 0;
    float* gout = D + l * sz + (int64_t)j * m + (int64_t)k * mn;
    float ring[kRing];
    float P = 0.0f;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int kWarps = 6 * TJ / 32;
    // the image tile of the chunk at i0 into Tb with 4-byte cp.async, one warp per
    // tile row (rows of both k planes); samples outside the volume are zero-filled
    // (no bytes read)
    auto load_tile = [&](int i0, float* Tb) {
        for (int row = warp; row < 2 * R; row += kWarps) {
            const int z = row / R, r = row - z * R;
            const int jr = j0 - QS + r, kz = k + z * QS;
            const bool row_ok = jr >= 0 && jr < n && kz < o;
            const float* src = im + (int64_t)(row_ok ? jr : 0) * m + (int64_t)(row_ok ? kz : 0) * mn;
            float* dst = Tb + row * W;
#pragma unroll
            for (int ip = lane; ip < WL; ip += 32) {
                const int ii = i0 - QS + ip;
                const bool ok = row_ok && ii >= 0 && ii < m;
                const unsigned d = (unsigned)__cvta_generic_to_shared(dst + ip);
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(ok ? src + ii : im),
                             "r"(ok ? 4 : 0)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load_tile(0, Tbuf);
    for (int i0 = 0, c = 0; i0 < m; i0 += CH, c++) {
        float* T = Tbuf + (c & 1) * 2 * R * W;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // this chunk's tile has landed; the previous chunk's tile is consumed
        if (i0 + CH < m) load_tile(i0 + CH, Tbuf + ((c + 1) & 1) * 2 * R * W);  // in flight during this chunk
        const int cend = min(CH, m - i0);
        // interior chunk: no line start or end, no shifted sample outside the line, all
        // CH samples present; the steps need no index checks
        const bool interior = i0 >= CH && i0 + CH + QS <= m;
        if (line_ok && interior) {
            const float* self = T + (jj + QS) * W + QS;
            // a partner line outside the volume compares the voxel with itself (d = 0)
            const float* oth = other_ok ? T + (kk * R + jj + QS + dx) * W + QS + dy : self;
            float* out = O + (l * TJ + jj) * (CH + 1);
#pragma unroll
            for (int u = 0; u < CH; u++) {
                const float d = oth[u] - self[u];
                P = P + d * d;
                ring[u & (kRing - 1)] = P;  // i0 is a multiple of kRing
                out[u] = P - ring[(u - 2 * QS - 1) & (kRing - 1)];
            }
        } else if (line_ok) {
            const float* self = T + (jj + QS) * W + QS;
            const float* oth = T + (kk * R + jj + QS + dx) * W + QS + dy;
            float* out = O + (l * TJ + jj) * (CH + 1);
#pragma unroll
            for (int u = 0; u < CH; u++) {
                if (u < cend) {
                    const int t = i0 + u;
                    const float s = self[u];
                    const float v = (other_ok && t + dy >= 0 && t + dy < m) ? oth[u] : s;
                    const float d = v - s;
                    const float x = d * d;
                    P = (t == 0) ? x : P + x;
                    ring[u & (kRing - 1)] = P;  // i0 is a multiple of kRing
                    const int i = t - QS;       // output position (lag r = QS)
                    if (i >= 0) out[u] = (i <= QS) ? P : P - ring[(u - 2 * QS - 1) & (kRing - 1)];
                    if (t == m - 1) {
                        // tail: i in [m-QS, m): P[m-1] - P[i-QS-1]
#pragma unroll
                        for (int s2 = 0; s2 < QS; s2++) gout[m - QS + s2] = P - ring[(u - 2 * QS + s2) & (kRing - 1)];
                    }
                }
            }
        }
        __syncwarp();  // a warp stores the output rows its own lanes wrote (warp = channel)
        // coalesced store of outputs i0-QS .. i0+cend-1-QS: the warp of channel l stores
        // its TJ lines, one lane per sample (CH == 32)
        {
            const int i = i0 + lane - QS;
            if (lane < cend && i >= 0) {
                const int nl = min(TJ, n - j0);
                float* dst = D + warp * sz + (int64_t)k * mn + (int64_t)j0 * m + i;
                const float* src = O + warp * TJ * (CH + 1) + lane;
#pragma unroll 8
                for (int jl = 0; jl < nl; jl++) dst[(int64_t)jl * m] = src[jl * (CH + 1)];
            }
        }
    }
}

// i- and j-axis passes in one: CTA = one k slice x one channel, a thread = one line
// (n <= kIJLines).  The slice is taken in strips of 32 outputs along i: the shifted
// squared differences of a strip go to shared memory with coalesced loads (lane =
// sample), each thread runs its line's box sum along the strip in place (prefix and
// ring stay in its registers from strip to strip; a strip's samples are those QS
// ahead of its outputs), then the first warp runs the 32 columns' box sums along j and
// stores them, coalesced along i.  The other warps wait for that one; the CTAs on the
// SM (six at 160 lines) fill in.
// D is written once in place of twice and a read, 378 MB less at 192x160x256, where the
// two passes took 89 + 63 us and this one takes 92 (radius 2; bound by issue, 36
// instructions a value, and the barriers).  Strips of 64: 116 us (five CTAs, three waves);
// 48 registers and eight CTAs: 182 us (the loads no longer hit L1); 40: 133 us (spills).
// Above kIJLines lines a thread would hold several lines' state: those volumes take the
// two separate passes.
constexpr int kIJLines = 512, kStrip = 32, kPitch = kStrip + 1;

template <int QS>
__global__ void __launch_bounds__(kIJLines, 2)
    k_pass_ij(const float* __restrict__ im, float* __restrict__ D, int m, int n, int o) {
    extern __shared__ float X[];  // [n][kPitch]
    const int k = blockIdx.x, l = blockIdx.y;
    const int64_t mn = (int64_t)m * n;
    const int dx = c_dx[l] * QS, dy = c_dy[l] * QS, dz = c_dz[l] * QS;
    const float* slice = im + k * mn;
    const int away = (int)(dz * mn) + dx * m + dy;  // a partner's distance in samples
    const bool slice_ok = k + dz < o;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int j = threadIdx.x;
    // squared difference of sample (t, row); a partner outside compares the voxel with itself
    auto sample = [&](int t, int row) {
        const int at = row * m + t;
        const bool ok = slice_ok && (unsigned)(row + dx) < (unsigned)n && (unsigned)(t + dy) < (unsigned)m;
        const float a = slice[at], d = slice[ok ? at + away : at] - a;
        return d * d;
    };
    float ring[kRing];
    float P = 0.0f;
    if (j < n) {
#pragma unroll
        for (int t = 0; t < QS; t++) {  // QS < m
            const float x = sample(t, j);
            P = t == 0 ? x : P + x;
            ring[t] = P;
        }
    }
    for (int i0 = 0; i0 < m; i0 += kStrip) {
        {
            const int t = min(i0 + QS + lane, m - 1);  // past the line's end: not used
            const bool ok_t = slice_ok && (unsigned)(t + dy) < (unsigned)m;
            float* x = X + lane;
            int row = warp;
            for (; row + 7 * warps < n; row += 8 * warps) {
                float a[8], b[8];
#pragma unroll
                for (int r = 0; r < 8; r++) {
                    const int rr = row + r * warps, at = rr * m + t;
                    a[r] = slice[at];
                    b[r] = slice[ok_t && (unsigned)(rr + dx) < (unsigned)n ? at + away : at];
                }
#pragma unroll
                for (int r = 0; r < 8; r++) {
                    const float d = b[r] - a[r];
                    x[(row + r * warps) * kPitch] = d * d;
                }
            }
            for (; row < n; row += warps) x[row * kPitch] = sample(t, row);
        }
        __syncthreads();
        if (j < n) {
            float* x = X + j * kPitch;
            if (i0 > 0 && i0 + kStrip + QS <= m) {  // no line start, no line end
#pragma unroll
                for (int u = 0; u < kStrip; u++) {
                    P = P + x[u];
                    ring[(QS + u) & (kRing - 1)] = P;
                    x[u] = P - ring[(u - QS - 1) & (kRing - 1)];
                }
            } else {
#pragma unroll
                for (int u = 0; u < kStrip; u++) {
                    const int i = i0 + u;
                    if (i + QS < m) P = P + x[u];  // past the line's end the prefix stays
                    ring[(QS + u) & (kRing - 1)] = P;
                    x[u] = i <= QS ? P : P - ring[(u - QS - 1) & (kRing - 1)];
                }
            }
        }
        __syncthreads();
        if (j < kStrip && i0 + j < m) {
            float* base = D + l * (mn * o) + k * mn + i0 + j;
            float rj[kRing], Q = 0.0f;
            for (int c0 = 0; c0 < n; c0 += kRing) {
                const float* x = X + c0 * kPitch + j;
                if (c0 > 0 && c0 + kRing < n) {
                    float* out = base + (int64_t)(c0 - QS) * m;
                    float y[kRing];
#pragma unroll
                    for (int u = 0; u < kRing; u++) y[u] = x[u * kPitch];
#pragma unroll
                    for (int u = 0; u < kRing; u++) {
                        Q = Q + y[u];
                        rj[u] = Q;
                        *out = Q - rj[(u - 2 * QS - 1) & (kRing - 1)];
                        out += m;
                    }
                } else {
#pragma unroll
                    for (int u = 0; u < kRing; u++) {
                        const int t = c0 + u;
                        if (t < n) {
                            const float y = x[u * kPitch];
                            Q = t == 0 ? y : Q + y;
                            rj[u] = Q;
                            const int jo = t - QS;
                            if (jo >= 0)
                                base[(int64_t)jo * m] = jo <= QS ? Q : Q - rj[(u - 2 * QS - 1) & (kRing - 1)];
                            if (t == n - 1) {
#pragma unroll
                                for (int s2 = 0; s2 < QS; s2++)
                                    base[(int64_t)(n - QS + s2) * m] = Q - rj[(u - 2 * QS + s2) & (kRing - 1)];
                            }
                        }
                    }
                }
            }
        }
        __syncthreads();  // the strip's tile is consumed
    }
}

// In-place box pass along j (axis=1) or k (axis=2); threads over consecutive i.
// Samples are loaded CHUNK at a time before any of the chunk's outputs (which
// lag by r) are stored, so the loads of a chunk are independent; with CHUNK a
// multiple of kRing and QS fixed at compile time the ring stays in registers.
template <int QS>
__global__ void k_pass_jk(float* __restrict__ D, int m, int n, int o, int axis) {
    constexpr int CHUNK = kRing;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = blockIdx.y;  // the other coordinate: k for axis 1, j for axis 2
    const int l = blockIdx.z;
    if (i >= m) return;
    const int64_t mn = (int64_t)m * n, sz = mn * o;
    float* base;
    int64_t stride;
    int L;
    if (axis == 1) { base = D + l * sz + i + b * mn; stride = m; L = n; }
    else { base = D + l * sz + i + (int64_t)b * m; stride = mn; L = o; }
    float ring[kRing];
    float P = 0.0f;
    for (int c0 = 0; c0 < L; c0 += CHUNK) {
        float x[CHUNK];
#pragma unroll
        for (int u = 0; u < CHUNK; u++) x[u] = (c0 + u < L) ? base[(c0 + u) * stride] : 0.0f;
#pragma unroll
        for (int u = 0; u < CHUNK; u++) {
            const int t = c0 + u;
            if (t < L) {
                P = (t == 0) ? x[u] : P + x[u];
                ring[u] = P;  // c0 is a multiple of kRing
                const int io = t - QS;
                if (io >= 0) base[io * stride] = (io <= QS) ? P : P - ring[(u - 2 * QS - 1) & (kRing - 1)];
                if (t == L - 1) {
#pragma unroll
                    for (int s2 = 0; s2 < QS; s2++)
                        base[(L - QS + s2) * stride] = P - ring[(u - 2 * QS + s2) & (kRing - 1)];
                }
            }
        }
    }
}

// The five quantisation thresholds and, around each, a window of 2^-20 relative
// width: the product y = v * RN(1/noise) is within 1.5 ulp of the correctly rounded
// quotient RN(v/noise), so a threshold whose window does not hold y compares with
// the quotient as it compares with y.
struct QuantThr {
    float t[5], lo[5], hi[5];
};

// The twelve SSC pairs (src/MINDSSCbox.h:136-140): pair l compares channel l / 2
// at the voxel's neighbour QS away along one axis (0: i, 1: j, 2: k) in direction
// kSign[l]; a neighbour outside the volume reads the voxel itself.  With QS a
// compile-time constant every offset is a constant multiple of the line and
// slice strides and each pair needs one bounds test.
__device__ __forceinline__ float exp2_approx(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float fmin3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// RN(x / 12) for finite x >= 0, up to results far below 1e-6: quotient estimate and
// Markstein's correction by the exact remainder (all 2^23 significands agree with the
// IEEE division; the exponent only scales).
__device__ __forceinline__ float twelfth(float x) {
    const float r = 1.0f / 12.0f, q = __fmul_rn(x, r);
    return __fmaf_rn(__fmaf_rn(-12.0f, q, x), r, q);
}
// `width` ones from bit `pos` on (width >= 0)
__device__ __forceinline__ uint32_t bit_mask(int pos, int width) {
    uint32_t r;
    asm("bmsk.clamp.b32 %0, %1, %2;" : "=r"(r) : "r"(pos), "r"(width));
    return r;
}

template <int QS, bool LOGTHR>
__global__ void __launch_bounds__(64) k_quantise(const float* __restrict__ D, uint64_t* __restrict__ codes, int m,
                                                 int n, int o, QuantThr th) {
    constexpr int kAxis[12] = {1, 0, 1, 0, 2, 1, 2, 0, 2, 1, 2, 0};
    constexpr int kSign[12] = {-1, -1, -1, 1, -1, 1, -1, 1, -1, -1, -1, -1};
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y;
    const int k = blockIdx.z;
    if (i >= m) return;
    const int64_t mn = (int64_t)m * n, sz = mn * o;
    // a pair's neighbour is in this slice, at a 32-bit index, or at the same place of the
    // slice QS below, whose base is the block's
    const uint32_t at = (uint32_t)j * m + i;
    const uint32_t near[2][2] = {{i >= QS ? at - QS : at, i + QS < m ? at + QS : at},
                            {j >= QS ? at - QS * m : at, j + QS < n ? at + QS * m : at}};
    const float* here = D + k * mn;
    const float* below = k >= QS ? here - QS * mn : here;
    static_assert(kSign[4] < 0 && kSign[6] < 0 && kSign[8] < 0 && kSign[10] < 0, "k neighbours are below");
    float v[12];
    auto load = [&]() {
#pragma unroll
        for (int l = 0; l < 12; l++) {
            const int ax = kAxis[l];
            v[l] = ax == 2 ? __ldg(below + (l >> 1) * sz + at) : __ldg(here + (l >> 1) * sz + near[ax][kSign[l] > 0]);
        }
    };
    load();
    // Finite values: the minimum in any order, and a sum that is below infinity.
    float noise = 0.0f;
    {
        float lowest = fmin3(v[0], v[1], v[2]);
#pragma unroll
        for (int l = 3; l < 11; l += 2) lowest = fmin3(lowest, v[l], v[l + 1]);
        lowest = fminf(lowest, v[11]);
#pragma unroll
        for (int l = 0; l < 12; l++) { v[l] = v[l] - lowest; noise = noise + v[l]; }
    }
    const bool finite = noise < INFINITY;
    if (!finite) {  // the reference's scan: a NaN first value stays, later ones are skipped
        load();
        float lowest = v[0];
#pragma unroll
        for (int l = 1; l < 12; l++) lowest = v[l] < lowest ? v[l] : lowest;
        noise = 0.0f;
#pragma unroll
        for (int l = 0; l < 12; l++) { v[l] = v[l] - lowest; noise = noise + v[l]; }
        noise = __fdiv_rn(noise, 12.0f);
    } else {
        noise = twelfth(noise);
    }
    noise = fmaxf(noise, 1e-6f);
    // The level only counts the thresholds above the correctly rounded quotient
    // RN(v / noise).  v * RN(1 / noise) is within 1.5 ulp of it (two roundings of
    // at most half an ulp each, relative 2^-24, on a quotient whose own rounding is
    // half an ulp), so unless a threshold lies within 2^-20 (relative, ~8 ulp) of
    // that product both give the same count; near a threshold the IEEE division
    // decides.  noise >= 1e-6 (fmaxf drops a NaN sum); NaN, infinite, zero and
    // tiny quotients fall on the same side of every threshold both ways.
    uint32_t w0 = 0, w1 = 0;  // the code's 60 bits, thermometer {0,1,3,7,15,31} of pair l at bit 5 l
    auto put = [&](int l, int lvl) {
        if (l < 6) w0 |= bit_mask(5 * l, lvl);
        else if (l > 6) w1 |= bit_mask(5 * l - 32, lvl);
        else {
            const uint32_t t = bit_mask(0, lvl);
            w0 |= t << 30;
            w1 |= t >> 2;
        }
    };
    bool exact = false;
    if (LOGTHR) {
        // thresholds -log((c+1.5)/6), c = 0..4: c counts when c < z = 6 exp(-x) - 1.5, so the
        // level is ceil(z), or 0 below.  z from the fast reciprocal and exponential is within
        // 2^-17 of the z of the quotient and of the float thresholds (the reciprocal is normal: a
        // finite sum leaves a noise below 2^125): relative errors of
        // 2^-22 (exponential), 2^-21.4 (its argument) and 2^-20 (thresholds), with y e^-y <=
        // 0.37, times 6.  One multiply-add places z + 1 at 2^-16 a unit of the mantissa, with
        // the ceiling above the low 16 bits; where those are within 4 of a whole number for
        // any pair, or the sum is not finite, the IEEE divisions decide.  (With a rounding, a
        // ceiling and a conversion for each pair the kernel was bound by the conversion pipe
        // and by issue, 435 instructions a voxel, 111 us at 192x160x256; now 280 and 72 us.)
        constexpr float kBase = 192.0f;  // [128, 256): a unit of the last place is 2^-16
        const float c2 = __fmul_rn(rcp_approx(noise), -1.44269504f);
        uint32_t z[12], low = 0xffffffffu;
#pragma unroll
        for (int l = 0; l < 12; l++) {
            const float e = exp2_approx(__fmul_rn(v[l], c2));
            z[l] = __float_as_uint(__fmaf_rn(6.0f, e, kBase - 1.5f + 1.0f + 4 * 0x1p-16f));
            put(l, max((int)(z[l] >> 16) - 0x4340, 0));
        }
#pragma unroll
        for (int l = 0; l < 12; l += 4)  // the low halves, two to a word
            low = __vimin3_u16x2(low, __byte_perm(z[l], z[l + 1], 0x5410), __byte_perm(z[l + 2], z[l + 3], 0x5410));
        exact = (low & 0xffffu) < 8u || low < 8u << 16 || !finite;
    } else {
        // y outside every threshold's window: each threshold is above or below the
        // quotient as it is above or below y; y inside a window: the IEEE division decides
        const float rcp = __frcp_rn(noise);
#pragma unroll
        for (int l = 0; l < 12; l++) {
            const float y = __fmul_rn(v[l], rcp);
            int lvl = 0, cnt = 0;
#pragma unroll
            for (int q = 0; q < 5; q++) {
                lvl += y < th.lo[q];
                cnt += y <= th.hi[q];
            }
            exact = exact || cnt != lvl;
            put(l, lvl);
        }
    }
    if (exact) {
        w0 = w1 = 0;
#pragma unroll
        for (int l = 0; l < 12; l++) {
            const float x = __fdiv_rn(v[l], noise);
            int lvl = 0;
#pragma unroll
            for (int q = 0; q < 5; q++) lvl += th.t[q] > x;
            put(l, lvl);
        }
    }
    codes[k * mn + at] = (uint64_t)w1 << 32 | w0;
}

}  // namespace

// One line per thread, and a partner's distance (up to QS + 1 slices) in 32 bits.
static bool mind_by_slice(int m, int n) { return n <= kIJLines && (int64_t)m * n < (1 << 28); }

template <int QS>
static void mind_passes(const float* d_im, int m, int n, int o, const float thr[5], float* d_scratch,
                        uint64_t* d_codes, cudaStream_t s) {
    // 64 i per block: the usual volume extents are multiples of 64, so no lane idles
    const bool by_slice = mind_by_slice(m, n);
    if (by_slice) {
        constexpr int most = kIJLines * kPitch * (int)sizeof(float);
        cudaFuncSetAttribute(k_pass_ij<QS>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        k_pass_ij<QS><<<dim3(o, 6), (n + 31) / 32 * 32, n * kPitch * sizeof(float), s>>>(d_im, d_scratch, m, n, o);
    } else {
        const size_t smem = (size_t)(4 * (TJ + 2 * QS) * (CH + 2 * QS + 1) + 6 * TJ * (CH + 1)) * sizeof(float);
        if (smem > 48 * 1024)
            cudaFuncSetAttribute(k_pass_i<QS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        k_pass_i<QS><<<dim3((n + TJ - 1) / TJ, o), 6 * TJ, smem, s>>>(d_im, d_scratch, m, n, o);
        k_pass_jk<QS><<<dim3((m + 63) / 64, o, 6), 64, 0, s>>>(d_scratch, m, n, o, 1);
    }
    k_pass_jk<QS><<<dim3((m + 63) / 64, n, 6), 64, 0, s>>>(d_scratch, m, n, o, 2);
    QuantThr th;
    for (int q = 0; q < 5; q++) {
        // a window of 2^-20 (relative) on either side of the threshold
        const float a = thr[q] * (1.0f - 0x1p-20f), b = thr[q] * (1.0f + 0x1p-20f);
        th.t[q] = thr[q];
        th.lo[q] = a < b ? a : b;
        th.hi[q] = a < b ? b : a;
    }
    // the reference's thresholds -logf((c+1.5)/6) (within 2^-20): the level from one exponential
    bool logthr = true;
    for (int q = 0; q < 5; q++) {
        const double ref = -std::log((q + 1.5) / 6.0);
        logthr = logthr && std::fabs((double)thr[q] - ref) <= 0x1p-20 * ref;
    }
    if (logthr) k_quantise<QS, true><<<dim3((m + 63) / 64, n, o), 64, 0, s>>>(d_scratch, d_codes, m, n, o, th);
    else k_quantise<QS, false><<<dim3((m + 63) / 64, n, o), 64, 0, s>>>(d_scratch, d_codes, m, n, o, th);
}

cudaError_t launch_mind_ssc(const float* d_im, int m, int n, int o, int qs, const float thr[5], float* d_scratch,
                            uint64_t* d_codes, cudaStream_t s) {
    switch (qs) {
        case 1: mind_passes<1>(d_im, m, n, o, thr, d_scratch, d_codes, s); break;
        case 2: mind_passes<2>(d_im, m, n, o, thr, d_scratch, d_codes, s); break;
        case 3: mind_passes<3>(d_im, m, n, o, thr, d_scratch, d_codes, s); break;
        case 4: mind_passes<4>(d_im, m, n, o, thr, d_scratch, d_codes, s); break;
        case 5: mind_passes<5>(d_im, m, n, o, thr, d_scratch, d_codes, s); break;
        case 6: mind_passes<6>(d_im, m, n, o, thr, d_scratch, d_codes, s); break;
        case 7: mind_passes<7>(d_im, m, n, o, thr, d_scratch, d_codes, s); break;
        default: return cudaErrorInvalidValue;
    }
    count_launches(mind_by_slice(m, n) ? 3 : 4);
    return cudaGetLastError();
}

}  // namespace deeds
