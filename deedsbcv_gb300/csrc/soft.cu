// Differentiable soft-min deeds level on sm_103a: forward and hand-written adjoint.
//
// There is no counterpart in the reference; the form relaxes one level of
// src/deedsBCV0.cpp:238-306 so that it is differentiable in both images and in
// the regularisation weight alpha.  With a zero prior field:
//   descriptor  s_l(p) = 6 exp(-(v_l - min v)/max(mean(v - min v), 1e-6)), v_l the
//               12 box-filtered self-similarity distances of MIND-SSC
//               (src/MINDSSCbox.h:127-201; the reference quantises exactly this
//               quantity: code = #{c : s > c + 1.5});
//   cost        C[c][l] = alpha1 sum_{samples p of c} sum_ch phi(sF_ch(p) - sM_ch(p + d(l))),
//               phi(x) = sqrt(x^2 + eps^2) - eps, alpha1 = 0.5 (g/(alpha q))/maxsamp,
//               sampling and clamp-to-edge of src/dataCostD.h:141-200;
//   upward      B_c = C_c + sum_children (M_k - min M_k),
//               M_c(lp) = -tau LSE_l(-(e_c B_c(l) + |lab(l) - lab(lp)|^2)/tau)
//               (src/regularisation.h:190-238 with min -> soft-min);
//   downward    log p_root = log softmax(-B_root/tau),
//               log p_c(l) = -e_c B_c(l)/tau + LSE_lp(log p_p(lp) + M_c(lp)/tau - |lab(l)-lab(lp)|^2/tau);
//   output      E_c = sum_l p_c(l) d(l), d(l) = (label - hw) q per axis (u = x, v = y, w = z).
//
// Both label-space transforms are the same operator S(x)(b) = LSE_a(x(a) - |a-b|^2/tau)
// over the len^3 label grid.  Because |a-b|^2 is a sum over the three axes, S is
// three one-axis passes in the log domain (len^4 terms per pass instead of len^6),
// each pass max-shifted so that nothing under- or overflows.  Its adjoint is three
// passes back, each weighting the incoming gradient with exp(in(a) - |a-b|^2/tau -
// out(b)) <= 1.  One CTA owns one tree node; its label vectors and the pass
// intermediates live in shared memory.  Tree nodes are processed one breadth level
// per launch (children before parents upward, parents before children downward).
//
// Backward recomputes the forward sweeps from the inputs (no message tensors are
// kept between forward and backward) and then runs, per breadth level:
//   marginal adjoint (leaves to root): h_c = dL/dlog p_c = (gE_c . d) p_c + sum_children R_k;
//       Bbar_c = -e_c h_c/tau (root: -(h - p sum h)/tau); R_c = S^T h_c (w.r.t. S's input);
//   message adjoint (root to leaves): Mbar_c = R_c/tau + Bbar_parent;
//       Bbar_c += e_c S^T(Mbar_c) (S taken at -e_c B_c/tau); cbar_c = Bbar_c;
// then the cost, descriptor, box-filter and squared-difference adjoints.  The min
// subtracted from each message shifts B_parent by a constant to which the marginals
// are invariant, so it carries no gradient.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace deeds {

namespace {

__constant__ int s_dx[6] = {1, 1, -1, 0, 1, 0};
__constant__ int s_dy[6] = {1, -1, 0, -1, 0, 1};
__constant__ int s_dz[6] = {0, 0, 1, 1, 1, 1};
__constant__ int s_sx[12] = {-1, 0, -1, 0, 0, 1, 0, 0, 0, -1, 0, 0};
__constant__ int s_sy[12] = {0, -1, 0, 1, 0, 0, 0, 1, 0, 0, 0, -1};
__constant__ int s_sz[12] = {0, 0, 0, 0, -1, 0, -1, 0, -1, 0, -1, 0};

__device__ __forceinline__ bool inside(int i, int j, int k, int m, int n, int o) {
    return i >= 0 && i < m && j >= 0 && j < n && k >= 0 && k < o;
}

inline unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

// ---------------------------------------------------------------------------
// Descriptor

// w_l(p) = (I(p + t_l) - I(p))^2, 0 where p + t_l leaves the volume (the reference's
// imshift keeps the voxel itself there, src/MINDSSCbox.h:79-124)
__global__ void k_soft_sqdiff(const float* __restrict__ im, float* __restrict__ w, int m, int n, int o, int qs) {
    const int64_t sz = (int64_t)m * n * o;
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= sz) return;
    const int i = (int)(p % m), j = (int)((p / m) % n), k = (int)(p / ((int64_t)m * n));
    const float c = im[p];
#pragma unroll
    for (int l = 0; l < 6; l++) {
        const int ii = i + s_dy[l] * qs, jj = j + s_dx[l] * qs, kk = k + s_dz[l] * qs;
        float d = 0.0f;
        if (inside(ii, jj, kk, m, n, o)) d = im[ii + (int64_t)jj * m + (int64_t)kk * m * n] - c;
        w[l * sz + p] = d * d;
    }
}

// Windowed sum over [max(0,i-r), min(L-1,i+r)] along one axis, out of place, summed
// directly (no prefix-sum differences, whose cancellation would cost the soft
// descriptor its float32 accuracy).  The operator is symmetric, so the same
// kernel is its own adjoint.  Grid: x over i, y over j (32 x 8 blocks), z over
// (k, channel): no index divisions by runtime sizes.  For radii above 3; below, k_soft_box3.
__global__ void k_soft_box(const float* __restrict__ in, float* __restrict__ out, int m, int n, int o, int r, int axis) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= m || j >= n) return;
    const int k = blockIdx.z % o, ch = blockIdx.z / o;
    const int64_t mn = (int64_t)m * n;
    const int64_t p = (int64_t)ch * mn * o + i + (int64_t)j * m + (int64_t)k * mn;
    int L, c;
    int64_t stride;
    if (axis == 0) { L = m; stride = 1; c = i; }
    else if (axis == 1) { L = n; stride = m; c = j; }
    else { L = o; stride = mn; c = k; }
    const float* x = in + (p - (int64_t)c * stride);
    float acc = 0.0f;
    const int a0 = max(0, c - r), a1 = min(L - 1, c + r);
    for (int a = a0; a <= a1; a++) acc += x[a * stride];
    out[p] = acc;
}

// The three windowed sums in one pass, radius R (a compile-time constant, up to 3), of
// six channels: of `in` (6 x sz), or (IMAGE) of the squared differences of k_soft_sqdiff
// made from the image `in` on the way.  A block marches along k over 32 x 8 columns: each
// plane's tile and halo go to shared memory (double-buffered, one barrier a plane, the
// next plane's loads in flight), a thread sums its window along i, then j, and keeps
// the last 2R + 1 planes' sums in registers for k.  Sums and their order are those of the
// three passes.  Bound by issue (about 50 instructions a value at R = 1).
// 96x80x112, radius 1: differences and three passes 73 us, one launch 29; three passes of
// given channels 63 us, one launch 16.
constexpr int kBoxPlanes = 32;  // planes a block outputs: 2R more are read

template <int R, bool IMAGE>
__global__ void __launch_bounds__(256) k_soft_box3(const float* __restrict__ in, float* __restrict__ out, int m, int n,
                                                   int o, int qs) {
    constexpr int TI = 32, TJ = 8, SI = TI + 2 * R, SJ = TJ + 2 * R, NE = (SI * SJ + 255) / 256;
    __shared__ float tile[2][SJ][SI];
    const int ch = blockIdx.z % 6, k0 = (int)(blockIdx.z / 6) * kBoxPlanes, k1 = min(o, k0 + kBoxPlanes);
    const int64_t mn = (int64_t)m * n, sz = mn * o;
    const float* vol = IMAGE ? in : in + ch * sz;
    const int ti = threadIdx.x % TI, tj = threadIdx.x / TI;
    const int i = blockIdx.x * TI + ti, j = blockIdx.y * TJ + tj;
    const int di = IMAGE ? s_dy[ch] * qs : 0, dj = IMAGE ? s_dx[ch] * qs : 0, dk = IMAGE ? s_dz[ch] * qs : 0;
    float next[NE];
    auto fetch = [&](int k) {
#pragma unroll
        for (int e = 0; e < NE; e++) {
            const int at = threadIdx.x + e * 256, b = at / SI, a = at - b * SI;
            const int ii = blockIdx.x * TI - R + a, jj = blockIdx.y * TJ - R + b;
            float v = 0.0f;
            if (at < SI * SJ && inside(ii, jj, k, m, n, o)) {
                const int64_t p = ii + (int64_t)jj * m + k * mn;
                v = __ldg(vol + p);
                if (IMAGE) {
                    const bool both = inside(ii + di, jj + dj, k + dk, m, n, o);
                    const float d = both ? __ldg(vol + p + di + (int64_t)dj * m + dk * mn) - v : 0.0f;
                    v = d * d;
                }
            }
            next[e] = v;
        }
    };
    float win[2 * R + 1];
#pragma unroll
    for (int d = 0; d <= 2 * R; d++) win[d] = 0.0f;
    fetch(k0 - R);
    for (int k = k0 - R, buf = 0; k < k1 + R; k++, buf ^= 1) {
#pragma unroll
        for (int e = 0; e < NE; e++) {
            const int at = threadIdx.x + e * 256;
            if (at < SI * SJ) tile[buf][0][at] = next[e];
        }
        __syncthreads();
        if (k + 1 < k1 + R) fetch(k + 1);
        float sj = 0.0f;
#pragma unroll
        for (int b = 0; b <= 2 * R; b++) {
            float si = 0.0f;
#pragma unroll
            for (int a = 0; a <= 2 * R; a++) si += tile[buf][tj + b][ti + a];
            sj += si;
        }
#pragma unroll
        for (int d = 0; d < 2 * R; d++) win[d] = win[d + 1];
        win[2 * R] = sj;
        if (k - R >= k0 && i < m && j < n) {
            float acc = 0.0f;
#pragma unroll
            for (int d = 0; d <= 2 * R; d++) acc += win[d];
            out[ch * sz + i + (int64_t)j * m + (k - R) * mn] = acc;
        }
    }
}

struct DescPoint {
    float v[12];
    int64_t q[12];
};

__device__ __forceinline__ void gather_desc(const float* __restrict__ d, int64_t p, int m, int n, int o, int qs,
                                            DescPoint& dp) {
    const int64_t sz = (int64_t)m * n * o;
    const int i = (int)(p % m), j = (int)((p / m) % n), k = (int)(p / ((int64_t)m * n));
#pragma unroll
    for (int l = 0; l < 12; l++) {
        const int ii = i + s_sy[l] * qs, jj = j + s_sx[l] * qs, kk = k + s_sz[l] * qs;
        dp.q[l] = inside(ii, jj, kk, m, n, o) ? ii + (int64_t)jj * m + (int64_t)kk * m * n : p;
        dp.v[l] = d[(l >> 1) * sz + dp.q[l]];
    }
}

// soft descriptor s (12 x sz) from the box-filtered channels d (6 x sz)
__global__ void k_soft_desc(const float* __restrict__ d, float* __restrict__ s, int m, int n, int o, int qs) {
    const int64_t sz = (int64_t)m * n * o;
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= sz) return;
    DescPoint dp;
    gather_desc(d, p, m, n, o, qs, dp);
    float mn = dp.v[0];
#pragma unroll
    for (int l = 1; l < 12; l++) mn = fminf(mn, dp.v[l]);
    float sum = 0.0f;
#pragma unroll
    for (int l = 0; l < 12; l++) sum += dp.v[l] - mn;
    const float noise = fmaxf(sum / 12.0f, 1e-6f);
#pragma unroll
    for (int l = 0; l < 12; l++) s[l * sz + p] = 6.0f * expf(-(dp.v[l] - mn) / noise);
}

// adjoint of k_soft_desc: sbar (12 x sz) -> dbar (6 x sz), accumulated with atomics
// (the twelve gathers of a voxel hit neighbours that other voxels also gather)
__global__ void k_soft_desc_adj(const float* __restrict__ d, const float* __restrict__ sbar, float* __restrict__ dbar,
                                int m, int n, int o, int qs) {
    const int64_t sz = (int64_t)m * n * o;
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= sz) return;
    DescPoint dp;
    gather_desc(d, p, m, n, o, qs, dp);
    float mn = dp.v[0];
    int am = 0;
#pragma unroll
    for (int l = 1; l < 12; l++)
        if (dp.v[l] < mn) { mn = dp.v[l]; am = l; }
    float sum = 0.0f;
#pragma unroll
    for (int l = 0; l < 12; l++) sum += dp.v[l] - mn;
    const bool clamped = sum / 12.0f < 1e-6f;
    const float noise = fmaxf(sum / 12.0f, 1e-6f);
    // x_l = (v_l - mn)/noise, noise = sum_l (v_l - mn)/12 unless clamped, mn = v_am
    float vb[12], nbar = 0.0f;
#pragma unroll
    for (int l = 0; l < 12; l++) {
        const float x = (dp.v[l] - mn) / noise;
        vb[l] = -6.0f * expf(-x) * sbar[l * sz + p];  // dL/dx_l
        nbar -= vb[l] * x / noise;
    }
    float tot = 0.0f;
#pragma unroll
    for (int l = 0; l < 12; l++) {
        vb[l] = vb[l] / noise + (clamped ? 0.0f : nbar / 12.0f);
        tot += vb[l];
    }
#pragma unroll
    for (int l = 0; l < 12; l++) atomicAdd(dbar + (l >> 1) * sz + dp.q[l], l == am ? vb[l] - tot : vb[l]);
}

// adjoint of k_soft_sqdiff: wbar (6 x sz) -> imbar (accumulated)
__global__ void k_soft_sqdiff_adj(const float* __restrict__ im, const float* __restrict__ wbar,
                                  float* __restrict__ imbar, int m, int n, int o, int qs) {
    const int64_t sz = (int64_t)m * n * o;
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= sz) return;
    const int i = (int)(p % m), j = (int)((p / m) % n), k = (int)(p / ((int64_t)m * n));
    const float c = im[p];
    float self = 0.0f;
#pragma unroll
    for (int l = 0; l < 6; l++) {
        const int ii = i + s_dy[l] * qs, jj = j + s_dx[l] * qs, kk = k + s_dz[l] * qs;
        if (inside(ii, jj, kk, m, n, o)) {
            const int64_t t = ii + (int64_t)jj * m + (int64_t)kk * m * n;
            const float gr = 2.0f * (im[t] - c) * wbar[l * sz + p];
            atomicAdd(imbar + t, gr);
            self -= gr;
        }
    }
    atomicAdd(imbar + p, self);
}

// ---------------------------------------------------------------------------
// Cost

// 4-byte asynchronous global->shared copies (cp.async, sm_80+): a thread issues all
// its staging copies back to back and waits once, instead of one load latency per
// element.  The caller waits with cp_async_wait_all() and then a block barrier.
__device__ __forceinline__ void cp_async4(float* smem_dst, const float* gsrc) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

struct SoftGeom {
    int m, n, o, g, hw, q, len, len3, m1, n1, o1, S, nx, nsamp;
    float alpha1, eps;
};

__device__ __forceinline__ float phi_grad(float x, float eps) { return x * rsqrtf(x * x + eps * eps); }

// C[c][l]: one CTA per node, the node's fixed samples in shared memory, threads over labels
__global__ void k_soft_cost(const float* __restrict__ sF, const float* __restrict__ sM, float* __restrict__ cost,
                            SoftGeom G) {
    extern __shared__ float fs[];  // [nsamp][12]
    const int node = blockIdx.x;
    const int y = node % G.m1, x = (node / G.m1) % G.n1, z = node / (G.m1 * G.n1);
    const int64_t mn = (int64_t)G.m * G.n, sz = mn * G.o;
    for (int e = threadIdx.x; e < G.nsamp * 12; e += blockDim.x) {
        const int c = e % 12, s = e / 12;
        const int ii = s % G.g, jj = (s / G.g) % G.nx, kk = s / (G.g * G.nx);
        const int64_t p = (y * G.g + ii) + (int64_t)(x * G.g + jj * G.S) * G.m + (int64_t)(z * G.g + kk * G.S) * mn;
        fs[e] = sF[c * sz + p];
    }
    __syncthreads();
    for (int l = threadIdx.x; l < G.len3; l += blockDim.x) {
        const int dy = (l % G.len - G.hw) * G.q, dx = ((l / G.len) % G.len - G.hw) * G.q,
                  dz = (l / (G.len * G.len) - G.hw) * G.q;
        float acc = 0.0f;
        int s = 0;
        for (int kk = 0; kk < G.nx; kk++) {
            const int qk = clampi(z * G.g + kk * G.S + dz, 0, G.o - 1);
            for (int jj = 0; jj < G.nx; jj++) {
                const int qj = clampi(x * G.g + jj * G.S + dx, 0, G.n - 1);
                for (int ii = 0; ii < G.g; ii++, s++) {
                    const int qi = clampi(y * G.g + ii + dy, 0, G.m - 1);
                    const float* mv = sM + qi + (int64_t)qj * G.m + (int64_t)qk * mn;
                    const float* fv = fs + s * 12;
#pragma unroll
                    for (int c = 0; c < 12; c++) {
                        const float dl = fv[c] - __ldg(mv + c * sz);
                        acc += sqrtf(dl * dl + G.eps * G.eps) - G.eps;
                    }
                }
            }
        }
        cost[(int64_t)node * G.len3 + l] = G.alpha1 * acc;
    }
}

// Adjoint of the cost w.r.t. the fixed descriptor (one CTA per node, one thread per
// (sample, channel); samples of different nodes are disjoint, so plain stores) and
// dot = sum(cbar * C) for the alpha gradient (C = alpha1 f, alpha1 ~ 1/alpha,
// dL/dalpha = -dot/alpha).
__global__ void k_soft_cost_adj_fixed(const float* __restrict__ sF, const float* __restrict__ sM,
                                      const float* __restrict__ cbar, const float* __restrict__ cost,
                                      float* __restrict__ sFbar, double* __restrict__ dot, SoftGeom G) {
    const int node = blockIdx.x;
    const int y = node % G.m1, x = (node / G.m1) % G.n1, z = node / (G.m1 * G.n1);
    const int64_t mn = (int64_t)G.m * G.n, sz = mn * G.o;
    const float* cb = cbar + (int64_t)node * G.len3;
    const float* cn = cost + (int64_t)node * G.len3;
    // The level is invariant to adding a constant to one node's costs, so the exact
    // cbar sums to zero over labels and sum(cbar * C) = sum(cbar * (C - mean C)); the
    // centred form keeps float32 rounding in cbar from being amplified by |mean C|.
    __shared__ double red[32];
    double csum = 0.0;
    for (int l = threadIdx.x; l < G.len3; l += blockDim.x) csum += (double)cn[l];
    for (int off = 16; off > 0; off >>= 1) csum += __shfl_xor_sync(0xffffffffu, csum, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = csum;
    __syncthreads();
    double cmean = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) cmean += red[w];
    cmean /= (double)G.len3;
    double part = 0.0;
    for (int l = threadIdx.x; l < G.len3; l += blockDim.x) part += (double)cb[l] * ((double)cn[l] - cmean);
    for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
    if ((threadIdx.x & 31) == 0) atomicAdd(dot, part);
    for (int e = threadIdx.x; e < G.nsamp * 12; e += blockDim.x) {
        const int c = e % 12, s = e / 12;
        const int ii = s % G.g, jj = (s / G.g) % G.nx, kk = s / (G.g * G.nx);
        const int pi = y * G.g + ii, pj = x * G.g + jj * G.S, pk = z * G.g + kk * G.S;
        const int64_t p = pi + (int64_t)pj * G.m + (int64_t)pk * mn;
        const float f = sF[c * sz + p];
        const float* mc = sM + c * sz;
        float gF = 0.0f;
        int l = 0;
        for (int lz = 0; lz < G.len; lz++) {
            const int qk = clampi(pk + (lz - G.hw) * G.q, 0, G.o - 1);
            for (int lx = 0; lx < G.len; lx++) {
                const int qj = clampi(pj + (lx - G.hw) * G.q, 0, G.n - 1);
                const float* row = mc + (int64_t)qj * G.m + (int64_t)qk * mn;
                for (int ly = 0; ly < G.len; ly++, l++) {
                    const int qi = clampi(pi + (ly - G.hw) * G.q, 0, G.m - 1);
                    gF += cb[l] * phi_grad(f - row[qi], G.eps);
                }
            }
        }
        sFbar[c * sz + p] = G.alpha1 * gF;
    }
}

// Range of p along one axis with clamp(p + d, 0, dim-1) == qv, intersected with the
// node-covered extent [0, cover) (empty when lo > hi).
__device__ __forceinline__ void preimage(int qv, int d, int dim, int cover, int& lo, int& hi) {
    lo = qv == 0 ? 0 : qv - d;
    hi = qv == dim - 1 ? dim - 1 : qv - d;
    if (qv == 0) hi = min(hi, -d);
    if (qv == dim - 1) lo = max(lo, dim - 1 - d);
    lo = max(lo, 0);
    hi = min(hi, cover - 1);
}

// Adjoint of the cost w.r.t. the moving descriptor as a gather (no atomics): one
// thread per moving voxel q (all 12 channels), over the labels and the samples p
// whose clamped displaced position is q.
__global__ void k_soft_cost_adj_moving(const float* __restrict__ sF, const float* __restrict__ sM,
                                       const float* __restrict__ cbar, float* __restrict__ sMbar, SoftGeom G) {
    const int64_t mn = (int64_t)G.m * G.n, sz = mn * G.o;
    const int64_t qv = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (qv >= sz) return;
    const int qi = (int)(qv % G.m), qj = (int)((qv / G.m) % G.n), qk = (int)(qv / mn);
    float mq[12], acc[12];
#pragma unroll
    for (int c = 0; c < 12; c++) {
        mq[c] = sM[c * sz + qv];
        acc[c] = 0.0f;
    }
    const int ci = G.m1 * G.g, cj = G.n1 * G.g, ck = G.o1 * G.g;
    for (int lz = 0; lz < G.len; lz++) {
        int k0, k1;
        preimage(qk, (lz - G.hw) * G.q, G.o, ck, k0, k1);
        for (int pk = k0; pk <= k1; pk++) {
            if ((pk % G.g) % G.S) continue;
            for (int lx = 0; lx < G.len; lx++) {
                int j0, j1;
                preimage(qj, (lx - G.hw) * G.q, G.n, cj, j0, j1);
                for (int pj = j0; pj <= j1; pj++) {
                    if ((pj % G.g) % G.S) continue;
                    const int nbase = (pj / G.g) * G.m1 + (pk / G.g) * G.m1 * G.n1;
                    const int lbase = lx * G.len + lz * G.len * G.len;
                    for (int ly = 0; ly < G.len; ly++) {
                        int i0, i1;
                        preimage(qi, (ly - G.hw) * G.q, G.m, ci, i0, i1);
                        for (int pi = i0; pi <= i1; pi++) {
                            const float cb = __ldg(cbar + (int64_t)(nbase + pi / G.g) * G.len3 + lbase + ly);
                            const float* fp = sF + pi + (int64_t)pj * G.m + (int64_t)pk * mn;
#pragma unroll
                            for (int c = 0; c < 12; c++) acc[c] += cb * phi_grad(__ldg(fp + c * sz) - mq[c], G.eps);
                        }
                    }
                }
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 12; c++) sMbar[c * sz + qv] = -G.alpha1 * acc[c];
}

// The same gather with the grid spacing, label width and quantisation fixed at
// compile time (the row-form level shapes): the label and sample loops unroll
// and the node and lattice arithmetic uses constants.
template <int G_, int LEN_, int Q_>
__global__ void __launch_bounds__(128) k_soft_cost_adj_moving_t(const float* __restrict__ sF,
                                                               const float* __restrict__ sM,
                                                               const float* __restrict__ cbar,
                                                               float* __restrict__ sMbar, SoftGeom G) {
    constexpr int S = G_ > 4 ? 2 : 1, HW = (LEN_ - 1) / 2, LEN3 = LEN_ * LEN_ * LEN_;
    const int64_t mn = (int64_t)G.m * G.n, sz = mn * G.o;
    const int64_t qv = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (qv >= sz) return;
    const int qi = (int)(qv % G.m), qj = (int)((qv / G.m) % G.n), qk = (int)(qv / mn);
    float mq[12], acc[12];
#pragma unroll
    for (int c = 0; c < 12; c++) {
        mq[c] = sM[c * sz + qv];
        acc[c] = 0.0f;
    }
    const int ci = G.m1 * G_, cj = G.n1 * G_, ck = G.o1 * G_;
    const float eps = G.eps;
    constexpr int R = HW * Q_;
    // away from the y faces every label has exactly one y preimage, qi - dy, inside
    // the node-covered extent: a straight-line path whose loads can be issued together
    const bool yint = qi >= (R > 1 ? R : 1) && qi <= min(ci - 1 - R, G.m - 2);
    for (int lz = 0; lz < LEN_; lz++) {
        int k0, k1;
        preimage(qk, (lz - HW) * Q_, G.o, ck, k0, k1);
        for (int pk = k0; pk <= k1; pk++) {
            if (S > 1 && (pk % G_) % S) continue;
            for (int lx = 0; lx < LEN_; lx++) {
                int j0, j1;
                preimage(qj, (lx - HW) * Q_, G.n, cj, j0, j1);
                for (int pj = j0; pj <= j1; pj++) {
                    if (S > 1 && (pj % G_) % S) continue;
                    const int nbase = (pj / G_) * G.m1 + (pk / G_) * G.m1 * G.n1;
                    const float* cbl = cbar + (int64_t)(lx * LEN_ + lz * LEN_ * LEN_);
                    const float* fpk = sF + (int64_t)pj * G.m + (int64_t)pk * mn;
                    if (yint) {
                        float cbv[LEN_];
#pragma unroll
                        for (int ly = 0; ly < LEN_; ly++) {
                            const int pi = qi - (ly - HW) * Q_;
                            cbv[ly] = __ldg(cbl + (int64_t)(nbase + pi / G_) * LEN3 + ly);
                        }
#pragma unroll
                        for (int ly = 0; ly < LEN_; ly++) {
                            const float* fp = fpk + qi - (ly - HW) * Q_;
#pragma unroll
                            for (int c = 0; c < 12; c++)
                                acc[c] += cbv[ly] * phi_grad(__ldg(fp + c * sz) - mq[c], eps);
                        }
                    } else {
                        for (int ly = 0; ly < LEN_; ly++) {
                            int i0, i1;
                            preimage(qi, (ly - HW) * Q_, G.m, ci, i0, i1);
                            for (int pi = i0; pi <= i1; pi++) {
                                const float cb = __ldg(cbl + (int64_t)(nbase + pi / G_) * LEN3 + ly);
                                const float* fp = fpk + pi;
#pragma unroll
                                for (int c = 0; c < 12; c++)
                                    acc[c] += cb * phi_grad(__ldg(fp + c * sz) - mq[c], eps);
                            }
                        }
                    }
                }
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 12; c++) sMbar[c * sz + qv] = -G.alpha1 * acc[c];
}

template <int G_, int LEN_, int Q_>
static cudaError_t run_adj_moving_t(const SoftGeom& G, const float* sF, const float* sM, const float* cbar,
                                    float* sMbar, cudaStream_t st) {
    const int64_t sz = (int64_t)G.m * G.n * G.o;
    k_soft_cost_adj_moving_t<G_, LEN_, Q_><<<(unsigned)((sz + 127) / 128), 128, 0, st>>>(sF, sM, cbar, sMbar, G);
    return cudaSuccess;
}

// ---------------------------------------------------------------------------
// Halo form of the cost and its adjoint.  The moving descriptor values that one
// node's samples reach under every label form one box (the node block grown by
// hw*q on each side, clipped to the volume: the reference's clamp-to-edge maps
// every displaced position into it).  The box of a group of channels is staged
// in shared memory with coalesced loads, so the len^3 x samples x channels terms
// read shared memory only.  For nodes whose box is not clipped the displaced
// position is a per-sample base plus a per-label offset; clipped (border) nodes
// clamp per axis.

struct Halo {
    int y0, x0, z0, HY, HX, HZ, H3;
    bool interior;
};

__device__ __forceinline__ Halo node_halo(const SoftGeom& G, int y, int x, int z) {
    const int R = G.hw * G.q;
    const int ylo = y * G.g - R, yhi = y * G.g + G.g - 1 + R;
    const int xlo = x * G.g - R, xhi = x * G.g + G.g - 1 + R;
    const int zlo = z * G.g - R, zhi = z * G.g + G.g - 1 + R;
    Halo h;
    h.y0 = max(0, ylo); h.HY = min(G.m - 1, yhi) - h.y0 + 1;
    h.x0 = max(0, xlo); h.HX = min(G.n - 1, xhi) - h.x0 + 1;
    h.z0 = max(0, zlo); h.HZ = min(G.o - 1, zhi) - h.z0 + 1;
    h.H3 = h.HY * h.HX * h.HZ;
    h.interior = ylo >= 0 && yhi < G.m && xlo >= 0 && xhi < G.n && zlo >= 0 && zhi < G.o;
    return h;
}

__device__ __forceinline__ int label_dy(const SoftGeom& G, int l) { return (l % G.len - G.hw) * G.q; }
__device__ __forceinline__ int label_dx(const SoftGeom& G, int l) { return ((l / G.len) % G.len - G.hw) * G.q; }
__device__ __forceinline__ int label_dz(const SoftGeom& G, int l) { return (l / (G.len * G.len) - G.hw) * G.q; }

// sample s of node (y,x,z): voxel coordinates
__device__ __forceinline__ void sample_pos(const SoftGeom& G, int y, int x, int z, int s, int& py, int& px, int& pz) {
    py = y * G.g + s % G.g;
    px = x * G.g + ((s / G.g) % G.nx) * G.S;
    pz = z * G.g + (s / (G.g * G.nx)) * G.S;
}

__device__ __forceinline__ int halo_clamped(const SoftGeom& G, const Halo& h, int py, int px, int pz, int l) {
    const int a = clampi(py + label_dy(G, l), 0, G.m - 1) - h.y0;
    const int b = clampi(px + label_dx(G, l), 0, G.n - 1) - h.x0;
    const int c = clampi(pz + label_dz(G, l), 0, G.o - 1) - h.z0;
    return a + h.HY * (b + h.HX * c);
}

// Stage channels [c0, c0+CG) of the node's halo (coalesced along y).
__device__ __forceinline__ void stage_halo(const SoftGeom& G, const Halo& h, const float* __restrict__ vol, int c0,
                                           int CG, float* hv) {
    const int64_t mn = (int64_t)G.m * G.n, sz = mn * G.o;
    for (int e = threadIdx.x; e < CG * h.H3; e += blockDim.x) {
        const int c = e / h.H3, r = e % h.H3;
        const int a = r % h.HY, b = (r / h.HY) % h.HX, cc = r / (h.HY * h.HX);
        hv[e] = vol[(int64_t)(c0 + c) * sz + (h.y0 + a) + (int64_t)(h.x0 + b) * G.m + (int64_t)(h.z0 + cc) * mn];
    }
}

constexpr int kHaloLPT = 3;  // labels per thread in the halo cost kernel (len^3 <= 3 * 512)

// C[node][l] from shared-memory halos; threads own labels, CG channels per stage.
__global__ void __launch_bounds__(512) k_soft_cost_halo(const float* __restrict__ sF, const float* __restrict__ sM,
                                                        float* __restrict__ cost, SoftGeom G, int CG, int H3max) {
    extern __shared__ float sh[];
    const int node = blockIdx.x;
    const int y = node % G.m1, x = (node / G.m1) % G.n1, z = node / (G.m1 * G.n1);
    const Halo h = node_halo(G, y, x, z);
    const int64_t mn = (int64_t)G.m * G.n, sz = mn * G.o;
    float* hv = sh;                                             // [CG][H3]
    float* fsm = sh + (size_t)CG * H3max;                       // [CG][nsamp]
    int* loff = reinterpret_cast<int*>(fsm + CG * G.nsamp);     // [len3]
    int* sb = loff + G.len3;                                    // [nsamp]
    for (int l = threadIdx.x; l < G.len3; l += blockDim.x)
        loff[l] = label_dy(G, l) + h.HY * (label_dx(G, l) + h.HX * label_dz(G, l));
    for (int s = threadIdx.x; s < G.nsamp; s += blockDim.x) {
        int py, px, pz;
        sample_pos(G, y, x, z, s, py, px, pz);
        sb[s] = (py - h.y0) + h.HY * ((px - h.x0) + h.HX * (pz - h.z0));
    }
    float acc[kHaloLPT];
#pragma unroll
    for (int k = 0; k < kHaloLPT; k++) acc[k] = 0.0f;
    const float eps2 = G.eps * G.eps;
    for (int c0 = 0; c0 < 12; c0 += CG) {
        __syncthreads();
        stage_halo(G, h, sM, c0, CG, hv);
        for (int e = threadIdx.x; e < CG * G.nsamp; e += blockDim.x) {
            const int c = e / G.nsamp, s = e % G.nsamp;
            int py, px, pz;
            sample_pos(G, y, x, z, s, py, px, pz);
            fsm[e] = sF[(int64_t)(c0 + c) * sz + py + (int64_t)px * G.m + (int64_t)pz * mn];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kHaloLPT; k++) {
            const int l = threadIdx.x + k * blockDim.x;
            if (l >= G.len3) break;
            float a = acc[k];
            if (h.interior) {
                const int lo = loff[l];
                for (int s = 0; s < G.nsamp; s++) {
                    const int base = sb[s] + lo;
                    for (int c = 0; c < CG; c++) {
                        const float d = fsm[c * G.nsamp + s] - hv[c * h.H3 + base];
                        const float x2 = d * d + eps2;
                        a += x2 * rsqrtf(x2);
                    }
                }
            } else {
                for (int s = 0; s < G.nsamp; s++) {
                    int py, px, pz;
                    sample_pos(G, y, x, z, s, py, px, pz);
                    const int base = halo_clamped(G, h, py, px, pz, l);
                    for (int c = 0; c < CG; c++) {
                        const float d = fsm[c * G.nsamp + s] - hv[c * h.H3 + base];
                        const float x2 = d * d + eps2;
                        a += x2 * rsqrtf(x2);
                    }
                }
            }
            acc[k] = a;
        }
    }
#pragma unroll
    for (int k = 0; k < kHaloLPT; k++) {
        const int l = threadIdx.x + k * blockDim.x;
        if (l < G.len3) cost[(int64_t)node * G.len3 + l] = G.alpha1 * (acc[k] - (float)(12 * G.nsamp) * G.eps);
    }
}

// Adjoint of the cost from shared-memory halos: threads own (channel, sample)
// items and walk the labels; each term's gradient goes to the fixed sample (a
// register) and, through a shared-memory atomic, to the halo position it read;
// the halo gradients are then added to the moving descriptor's gradient
// (neighbouring nodes' halos overlap).  Also dot = sum(cbar * C) for alpha.
__global__ void __launch_bounds__(256) k_soft_cost_adj_halo(const float* __restrict__ sF,
                                                            const float* __restrict__ sM,
                                                            const float* __restrict__ cbar,
                                                            const float* __restrict__ cost, float* __restrict__ sFbar,
                                                            float* __restrict__ sMbar, double* __restrict__ dot,
                                                            SoftGeom G, int CG, int H3max) {
    extern __shared__ float sh[];
    __shared__ double red[32];
    const int node = blockIdx.x;
    const int y = node % G.m1, x = (node / G.m1) % G.n1, z = node / (G.m1 * G.n1);
    const Halo h = node_halo(G, y, x, z);
    const int64_t mn = (int64_t)G.m * G.n, sz = mn * G.o;
    float* hv = sh;                                        // [CG][H3]
    float* hg = sh + (size_t)CG * H3max;                   // [CG][H3]
    float* cb = hg + (size_t)CG * H3max;                   // [len3]
    int* loff = reinterpret_cast<int*>(cb + G.len3);       // [len3]
    int* sb = loff + G.len3;                               // [nsamp]
    const float* cbn = cbar + (int64_t)node * G.len3;
    const float* cn = cost + (int64_t)node * G.len3;
    // alpha: centred dot product (the exact cbar sums to zero over labels)
    double csum = 0.0;
    for (int l = threadIdx.x; l < G.len3; l += blockDim.x) {
        csum += (double)cn[l];
        cb[l] = cbn[l];
        loff[l] = label_dy(G, l) + h.HY * (label_dx(G, l) + h.HX * label_dz(G, l));
    }
    for (int off = 16; off > 0; off >>= 1) csum += __shfl_xor_sync(0xffffffffu, csum, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = csum;
    for (int s = threadIdx.x; s < G.nsamp; s += blockDim.x) {
        int py, px, pz;
        sample_pos(G, y, x, z, s, py, px, pz);
        sb[s] = (py - h.y0) + h.HY * ((px - h.x0) + h.HX * (pz - h.z0));
    }
    __syncthreads();
    double cmean = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) cmean += red[w];
    cmean /= (double)G.len3;
    double part = 0.0;
    for (int l = threadIdx.x; l < G.len3; l += blockDim.x) part += (double)cb[l] * ((double)cn[l] - cmean);
    for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
    if ((threadIdx.x & 31) == 0) atomicAdd(dot, part);
    const float eps2 = G.eps * G.eps;
    for (int c0 = 0; c0 < 12; c0 += CG) {
        __syncthreads();
        stage_halo(G, h, sM, c0, CG, hv);
        for (int e = threadIdx.x; e < CG * h.H3; e += blockDim.x) hg[e] = 0.0f;
        __syncthreads();
        for (int item = threadIdx.x; item < CG * G.nsamp; item += blockDim.x) {
            const int c = item / G.nsamp, s = item % G.nsamp;
            int py, px, pz;
            sample_pos(G, y, x, z, s, py, px, pz);
            const int64_t p = py + (int64_t)px * G.m + (int64_t)pz * mn;
            const float f = sF[(int64_t)(c0 + c) * sz + p];
            const float* hvc = hv + c * h.H3;
            float* hgc = hg + c * h.H3;
            float gF = 0.0f;
            if (h.interior) {
                const int base = sb[s];
                for (int l = 0; l < G.len3; l++) {
                    const int idx = base + loff[l];
                    const float d = f - hvc[idx];
                    const float gr = cb[l] * d * rsqrtf(d * d + eps2);
                    gF += gr;
                    atomicAdd(hgc + idx, -gr);
                }
            } else {
                for (int l = 0; l < G.len3; l++) {
                    const int idx = halo_clamped(G, h, py, px, pz, l);
                    const float d = f - hvc[idx];
                    const float gr = cb[l] * d * rsqrtf(d * d + eps2);
                    gF += gr;
                    atomicAdd(hgc + idx, -gr);
                }
            }
            sFbar[(int64_t)(c0 + c) * sz + p] = G.alpha1 * gF;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < CG * h.H3; e += blockDim.x) {
            const float v = hg[e];
            if (v == 0.0f) continue;
            const int c = e / h.H3, r = e % h.H3;
            const int a = r % h.HY, b = (r / h.HY) % h.HX, cc = r / (h.HY * h.HX);
            atomicAdd(sMbar + (int64_t)(c0 + c) * sz + (h.y0 + a) + (int64_t)(h.x0 + b) * G.m +
                          (int64_t)(h.z0 + cc) * mn,
                      G.alpha1 * v);
        }
    }
}

// Column form, for compile-time grid spacing, label width
// and quantisation.  Each node stages a full NA^3 box (NA = g + 2hw*q) of the
// moving descriptor whose entry (a, b, c) holds the voxel at the clamped
// coordinates (y*g - hw*q + a, ...): the reference's clamp-to-edge is baked into
// the staged data, so every displaced sample position is plain box arithmetic.  A
// thread owns one sampled column of the node (fixed x and z sample offsets, its g
// samples along y) and one (lx, lz) label pair, and walks the len y-labels: the
// displaced y positions i + ly*q of its g samples are NA consecutive box entries,
// loaded once per channel.

// Block size (whole warps, 128..256) that leaves the fewest idle item slots.
constexpr int balanced_block(int items) {
    int best = 256, waste = (items + 255) / 256 * 256 - items;
    for (int b = 224; b >= 128; b -= 32) {
        const int w = (items + b - 1) / b * b - items;
        if (w * 256 < waste * b) { best = b; waste = w; }
    }
    return best;
}

template <int G_, int LEN_, int Q_>
struct ColGeom {
    static constexpr int GS = G_, HW = (LEN_ - 1) / 2, R = HW * Q_, NA = G_ + 2 * R, NA3 = NA * NA * NA;
    static constexpr int S = G_ > 4 ? 2 : 1, NX = (G_ + S - 1) / S, NSAMP = NX * NX * G_;
    static constexpr int ITEMS = NX * NX * LEN_ * LEN_, LEN3 = LEN_ * LEN_ * LEN_;
    // forward items: (channel half, column, lx, lz)
    static constexpr int FWD_ITEMS = 2 * ITEMS, FWD_BLOCK = balanced_block(FWD_ITEMS);
};

// Stage channels [c0, c0+CG) of the node's clamped box and, when fs is given, all
// 12 channels of its fixed samples.
template <class CGm>
__device__ __forceinline__ void stage_box(const SoftGeom& G, int y, int x, int z, const float* __restrict__ sM, int c0,
                                          int CG, float* hv, const float* __restrict__ sF, float* fs) {
    const int64_t mn = (int64_t)G.m * G.n, sz = mn * G.o;
    const int yb = y * G.g - CGm::R, xb = x * G.g - CGm::R, zb = z * G.g - CGm::R;
    // a warp stages 32/NA box rows at a time: lane -> (row within the group, y offset)
    constexpr int RPW = 32 / CGm::NA;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int sub = lane / CGm::NA, a = lane - sub * CGm::NA;
    const int ya = clampi(yb + a, 0, G.m - 1);
    const int nrows = CG * CGm::NA * CGm::NA;
    if (sub < RPW)
        for (int r = warp * RPW + sub; r < nrows; r += nw * RPW) {
            const int b = r % CGm::NA, t = r / CGm::NA, cc = t % CGm::NA, c = t / CGm::NA;
            cp_async4(hv + r * CGm::NA + a, sM + (int64_t)(c0 + c) * sz + ya + (int64_t)clampi(xb + b, 0, G.n - 1) * G.m +
                                                (int64_t)clampi(zb + cc, 0, G.o - 1) * mn);
        }
    if (fs)
        for (int e = threadIdx.x; e < 12 * CGm::NSAMP; e += blockDim.x) {
            const int c = e / CGm::NSAMP, s = e % CGm::NSAMP;
            const int py = y * CGm::GS + s % CGm::GS, px = x * CGm::GS + ((s / CGm::GS) % CGm::NX) * CGm::S,
                      pz = z * CGm::GS + (s / (CGm::GS * CGm::NX)) * CGm::S;
            cp_async4(fs + e, sF + (int64_t)c * sz + py + (int64_t)px * G.m + (int64_t)pz * mn);
        }
    cp_async_wait_all();
}

template <int G_, int LEN_, int Q_>
__global__ void __launch_bounds__(ColGeom<G_, LEN_, Q_>::FWD_BLOCK, 4)
    k_soft_cost_col(const float* __restrict__ sF, const float* __restrict__ sM, float* __restrict__ cost, SoftGeom G) {
    using CGm = ColGeom<G_, LEN_, Q_>;
    extern __shared__ float sh[];
    const int node = blockIdx.x;
    const int y = node % G.m1, x = (node / G.m1) % G.n1, z = node / (G.m1 * G.n1);
    float* hv = sh;                      // [12][NA3]
    float* fs = sh + 12 * CGm::NA3;      // [12][NSAMP]
    float* acc = fs + 12 * CGm::NSAMP;   // [LEN3]
    stage_box<CGm>(G, y, x, z, sM, 0, 12, hv, sF, fs);
    for (int l = threadIdx.x; l < CGm::LEN3; l += blockDim.x) acc[l] = 0.0f;
    __syncthreads();
    const float eps2 = G.eps * G.eps;
    // items are (column, lab, channel half) with the column fastest: the NX^2 = 16
    // columns of one (lab, half) are the 16 lanes of a half-warp (the block is a
    // multiple of 16 threads), whose label sums are reduced with shuffles before
    // one shared-memory add per label
    static_assert(CGm::NX * CGm::NX == 16, "column kernels assume 16 sampled columns per node");
    for (int base = 0; base < CGm::FWD_ITEMS; base += blockDim.x) {
        const int item = base + threadIdx.x;
        const bool valid = item < CGm::FWD_ITEMS;
        const int it = valid ? item : 0;
        const int col = it % 16, lab = (it / 16) % (LEN_ * LEN_);
        const int half = it / CGm::ITEMS;
        const int jj = col % CGm::NX, kk = col / CGm::NX, lx = lab % LEN_, lz = lab / LEN_;
        const int plane = CGm::NA * ((jj * CGm::S + lx * Q_) + CGm::NA * (kk * CGm::S + lz * Q_));
        float sums[LEN_][2];
#pragma unroll
        for (int ly = 0; ly < LEN_; ly++) sums[ly][0] = sums[ly][1] = 0.0f;
        if (valid)
            for (int c = 6 * half; c < 6 * half + 6; c++) {
                const float* hvc = hv + c * CGm::NA3 + plane;
                const float* fsc = fs + c * CGm::NSAMP + G_ * col;
                float v[CGm::NA], f[G_];
#pragma unroll
                for (int a = 0; a < CGm::NA; a++) v[a] = hvc[a];
#pragma unroll
                for (int i = 0; i < G_; i++) f[i] = fsc[i];
#pragma unroll
                for (int ly = 0; ly < LEN_; ly++)
#pragma unroll
                    for (int i = 0; i < G_; i++) {
                        const float d = f[i] - v[i + ly * Q_];
                        const float x2 = d * d + eps2;
                        sums[ly][i & 1] += x2 * rsqrtf(x2);
                    }
            }
#pragma unroll
        for (int ly = 0; ly < LEN_; ly++) {
            float v = sums[ly][0] + sums[ly][1];
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
            if (valid && col == 0) atomicAdd(acc + ly + LEN_ * lab, v);
        }
    }
    __syncthreads();
    for (int l = threadIdx.x; l < CGm::LEN3; l += blockDim.x)
        cost[(int64_t)node * CGm::LEN3 + l] = G.alpha1 * (acc[l] - (float)(12 * CGm::NSAMP) * G.eps);
}

// Two floats in a register pair: one instruction does both lanes' operation, each
// rounded as the scalar one.
__device__ __forceinline__ uint64_t f2_pack(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_split(uint64_t v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// Adjoint of the column form.  A CTA takes one node's half of the channels, a warp one
// pair of channels (two floats per register pair, as they lie in shared memory), a lane
// one of the 16 sampled columns; the two half-warps take two label columns (lx, lz) whose
// box rows (jj + lx, kk + lz) cannot meet: lx or lz four apart.  So a row's gradient is
// added to shared memory by one lane at a time with plain loads and stores, and the fixed
// samples with their gradients stay in the lane's registers throughout.
// Bound by the reciprocal square roots, 16 a clock and SM: at 160x160x192, 343 labels,
// 20.2 G of them take 4.4 ms (0.78 ms at 96x80x112); 57 % of that rate is reached with the
// 12 warps an SM has room for.  Shared-memory float adds, a compare-and-swap loop each and
// 10 of them per 28 terms, took more than the terms: 11.2 ms (2.00 ms) before, 6.9 ms
// (1.22 ms) now.
template <int LEN_, int Q_>
struct AdjGeom {
    static constexpr int GS = 4, R = (LEN_ - 1) / 2 * Q_, NA = GS + 2 * R, LEN3 = LEN_ * LEN_ * LEN_;
    static_assert(NA % 2 == 0 && Q_ == 1, "rows are read as 16-byte pairs of entries");
    // pitches in 16-byte units (two entries): a phase of a 16-byte access is eight lanes,
    // rows jj = 0..3 of planes kk and kk + 1, which must fall into eight different units
    static constexpr int RU = NA / 2 % 8 == 4 ? NA / 2 + 1 : NA / 2;
    static constexpr int ODD = RU % 2;  // odd: the four rows leave a gap of four; even: of one
    static constexpr int PU = ODD ? (NA * RU + 3) / 8 * 8 + 4 : NA * RU + 1 - NA * RU % 2;
    static constexpr int CU = NA * PU;  // units of a channel pair
    static constexpr int WP = (LEN_ + 3) / 4 * 4;
    // label columns taken two at a time: lx in [0, PX) with lx + 4; the rest by lz
    static constexpr int PX = LEN_ < 8 ? LEN_ - 4 : 4, NR = LEN_ - 2 * PX;
    static constexpr int STEPS = PX * LEN_ + NR * (PX + NR);
    static constexpr size_t SMEM = 16 * (size_t)(6 * CU) + 4 * (size_t)(LEN_ * LEN_ * WP);
};

template <int LEN_, int Q_>
__global__ void __launch_bounds__(96)
    k_soft_cost_adj_col(const float* __restrict__ sF, const float* __restrict__ sM, const float* __restrict__ cbar,
                        const float* __restrict__ cost, float* __restrict__ sFbar, float* __restrict__ sMbar,
                        double* __restrict__ dot, SoftGeom G) {
    using A = AdjGeom<LEN_, Q_>;
    extern __shared__ __align__(16) float sh[];
    __shared__ double red[3];
    __shared__ int64_t ox[A::NA], oz[A::NA];  // offsets of the box's clamped x and z
    const int node = blockIdx.x >> 1, half = blockIdx.x & 1;
    const int y = node % G.m1, x = (node / G.m1) % G.n1, z = node / (G.m1 * G.n1);
    const int64_t mn = (int64_t)G.m * G.n, sz = mn * G.o;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c0 = 6 * half + 2 * warp;  // this warp's channels c0, c0 + 1
    float* hv = sh + 4 * A::CU * warp;   // [NA][PU], [NA][RU] of two entries, [2] channels
    float* hg = hv + 4 * A::CU * 3;
    float* cb = sh + 4 * A::CU * 6;      // [LEN^2][WP]
    const int yb = y * 4 - A::R, xb = x * 4 - A::R, zb = z * 4 - A::R;
    // a warp moves 32/NA box rows at a time: lane -> (row within the group, y offset)
    constexpr int RPW = 32 / A::NA;
    const int sub = lane / A::NA, la = lane - sub * A::NA;
    const int64_t ya = clampi(yb + la, 0, G.m - 1) + (int64_t)c0 * sz;
    if (threadIdx.x < A::NA) ox[threadIdx.x] = (int64_t)clampi(xb + threadIdx.x, 0, G.n - 1) * G.m;
    else if (threadIdx.x >= 32 && threadIdx.x < 32 + A::NA)
        oz[threadIdx.x - 32] = (int64_t)clampi(zb + threadIdx.x - 32, 0, G.o - 1) * mn;
    __syncthreads();
    if (sub < RPW)
#pragma unroll 4
        for (int b = sub, cc = 0; cc < A::NA;) {
            const float* g = sM + ya + ox[b] + oz[cc];
            float* d = hv + 4 * (cc * A::PU + b * A::RU) + 2 * la;
            cp_async4(d, g);
            cp_async4(d + 1, g + sz);
            if ((b += RPW) >= A::NA) {
                b -= A::NA;
                cc++;
            }
        }
    for (int e = lane; e < A::CU; e += 32) reinterpret_cast<float4*>(hg)[e] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float* cbn = cbar + (int64_t)node * A::LEN3;
    const float* cn = cost + (int64_t)node * A::LEN3;
    double csum = 0.0;
    for (int l = threadIdx.x; l < A::LEN3; l += 96) {
        cb[(l / LEN_) * A::WP + l % LEN_] = cbn[l];
        if (half == 0) csum += (double)cn[l];
    }
    // alpha: centred dot product (the exact cbar sums to zero over labels)
    if (half == 0) {
        for (int off = 16; off > 0; off >>= 1) csum += __shfl_xor_sync(0xffffffffu, csum, off);
        if (lane == 0) red[warp] = csum;
    }
    // the lane's column: its fixed samples and their gradients
    const int col = lane & 15, hw = lane >> 4, jj = col & 3, kk = col >> 2;
    const int64_t fp = (int64_t)c0 * sz + y * 4 + (int64_t)(x * 4 + jj) * G.m + (int64_t)(z * 4 + kk) * mn;
    uint64_t f[4], gf[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        f[i] = f2_pack(sF[fp + i], sF[fp + i + sz]);
        gf[i] = 0;
    }
    cp_async_wait_all();
    __syncthreads();
    if (half == 0) {
        const double cmean = (red[0] + red[1] + red[2]) / (double)A::LEN3;
        double part = 0.0;
        for (int l = threadIdx.x; l < A::LEN3; l += 96)
            part += (double)cb[(l / LEN_) * A::WP + l % LEN_] * ((double)cn[l] - cmean);
        for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
        if (lane == 0) atomicAdd(dot, part);
    }
    const uint64_t eps2 = f2_pack(G.eps * G.eps, G.eps * G.eps), minus = f2_pack(-1.0f, -1.0f);
#pragma unroll 1
    for (int s = 0; s < A::STEPS; s++) {
        int lx, lz;
        bool valid = true;
        if (s < A::PX * LEN_) {
            lx = s / LEN_ + 4 * hw;
            lz = s % LEN_;
        } else {
            const int t = s - A::PX * LEN_, r = t / (A::PX + A::NR), u = t % (A::PX + A::NR);
            lx = LEN_ < 8 ? A::PX + r : 8 + r;
            lz = u < A::PX ? u + 4 * hw : (LEN_ < 8 ? u : 8 + u - A::PX);
            valid = u < A::PX || hw == 0;
        }
        if (valid) {
            const int row = (kk + lz) * A::PU + (jj + lx) * A::RU;
            const ulonglong2* hvr = reinterpret_cast<const ulonglong2*>(hv) + row;
            ulonglong2* hgr = reinterpret_cast<ulonglong2*>(hg) + row;
            const float* w = cb + A::WP * (lx + LEN_ * lz);
            uint64_t v[A::NA], gm[A::NA];
#pragma unroll
            for (int a = 0; a < A::NA; a += 2) {
                const ulonglong2 t = hvr[a / 2];
                v[a] = t.x;
                v[a + 1] = t.y;
                gm[a] = gm[a + 1] = 0;
            }
#pragma unroll
            for (int ly = 0; ly < LEN_; ly++) {
                const uint64_t w2 = f2_pack(w[ly], w[ly]);
                uint64_t d[4], t[4];
                float q[8];
#pragma unroll
                for (int i = 0; i < 4; i++) d[i] = f2_fma(v[i + ly], minus, f[i]);
#pragma unroll
                for (int i = 0; i < 4; i++) f2_split(f2_fma(d[i], d[i], eps2), q[2 * i], q[2 * i + 1]);
#pragma unroll
                for (int i = 0; i < 8; i++) q[i] = rsqrtf(q[i]);
#pragma unroll
                for (int i = 0; i < 4; i++) t[i] = f2_mul(d[i], f2_pack(q[2 * i], q[2 * i + 1]));  // phi'(d)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    gf[i] = f2_fma(w2, t[i], gf[i]);
                    gm[i + ly] = f2_fma(w2, t[i], gm[i + ly]);
                }
            }
#pragma unroll
            for (int a = 0; a < A::NA; a += 2) {
                ulonglong2 t = hgr[a / 2];
                t.x = f2_add(t.x, gm[a]);
                t.y = f2_add(t.y, gm[a + 1]);
                hgr[a / 2] = t;
            }
        }
        __syncwarp();  // the next step's rows are other lanes' of this one
    }
    // the moving side's gradient is -hg
    if (sub < RPW)
#pragma unroll 4
        for (int b = sub, cc = 0; cc < A::NA;) {
            const float2 gv = *reinterpret_cast<const float2*>(hg + 4 * (cc * A::PU + b * A::RU) + 2 * la);
            float* g = sMbar + ya + ox[b] + oz[cc];
            if (gv.x != 0.0f) atomicAdd(g, -G.alpha1 * gv.x);
            if (gv.y != 0.0f) atomicAdd(g + sz, -G.alpha1 * gv.y);
            if ((b += RPW) >= A::NA) {
                b -= A::NA;
                cc++;
            }
        }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float g0, g1;
        f2_split(gf[i], g0, g1);
        g0 += __shfl_xor_sync(0xffffffffu, g0, 16);
        g1 += __shfl_xor_sync(0xffffffffu, g1, 16);
        if (hw == 0) {
            sFbar[fp + i] = G.alpha1 * g0;
            sFbar[fp + i + sz] = G.alpha1 * g1;
        }
    }
}

// ---------------------------------------------------------------------------
// Row form for the coarser levels (grid > 4: nine sampled columns per node, and
// label quantisation > 1).  An item is one label pair (lx, lz) of one sampled
// column; its displaced samples read one row of the moving descriptor: NA = g +
// (len-1) q consecutive voxels along y at clamped (x, z).  At these shapes no
// two items of a node read the same row, so a node's rows are staged compactly,
// row t at slot t with an odd pitch: the staging copies are coalesced along y
// (a warp per row, cp.async) and each thread then reads its own row from shared
// memory without bank conflicts (consecutive threads, rows PY apart, PY odd).  A thread keeps its item's len sums (forward)
// or the label weights (adjoint) in registers across all channel groups.  The
// moving-side gradient is the gather kernel k_soft_cost_adj_moving.

struct RowPlan {
    int PY, CG;  // row pitch (floats, odd), channels per stage
};

template <int G_, int LEN_, int Q_>
struct RowGeom {
    static constexpr int S = G_ > 4 ? 2 : 1, NX = (G_ + S - 1) / S, NCOL = NX * NX, NSAMP = NCOL * G_;
    static constexpr int NA = G_ + (LEN_ - 1) * Q_, LEN2 = LEN_ * LEN_, LEN3 = LEN2 * LEN_;
    static constexpr int ITEMS = LEN2 * NCOL;
    static constexpr int BLOCK = (ITEMS + 31) / 32 * 32;
    static constexpr int PY = NA | 1;
    static_assert(ITEMS <= 1024 && NA <= 32, "one item per thread, one row per warp");
};

// Item t of a node: label pair (lab = lx + len*lz) and sampled column (jj, kk).
// Label-fastest order (forward: a warp's items share a column, its label sums go
// to distinct addresses) or column-fastest order (adjoint: a warp's items spread
// over the nine columns, so its sample-gradient atomics hit a column <= 4 times).
template <class RG, int LEN_, int Q_, bool COL_FAST>
__device__ __forceinline__ void row_item(int t, int& lab, int& col, int& bx, int& bz) {
    lab = COL_FAST ? t / RG::NCOL : t % RG::LEN2;
    col = COL_FAST ? t % RG::NCOL : t / RG::LEN2;
    const int lx = lab % LEN_, lz = lab / LEN_, jj = col % RG::NX, kk = col / RG::NX;
    bx = jj * RG::S + lx * Q_;
    bz = kk * RG::S + lz * Q_;
}

// Stage channels [c0, c0+CG) of the node's item rows: rows[c][t][a], pitch PY.
// goff[t] holds item t's clamped (x, z) offset in one channel.
template <class RG>
__device__ __forceinline__ void stage_rows(const SoftGeom& G, int yb, const float* __restrict__ sM, int c0, int CG,
                                           const int* goff, float* rows) {
    const int64_t sz = (int64_t)G.m * G.n * G.o;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int ya = clampi(yb + lane, 0, G.m - 1);
    if (lane < RG::NA)
        for (int c = 0; c < CG; c++) {
            const float* src = sM + (int64_t)(c0 + c) * sz + ya;
            float* dst = rows + c * (RG::ITEMS * RG::PY) + lane;
            for (int r = warp; r < RG::ITEMS; r += nw) cp_async4(dst + r * RG::PY, src + goff[r]);
        }
    cp_async_wait_all();
}

template <class RG>
__device__ __forceinline__ void stage_fixed_samples(const SoftGeom& G, int y, int x, int z,
                                                    const float* __restrict__ sF, float* fs) {
    const int64_t mn = (int64_t)G.m * G.n, sz = mn * G.o;
    for (int e = threadIdx.x; e < 12 * RG::NSAMP; e += blockDim.x) {
        const int c = e / RG::NSAMP, s = e % RG::NSAMP;
        const int col = s / G.g, i = s % G.g;
        const int py = y * G.g + i, px = x * G.g + (col % RG::NX) * RG::S, pz = z * G.g + (col / RG::NX) * RG::S;
        cp_async4(fs + e, sF + (int64_t)c * sz + py + (int64_t)px * G.m + (int64_t)pz * mn);
    }
    cp_async_wait_all();
}

// Each thread writes its item's clamped (x, z) row offset; returns the box's y origin.
template <class RG, int LEN_, int Q_, bool COL_FAST>
__device__ __forceinline__ int row_offsets(const SoftGeom& G, int y, int x, int z, int* goff) {
    const int R = (RG::NA - G.g) / 2;
    const int t = threadIdx.x;
    if (t < RG::ITEMS) {
        int lab, col, bx, bz;
        row_item<RG, LEN_, Q_, COL_FAST>(t, lab, col, bx, bz);
        goff[t] = clampi(x * G.g - R + bx, 0, G.n - 1) * G.m + clampi(z * G.g - R + bz, 0, G.o - 1) * G.m * G.n;
    }
    return y * G.g - R;
}

template <int G_, int LEN_, int Q_>
__global__ void __launch_bounds__(RowGeom<G_, LEN_, Q_>::BLOCK, 2)
    k_soft_cost_rows(const float* __restrict__ sF, const float* __restrict__ sM, float* __restrict__ cost, SoftGeom G,
                     RowPlan P) {
    using RG = RowGeom<G_, LEN_, Q_>;
    extern __shared__ float sh[];
    const int node = blockIdx.x;
    const int y = node % G.m1, x = (node / G.m1) % G.n1, z = node / (G.m1 * G.n1);
    float* rows = sh;                                  // [CG][ITEMS][PY]
    float* fs = rows + P.CG * RG::ITEMS * RG::PY;      // [12][NSAMP]
    float* acc = fs + 12 * RG::NSAMP;                  // [LEN3]
    int* goff = reinterpret_cast<int*>(acc + RG::LEN3);  // [ITEMS]
    const int yb = row_offsets<RG, LEN_, Q_, false>(G, y, x, z, goff);
    for (int l = threadIdx.x; l < RG::LEN3; l += blockDim.x) acc[l] = 0.0f;
    stage_fixed_samples<RG>(G, y, x, z, sF, fs);
    const float eps2 = G.eps * G.eps;
    const int t = threadIdx.x;
    const bool active = t < RG::ITEMS;
    int lab = 0, col = 0, bx, bz;
    row_item<RG, LEN_, Q_, false>(active ? t : 0, lab, col, bx, bz);
    float sums[LEN_];
#pragma unroll
    for (int ly = 0; ly < LEN_; ly++) sums[ly] = 0.0f;
    for (int c0 = 0; c0 < 12; c0 += P.CG) {
        __syncthreads();  // goff written / previous rows consumed
        stage_rows<RG>(G, yb, sM, c0, P.CG, goff, rows);
        __syncthreads();
        if (active)
            for (int c = 0; c < P.CG; c++) {
                const float* row = rows + (c * RG::ITEMS + t) * RG::PY;
                const float* fc = fs + (c0 + c) * RG::NSAMP + col * G_;
                float v[RG::NA], f[G_];
#pragma unroll
                for (int a = 0; a < RG::NA; a++) v[a] = row[a];
#pragma unroll
                for (int i = 0; i < G_; i++) f[i] = fc[i];
#pragma unroll
                for (int ly = 0; ly < LEN_; ly++)
#pragma unroll
                    for (int i = 0; i < G_; i++) {
                        const float d = f[i] - v[i + ly * Q_];
                        const float x2 = d * d + eps2;
                        sums[ly] += x2 * rsqrtf(x2);
                    }
            }
    }
    if (active)
#pragma unroll
        for (int ly = 0; ly < LEN_; ly++) atomicAdd(acc + ly + LEN_ * lab, sums[ly]);
    __syncthreads();
    for (int l = threadIdx.x; l < RG::LEN3; l += blockDim.x)
        cost[(int64_t)node * RG::LEN3 + l] = G.alpha1 * (acc[l] - (float)(12 * RG::NSAMP) * G.eps);
}

// Fixed-side adjoint and the alpha dot product in row form: an item's len label
// weights stay in registers, its g sample gradients are summed over its labels
// per channel and added to the node's shared sample gradients.
template <int G_, int LEN_, int Q_>
__global__ void __launch_bounds__(RowGeom<G_, LEN_, Q_>::BLOCK, 2)
    k_soft_cost_adjF_rows(const float* __restrict__ sF, const float* __restrict__ sM, const float* __restrict__ cbar,
                          const float* __restrict__ cost, float* __restrict__ sFbar, double* __restrict__ dot,
                          SoftGeom G, RowPlan P) {
    using RG = RowGeom<G_, LEN_, Q_>;
    extern __shared__ float sh[];
    __shared__ double red[32];
    const int node = blockIdx.x;
    const int y = node % G.m1, x = (node / G.m1) % G.n1, z = node / (G.m1 * G.n1);
    const int64_t mn = (int64_t)G.m * G.n, sz = mn * G.o;
    float* rows = sh;                                  // [CG][ITEMS][PY]
    float* fs = rows + P.CG * RG::ITEMS * RG::PY;      // [12][NSAMP]
    float* gfs = fs + 12 * RG::NSAMP;                  // [12][NSAMP]
    float* cb = gfs + 12 * RG::NSAMP;                  // [LEN3]
    int* goff = reinterpret_cast<int*>(cb + RG::LEN3);  // [ITEMS]
    const float* cbn = cbar + (int64_t)node * RG::LEN3;
    const float* cn = cost + (int64_t)node * RG::LEN3;
    const int yb = row_offsets<RG, LEN_, Q_, true>(G, y, x, z, goff);
    // alpha: centred dot product (the exact cbar sums to zero over labels)
    double csum = 0.0;
    for (int l = threadIdx.x; l < RG::LEN3; l += blockDim.x) {
        csum += (double)cn[l];
        cb[l] = cbn[l];
    }
    for (int off = 16; off > 0; off >>= 1) csum += __shfl_xor_sync(0xffffffffu, csum, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = csum;
    for (int e = threadIdx.x; e < 12 * RG::NSAMP; e += blockDim.x) gfs[e] = 0.0f;
    stage_fixed_samples<RG>(G, y, x, z, sF, fs);
    __syncthreads();
    double cmean = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) cmean += red[w];
    cmean /= (double)RG::LEN3;
    double part = 0.0;
    for (int l = threadIdx.x; l < RG::LEN3; l += blockDim.x) part += (double)cb[l] * ((double)cn[l] - cmean);
    for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
    if ((threadIdx.x & 31) == 0) atomicAdd(dot, part);
    const float eps2 = G.eps * G.eps;
    const int t = threadIdx.x;
    const bool active = t < RG::ITEMS;
    int lab = 0, col = 0, bx, bz;
    row_item<RG, LEN_, Q_, true>(active ? t : 0, lab, col, bx, bz);
    float w[LEN_];
#pragma unroll
    for (int ly = 0; ly < LEN_; ly++) w[ly] = cb[ly + LEN_ * lab];
    for (int c0 = 0; c0 < 12; c0 += P.CG) {
        __syncthreads();
        stage_rows<RG>(G, yb, sM, c0, P.CG, goff, rows);
        __syncthreads();
        if (active)
            for (int c = 0; c < P.CG; c++) {
                const float* row = rows + (c * RG::ITEMS + t) * RG::PY;
                const float* fc = fs + (c0 + c) * RG::NSAMP + col * G_;
                float* gfc = gfs + (c0 + c) * RG::NSAMP + col * G_;
                float v[RG::NA], f[G_], gf[G_];
#pragma unroll
                for (int a = 0; a < RG::NA; a++) v[a] = row[a];
#pragma unroll
                for (int i = 0; i < G_; i++) {
                    f[i] = fc[i];
                    gf[i] = 0.0f;
                }
#pragma unroll
                for (int ly = 0; ly < LEN_; ly++)
#pragma unroll
                    for (int i = 0; i < G_; i++) {
                        const float d = f[i] - v[i + ly * Q_];
                        gf[i] += w[ly] * d * rsqrtf(d * d + eps2);
                    }
#pragma unroll
                for (int i = 0; i < G_; i++) atomicAdd(gfc + i, gf[i]);
            }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 12 * RG::NSAMP; e += blockDim.x) {
        const int c = e / RG::NSAMP, s = e % RG::NSAMP;
        const int cl = s / G.g, i = s % G.g;
        const int py = y * G.g + i, px = x * G.g + (cl % RG::NX) * RG::S, pz = z * G.g + (cl / RG::NX) * RG::S;
        sFbar[(int64_t)c * sz + py + (int64_t)px * G.m + (int64_t)pz * mn] = G.alpha1 * gfs[e];
    }
}

// ---------------------------------------------------------------------------
// Tree sweeps

struct SoftTree {
    int len, len3, hw, sz, root, q;
    float tau, itau;
    const int* parents;
    const float* edgemst;
    const int* child_ptr;
    const int* children;
    const float* off;  // nullable: (3, sz) label-unit offsets x|y|z of each node's edge, (prior[parent]-prior[node])/q
    float* offbar;     // nullable (backward): dL/doff, (3, sz)
};

// The offset of node c's edge along label axis s (stride 1 = y, len = x, len^2 = z).
__device__ __forceinline__ float edge_off(const SoftTree& t, int c, int axis) {
    if (!t.off) return 0.0f;
    const int comp = axis == 0 ? 1 : (axis == 1 ? 0 : 2);  // off is stored x|y|z
    return t.off[comp * t.sz + c];
}

__device__ float block_max(float v, float* red) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float r = -INFINITY;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) r = fmaxf(r, red[w]);
    __syncthreads();
    return r;
}

// (max, sum exp(x - max)) of the block's values in one reduction; returns the LSE.
// red needs 64 floats.
__device__ float block_lse(float mx, float se, float* red) {
    for (int o = 16; o > 0; o >>= 1) {
        const float om = __shfl_xor_sync(0xffffffffu, mx, o), os = __shfl_xor_sync(0xffffffffu, se, o);
        const float nm = fmaxf(mx, om);
        se = (mx == -INFINITY ? 0.0f : se * __expf(mx - nm)) + (om == -INFINITY ? 0.0f : os * __expf(om - nm));
        mx = nm;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5] = mx;
        red[32 + (threadIdx.x >> 5)] = se;
    }
    __syncthreads();
    float m = -INFINITY;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) m = fmaxf(m, red[w]);
    float t = 0.0f;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++)
        if (red[w] != -INFINITY) t += red[32 + w] * __expf(red[w] - m);
    __syncthreads();
    return m + __logf(t);
}

// three sums in one reduction; red needs 96 floats
__device__ void block_sum3(float& a, float& b, float& c, float* red) {
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
        c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5] = a;
        red[32 + (threadIdx.x >> 5)] = b;
        red[64 + (threadIdx.x >> 5)] = c;
    }
    __syncthreads();
    a = b = c = 0.0f;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
        a += red[w];
        b += red[32 + w];
        c += red[64 + w];
    }
    __syncthreads();
}

__device__ float block_sum(float v, float* red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float r = 0.0f;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) r += red[w];
    __syncthreads();
    return r;
}

// out(o) = LSE_a in(line(o), a) - d(a, b)^2/tau along the axis of stride s, with b =
// o's coordinate on that axis and d = sgn (b - a) + off (the prior field's offset of
// the edge; sgn = +1 when b indexes the parent label, -1 when it indexes the child's).
// Ends with a barrier.
__device__ void lse_axis(const float* in, float* out, int len, int len3, int s, float itau, float off, float sgn) {
    for (int o = threadIdx.x; o < len3; o += blockDim.x) {
        const int b = (o / s) % len;
        const float* line = in + (o - b * s);
        float mx = -INFINITY;
        for (int a = 0; a < len; a++) {
            const float d = sgn * (float)(b - a) + off;
            mx = fmaxf(mx, line[a * s] - d * d * itau);
        }
        float acc = 0.0f;
        for (int a = 0; a < len; a++) {
            const float d = sgn * (float)(b - a) + off;
            acc += __expf(line[a * s] - d * d * itau - mx);
        }
        out[o] = mx + __logf(acc);
    }
    __syncthreads();
}

// adjoint of one pass: inbar(a) = sum_b outbar(b) w(a, b), w = exp(in(a) - d^2/tau - out(b));
// returns this thread's part of dL/doff = sum_{a,b} outbar(b) w(a, b) (-2 d / tau).
__device__ float lse_axis_adj(const float* in, const float* out, const float* outbar, float* inbar, int len, int len3,
                              int s, float itau, float off, float sgn) {
    float dof = 0.0f;
    for (int o = threadIdx.x; o < len3; o += blockDim.x) {
        const int a = (o / s) % len;
        const int base = o - a * s;
        const float x = in[o];
        float acc = 0.0f;
        for (int b = 0; b < len; b++) {
            const float d = sgn * (float)(b - a) + off;
            const float wb = outbar[base + b * s] * __expf(x - d * d * itau - out[base + b * s]);
            acc += wb;
            dof += wb * d;
        }
        inbar[o] = acc;
    }
    __syncthreads();
    return -2.0f * itau * dof;
}

// S = pass z o pass x o pass y; keeps t1, t2 for the adjoint (out may alias in).
// off3 = (y, x, z) offsets of the node's edge.
__device__ __forceinline__ void sep_lse(const float* in, float* t1, float* t2, float* out, int len, int len3,
                                        float itau, const float* off3, float sgn) {
    lse_axis(in, t1, len, len3, 1, itau, off3[0], sgn);
    lse_axis(t1, t2, len, len3, len, itau, off3[1], sgn);
    lse_axis(t2, out, len, len3, len * len, itau, off3[2], sgn);
}

// inbar = S^T outbar.  wa is scratch; wb may alias outbar and inbar may alias wa.
// dof3 (y, x, z) receives this thread's parts of dL/doff.
__device__ __forceinline__ void sep_lse_adj(const float* in, const float* t1, const float* t2, const float* out,
                                            const float* outbar, float* wa, float* wb, float* inbar, int len,
                                            int len3, float itau, const float* off3, float sgn, float* dof3) {
    dof3[2] = lse_axis_adj(t2, out, outbar, wa, len, len3, len * len, itau, off3[2], sgn);
    dof3[1] = lse_axis_adj(t1, t2, wa, wb, len, len3, len, itau, off3[1], sgn);
    dof3[0] = lse_axis_adj(in, t1, wb, inbar, len, len3, 1, itau, off3[0], sgn);
}

// Adds this block's dL/doff of node c (scaled) into t.offbar (x|y|z layout); red: 96 floats.
__device__ void add_offbar(const SoftTree& t, int c, float* dof3, float scale, float* red) {
    if (!t.offbar) return;
    block_sum3(dof3[0], dof3[1], dof3[2], red);
    if (threadIdx.x == 0) {
        t.offbar[t.sz + c] += scale * dof3[0];      // y
        t.offbar[c] += scale * dof3[1];             // x
        t.offbar[2 * t.sz + c] += scale * dof3[2];  // z
    }
}

// ---- per-node bodies (one CTA per node; data of other nodes written in the same
// sweep is read with __ldcg, after the producer's release has been observed)
//
// What a node reads that does not come from this sweep (its own rows from the
// forward or earlier sweeps, its child list) is loaded before the dependency
// wait into NodePre — one label per thread, the label threadIdx.x — so that after
// the wait only the rows produced in this sweep remain on the critical path, and
// the children's rows are then loaded together rather than one child after another.

constexpr int kMaxChildren = 6;  // a 6-connected grid tree: at most 6 children (the root)

struct NodePre {
    float v0, v1, v2;  // own values at label threadIdx.x (meaning depends on the sweep)
    int nch;
    int ch[kMaxChildren];
};

// Own value at label l: prefetched for the thread's first label, else loaded.
__device__ __forceinline__ float own(int l, float pre, const float* __restrict__ row) {
    return l == (int)threadIdx.x ? pre : row[l];
}

__device__ __forceinline__ void load_children(const SoftTree& t, int c, NodePre& pre) {
    const int k0 = t.child_ptr[c], k1 = t.child_ptr[c + 1];
    pre.nch = k1 - k0;
#pragma unroll
    for (int i = 0; i < kMaxChildren; i++) pre.ch[i] = i < pre.nch ? t.children[k0 + i] : 0;
}

// v + sum over children in child order of (X[k][l] - xmin[k]) (xmin may be null):
// all children's values are loaded before the in-order sum.
__device__ __forceinline__ float add_children(const SoftTree& t, int c, const NodePre& pre, int l, float v,
                                              const float* __restrict__ X, const float* __restrict__ xmin) {
    const int L3 = t.len3;
    if (pre.nch <= kMaxChildren) {
        float xs[kMaxChildren], ms[kMaxChildren];
#pragma unroll
        for (int i = 0; i < kMaxChildren; i++) {
            xs[i] = i < pre.nch ? __ldcg(X + (int64_t)pre.ch[i] * L3 + l) : 0.0f;
            ms[i] = (xmin && i < pre.nch) ? __ldcg(xmin + pre.ch[i]) : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < kMaxChildren; i++)
            if (i < pre.nch) v += xmin ? xs[i] - ms[i] : xs[i];
        return v;
    }
    for (int ci = t.child_ptr[c]; ci < t.child_ptr[c + 1]; ci++) {
        const int k = t.children[ci];
        v += xmin ? __ldcg(X + (int64_t)k * L3 + l) - __ldcg(xmin + k) : __ldcg(X + (int64_t)k * L3 + l);
    }
    return v;
}

// The bodies below are for label widths above 9; k_sweep has those up to 9.

// Upward: B_c = C_c + sum_children (M_k - min M_k), stored minus its minimum (the
// marginals and the parent's (message - min) are invariant to a constant shift of
// B_c, and the centred values keep the exponents of the label-space transforms
// small where the probability mass is); M_c = -tau S(-e_c B_c / tau).
__device__ void node_up(const SoftTree& t, int c, const NodePre& pre, const float* __restrict__ cost,
                        float* __restrict__ B, float* __restrict__ M, float* __restrict__ Mmin, float* sh) {
    const int L3 = t.len3;
    float* f = sh;
    float* t1 = sh + L3;
    float* t2 = sh + 2 * L3;
    float* red = sh + 3 * L3;
    const float e = c == t.root ? 0.0f : t.edgemst[c];
    float bmin = INFINITY;
    for (int l = threadIdx.x; l < L3; l += blockDim.x) {
        const float v = add_children(t, c, pre, l, own(l, pre.v0, cost + (int64_t)c * L3), M, Mmin);
        f[l] = v;
        bmin = fminf(bmin, v);
    }
    bmin = -block_max(-bmin, red);
    for (int l = threadIdx.x; l < L3; l += blockDim.x) {
        const float v = f[l] - bmin;
        B[(int64_t)c * L3 + l] = v;
        f[l] = -e * v * t.itau;
    }
    __syncthreads();
    if (c == t.root) return;
    const float off3[3] = {edge_off(t, c, 0), edge_off(t, c, 1), edge_off(t, c, 2)};
    sep_lse(f, t1, t2, f, t.len, L3, t.itau, off3, 1.0f);  // output index = parent label
    float mn = INFINITY;
    for (int lp = threadIdx.x; lp < L3; lp += blockDim.x) {
        const float msg = -t.tau * f[lp];
        M[(int64_t)c * L3 + lp] = msg;
        mn = fminf(mn, msg);
    }
    mn = -block_max(-mn, red);
    if (threadIdx.x == 0) Mmin[c] = mn;
}

// Downward marginals; writes log p_c and the expected displacement.  log p_c is
// normalised in exact arithmetic; renormalising stops float rounding from drifting
// along root-to-leaf paths (no effect on the exact gradient, whose parameter
// derivatives are tangent to the normalised set).
__device__ void node_down(const SoftTree& t, int c, const NodePre& pre, const float* __restrict__ B,
                          const float* __restrict__ M, float* __restrict__ logp, float* __restrict__ disp, float* sh) {
    const int L3 = t.len3, len = t.len;
    float* r = sh;
    float* t1 = sh + L3;
    float* t2 = sh + 2 * L3;
    float* red = sh + 3 * L3;
    float* lc = logp + (int64_t)c * L3;
    const float* bc = B + (int64_t)c * L3;
    if (c == t.root) {
        for (int l = threadIdx.x; l < L3; l += blockDim.x) r[l] = -own(l, pre.v1, bc) * t.itau;
    } else {
        const int p = t.parents[c];
        const float e = t.edgemst[c];
        for (int lp = threadIdx.x; lp < L3; lp += blockDim.x)
            r[lp] = __ldcg(logp + (int64_t)p * L3 + lp) + own(lp, pre.v0, M + (int64_t)c * L3) * t.itau;
        __syncthreads();
        const float off3[3] = {edge_off(t, c, 0), edge_off(t, c, 1), edge_off(t, c, 2)};
        sep_lse(r, t1, t2, r, len, L3, t.itau, off3, -1.0f);  // output index = child label
        for (int l = threadIdx.x; l < L3; l += blockDim.x) r[l] += -e * own(l, pre.v1, bc) * t.itau;
    }
    float mx = -INFINITY;
    for (int l = threadIdx.x; l < L3; l += blockDim.x) mx = fmaxf(mx, r[l]);
    float se = 0.0f;
    for (int l = threadIdx.x; l < L3; l += blockDim.x) se += __expf(r[l] - mx);
    const float lz = block_lse(mx, se, red);
    float eu = 0.0f, ev = 0.0f, ew = 0.0f;
    for (int l = threadIdx.x; l < L3; l += blockDim.x) {
        const float lp = r[l] - lz;
        lc[l] = lp;
        const float pl = __expf(lp);
        eu += pl * (float)(((l / len) % len - t.hw) * t.q);
        ev += pl * (float)((l % len - t.hw) * t.q);
        ew += pl * (float)((l / (len * len) - t.hw) * t.q);
    }
    block_sum3(eu, ev, ew, red);
    if (threadIdx.x == 0) {
        disp[c] = eu;
        disp[t.sz + c] = ev;
        disp[2 * t.sz + c] = ew;
    }
}

// Adjoint of the marginals (leaves to root):
//   h(l) = gE_c . d(l) p_c(l) + sum_children R_k(l)    (= dL/dlog p_c)
//   Bbar_c = -e h/tau (root: -(h - p sum h)/tau, projected to zero mean);  R_c = S^T h w.r.t. r
__device__ void node_down_adj(const SoftTree& t, int c, const NodePre& pre, const float* __restrict__ M,
                              const float* __restrict__ logp, const float* __restrict__ gdisp, float* __restrict__ R,
                              float* __restrict__ Bbar, float* sh) {
    const int L3 = t.len3, len = t.len;
    float* r = sh;
    float* t1 = sh + L3;
    float* t2 = sh + 2 * L3;
    float* G = sh + 3 * L3;
    float* h = sh + 4 * L3;
    float* wa = sh + 5 * L3;
    float* red = sh + 6 * L3;
    const float* lc = logp + (int64_t)c * L3;
    const float gu = gdisp[c], gv = gdisp[t.sz + c], gw = gdisp[2 * t.sz + c];
    float tot = 0.0f;
    for (int l = threadIdx.x; l < L3; l += blockDim.x) {
        const float du = (float)(((l / len) % len - t.hw) * t.q), dv = (float)((l % len - t.hw) * t.q),
                    dw = (float)((l / (len * len) - t.hw) * t.q);
        const float v = add_children(t, c, pre, l, (gu * du + gv * dv + gw * dw) * __expf(own(l, pre.v0, lc)), R,
                                     nullptr);
        h[l] = v;
        tot += v;
    }
    float* bb = Bbar + (int64_t)c * L3;
    if (c == t.root) {
        tot = block_sum(tot, red);
        float mean = 0.0f;
        for (int l = threadIdx.x; l < L3; l += blockDim.x) {
            wa[l] = -(h[l] - __expf(own(l, pre.v0, lc)) * tot) * t.itau;
            mean += wa[l];
        }
        mean = block_sum(mean, red) / (float)L3;
        for (int l = threadIdx.x; l < L3; l += blockDim.x) bb[l] = wa[l] - mean;
        return;
    }
    const int p = t.parents[c];
    const float e = t.edgemst[c];
    for (int l = threadIdx.x; l < L3; l += blockDim.x) {
        bb[l] = -e * t.itau * h[l];
        r[l] = own(l, pre.v2, logp + (int64_t)p * L3) + own(l, pre.v1, M + (int64_t)c * L3) * t.itau;
    }
    __syncthreads();
    const float off3[3] = {edge_off(t, c, 0), edge_off(t, c, 1), edge_off(t, c, 2)};
    float dof3[3];
    sep_lse(r, t1, t2, G, len, L3, t.itau, off3, -1.0f);
    sep_lse_adj(r, t1, t2, G, h, wa, h, wa, len, L3, t.itau, off3, -1.0f, dof3);
    float* rc = R + (int64_t)c * L3;
    for (int l = threadIdx.x; l < L3; l += blockDim.x) rc[l] = wa[l];
    add_offbar(t, c, dof3, 1.0f, red);
}

// Adjoint of the upward recursion (root to leaves, root excluded):
//   Mbar_c = R_c/tau + Bbar_parent; M_c = -tau S(f), f = -e B_c/tau, so
//   dL/dB_c += -e/tau S^T(-tau Mbar_c) = e S^T(Mbar_c).  Bbar_c is final afterwards
// (= dL/dC_c); the exact value sums to zero over labels (shift invariance), and
// projecting keeps rounding from accumulating as a common mode down the tree.
__device__ void node_up_adj(const SoftTree& t, int c, const NodePre& pre, const float* __restrict__ B,
                            const float* __restrict__ R, float* __restrict__ Bbar, float* sh) {
    if (c == t.root) return;
    const int L3 = t.len3, len = t.len;
    float* f = sh;
    float* t1 = sh + L3;
    float* t2 = sh + 2 * L3;
    float* out = sh + 3 * L3;
    float* mb = sh + 4 * L3;
    float* wa = sh + 5 * L3;
    float* red = sh + 6 * L3;
    const int p = t.parents[c];
    const float e = t.edgemst[c];
    for (int l = threadIdx.x; l < L3; l += blockDim.x) {
        f[l] = -e * own(l, pre.v0, B + (int64_t)c * L3) * t.itau;
        mb[l] = own(l, pre.v1, R + (int64_t)c * L3) * t.itau + __ldcg(Bbar + (int64_t)p * L3 + l);
    }
    __syncthreads();
    const float off3[3] = {edge_off(t, c, 0), edge_off(t, c, 1), edge_off(t, c, 2)};
    float dof3[3];
    sep_lse(f, t1, t2, out, len, L3, t.itau, off3, 1.0f);
    sep_lse_adj(f, t1, t2, out, mb, wa, mb, wa, len, L3, t.itau, off3, 1.0f, dof3);
    // M = -tau out: dL/dout = -tau Mbar, so the offset gradient computed with Mbar scales by -tau
    add_offbar(t, c, dof3, -t.tau, red);
    float* bb = Bbar + (int64_t)c * L3;
    float mean = 0.0f;
    for (int l = threadIdx.x; l < L3; l += blockDim.x) {
        wa[l] = own(l, pre.v2, bb) + e * wa[l];
        mean += wa[l];
    }
    mean = block_sum(mean, red) / (float)L3;
    for (int l = threadIdx.x; l < L3; l += blockDim.x) bb[l] = wa[l] - mean;
}

// ---- persistent sweeps
//
// One launch per sweep.  CTAs claim nodes with a global ticket in breadth order
// (top-down sweeps) or reverse breadth order (bottom-up sweeps), wait until the
// node's parent (top-down) or all of its children (bottom-up) are finished, run the
// node body and release it.  A node only waits on nodes with smaller tickets,
// which were claimed by CTAs that are running and wait only on smaller tickets
// still, so the sweep always progresses; there are no per-level launches.  Each
// wait is bounded: on expiry the sweep records an error (reported as a timeout by
// the host) and carries on without further waits, so no CTA can hang.  (A
// wait-free variant for the bottom-up sweeps, in which the CTA completing a
// node's children continues with the node, measured 6-9 % slower: claiming in
// breadth order keeps each level's nodes in flight together.)


struct SweepState {
    int* ticket;  // next ticket
    int* done;    // top-down: 1 when the node is finished; bottom-up: children finished
    int* err;     // set when a wait gave up
};

__device__ __forceinline__ int ld_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

enum SweepKind { kSweepUp = 0, kSweepDown = 1, kSweepDownAdj = 2, kSweepUpAdj = 3 };

// Publishing a finished node: a release store (top-down: the node is done) or a
// release reduction (bottom-up: one more child of the parent has arrived) at GPU
// scope; the preceding block barrier makes every thread's writes of the node part
// of what is released, and waiters read the flag with ld.acquire.
__device__ __forceinline__ void st_release(int* p, int v) {
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void red_release_add(int* p, int v) {
    asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

constexpr int kSweepSpinLimit = 1 << 21;  // polls of an L2 round trip each: 0.4 s

// Polls until ready(); gives up after the limit (setting *err) or soon after another
// thread did, and returns false then (the caller carries on with what it has).
template <class Ready>
__device__ __forceinline__ bool bounded_poll(Ready ready, int* err) {
    for (int it = 1; !ready(); it++) {
        if (it > kSweepSpinLimit) {
            atomicExch(err, 1);
            return false;
        }
        if (it % 256 == 0 && ld_acquire(err)) return false;
    }
    return true;
}

__device__ __forceinline__ bool bounded_wait_geq(const int* flag, int need, int* err) {
    return bounded_poll([&] { return ld_acquire(flag) >= need; }, err);
}

// A row that other nodes of the same sweep wait for is its own flag: it starts as
// kNotYet in every word, each word is stored once, and a reader polls the words that
// it uses.  No word depends on another, so nothing has to be ordered.  The lanes of a warp
// see their words at different times and are brought together again behind the poll.
// (The store never writes kNotYet itself: a NaN with just these bits becomes the usual one.)
constexpr uint32_t kNotYet = 0xffffffffu;

__device__ __forceinline__ uint32_t ld_word(const float* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_word(float* p, float v) {
    const uint32_t b = __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(b == kNotYet ? 0x7fffffffu : b) : "memory");
}
__device__ __forceinline__ float wait_word(const float* p, int* err) {
    uint32_t v;
    bounded_poll([&] { return (v = ld_word(p)) != kNotYet; }, err);
    __syncwarp();
    return __uint_as_float(v);
}

struct SweepArgs {
    const float* cost;
    float* B;
    float* M;
    float* Mmin;
    float* logp;
    float* disp;
    const float* gdisp;
    float* R;
    float* Bbar;
    float* Bpart;  // k_sweep: the downward adjoint's part of Bbar (Bbar itself is waited for)
};

template <int KIND>
__device__ __forceinline__ void run_node(const SoftTree& t, int c, const NodePre& pre, const SweepArgs& a,
                                         float* sh) {
    if (KIND == kSweepUp) node_up(t, c, pre, a.cost, a.B, a.M, a.Mmin, sh);
    else if (KIND == kSweepDown) node_down(t, c, pre, a.B, a.M, a.logp, a.disp, sh);
    else if (KIND == kSweepDownAdj) node_down_adj(t, c, pre, a.M, a.logp, a.gdisp, a.R, a.Bbar, sh);
    else node_up_adj(t, c, pre, a.B, a.R, a.Bbar, sh);
}

// The node's inputs that precede this sweep (see NodePre), loaded before the wait.
template <int KIND>
__device__ __forceinline__ NodePre prefetch_node(const SoftTree& t, int c, const SweepArgs& a) {
    NodePre pre;
    pre.v0 = pre.v1 = pre.v2 = 0.0f;
    pre.nch = 0;
    const int l = threadIdx.x;
    const bool in = l < t.len3;
    const int64_t row = (int64_t)c * t.len3 + l;
    const bool root = c == t.root;
    if (KIND == kSweepUp) {
        if (in) pre.v0 = a.cost[row];
        load_children(t, c, pre);
    } else if (KIND == kSweepDown) {
        if (in) {
            if (!root) pre.v0 = a.M[row];
            pre.v1 = a.B[row];
        }
    } else if (KIND == kSweepDownAdj) {
        if (in) {
            pre.v0 = a.logp[row];
            if (!root) {
                pre.v1 = a.M[row];
                pre.v2 = a.logp[(int64_t)t.parents[c] * t.len3 + l];
            }
        }
        load_children(t, c, pre);
    } else if (!root && in) {
        pre.v0 = a.B[row];
        pre.v1 = a.R[row];
        pre.v2 = a.Bbar[row];
    }
    return pre;
}

template <int KIND>
__global__ void k_soft_sweep(SoftTree t, const int* __restrict__ ordered, SweepArgs a, SweepState st) {
    extern __shared__ float sh[];
    __shared__ int s_tk;
    constexpr bool kTopDown = KIND == kSweepDown || KIND == kSweepUpAdj;
    for (;;) {
        if (threadIdx.x == 0) s_tk = atomicAdd(st.ticket, 1);
        __syncthreads();
        const int tk = s_tk;
        if (tk >= t.sz) break;
        const int c = ordered[kTopDown ? tk : t.sz - 1 - tk];
        const NodePre pre = prefetch_node<KIND>(t, c, a);
        if (threadIdx.x == 0 && ld_acquire(st.err) == 0) {
            // top-down: the parent is released (done = 1); bottom-up: every child has arrived
            const int* flag = kTopDown ? (c == t.root ? nullptr : st.done + t.parents[c]) : st.done + c;
            const int need = kTopDown ? 1 : t.child_ptr[c + 1] - t.child_ptr[c];
            if (flag && need > 0) bounded_wait_geq(flag, need, st.err);
        }
        __syncthreads();
        run_node<KIND>(t, c, pre, a, sh);
        __syncthreads();
        if (threadIdx.x == 0) {
            if (kTopDown) st_release(st.done + c, 1);
            else if (c != t.root) red_release_add(st.done + t.parents[c], 1);
        }
    }
}

// ---- label widths 3 to 9: one thread per label, the label width known to the compiler
//
// A sweep is a chain of dependent nodes (the tree's depth, hundreds at grid 4), so what
// counts is the time from a finished parent (children) to the next one.  Against the
// bodies above: the width is a constant (no division, the line's values in registers,
// one pass for maximum and sum), a block reduction costs one barrier, and everything
// that does not depend on this sweep is done before the wait; in the two adjoint sweeps
// that is the whole forward transform and all its weights exp(in - d^2/tau - out), so
// that behind the wait each axis is LEN products from shared memory.  What no other node
// reads comes last.  A node's row is its own flag (see kNotYet): a round trip to L2 from the
// parent's store to this node's value, in place of store, fence, flag, poll, barrier, load.
// Measured, 343 labels at grid 4, up/down/adjoint down/adjoint up.  96x80x112 (13440
// nodes): the bodies above 1.3 to 1.7 ms each, this form with flags 0.66/0.67/0.56/0.51 ms,
// with rows as flags 0.46/0.45/0.36/0.35 ms.  Four pairs of 160x160x192 (76800 nodes) in
// flight together: about 22 ms each, 8.8/8.6/7.3/6.9 ms (one CTA to an SM: 9.8 for the
// third), 6.1/6.2/5.3/5.0 ms.  The arithmetic and its order are those of the bodies above.
// Wider label sets keep those: past 1024 labels there is more than one label per thread.
template <int LEN>
struct SweepShared {
    static constexpr int L2 = LEN * LEN, L3 = LEN * LEN * LEN, W = (L3 + 31) / 32;
    float x[L3], y[L3], z[L3], w[L3];
    float red[5][W];
};

// d(i) = sgn (own - i) + off (forward), sgn (i - own) + off (adjoint)
__device__ __forceinline__ float fwd_dist(int own, int i, float sgn, float off) { return sgn * (float)(own - i) + off; }
__device__ __forceinline__ float adj_dist(int own, int i, float sgn, float off) { return sgn * (float)(i - own) + off; }

template <int LEN>
__device__ __forceinline__ float lse_values(float (&v)[LEN], int own, float itau, float sgn, float off) {
    float mx = -INFINITY, acc = 0.0f;
#pragma unroll
    for (int a = 0; a < LEN; a++) {
        const float d = fwd_dist(own, a, sgn, off);
        v[a] -= d * d * itau;
        mx = fmaxf(mx, v[a]);
    }
#pragma unroll
    for (int a = 0; a < LEN; a++) acc += __expf(v[a] - mx);
    return mx + __logf(acc);
}

template <int LEN, int S>
__device__ __forceinline__ float lse_line(const float* line, int own, float itau, float sgn, float off) {
    float v[LEN];
#pragma unroll
    for (int a = 0; a < LEN; a++) v[a] = line[a * S];
    return lse_values<LEN>(v, own, itau, sgn, off);
}

// w[b] = exp(x - d^2/tau - out(b)) along the line
template <int LEN, int S>
__device__ __forceinline__ void adj_weights(float (&w)[LEN], float x, const float* out, int own, float itau, float sgn,
                                            float off) {
#pragma unroll
    for (int b = 0; b < LEN; b++) {
        const float d = adj_dist(own, b, sgn, off);
        w[b] = __expf(x - d * d * itau - out[b * S]);
    }
}

template <int LEN, int S>
__device__ __forceinline__ float adj_line(const float (&w)[LEN], const float* outbar, int own, float sgn, float off,
                                          bool want, float& dof) {
    float wb[LEN], acc = 0.0f;
#pragma unroll
    for (int b = 0; b < LEN; b++) wb[b] = outbar[b * S] * w[b];
#pragma unroll
    for (int b = 0; b < LEN; b++) acc += wb[b];
    if (want) {
#pragma unroll
        for (int b = 0; b < LEN; b++) dof += wb[b] * adj_dist(own, b, sgn, off);
    }
    return acc;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_add(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// v + sum over children in child order of (X[k][l] - xmin[k]) (xmin may be null), each
// word waited for; up to six children's words are polled together.
__device__ __forceinline__ float wait_children(const SoftTree& t, int c, const NodePre& pre, int l, float v,
                                               const float* X, const float* xmin, int* err) {
    const int L3 = t.len3;
    if (pre.nch <= kMaxChildren) {
        uint32_t xs[kMaxChildren], ms[kMaxChildren];
        bounded_poll([&] {
            bool ok = true;
#pragma unroll
            for (int i = 0; i < kMaxChildren; i++)
                if (i < pre.nch) {
                    xs[i] = ld_word(X + (int64_t)pre.ch[i] * L3 + l);
                    ms[i] = xmin ? ld_word(xmin + pre.ch[i]) : 0u;
                }
#pragma unroll
            for (int i = 0; i < kMaxChildren; i++)
                if (i < pre.nch) ok = ok && xs[i] != kNotYet && ms[i] != kNotYet;
            return ok;
        }, err);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kMaxChildren; i++)
            if (i < pre.nch) v += xmin ? __uint_as_float(xs[i]) - __uint_as_float(ms[i]) : __uint_as_float(xs[i]);
        return v;
    }
    for (int ci = t.child_ptr[c]; ci < t.child_ptr[c + 1]; ci++) {
        const int k = t.children[ci];
        const float x = wait_word(X + (int64_t)k * L3 + l, err);
        v += xmin ? x - wait_word(xmin + k, err) : x;
    }
    return v;
}

// The block barrier of the sweeps whose lanes poll: it wants a warp's lanes together.  (Lanes
// that left a poll at different times went on separately.  About one backward pass in a
// thousand then gave up: a block had gone on to its next node while the words of a row's
// last warp, 320 to 342 of 343, had never been stored.)
__device__ __forceinline__ void block_sync() {
    __syncwarp();
    __syncthreads();
}

// Block reductions with one barrier; red is not written again before two barriers.
template <int W>
__device__ __forceinline__ float all_max(float v, float* red) {
    v = warp_max(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    block_sync();
    float r = red[0];
#pragma unroll
    for (int w = 1; w < W; w++) r = fmaxf(r, red[w]);
    return r;
}
template <int W>
__device__ __forceinline__ float all_sum(float v, float* red) {
    v = warp_add(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    block_sync();
    float r = red[0];
#pragma unroll
    for (int w = 1; w < W; w++) r += red[w];
    return r;
}

// (max, sum exp(x - max)) of the block; returns the LSE
template <int W>
__device__ __forceinline__ float all_lse(float mx, float se, float* rmx, float* rse) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float om = __shfl_xor_sync(0xffffffffu, mx, o), os = __shfl_xor_sync(0xffffffffu, se, o);
        const float nm = fmaxf(mx, om);
        se = (mx == -INFINITY ? 0.0f : se * __expf(mx - nm)) + (om == -INFINITY ? 0.0f : os * __expf(om - nm));
        mx = nm;
    }
    if ((threadIdx.x & 31) == 0) {
        rmx[threadIdx.x >> 5] = mx;
        rse[threadIdx.x >> 5] = se;
    }
    block_sync();
    float m = -INFINITY, t = 0.0f;
#pragma unroll
    for (int w = 0; w < W; w++) m = fmaxf(m, rmx[w]);
#pragma unroll
    for (int w = 0; w < W; w++)
        if (rmx[w] != -INFINITY) t += rse[w] * __expf(rmx[w] - m);
    return m + __logf(t);
}

template <int KIND, int LEN>
__global__ void __launch_bounds__(SweepShared<LEN>::W * 32, LEN <= 7 ? 2 : 1)
    k_sweep(SoftTree t, const int* __restrict__ ordered, SweepArgs a, SweepState st) {
    using SH = SweepShared<LEN>;
    constexpr int L2 = SH::L2, L3 = SH::L3, W = SH::W;
    constexpr bool kTopDown = KIND == kSweepDown || KIND == kSweepUpAdj;
    constexpr bool kAdj = KIND == kSweepDownAdj || KIND == kSweepUpAdj;
    constexpr float sgn = KIND == kSweepUp || KIND == kSweepUpAdj ? 1.0f : -1.0f;
    __shared__ SH sh;
    __shared__ int s_tk[2];  // in turn: the next ticket may be written while this one is being read
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool in = tid < L3;
    const int l = in ? tid : L3 - 1;  // threads past the last label repeat it and write nothing
    const int ly = l % LEN, lx = (l / LEN) % LEN, lz = l / L2;
    const int by = l - ly, bx = l - lx * LEN, bz = l - lz * L2;
    const float itau = t.itau;
    for (int turn = 0;; turn ^= 1) {
        if (tid == 0) s_tk[turn] = atomicAdd(st.ticket, 1);
        block_sync();
        const int tk = s_tk[turn];
        if (tk >= t.sz) break;
        const int c = ordered[kTopDown ? tk : t.sz - 1 - tk];
        const bool root = c == t.root;
        const int64_t row = (int64_t)c * L3 + l;

        // ---- before the wait: what earlier sweeps left
        const int p = root ? c : t.parents[c];
        const float e = root ? 0.0f : t.edgemst[c];
        const float oy = edge_off(t, c, 0), ox = edge_off(t, c, 1), oz = edge_off(t, c, 2);
        NodePre pre;
        pre.nch = 0;
        float v0 = 0.0f, v1 = 0.0f;      // own values
        float wy[LEN], wx[LEN], wz[LEN];  // adjoint weights
        float gu = 0.0f, gv = 0.0f, gw = 0.0f;
        if (KIND == kSweepUp) {
            v0 = a.cost[row];
            load_children(t, c, pre);
        } else if (KIND == kSweepDown) {
            if (!root) v0 = a.M[row];
            v1 = a.B[row];
        } else if (KIND == kSweepDownAdj) {
            v0 = a.logp[row];
            load_children(t, c, pre);
            gu = a.gdisp[c];
            gv = a.gdisp[t.sz + c];
            gw = a.gdisp[2 * t.sz + c];
        } else if (!root) {
            v0 = a.R[row];
            v1 = a.Bpart[row];
        }
        if (kAdj && !root) {
            const float r = KIND == kSweepDownAdj ? a.logp[(int64_t)p * L3 + l] + a.M[row] * itau
                                                  : __fmul_rn(-e * a.B[row], itau);
            if (in) sh.x[tid] = r;
            block_sync();
            const float t1 = lse_line<LEN, 1>(sh.x + by, ly, itau, sgn, oy);
            if (in) sh.y[tid] = t1;
            block_sync();
            const float t2 = lse_line<LEN, LEN>(sh.y + bx, lx, itau, sgn, ox);
            if (in) sh.z[tid] = t2;
            block_sync();
            const float t3 = lse_line<LEN, L2>(sh.z + bz, lz, itau, sgn, oz);
            if (in) sh.w[tid] = t3;
            block_sync();
            adj_weights<LEN, L2>(wz, t2, sh.w + bz, lz, itau, sgn, oz);
            adj_weights<LEN, LEN>(wx, t1, sh.z + bx, lx, itau, sgn, ox);
            adj_weights<LEN, 1>(wy, r, sh.y + by, ly, itau, sgn, oy);
        }
        // ---- what others wait for
        float dof[3] = {0.0f, 0.0f, 0.0f};  // y, x, z
        float pl = 0.0f;                    // this label's probability (down)
        if (KIND == kSweepUp) {
            const float v = wait_children(t, c, pre, l, v0, a.M, a.Mmin, st.err);
            if (in) sh.x[tid] = v;
            const float bmin = -all_max<W>(-v, sh.red[0]);
            if (in) a.B[row] = v - bmin;
            if (!root) {
                float f[LEN];
#pragma unroll
                for (int i = 0; i < LEN; i++) f[i] = __fmul_rn(-e * (sh.x[by + i] - bmin), itau);
                const float t1 = lse_values<LEN>(f, ly, itau, sgn, oy);
                if (in) sh.y[tid] = t1;
                block_sync();
                const float t2 = lse_line<LEN, LEN>(sh.y + bx, lx, itau, sgn, ox);
                if (in) sh.z[tid] = t2;
                block_sync();
                const float msg = -t.tau * lse_line<LEN, L2>(sh.z + bz, lz, itau, sgn, oz);
                if (in) st_word(a.M + row, msg);
                const float mn = -warp_max(-msg);
                if (lane == 0) sh.red[1][warp] = mn;
            }
        } else if (KIND == kSweepDown) {
            float r;
            if (root) {
                r = -v1 * itau;
            } else {
                const float x = wait_word(a.logp + (int64_t)p * L3 + l, st.err) + v0 * itau;
                if (in) sh.x[tid] = x;
                block_sync();
                const float t1 = lse_line<LEN, 1>(sh.x + by, ly, itau, sgn, oy);
                if (in) sh.y[tid] = t1;
                block_sync();
                const float t2 = lse_line<LEN, LEN>(sh.y + bx, lx, itau, sgn, ox);
                if (in) sh.z[tid] = t2;
                block_sync();
                r = lse_line<LEN, L2>(sh.z + bz, lz, itau, sgn, oz) - e * v1 * itau;
            }
            const float lp = r - all_lse<W>(in ? r : -INFINITY, in ? 1.0f : 0.0f, sh.red[0], sh.red[1]);
            if (in) st_word(a.logp + row, lp);
            pl = in ? __expf(lp) : 0.0f;
        } else if (KIND == kSweepDownAdj) {
            const float du = (float)((lx - t.hw) * t.q), dv = (float)((ly - t.hw) * t.q), dw = (float)((lz - t.hw) * t.q);
            const float pc = __expf(v0);
            const float h = wait_children(t, c, pre, l, (gu * du + gv * dv + gw * dw) * pc, a.R, nullptr, st.err);
            if (root) {
                const float tot = all_sum<W>(in ? h : 0.0f, sh.red[0]);
                const float b = -(h - pc * tot) * itau;
                const float mean = all_sum<W>(in ? b : 0.0f, sh.red[1]) / (float)L3;
                if (in) a.Bbar[row] = b - mean;
            } else {
                if (in) {
                    sh.x[tid] = h;
                    a.Bpart[row] = -e * itau * h;
                }
                block_sync();
                const float gz = adj_line<LEN, L2>(wz, sh.x + bz, lz, sgn, oz, t.offbar, dof[2]);
                if (in) sh.y[tid] = gz;
                block_sync();
                const float gx = adj_line<LEN, LEN>(wx, sh.y + bx, lx, sgn, ox, t.offbar, dof[1]);
                if (in) sh.z[tid] = gx;
                block_sync();
                const float gy = adj_line<LEN, 1>(wy, sh.z + by, ly, sgn, oy, t.offbar, dof[0]);
                if (in) st_word(a.R + row, gy);
            }
        } else if (!root) {
            const float x = v0 * itau + wait_word(a.Bbar + (int64_t)p * L3 + l, st.err);
            if (in) sh.x[tid] = x;
            block_sync();
            const float gz = adj_line<LEN, L2>(wz, sh.x + bz, lz, sgn, oz, t.offbar, dof[2]);
            if (in) sh.y[tid] = gz;
            block_sync();
            const float gx = adj_line<LEN, LEN>(wx, sh.y + bx, lx, sgn, ox, t.offbar, dof[1]);
            if (in) sh.z[tid] = gx;
            block_sync();
            const float gy = adj_line<LEN, 1>(wy, sh.z + by, ly, sgn, oy, t.offbar, dof[0]);
            const float b = v1 + e * gy;
            const float mean = all_sum<W>(in ? b : 0.0f, sh.red[0]) / (float)L3;
            if (in) st_word(a.Bbar + row, b - mean);
        }
        if (KIND == kSweepUp && !root) {
            block_sync();
            if (tid == 0) {
                float mn = sh.red[1][0];
#pragma unroll
                for (int w = 1; w < W; w++) mn = fminf(mn, sh.red[1][w]);
                st_word(a.Mmin + c, mn);
            }
        }

        // ---- sums that no other node reads
        if (KIND == kSweepDown || (kAdj && t.offbar && !root)) {
            float s0, s1, s2;  // x, y, z
            if (KIND == kSweepDown) {
                s0 = pl * (float)((lx - t.hw) * t.q);
                s1 = pl * (float)((ly - t.hw) * t.q);
                s2 = pl * (float)((lz - t.hw) * t.q);
            } else {
                // M = -tau out in the upward recursion: its offset gradient scales by -tau
                const float scale = -2.0f * itau * (KIND == kSweepUpAdj ? -t.tau : 1.0f);
                s0 = in ? scale * dof[1] : 0.0f;
                s1 = in ? scale * dof[0] : 0.0f;
                s2 = in ? scale * dof[2] : 0.0f;
            }
            s0 = warp_add(s0);
            s1 = warp_add(s1);
            s2 = warp_add(s2);
            if (lane == 0) {
                sh.red[2][warp] = s0;
                sh.red[3][warp] = s1;
                sh.red[4][warp] = s2;
            }
            block_sync();
            if (tid < 3) {
                float s = 0.0f;
                for (int w = 0; w < W; w++) s += sh.red[2 + tid][w];
                if (KIND == kSweepDown) a.disp[(int64_t)tid * t.sz + c] = s;
                else t.offbar[(int64_t)tid * t.sz + c] += s;
            }
        }
    }
}

int soft_threads(int len) { return len * len * len <= 343 ? 128 : 256; }

// one thread per label (rounded to whole warps): the per-node passes are latency bound
int tree_threads(int len) { return std::min(1024, (len * len * len + 31) / 32 * 32); }

SoftGeom make_geom(int m, int n, int o, int g, int hw, int q, float alpha1, float eps) {
    SoftGeom G;
    G.m = m; G.n = n; G.o = o; G.g = g; G.hw = hw; G.q = q;
    G.len = 2 * hw + 1; G.len3 = G.len * G.len * G.len;
    G.m1 = m / g; G.n1 = n / g; G.o1 = o / g;
    G.S = g > 4 ? 2 : 1;
    G.nx = (g + G.S - 1) / G.S;
    G.nsamp = G.nx * G.nx * g;
    G.alpha1 = alpha1;
    G.eps = eps;
    return G;
}

SoftTree make_tree(const SoftTreeDev& d) {
    SoftTree t;
    t.len = d.len; t.len3 = d.len * d.len * d.len; t.hw = (d.len - 1) / 2; t.sz = d.sz; t.root = d.root;
    t.q = d.q; t.tau = d.tau; t.itau = 1.0f / d.tau;
    t.parents = d.parents; t.edgemst = d.edgemst; t.child_ptr = d.child_ptr; t.children = d.children;
    t.off = d.off; t.offbar = d.offbar;
    return t;
}

}  // namespace

// off (x|y|z) of node c's edge = (prior[parent] - prior[c]) / q; the root has none
__global__ void k_soft_offsets(const float* __restrict__ prior, const int* __restrict__ parents, int root, int sz,
                               float q, float* __restrict__ off) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= sz) return;
    const int p = c == root ? c : parents[c];
#pragma unroll
    for (int a = 0; a < 3; a++) off[a * sz + c] = (prior[a * sz + p] - prior[a * sz + c]) / q;
}

// dL/dprior from dL/doff: each edge's offset depends on its two end nodes
__global__ void k_soft_offbar_to_prior(const float* __restrict__ offbar, const int* __restrict__ parents, int root,
                                       int sz, float q, float* __restrict__ gprior) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= sz || c == root) return;
    const int p = parents[c];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const float g = offbar[a * sz + c] / q;
        atomicAdd(gprior + a * sz + p, g);
        atomicAdd(gprior + a * sz + c, -g);
    }
}

// ---------------------------------------------------------------------------
// Host drivers

// The windowed sums of six channels into b: of the channels in a, or with an image of its
// squared differences (a is scratch for radii above 3).  Counts its launches.
static void box3(const float* image, float* a, float* b, int m, int n, int o, int r, cudaStream_t st) {
    const dim3 blk3(blocks_for(m, 32), blocks_for(n, 8), 6 * blocks_for(o, kBoxPlanes));
    switch (image ? -r : r) {
        case -1: k_soft_box3<1, true><<<blk3, 256, 0, st>>>(image, b, m, n, o, r); count_launches(1); return;
        case -2: k_soft_box3<2, true><<<blk3, 256, 0, st>>>(image, b, m, n, o, r); count_launches(1); return;
        case -3: k_soft_box3<3, true><<<blk3, 256, 0, st>>>(image, b, m, n, o, r); count_launches(1); return;
        case 1: k_soft_box3<1, false><<<blk3, 256, 0, st>>>(a, b, m, n, o, r); count_launches(1); return;
        case 2: k_soft_box3<2, false><<<blk3, 256, 0, st>>>(a, b, m, n, o, r); count_launches(1); return;
        case 3: k_soft_box3<3, false><<<blk3, 256, 0, st>>>(a, b, m, n, o, r); count_launches(1); return;
        default: break;
    }
    if (image) {
        const int64_t sz = (int64_t)m * n * o;
        k_soft_sqdiff<<<blocks_for(sz, 256), 256, 0, st>>>(image, a, m, n, o, r);
        count_launches(1);
    }
    const dim3 blk(32, 8), grid(blocks_for(m, 32), blocks_for(n, 8), 6 * o);
    k_soft_box<<<grid, blk, 0, st>>>(a, b, m, n, o, r, 0);
    k_soft_box<<<grid, blk, 0, st>>>(b, a, m, n, o, r, 1);
    k_soft_box<<<grid, blk, 0, st>>>(a, b, m, n, o, r, 2);
    count_launches(3);
}

cudaError_t launch_soft_offsets(const float* prior, const int* parents, int root, int sz, float q, float* off,
                                cudaStream_t st) {
    k_soft_offsets<<<blocks_for(sz, 256), 256, 0, st>>>(prior, parents, root, sz, q, off);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_soft_offbar_to_prior(const float* offbar, const int* parents, int root, int sz, float q,
                                        float* gprior, cudaStream_t st) {
    k_soft_offbar_to_prior<<<blocks_for(sz, 256), 256, 0, st>>>(offbar, parents, root, sz, q, gprior);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_soft_descriptor(const float* d_im, float* w6a, float* w6b, float* s12, int m, int n, int o, int qs,
                                   cudaStream_t st) {
    const int64_t sz = (int64_t)m * n * o;
    box3(d_im, w6a, w6b, m, n, o, qs, st);
    k_soft_desc<<<blocks_for(sz, 256), 256, 0, st>>>(w6b, s12, m, n, o, qs);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_soft_descriptor_adj(const float* d_im, float* w6a, float* w6b, const float* sbar12, float* dbar6,
                                       float* imbar, int m, int n, int o, int qs, cudaStream_t st) {
    const int64_t sz = (int64_t)m * n * o;
    box3(d_im, w6a, w6b, m, n, o, qs, st);
    cudaError_t err = cudaMemsetAsync(dbar6, 0, sizeof(float) * 6 * sz, st);
    if (err != cudaSuccess) return err;
    k_soft_desc_adj<<<blocks_for(sz, 256), 256, 0, st>>>(w6b, sbar12, dbar6, m, n, o, qs);
    box3(nullptr, dbar6, w6b, m, n, o, qs, st);  // adjoint of the box filter: the same operator
    k_soft_sqdiff_adj<<<blocks_for(sz, 256), 256, 0, st>>>(d_im, w6b, imbar, m, n, o, qs);
    count_launches(2);
    return cudaGetLastError();
}

// Channels per halo stage so that the kernel's shared memory stays within ~110 KB
// (two CTAs per SM); 0 when even one channel does not fit (generic kernels).
static int halo_channels(const SoftGeom& G, int H3max, int arrays, size_t extra_bytes) {
    static const int cands[6] = {12, 6, 4, 3, 2, 1};
    for (int c : cands)
        if ((size_t)arrays * c * H3max * sizeof(float) + extra_bytes + (arrays == 1 ? (size_t)c * G.nsamp * 4 : 0) <=
            110 * 1024)
            return c;
    return 0;
}

static int halo_h3max(const SoftGeom& G) {
    const int R = G.hw * G.q;
    return std::min(G.g + 2 * R, G.m) * std::min(G.g + 2 * R, G.n) * std::min(G.g + 2 * R, G.o);
}

// Column kernels are instantiated for the finest-level shapes (grid 4, quant 1,
// label widths 5/7/9); other shapes use the generic halo kernels.
template <int G_, int LEN_, int Q_>
static cudaError_t run_cost_col(const SoftGeom& G, const float* sF, const float* sM, float* cost, cudaStream_t st) {
    using CGm = ColGeom<G_, LEN_, Q_>;
    const size_t smem = sizeof(float) * (12 * (size_t)CGm::NA3 + 12 * CGm::NSAMP + CGm::LEN3);
    if (smem > 200 * 1024) return cudaErrorNotSupported;
    cudaError_t e = cudaFuncSetAttribute(k_soft_cost_col<G_, LEN_, Q_>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    k_soft_cost_col<G_, LEN_, Q_><<<G.m1 * G.n1 * G.o1, CGm::FWD_BLOCK, smem, st>>>(sF, sM, cost, G);
    return cudaSuccess;
}

template <int LEN_, int Q_>
static cudaError_t run_cost_adj_col(const SoftGeom& G, const float* sF, const float* sM, const float* cbar,
                                    const float* cost, float* sFbar, float* sMbar, double* dot, cudaStream_t st) {
    constexpr size_t smem = AdjGeom<LEN_, Q_>::SMEM;
    static_assert(smem <= 200 * 1024, "fits an SM");
    cudaError_t e = cudaFuncSetAttribute(k_soft_cost_adj_col<LEN_, Q_>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    k_soft_cost_adj_col<LEN_, Q_><<<2 * G.m1 * G.n1 * G.o1, 96, smem, st>>>(sF, sM, cbar, cost, sFbar, sMbar, dot, G);
    return cudaSuccess;
}

// Channels per stage of the row kernels: as many as fit in 64 KB of rows.
template <int G_, int LEN_, int Q_>
static RowPlan row_plan() {
    using RG = RowGeom<G_, LEN_, Q_>;
    static const int cands[6] = {12, 6, 4, 3, 2, 1};
    RowPlan P{RG::PY, 1};
    for (int c : cands)
        if ((size_t)c * RG::ITEMS * RG::PY * sizeof(float) <= 64 * 1024) { P.CG = c; break; }
    return P;
}

template <int G_, int LEN_, int Q_>
static cudaError_t run_cost_rows(const SoftGeom& G, const float* sF, const float* sM, float* cost, cudaStream_t st) {
    using RG = RowGeom<G_, LEN_, Q_>;
    const RowPlan P = row_plan<G_, LEN_, Q_>();
    const size_t smem = sizeof(float) * ((size_t)P.CG * RG::ITEMS * RG::PY + 12 * RG::NSAMP + RG::LEN3) +
                        sizeof(int) * RG::ITEMS;
    cudaError_t e = cudaFuncSetAttribute(k_soft_cost_rows<G_, LEN_, Q_>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    k_soft_cost_rows<G_, LEN_, Q_><<<G.m1 * G.n1 * G.o1, RG::BLOCK, smem, st>>>(sF, sM, cost, G, P);
    return cudaSuccess;
}

template <int G_, int LEN_, int Q_>
static cudaError_t run_cost_adjF_rows(const SoftGeom& G, const float* sF, const float* sM, const float* cbar,
                                      const float* cost, float* sFbar, double* dot, cudaStream_t st) {
    using RG = RowGeom<G_, LEN_, Q_>;
    const RowPlan P = row_plan<G_, LEN_, Q_>();
    const size_t smem = sizeof(float) * ((size_t)P.CG * RG::ITEMS * RG::PY + 24 * RG::NSAMP + RG::LEN3) +
                        sizeof(int) * RG::ITEMS;
    cudaError_t e = cudaFuncSetAttribute(k_soft_cost_adjF_rows<G_, LEN_, Q_>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k_soft_cost_adjF_rows<G_, LEN_, Q_><<<G.m1 * G.n1 * G.o1, RG::BLOCK, smem, st>>>(sF, sM, cbar, cost, sFbar,
                                                                                      dot, G, P);
    return cudaSuccess;
}

// Row kernels are instantiated for the coarse soft levels in use (grid 6 / quant
// 3 or 2, grid 5 / quant 2, label widths 5 and 7).  Every item stages its own
// row; where two items of a node read the same row (quant 2: x offsets 2jj + 2lx
// repeat) that row is simply staged twice.
static int row_shape(const SoftGeom& G) {
    if (G.len != 5 && G.len != 7) return 0;
    if (G.g == 6 && G.q == 3) return 60 + G.len;
    if (G.g == 6 && G.q == 2) return 600 + G.len;
    if (G.g == 5 && G.q == 2) return 50 + G.len;
    return 0;
}

#define DEEDS_ROW_CASES(FN, ...)                                                   \
    case 65: e = FN<6, 5, 3>(__VA_ARGS__); break;                                  \
    case 67: e = FN<6, 7, 3>(__VA_ARGS__); break;                                  \
    case 605: e = FN<6, 5, 2>(__VA_ARGS__); break;                                 \
    case 607: e = FN<6, 7, 2>(__VA_ARGS__); break;                                 \
    case 55: e = FN<5, 5, 2>(__VA_ARGS__); break;                                  \
    case 57: e = FN<5, 7, 2>(__VA_ARGS__); break;

static int col_shape(const SoftGeom& G) {
    if (G.g != 4 || G.q != 1) return 0;
    return G.len == 5 || G.len == 7 || G.len == 9 ? G.len : 0;
}

cudaError_t launch_soft_cost(const float* sF, const float* sM, float* cost, int m, int n, int o, int g, int hw, int q,
                             float alpha1, float eps, cudaStream_t st) {
    const SoftGeom G = make_geom(m, n, o, g, hw, q, alpha1, eps);
    const int H3max = halo_h3max(G);
    {
        cudaError_t e = cudaErrorNotSupported;
        switch (col_shape(G)) {
            case 5: e = run_cost_col<4, 5, 1>(G, sF, sM, cost, st); break;
            case 7: e = run_cost_col<4, 7, 1>(G, sF, sM, cost, st); break;
            case 9: e = run_cost_col<4, 9, 1>(G, sF, sM, cost, st); break;
            default: break;
        }
        if (e == cudaSuccess) {
            count_launches(1);
            return cudaGetLastError();
        }
        if (e != cudaErrorNotSupported) return e;
    }
    if (const int rs = row_shape(G)) {
        cudaError_t e = cudaErrorNotSupported;
        switch (rs) { DEEDS_ROW_CASES(run_cost_rows, G, sF, sM, cost, st) default: break; }
        if (e != cudaSuccess) return e;
        count_launches(1);
        return cudaGetLastError();
    }
    const size_t extra = sizeof(int) * (size_t)(G.len3 + G.nsamp);
    const int CG = G.len3 <= kHaloLPT * 512 ? halo_channels(G, H3max, 1, extra) : 0;
    if (CG > 0) {
        const size_t smem = sizeof(float) * ((size_t)CG * H3max + (size_t)CG * G.nsamp) + extra;
        cudaError_t e = cudaFuncSetAttribute(k_soft_cost_halo, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        const int threads = std::min(512, (G.len3 + 31) / 32 * 32);
        k_soft_cost_halo<<<G.m1 * G.n1 * G.o1, threads, smem, st>>>(sF, sM, cost, G, CG, H3max);
    } else {
        k_soft_cost<<<G.m1 * G.n1 * G.o1, soft_threads(G.len), sizeof(float) * G.nsamp * 12, st>>>(sF, sM, cost, G);
    }
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_soft_cost_adj(const float* sF, const float* sM, const float* cbar, const float* cost, float* sFbar,
                                 float* sMbar, double* dot, int m, int n, int o, int g, int hw, int q, float alpha1,
                                 float eps, cudaStream_t st) {
    const SoftGeom G = make_geom(m, n, o, g, hw, q, alpha1, eps);
    const int64_t sz = (int64_t)m * n * o;
    cudaError_t err = cudaMemsetAsync(sFbar, 0, sizeof(float) * 12 * sz, st);
    if (err == cudaSuccess) err = cudaMemsetAsync(dot, 0, sizeof(double), st);
    if (err != cudaSuccess) return err;
    if (const int rs = row_shape(G)) {  // fixed side in row form, moving side as a gather (no atomics)
        cudaError_t e = cudaErrorNotSupported;
        switch (rs) { DEEDS_ROW_CASES(run_cost_adjF_rows, G, sF, sM, cbar, cost, sFbar, dot, st) default: break; }
        if (e != cudaSuccess) return e;
        switch (rs) { DEEDS_ROW_CASES(run_adj_moving_t, G, sF, sM, cbar, sMbar, st) default: break; }
        if (e != cudaSuccess) return e;
        count_launches(2);
        return cudaGetLastError();
    }
    const int H3max = halo_h3max(G);
    const size_t extra = sizeof(float) * (size_t)G.len3 + sizeof(int) * (size_t)(G.len3 + G.nsamp);
    const int CG = halo_channels(G, H3max, 2, extra);
    if (col_shape(G) || CG > 0) {
        err = cudaMemsetAsync(sMbar, 0, sizeof(float) * 12 * sz, st);
        if (err != cudaSuccess) return err;
    }
    {
        cudaError_t e = cudaErrorNotSupported;
        switch (col_shape(G)) {
            case 5: e = run_cost_adj_col<5, 1>(G, sF, sM, cbar, cost, sFbar, sMbar, dot, st); break;
            case 7: e = run_cost_adj_col<7, 1>(G, sF, sM, cbar, cost, sFbar, sMbar, dot, st); break;
            case 9: e = run_cost_adj_col<9, 1>(G, sF, sM, cbar, cost, sFbar, sMbar, dot, st); break;
            default: break;
        }
        if (e == cudaSuccess) {
            count_launches(1);
            return cudaGetLastError();
        }
        if (e != cudaErrorNotSupported) return e;
    }
    if (CG > 0) {
        const size_t smem = sizeof(float) * 2 * (size_t)CG * H3max + extra;
        err = cudaFuncSetAttribute(k_soft_cost_adj_halo, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (err != cudaSuccess) return err;
        k_soft_cost_adj_halo<<<G.m1 * G.n1 * G.o1, 256, smem, st>>>(sF, sM, cbar, cost, sFbar, sMbar, dot, G, CG,
                                                                     H3max);
        count_launches(1);
    } else {
        k_soft_cost_adj_fixed<<<G.m1 * G.n1 * G.o1, 256, 0, st>>>(sF, sM, cbar, cost, sFbar, dot, G);
        k_soft_cost_adj_moving<<<blocks_for(sz, 128), 128, 0, st>>>(sF, sM, cbar, sMbar, G);
        count_launches(2);
    }
    return cudaGetLastError();
}

// Resident sweep CTAs per SM.  A sweep is bound by the latency along the
// deepest root-leaf path (hundreds of nodes at grid 4), and most of its CTAs wait;
// two per SM keep the sweep as fast as a full grid (measured 1-2 % faster at
// 160x160x192, label set 7^3) and leave the rest of each SM to kernels of other
// pairs running on other streams.
constexpr int kSweepCtasPerSm = 2;

// the widths of k_sweep
bool soft_tree_needs_bpart(int len) { return len <= 9; }
size_t soft_tree_smem(int len) { return sizeof(float) * (6 * (size_t)len * len * len + 96); }

template <int KIND>
static cudaError_t run_sweep(const SoftTree& t, const int* ordered, const SweepArgs& a, const SweepState& st,
                             int* sweep_mem, cudaStream_t s) {
    const int threads = tree_threads(t.len);
    size_t smem = 0, flags = 0;
    void (*kern)(SoftTree, const int*, SweepArgs, SweepState) = nullptr;
    if (t.len == 3) kern = k_sweep<KIND, 3>;
    else if (t.len == 5) kern = k_sweep<KIND, 5>;
    else if (t.len == 7) kern = k_sweep<KIND, 7>;
    else if (t.len == 9) kern = k_sweep<KIND, 9>;
    else {
        kern = k_soft_sweep<KIND>;
        smem = sizeof(float) * ((KIND == kSweepUp || KIND == kSweepDown ? 3 : 6) * (size_t)t.len3 + 96);
        flags = t.sz;
    }
    cudaError_t e;
    if (smem && (e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess)
        return e;
    int dev = 0, sms = 0, per_sm = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem)) != cudaSuccess) return e;
    per_sm = std::min(per_sm, kSweepCtasPerSm);
    const int grid = std::max(1, std::min(t.sz, sms * std::max(per_sm, 1)));
    // the ticket, and the general form's per-node flags, start at zero (the error word is
    // cleared by the caller); the rows that a sweep waits for start as kNotYet
    if ((e = cudaMemsetAsync(sweep_mem, 0, sizeof(int) * (flags + 1), s)) != cudaSuccess) return e;
    if (!flags) {
        const size_t rows = sizeof(float) * (size_t)t.sz * t.len3;
        if (KIND == kSweepUp) {
            if ((e = cudaMemsetAsync(a.M, 0xff, rows, s)) != cudaSuccess) return e;
            if ((e = cudaMemsetAsync(a.Mmin, 0xff, sizeof(float) * t.sz, s)) != cudaSuccess) return e;
        } else if (KIND == kSweepDown) {
            if ((e = cudaMemsetAsync(a.logp, 0xff, rows, s)) != cudaSuccess) return e;
        } else if (KIND == kSweepDownAdj) {
            if ((e = cudaMemsetAsync(a.R, 0xff, rows, s)) != cudaSuccess) return e;
            if ((e = cudaMemsetAsync(a.Bbar, 0xff, rows, s)) != cudaSuccess) return e;
        }
    }
    kern<<<grid, threads, smem, s>>>(t, ordered, a, st);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_soft_tree_forward(const SoftTreeDev& d, int* sweep_mem, const float* cost, float* B, float* M,
                                     float* Mmin, float* logp, float* disp, cudaStream_t s) {
    const SoftTree t = make_tree(d);
    SweepArgs a{cost, B, M, Mmin, logp, disp, nullptr, nullptr, nullptr, nullptr};
    const SweepState st{sweep_mem, sweep_mem + 1, sweep_mem + t.sz + 1};
    cudaError_t e = run_sweep<kSweepUp>(t, d.ordered, a, st, sweep_mem, s);
    if (e == cudaSuccess) e = run_sweep<kSweepDown>(t, d.ordered, a, st, sweep_mem, s);
    return e;
}

cudaError_t launch_soft_tree_backward(const SoftTreeDev& d, int* sweep_mem, const float* B, const float* M,
                                      const float* logp, const float* gdisp, float* R, float* Bbar, float* Bpart,
                                      cudaStream_t s) {
    const SoftTree t = make_tree(d);
    SweepArgs a{nullptr, const_cast<float*>(B), const_cast<float*>(M), nullptr, const_cast<float*>(logp), nullptr,
                gdisp, R, Bbar, Bpart};
    const SweepState st{sweep_mem, sweep_mem + 1, sweep_mem + t.sz + 1};
    cudaError_t e = run_sweep<kSweepDownAdj>(t, d.ordered, a, st, sweep_mem, s);
    if (e == cudaSuccess) e = run_sweep<kSweepUpAdj>(t, d.ordered, a, st, sweep_mem, s);
    return e;
}

// Self-test of the sweeps' bounded wait: one thread waits on a flag that nothing
// sets; status = 1 if the wait gave up and set the error word, 2 otherwise.
__global__ void k_selftest_flag_wait(const int* flag, int* err, int* status) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *status = bounded_wait_geq(flag, 1, err) ? 2 : 1;
}

cudaError_t launch_selftest_flag_wait(const int* flag, int* err, int* status, cudaStream_t s) {
    k_selftest_flag_wait<<<1, 32, 0, s>>>(flag, err, status);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace deeds
