// Field and image transforms on sm_103a (replaces upsampleDeformationsCL,
// interp3, warpAffine, warpImageCL, warpAffineS, consistentMappingCL and jacobian;
// src/transformations.h:5-279, src/dataCostD.h:213-315).
//
// The full-resolution field is never materialised on the hot path: a warp kernel
// evaluates upsampleDeformationsCL's trilinear grid interpolation for its own
// voxel (identical arithmetic) and immediately warps the image.  Interpolation
// weights are evaluated in FP64 exactly where the reference's C++ promotes to
// double (see common.cuh).  The blends run in float-float first and take the
// double evaluation only where the float-float value cannot prove the
// reference's rounding (ff_blend8): GB300's FP64 rate would otherwise bound
// these kernels (~80 DP operations per voxel for field + image).  Roofline: per
// voxel 4 B image gather (L2) + 4 B write; the grid field is L2-resident.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace deeds {

namespace {

struct Grid3 {
    const float* u;
    const float* v;
    const float* w;
    int m, n, o;
    float sm, sn, so;  // (float)full / (float)grid per axis
};

// upsampleDeformationsCL at voxel (i,j,k) of the full-resolution grid
// (src/transformations.h:248-267): coordinate index/scale, floor, trilinear.
__device__ __forceinline__ void upsample_at(const Grid3& g, int i, int j, int k, float& u, float& v, float& w) {
    int x, y, z;
    float dx, dy, dz;
    split_coord(__fdiv_rn((float)j, g.sn), x, dx);
    split_coord(__fdiv_rn((float)i, g.sm), y, dy);
    split_coord(__fdiv_rn((float)k, g.so), z, dz);
    const Corners c = corners(y, x, z, g.m, g.n, g.o);
    const FFWeights b = ff_weights(dx, dy, dz);
    u = sample_ff(g.u, c, b, dx, dy, dz);
    v = sample_ff(g.v, c, b, dx, dy, dz);
    w = sample_ff(g.w, c, b, dx, dy, dz);
}

struct Affine12 {
    float x[12];
};

__global__ void k_shift(const float* __restrict__ in, float* __restrict__ out, int64_t n, float neg_shift) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < n) out[p] = __fsub_rn(in[p], neg_shift);
}

// ---- The grid field along rows (j, k) of voxels, staged per block
//
// The voxels of a row share x, z and their fractions, so the blend of upsample_at
// factors over the nodes y of the row.  With c(y, x, z) a corner and
//   Q[y] = (1-dx)(1-dz) c(y,x0,z0) + (1-dx) dz c(y,x0,z1),
//   P[y] = Q[y] + dx (1-dz) c(y,x1,z0) + dx dz c(y,x1,z1),   R[y] = (1-dz) c(y,x1,z0)
// (float-float, once per node and component) a voxel's value is
//   (1-dy) P[y0] + dy Q[y1] + fl(dx dy) R[y1] + fl(fl(fl(dx dy) dz) c(y1,x1,z1)),
// the same exact expression as blend8_apply's: three float-float products and sums a
// component in place of eight.  The errors stay below ff_blend8's 2^-40 S (fewer steps
// of the same size), so the same proof decides.
//
// Where it cannot, the value usually is a tie: at fractions that are multiples of 2^-3
// every term is a multiple of U = 2^(e - 32), e the smallest exponent among the non-zero
// corners, and with no corner above 2^10 times that all sums stay below 2^46 U.  Every
// high part is then rounded to at least 2^-24 of its value and every low part is a
// multiple of U below 2^24 U, so all float-float steps are exact, the reference's
// double evaluation is exact too, and the sum rounded once is its result.  Anything
// else goes to blend8_exact.
// Bound: FP32 issue.  Upsampling grid 4 / 5 / 8 to 192x160x256: 1282 / 243 / 619 us with
// eight-term blends and FP64 at the ties, 397 / 201 / 286 us with one row and one voxel a
// thread, 192 / 189 / 168 us with four rows a block and three voxels a thread.
constexpr int kRowThreads = 64;  // threads per row: three voxels each at 192, which share a row's weights

struct RowStage {
    float4* pn;     // [3][g.m]: P.hi, P.lo, S (sum of |corner|, +0 only if all four are +0), c(y,x1,z1)
    float4* qr;     // [3][g.m]: Q.hi, Q.lo, R.hi, R.lo
    uint32_t* ex;   // [3][g.m]: smallest exponent of a non-zero corner | largest << 8
    int x, z;
    float dx, dz;
    bool dyadic;    // dx and dz multiples of 2^-3
};

__device__ __forceinline__ bool eighths(float f) { return f * 8.0f == rintf(f * 8.0f); }
constexpr size_t kRowBytes = 3 * (2 * sizeof(float4) + sizeof(uint32_t));  // per node

__device__ __forceinline__ RowStage stage_row(const Grid3& g, int j, int k, char* smem) {
    RowStage r;
    r.pn = reinterpret_cast<float4*>(smem + (size_t)threadIdx.y * ((kRowBytes * g.m + 15) & ~(size_t)15));
    r.qr = r.pn + 3 * g.m;
    r.ex = reinterpret_cast<uint32_t*>(r.qr + 3 * g.m);
    split_coord(__fdiv_rn((float)j, g.sn), r.x, r.dx);
    split_coord(__fdiv_rn((float)k, g.so), r.z, r.dz);
    r.dyadic = eighths(r.dx) && eighths(r.dz);
    const int x0 = clampi(r.x, 0, g.n - 1), x1 = clampi(r.x + 1, 0, g.n - 1);
    const int z0 = clampi(r.z, 0, g.o - 1), z1 = clampi(r.z + 1, 0, g.o - 1);
    const int64_t mn = (int64_t)g.m * g.n;
    const int64_t o00 = (int64_t)x0 * g.m + z0 * mn, o10 = (int64_t)x1 * g.m + z0 * mn, o01 = (int64_t)x0 * g.m + z1 * mn,
                  o11 = (int64_t)x1 * g.m + z1 * mn;
    const FF a = ff_two_sum(1.0f, -r.dx), c = ff_two_sum(1.0f, -r.dz);
    const FF wa = ff_mul(a, c), wb = ff_mul_f(c, r.dx), wc = ff_mul_f(a, r.dz), wd = ff_prod(r.dx, r.dz);
    for (int y = threadIdx.x; y < g.m; y += kRowThreads) {
#pragma unroll
        for (int comp = 0; comp < 3; comp++) {
            const float* v = (comp == 0 ? g.u : comp == 1 ? g.v : g.w) + y;
            const float c00 = __ldg(v + o00), c10 = __ldg(v + o10), c01 = __ldg(v + o01), c11 = __ldg(v + o11);
            const FF q = ff_add(ff_mul_f(wa, c00), ff_mul_f(wc, c01));
            const FF p = ff_add(ff_add(q, ff_mul_f(wb, c10)), ff_mul_f(wd, c11));
            const FF rr = ff_mul_f(c, c10);
            const uint32_t b[4] = {__float_as_uint(c00), __float_as_uint(c10), __float_as_uint(c01), __float_as_uint(c11)};
            float S = fabsf(c00) + fabsf(c10) + fabsf(c01) + fabsf(c11);
            if (S == 0.0f && (b[0] | b[1] | b[2] | b[3])) S = __int_as_float(0x7fc00000);  // a -0: blend8_exact decides
            uint32_t lo = 255u, hi = 0u;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t e = (b[i] >> 23) & 255u;
                lo = (b[i] & 0x7fffffffu) ? min(lo, e) : lo;
                hi = max(hi, e);
            }
            r.pn[comp * g.m + y] = make_float4(p.hi, p.lo, S, c11);
            r.qr[comp * g.m + y] = make_float4(q.hi, q.lo, rr.hi, rr.lo);
            r.ex[comp * g.m + y] = lo | hi << 8;
        }
    }
    return r;
}

__device__ __forceinline__ float row_value(const RowStage& r, const Grid3& g, int comp, int y, int y0, int y1, float dy,
                                           FF one_dy, float dxdy, float dxdydz) {
    const float4 p0 = r.pn[comp * g.m + y0], p1 = r.pn[comp * g.m + y1], q1 = r.qr[comp * g.m + y1];
    const float S = p0.z + p1.z;
    if (S >= 0x1p-60f && S <= 0x1p+100f) {
        FF acc = ff_mul(one_dy, FF{p0.x, p0.y});
        acc = ff_add(acc, ff_mul_f(FF{q1.x, q1.y}, dy));
        acc = ff_add(acc, ff_mul_f(FF{q1.z, q1.w}, dxdy));
        acc = ff_add(acc, FF{__fmul_rn(dxdydz, p1.w), 0.0f});
        float out;
        if (ff_round_safe(acc, S * 0x1p-40f, out)) return out;
        if (r.dyadic && eighths(dy) && acc.hi != 0.0f) {
            const uint32_t e0 = r.ex[comp * g.m + y0], e1 = r.ex[comp * g.m + y1];
            const uint32_t lo = min(e0 & 255u, e1 & 255u), hi = max(e0 >> 8, e1 >> 8);
            if (lo >= 64u && hi <= 190u && hi <= lo + 10u) return __fadd_rn(acc.hi, acc.lo);
        }
    } else if (S == 0.0f) {
        return 0.0f;
    }
    const float* v = comp == 0 ? g.u : comp == 1 ? g.v : g.w;
    const Corners c = corners(y, r.x, r.z, g.m, g.n, g.o);
    return blend8_exact(r.dx, dy, r.dz, __ldg(v + c.o000), __ldg(v + c.o100), __ldg(v + c.o010), __ldg(v + c.o001),
                        __ldg(v + c.o110), __ldg(v + c.o101), __ldg(v + c.o011), __ldg(v + c.o111));
}

// Field of voxel (i, j, k): mode 0 zero, 1 full-resolution arrays, 2 grid (eight-term
// blends), 3 grid staged along the row.
template <int MODE>
__device__ __forceinline__ void field_at(const Grid3& g, const RowStage& r, const float* __restrict__ fu,
                                         const float* __restrict__ fv, const float* __restrict__ fw, int i, int j, int k,
                                         int64_t p, float& u, float& v, float& w) {
    u = v = w = 0.0f;
    if (MODE == 1) { u = fu[p]; v = fv[p]; w = fw[p]; }
    if (MODE == 2) upsample_at(g, i, j, k, u, v, w);
    if (MODE == 3) {
        int y;
        float dy;
        split_coord(__fdiv_rn((float)i, g.sm), y, dy);
        const int y0 = clampi(y, 0, g.m - 1), y1 = clampi(y + 1, 0, g.m - 1);
        const FF one_dy = ff_two_sum(1.0f, -dy);
        const float dxdy = r.dx * dy, dxdydz = dxdy * r.dz;
        u = row_value(r, g, 0, y, y0, y1, dy, one_dy, dxdy, dxdydz);
        v = row_value(r, g, 1, y, y0, y1, dy, one_dy, dxdy, dxdydz);
        w = row_value(r, g, 2, y, y0, y1, dy, one_dy, dxdy, dxdydz);
    }
}

// A block covers blockDim.y rows, kRowThreads threads each: body(i, j, k, p) for its voxels.
template <int MODE, class Body>
__device__ __forceinline__ void for_rows(const Grid3& g, int m, int n, Body body) {
    extern __shared__ __align__(16) char s_row[];
    const int j = blockIdx.x * blockDim.y + threadIdx.y, k = blockIdx.y;
    RowStage r{};
    if (MODE == 3) {
        if (j < n) r = stage_row(g, j, k, s_row);
        __syncthreads();
    }
    if (j >= n) return;
    for (int i = threadIdx.x; i < m; i += kRowThreads) body(r, i, j, k, i + (int64_t)j * m + (int64_t)k * m * n);
}

template <int MODE>
__global__ void k_upsample(Grid3 g, float* __restrict__ u, float* __restrict__ v, float* __restrict__ w, int m, int n,
                           int o) {
    for_rows<MODE>(g, m, n, [&](const RowStage& r, int i, int j, int k, int64_t p) {
        float a, b, c;
        field_at<MODE>(g, r, nullptr, nullptr, nullptr, i, j, k, p, a, b, c);
        u[p] = a; v[p] = b; w[p] = c;
    });
}

// warpAffine (src/dataCostD.h:278-295) with the field of field_at.
template <int MODE>
__global__ void k_warp_affine(const float* __restrict__ in, Affine12 X, Grid3 g, const float* __restrict__ fu,
                              const float* __restrict__ fv, const float* __restrict__ fw, float* __restrict__ out, int m,
                              int n, int o, float* __restrict__ keep_u, float* __restrict__ keep_v,
                              float* __restrict__ keep_w) {
    for_rows<MODE>(g, m, n, [&](const RowStage& r, int i, int j, int k, int64_t p) {
        float u, v, w;
        field_at<MODE>(g, r, fu, fv, fw, i, j, k, p, u, v, w);
        if (keep_u) { keep_u[p] = u; keep_v[p] = v; keep_w[p] = w; }
        const float fi = (float)i, fj = (float)j, fk = (float)k;
        const float y1 = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(fi, X.x[0]), __fmul_rn(fj, X.x[1])), __fmul_rn(fk, X.x[2])), X.x[3]), v);
        const float x1 = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(fi, X.x[4]), __fmul_rn(fj, X.x[5])), __fmul_rn(fk, X.x[6])), X.x[7]), u);
        const float z1 = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(fi, X.x[8]), __fmul_rn(fj, X.x[9])), __fmul_rn(fk, X.x[10])), X.x[11]), w);
        int x, y, z;
        float dx, dy, dz;
        split_coord(x1, x, dx);
        split_coord(y1, y, dy);
        split_coord(z1, z, dz);
        out[p] = sample_ff(in, corners(y, x, z, m, n, o), ff_weights(dx, dy, dz), dx, dy, dz);
    });
}

// warpImageCL = interp3(flag=true) (src/dataCostD.h:213-223, src/transformations.h:9-22)
// with the field of field_at.
template <int MODE>
__global__ void k_warp_image(const float* __restrict__ in, Grid3 g, const float* __restrict__ fu,
                             const float* __restrict__ fv, const float* __restrict__ fw, float* __restrict__ out, int m,
                             int n, int o) {
    for_rows<MODE>(g, m, n, [&](const RowStage& r, int i, int j, int k, int64_t p) {
        float u, v, w;
        field_at<MODE>(g, r, fu, fv, fw, i, j, k, p, u, v, w);
        int x, y, z;
        float dx, dy, dz;
        split_coord(u, x, dx);
        split_coord(v, y, dy);
        split_coord(w, z, dz);
        const Corners c = corners(displaced(i, y, m), displaced(j, x, n), displaced(k, z, o), m, n, o);
        out[p] = sample_ff(in, c, ff_weights(dx, dy, dz), dx, dy, dz);
    });
}

// warpAffineS (src/dataCostD.h:241-266): nearest neighbour, round half away from zero.
template <int MODE>
__global__ void k_warp_seg(const short* __restrict__ in, Affine12 X, Grid3 g, const float* __restrict__ fu,
                           const float* __restrict__ fv, const float* __restrict__ fw, short* __restrict__ out, int m,
                           int n, int o) {
    for_rows<MODE>(g, m, n, [&](const RowStage& r, int i, int j, int k, int64_t p) {
        float u, v, w;
        field_at<MODE>(g, r, fu, fv, fw, i, j, k, p, u, v, w);
        const float fi = (float)i, fj = (float)j, fk = (float)k;
        const float y1 = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(fi, X.x[0]), __fmul_rn(fj, X.x[1])), __fmul_rn(fk, X.x[2])), X.x[3]), v);
        const float x1 = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(fi, X.x[4]), __fmul_rn(fj, X.x[5])), __fmul_rn(fk, X.x[6])), X.x[7]), u);
        const float z1 = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(fi, X.x[8]), __fmul_rn(fj, X.x[9])), __fmul_rn(fk, X.x[10])), X.x[11]), w);
        const int x = __float2int_rz(roundf(x1)), y = __float2int_rz(roundf(y1)), z = __float2int_rz(roundf(z1));
        out[p] = in[clampi(y, 0, m - 1) + (int64_t)clampi(x, 0, n - 1) * m + (int64_t)clampi(z, 0, o - 1) * (int64_t)m * n];
    });
}

__global__ void k_scale6(const float* __restrict__ a0, const float* __restrict__ a1, const float* __restrict__ a2,
                         const float* __restrict__ a3, const float* __restrict__ a4, const float* __restrict__ a5,
                         float* __restrict__ b0, float* __restrict__ b1, float* __restrict__ b2, float* __restrict__ b3,
                         float* __restrict__ b4, float* __restrict__ b5, int64_t n, float f) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    b0[p] = __fmul_rn(a0[p], f); b1[p] = __fmul_rn(a1[p], f); b2[p] = __fmul_rn(a2[p], f);
    b3[p] = __fmul_rn(a3[p], f); b4[p] = __fmul_rn(a4[p], f); b5[p] = __fmul_rn(a5[p], f);
}

// (float)(0.5 * (double)a - 0.5 * (double)b): the double difference of two floats is
// exact unless their exponents lie more than 29 apart, and then a/2 alone is nowhere
// near a float midpoint, so one float subtraction of the exact halves rounds alike;
// tiny values, whose halves may not be exact, take the double expression.
__device__ __forceinline__ float half_difference(float a, float b) {
    const float m = fminf(a == 0.0f ? 1.0f : fabsf(a), b == 0.0f ? 1.0f : fabsf(b));
    if (m >= 0x1p-100f) return __fsub_rn(0.5f * a, 0.5f * b);
    return (float)(0.5 * (double)a - 0.5 * (double)b);
}

// One consistentMappingCL iteration (src/transformations.h:203-226): both new
// fields from the previous ones, u <- 0.5*us - 0.5*(us2 at x+us), and back.
__global__ void k_consistent_step(const float* __restrict__ us, const float* __restrict__ vs,
                                  const float* __restrict__ ws, const float* __restrict__ us2,
                                  const float* __restrict__ vs2, const float* __restrict__ ws2, float* __restrict__ nu,
                                  float* __restrict__ nv, float* __restrict__ nw, float* __restrict__ nu2,
                                  float* __restrict__ nv2, float* __restrict__ nw2, int m, int n, int o) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, k = blockIdx.z;
    if (i >= m) return;
    const int64_t p = i + (int64_t)j * m + (int64_t)k * m * n;
    {
        int x, y, z;
        float dx, dy, dz;
        split_coord(us[p], x, dx);
        split_coord(vs[p], y, dy);
        split_coord(ws[p], z, dz);
        const Corners c = corners(displaced(i, y, m), displaced(j, x, n), displaced(k, z, o), m, n, o);
        const FFWeights b = ff_weights(dx, dy, dz);
        nu[p] = half_difference(us[p], sample_ff(us2, c, b, dx, dy, dz));
        nv[p] = half_difference(vs[p], sample_ff(vs2, c, b, dx, dy, dz));
        nw[p] = half_difference(ws[p], sample_ff(ws2, c, b, dx, dy, dz));
    }
    {
        int x, y, z;
        float dx, dy, dz;
        split_coord(us2[p], x, dx);
        split_coord(vs2[p], y, dy);
        split_coord(ws2[p], z, dz);
        const Corners c = corners(displaced(i, y, m), displaced(j, x, n), displaced(k, z, o), m, n, o);
        const FFWeights b = ff_weights(dx, dy, dz);
        nu2[p] = half_difference(us2[p], sample_ff(us, c, b, dx, dy, dz));
        nv2[p] = half_difference(vs2[p], sample_ff(vs, c, b, dx, dy, dz));
        nw2[p] = half_difference(ws2[p], sample_ff(ws, c, b, dx, dy, dz));
    }
}

// Jacobian determinant per node (src/transformations.h:118-158): central
// differences with replicate padding, /g, +1 on the diagonal; accumulates
// sum J, sum J^2 and count(J<0) for the diagnostic print.
__global__ void k_jacobian(const float* __restrict__ u, const float* __restrict__ v, const float* __restrict__ w,
                           int m, int n, int o, float f1, double* __restrict__ acc) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, k = blockIdx.z;
    double sj = 0.0, sj2 = 0.0, neg = 0.0;
    if (i < m) {
        const int64_t mn = (int64_t)m * n;
        auto at = [&](const float* a, int ii, int jj, int kk) {
            return a[clampi(ii, 0, m - 1) + (int64_t)clampi(jj, 0, n - 1) * m + (int64_t)clampi(kk, 0, o - 1) * mn];
        };
        auto d = [&](const float* a, int axis) {
            float r = 0.0f;
            const float gr[3] = {-0.5f, 0.0f, 0.5f};
            for (int f = 0; f < 3; f++) {
                const float s = axis == 1 ? at(a, i + f - 1, j, k) : (axis == 2 ? at(a, i, j + f - 1, k) : at(a, i, j, k + f - 1));
                r = __fadd_rn(r, __fmul_rn(gr[f], s));
            }
            return r;
        };
        const float a11 = (float)((double)__fmul_rn(d(u, 2), f1) + 1.0), a12 = __fmul_rn(d(u, 1), f1), a13 = __fmul_rn(d(u, 3), f1);
        const float a21 = __fmul_rn(d(v, 2), f1), a22 = (float)((double)__fmul_rn(d(v, 1), f1) + 1.0), a23 = __fmul_rn(d(v, 3), f1);
        const float a31 = __fmul_rn(d(w, 2), f1), a32 = __fmul_rn(d(w, 1), f1), a33 = (float)((double)__fmul_rn(d(w, 3), f1) + 1.0);
        const float J = a11 * (a22 * a33 - a23 * a32) - a21 * (a12 * a33 - a13 * a32) + a31 * (a12 * a23 - a13 * a22);
        sj = J; sj2 = (double)J * J; neg = J < 0.0f ? 1.0 : 0.0;
    }
    for (int off = 16; off > 0; off >>= 1) {
        sj += __shfl_xor_sync(0xffffffffu, sj, off);
        sj2 += __shfl_xor_sync(0xffffffffu, sj2, off);
        neg += __shfl_xor_sync(0xffffffffu, neg, off);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(acc + 0, sj);
        atomicAdd(acc + 1, sj2);
        atomicAdd(acc + 2, neg);
    }
}

inline dim3 vol_grid(int m, int n, int o, int threads) { return dim3((m + threads - 1) / threads, n, o); }

inline Grid3 make_grid(const float* u, const float* v, const float* w, int m2, int n2, int o2, int m, int n, int o) {
    Grid3 g;
    g.u = u; g.v = v; g.w = w;
    g.m = m2; g.n = n2; g.o = o2;
    g.sm = (float)m / (float)m2; g.sn = (float)n / (float)n2; g.so = (float)o / (float)o2;
    return g;
}

inline Affine12 make_affine(const float* X) {
    Affine12 a;
    for (int i = 0; i < 12; i++) a.x[i] = X[i];
    return a;
}

}  // namespace

cudaError_t launch_shift(const float* d_in, float* d_out, int64_t n, float shift, cudaStream_t s) {
    k_shift<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d_in, d_out, n, -shift);
    count_launches(1);
    return cudaGetLastError();
}

namespace {
// Rows per block, and whether a grid's rows are staged (mode 3): where two voxels or
// more share a node (below that, as between neighbouring levels' grids, staging costs
// more than it saves) and a row of nodes fits the default 48 KB.
constexpr int kRowsPerBlock = 4;
bool staged(const Grid3& g) { return g.sm >= 2.0f && kRowBytes * g.m + 16 <= 48 * 1024; }
int rows_per_block(int n, int mode, const Grid3& g, size_t& smem) {
    const size_t each = mode == 3 ? (kRowBytes * g.m + 15) & ~(size_t)15 : 0;
    int rows = std::min(kRowsPerBlock, n);
    while (rows > 1 && rows * each > 48 * 1024) rows--;
    smem = rows * each;
    return rows;
}
}  // namespace

#define DEEDS_ROWS(KERNEL, MODE, ...)                                                                    \
    do {                                                                                                \
        size_t smem;                                                                                    \
        const int rows = rows_per_block(n, MODE, g, smem);                                              \
        KERNEL<MODE><<<dim3((n + rows - 1) / rows, o), dim3(kRowThreads, rows), smem, s>>>(__VA_ARGS__); \
        count_launches(1);                                                                              \
        return cudaGetLastError();                                                                      \
    } while (0)
#define DEEDS_BY_MODE(KERNEL, ...)                           \
    do {                                                     \
        if (f.mode == 0) DEEDS_ROWS(KERNEL, 0, __VA_ARGS__); \
        if (f.mode == 1) DEEDS_ROWS(KERNEL, 1, __VA_ARGS__); \
        if (staged(g)) DEEDS_ROWS(KERNEL, 3, __VA_ARGS__);   \
        DEEDS_ROWS(KERNEL, 2, __VA_ARGS__);                  \
    } while (0)

cudaError_t launch_upsample(const float* u0, const float* v0, const float* w0, int m2, int n2, int o2, float* u,
                            float* v, float* w, int m, int n, int o, cudaStream_t s) {
    const Grid3 g = make_grid(u0, v0, w0, m2, n2, o2, m, n, o);
    if (staged(g)) DEEDS_ROWS(k_upsample, 3, g, u, v, w, m, n, o);
    DEEDS_ROWS(k_upsample, 2, g, u, v, w, m, n, o);
}

cudaError_t launch_warp_affine(const float* d_in, const float* X, const FieldRef& f, int m, int n, int o, float* d_out,
                               float* keep_u, float* keep_v, float* keep_w, cudaStream_t s) {
    const Grid3 g = f.mode == 2 ? make_grid(f.u, f.v, f.w, f.m1, f.n1, f.o1, m, n, o) : Grid3{};
    DEEDS_BY_MODE(k_warp_affine, d_in, make_affine(X), g, f.u, f.v, f.w, d_out, m, n, o, keep_u, keep_v, keep_w);
}

cudaError_t launch_warp_image(const float* d_in, const FieldRef& f, int m, int n, int o, float* d_out, cudaStream_t s) {
    const Grid3 g = f.mode == 2 ? make_grid(f.u, f.v, f.w, f.m1, f.n1, f.o1, m, n, o) : Grid3{};
    DEEDS_BY_MODE(k_warp_image, d_in, g, f.u, f.v, f.w, d_out, m, n, o);
}

cudaError_t launch_warp_seg(const short* d_in, const float* X, const FieldRef& f, int m, int n, int o, short* d_out,
                            cudaStream_t s) {
    const Grid3 g = f.mode == 2 ? make_grid(f.u, f.v, f.w, f.m1, f.n1, f.o1, m, n, o) : Grid3{};
    DEEDS_BY_MODE(k_warp_seg, d_in, make_affine(X), g, f.u, f.v, f.w, d_out, m, n, o);
}
#undef DEEDS_BY_MODE
#undef DEEDS_ROWS

cudaError_t launch_consistent(float* u, float* v, float* w, float* u2, float* v2, float* w2, int m, int n, int o, int g,
                              float* scratch /* 12*sz */, cudaStream_t s) {
    const int64_t sz = (int64_t)m * n * o;
    float* A[6];
    float* B[6];
    for (int i = 0; i < 6; i++) { A[i] = scratch + i * sz; B[i] = scratch + (6 + i) * sz; }
    const float f1 = (float)(1.0 / (float)g);
    const unsigned nb = (unsigned)((sz + 255) / 256);
    k_scale6<<<nb, 256, 0, s>>>(u, v, w, u2, v2, w2, A[0], A[1], A[2], A[3], A[4], A[5], sz, f1);
    for (int it = 0; it < 10; it++) {
        k_consistent_step<<<vol_grid(m, n, o, 64), 64, 0, s>>>(A[0], A[1], A[2], A[3], A[4], A[5], B[0], B[1], B[2],
                                                               B[3], B[4], B[5], m, n, o);
        for (int i = 0; i < 6; i++) { float* t = A[i]; A[i] = B[i]; B[i] = t; }
    }
    k_scale6<<<nb, 256, 0, s>>>(A[0], A[1], A[2], A[3], A[4], A[5], u, v, w, u2, v2, w2, sz, (float)g);
    count_launches(12);
    return cudaGetLastError();
}

cudaError_t launch_jacobian(const float* u, const float* v, const float* w, int m, int n, int o, int g, double* d_acc,
                            cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(d_acc, 0, 3 * sizeof(double), s);
    if (e != cudaSuccess) return e;
    const float f1 = (float)(1.0 / (float)g);
    k_jacobian<<<vol_grid(m, n, o, 64), 64, 0, s>>>(u, v, w, m, n, o, f1, d_acc);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace deeds
