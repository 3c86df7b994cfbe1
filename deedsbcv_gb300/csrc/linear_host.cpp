// Host half of linearBCV (see linear_host.h).  The fit works on at most a few
// ten thousand points, so it stays on the CPU next to the level loop; its
// arithmetic follows the reference's types exactly (compiled without FMA
// contraction): float accumulations, pow(x, 2) of a float evaluated in double
// (exact), the float overload of sqrt, double where a double literal appears.
#include "linear_host.h"

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <cstring>

namespace deeds {

namespace {

// Column view of a point set: column c of `len` entries at p + c*len.
struct Cols {
    const float* p;
    int len;
    const float* col(int c) const { return p + (size_t)c * len; }
};

float sq_norm_sqrt(const float* v, int len) {  // norm, src/QRsolve.h:2-8
    float acc = 0.0f;
    for (int i = 0; i < len; i++) acc = (float)((double)acc + (double)v[i] * (double)v[i]);
    return std::sqrt(acc);
}

float dotf(const float* a, const float* b, int len) {  // dotprod, src/QRsolve.h:10-16
    float acc = 0.0f;
    for (int i = 0; i < len; i++) acc += a[i] * b[i];
    return acc;
}

// One-sided Jacobi rotations on the columns of a 3x3 matrix, four sweeps
// (jacobiSVD3, src/QRsolve.h:86-141); U gets the normalised columns, V the
// accumulated rotations.
void jacobi3(const float* A, float* U, float* V) {
    for (int i = 0; i < 9; i++) { U[i] = A[i]; V[i] = 0.0f; }
    V[0] = V[4] = V[8] = 1.0f;
    for (int sweep = 0; sweep < 4; sweep++)
        for (int j = 1; j < 3; j++)
            for (int i = 0; i < j; i++) {
                float* ui = U + 3 * i;
                float* uj = U + 3 * j;
                const float a = dotf(ui, ui, 3), b = dotf(uj, uj, 3), gm = dotf(ui, uj, 3);
                const float zeta = (float)((double)(b - a) / (2.0 * (double)gm));
                const double sgn = zeta > 0 ? 1.0 : -1.0;
                const float t = (float)(sgn / ((double)std::fabs(zeta) + std::sqrt(1.0 + (double)(zeta * zeta))));
                const float c = (float)(1.0 / (double)std::sqrt(1.0f + t * t));
                const float s = c * t;
                float* vi = V + 3 * i;
                float* vj = V + 3 * j;
                for (int k = 0; k < 3; k++) {
                    const float ti = ui[k];
                    ui[k] = c * ti - s * uj[k];
                    uj[k] = s * ti + c * uj[k];
                }
                for (int k = 0; k < 3; k++) {
                    const float ti = vi[k];
                    vi[k] = c * ti - s * vj[k];
                    vj[k] = s * ti + c * vj[k];
                }
            }
    for (int j = 0; j < 3; j++) {
        const float sv = sq_norm_sqrt(U + 3 * j, 3);
        for (int i = 0; i < 3; i++) U[i + 3 * j] /= sv;
    }
}

// findRigid (src/QRsolve.h:143-254): rotation R = sum_k u_k v_k^T from the SVD of
// the cross-covariance, translation through R's QR solve of the second point
// set; RT gets R^T and the translation.
void find_rigid(float* RT, Cols a, Cols b) {
    const int len = a.len;
    std::vector<float> pa(4 * (size_t)len), pb(4 * (size_t)len);  // point-major (x4)
    for (int c = 0; c < 4; c++)
        for (int k = 0; k < len; k++) {
            pa[c + 4 * (size_t)k] = a.col(c)[k];
            pb[c + 4 * (size_t)k] = b.col(c)[k];
        }
    float ma[3] = {0.0f, 0.0f, 0.0f}, mb[3] = {0.0f, 0.0f, 0.0f};
    for (int k = 0; k < len; k++)
        for (int c = 0; c < 3; c++) {
            ma[c] += pa[c + 4 * (size_t)k];
            mb[c] += pb[c + 4 * (size_t)k];
        }
    for (int c = 0; c < 3; c++) {
        ma[c] /= (float)len;
        mb[c] /= (float)len;
    }
    float K[9] = {0.0f}, U[9], V[9], R[16] = {0.0f};
    for (int k = 0; k < len; k++)
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++) K[i + 3 * j] += (pa[j + 4 * (size_t)k] - ma[j]) * (pb[i + 4 * (size_t)k] - mb[i]);
    jacobi3(K, U, V);
    std::fill(RT, RT + 16, 0.0f);
    R[15] = 1.0f;
    RT[15] = 1.0f;
    for (int k = 0; k < 3; k++)
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++) R[j + 4 * i] += U[j + 3 * k] * V[i + 3 * k];
    std::vector<float> rb(4 * (size_t)len);
    lin_qrsolve(rb.data(), R, pb.data(), 4, len);
    float t1[3] = {0.0f, 0.0f, 0.0f};
    for (int k = 0; k < len; k++)
        for (int c = 0; c < 3; c++) t1[c] += rb[c + 4 * (size_t)k];
    for (int c = 0; c < 3; c++) t1[c] = t1[c] / (float)len - ma[c];
    float t0[3] = {0.0f, 0.0f, 0.0f};
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) t0[i] += R[i + 4 * j] * t1[j];
    for (int i = 0; i < 3; i++) {
        for (int j = 0; j < 3; j++) RT[i + 4 * j] += R[j + 4 * i];
        RT[3 + 4 * i] = t0[i];
    }
}

// The k-th smallest of n non-negative floats (squared residuals): their bit patterns
// order like the values, so counting the top 12 bits, then the next 10 and the last 10
// of those that share them, finds it exactly, in place of nth_element (whose answer is
// the same value).  scratch holds the patterns that are still in question.
float kth_smallest_nonneg(const float* v, size_t n, int k, std::vector<uint32_t>& scratch) {
    scratch.resize(n);
    uint32_t* s = scratch.data();
    std::memcpy(s, v, n * sizeof(float));
    uint32_t want = (uint32_t)k, r = 0;
    const int shift[3] = {20, 10, 0};
    const uint32_t mask[3] = {0xfffu, 0x3ffu, 0x3ffu};
    uint32_t hist[2][4096];
    for (int pass = 0; pass < 3; pass++) {
        const int sh = shift[pass];
        const uint32_t mk = mask[pass];
        for (int h = 0; h < 2; h++) std::fill(hist[h], hist[h] + mk + 1, 0u);
        size_t i = 0;
        for (; i + 1 < n; i += 2) {  // two tables: equal neighbours do not wait for each other
            hist[0][(s[i] >> sh) & mk]++;
            hist[1][(s[i + 1] >> sh) & mk]++;
        }
        if (i < n) hist[0][(s[i] >> sh) & mk]++;
        uint32_t b = 0;
        for (;; b++) {
            const uint32_t c = hist[0][b] + hist[1][b];
            if (c > want) break;
            want -= c;
        }
        r |= b << sh;
        size_t kept = 0;
        for (i = 0; i < n; i++) {
            const uint32_t x = s[i];
            s[kept] = x;
            kept += ((x >> sh) & mk) == b;
        }
        n = kept;
    }
    float out;
    std::memcpy(&out, &r, sizeof(out));
    return out;
}

// Points are taken a block at a time: what is independent from point to point (vector
// updates, quotients, products) in loops that the compiler turns into vector code, into
// small arrays from which the sequential sums then read.
constexpr int kBlock = 64;

// acc = (float)((double)acc + (double)v[i] * (double)v[i]) for i = 0 .. n - 1.
// With a fused multiply-add the chain is one instruction a point: its single rounding
// gives the same float unless the double sum is inexact and itself half way between two
// floats (or so small that the float is subnormal), which a second, independent loop
// looks for; a block with such a point takes the chain of doubles.
float add_squares(float acc, const float* __restrict v, int n) {
#ifdef __FP_FAST_FMAF
    float a[kBlock + 1];
    a[0] = acc;
    for (int i = 0; i < n; i++) a[i + 1] = __builtin_fmaf(v[i], v[i], a[i]);
    uint64_t bad = 0;
    for (int i = 0; i < n; i++) {
        const double x = a[i], y = (double)v[i] * (double)v[i], s = x + y;  // y is exact
        const double t = s - x, e = (x - (s - t)) + (y - t);                // the sum's rounding error
        uint64_t b;
        std::memcpy(&b, &s, sizeof(b));
        bad |= (uint64_t)(((b & 0x1fffffffu) == 0x10000000u) & !(e == 0.0)) | (uint64_t)(!(s >= 0x1p-120) & !(s == 0.0));
    }
    if (!bad) return a[n];
#endif
    for (int i = 0; i < n; i++) acc = (float)((double)acc + (double)v[i] * (double)v[i]);
    return acc;
}

void fit(float* RT, Cols a, Cols b, bool rigid) {
    if (rigid) find_rigid(RT, a, b);
    else lin_qrsolve(RT, a.p, b.p, a.len, 4);
}

}  // namespace

// The Gram-Schmidt QR with every sum kept in its own sequential accumulator, in
// index order, exactly as the reference evaluates it; what changes is only that
// independent sums (and the vector updates feeding them) share one pass over
// the points, so their dependency chains overlap instead of running one after
// another.  Same bits, several times fewer passes.
// A Grace core, the 16 fits to 60000 points: 10.4 ms, 14.5 ms with the loops point by
// point and the squares' sum in doubles.
void lin_qrsolve(float* X, const float* A, const float* b, int len, int nrhs) {
    std::vector<float> Qv(4 * (size_t)len);  // while columns are made: one after the other
    float* __restrict q0 = Qv.data();
    float* __restrict q1 = q0 + len;
    float* __restrict q2 = q1 + len;
    float* __restrict q3 = q2 + len;
    const float* __restrict a0 = A;
    const float* __restrict a1 = A + len;
    const float* __restrict a2 = A + 2 * (size_t)len;
    const float* __restrict a3 = A + 3 * (size_t)len;
    float p1[kBlock], p2[kBlock], p3[kBlock];
    auto blocks = [len](auto body) {
        for (int i = 0; i < len; i += kBlock) body(i, std::min(kBlock, len - i));
    };
    // column 1
    float n0 = 0.0f;
    blocks([&](int i0, int n) { n0 = add_squares(n0, a0 + i0, n); });
    const float r11 = std::sqrt(n0);
    float r12 = 0.0f, r13 = 0.0f, r14 = 0.0f;
    blocks([&](int i0, int n) {
        for (int i = 0; i < n; i++) {
            const float q = a0[i0 + i] / r11;
            q0[i0 + i] = q;
            p1[i] = q * a1[i0 + i];
            p2[i] = q * a2[i0 + i];
            p3[i] = q * a3[i0 + i];
        }
        for (int i = 0; i < n; i++) {
            r12 += p1[i];
            r13 += p2[i];
            r14 += p3[i];
        }
    });
    // column 2 (q2, q3 hold the partially orthogonalised columns 3 and 4)
    float n1 = 0.0f;
    blocks([&](int i0, int n) {
        for (int i = i0; i < i0 + n; i++) {
            q1[i] = a1[i] - q0[i] * r12;
            q2[i] = a2[i] - q0[i] * r13;
            q3[i] = a3[i] - q0[i] * r14;
        }
        n1 = add_squares(n1, q1 + i0, n);
    });
    const float r22 = std::sqrt(n1);
    float r23 = 0.0f, r24 = 0.0f;
    blocks([&](int i0, int n) {
        for (int i = 0; i < n; i++) {
            const float q = q1[i0 + i] / r22;
            q1[i0 + i] = q;
            p1[i] = q * a2[i0 + i];
            p2[i] = q * a3[i0 + i];
        }
        for (int i = 0; i < n; i++) {
            r23 += p1[i];
            r24 += p2[i];
        }
    });
    // column 3
    float n2 = 0.0f;
    blocks([&](int i0, int n) {
        for (int i = i0; i < i0 + n; i++) {
            q2[i] = a2[i] - q0[i] * r13 - q1[i] * r23;
            q3[i] = a3[i] - q0[i] * r14 - q1[i] * r24;
        }
        n2 = add_squares(n2, q2 + i0, n);
    });
    const float r33 = std::sqrt(n2);
    float r34 = 0.0f;
    blocks([&](int i0, int n) {
        for (int i = 0; i < n; i++) {
            const float q = q2[i0 + i] / r33;
            q2[i0 + i] = q;
            p1[i] = q * a3[i0 + i];
        }
        for (int i = 0; i < n; i++) r34 += p1[i];
    });
    // column 4
    float n3 = 0.0f;
    blocks([&](int i0, int n) {
        for (int i = i0; i < i0 + n; i++) q3[i] = a3[i] - q0[i] * r14 - q1[i] * r24 - q2[i] * r34;
        n3 = add_squares(n3, q3 + i0, n);
    });
    const float r44 = std::sqrt(n3);
    for (int i = 0; i < len; i++) q3[i] = q3[i] / r44;
    // right-hand sides: 4 dot products each, up to four right-hand sides per pass
    for (int j0 = 0; j0 < nrhs; j0 += 4) {
        const int nj = std::min(4, nrhs - j0);
        float d[4][4] = {{0.0f}};
        if (nj == 4) {
            const float* b0 = b + (size_t)j0 * len;
            const float* b1 = b0 + len;
            const float* b2 = b1 + len;
            const float* b3 = b2 + len;
            // a vector of four sums, one for each column of Q, per right-hand side
            typedef float V4 __attribute__((vector_size(16)));
            V4 s0 = {0.0f, 0.0f, 0.0f, 0.0f}, s1 = s0, s2 = s0, s3 = s0;
            for (int i = 0; i < len; i++) {
                const V4 q = {q0[i], q1[i], q2[i], q3[i]};
                s0 += q * b0[i];
                s1 += q * b1[i];
                s2 += q * b2[i];
                s3 += q * b3[i];
            }
            for (int c = 0; c < 4; c++) {
                d[0][c] = s0[c];
                d[1][c] = s1[c];
                d[2][c] = s2[c];
                d[3][c] = s3[c];
            }
        } else {
            for (int j = 0; j < nj; j++) {
                const float* bj = b + (size_t)(j0 + j) * len;
                for (int i = 0; i < len; i++) {
                    d[j][0] += q0[i] * bj[i];
                    d[j][1] += q1[i] * bj[i];
                    d[j][2] += q2[i] * bj[i];
                    d[j][3] += q3[i] * bj[i];
                }
            }
        }
        for (int j = 0; j < nj; j++) {
            const float x4 = d[j][3] / r44;
            const float x3 = (d[j][2] - r34 * x4) / r33;
            const float x2 = (d[j][1] - r23 * x3 - r24 * x4) / r22;
            const float x1 = (d[j][0] - r12 * x2 - r13 * x3 - r14 * x4) / r11;
            float* Xj = X + 4 * (size_t)(j0 + j);
            Xj[0] = x1;
            Xj[1] = x2;
            Xj[2] = x3;
            Xj[3] = x4;
        }
    }
}

void lin_affine_robust(float* RT, const float* p1, const float* p2, int len, bool rigid) {
    if (len < kMinFitPoints) return;  // the trimmed half would be empty (the reference reads outside its arrays)
    const Cols A{p1, len}, B{p2, len};
    fit(RT, A, B, rigid);
    const int half = len / 2;
    std::vector<float> errv(len);
    std::vector<uint32_t> scratch;
    std::vector<float> ha(4 * (size_t)half, 1.0f), hb(4 * (size_t)half, 1.0f);  // the kept half; column 3 stays 1
    const float* __restrict A0 = A.col(0);
    const float* __restrict A1 = A.col(1);
    const float* __restrict A2 = A.col(2);
    const float* __restrict A3 = A.col(3);
    const float* __restrict B0 = B.col(0);
    const float* __restrict B1 = B.col(1);
    const float* __restrict B2 = B.col(2);
    float* __restrict err = errv.data();
    for (int iter = 0; iter < 15; iter++) {
        float R[12];
        std::memcpy(R, RT, sizeof(R));
        for (int l = 0; l < len; l++) {
            const float v0 = A0[l], v1 = A1[l], v2 = A2[l], h = A3[l];
            const float y = (((0.0f + v0 * R[0]) + v1 * R[1]) + v2 * R[2]) + h * R[3];
            const float x = (((0.0f + v0 * R[4]) + v1 * R[5]) + v2 * R[6]) + h * R[7];
            const float z = (((0.0f + v0 * R[8]) + v1 * R[9]) + v2 * R[10]) + h * R[11];
            const double ey = (double)(y - B0[l]), ex = (double)(x - B1[l]), ez = (double)(z - B2[l]);
            err[l] = (float)(ey * ey + ex * ex + ez * ez);
        }
        const float median = kth_smallest_nonneg(err, len, len / 2, scratch);
        // points at or below the median, in order; any beyond the half overwrite the last slot
        auto put = [&](int slot, int i) {
            ha[slot] = A0[i];
            ha[slot + (size_t)half] = A1[i];
            ha[slot + 2 * (size_t)half] = A2[i];
            hb[slot] = B0[i];
            hb[slot + (size_t)half] = B1[i];
            hb[slot + 2 * (size_t)half] = B2[i];
        };
        if (median == median) {  // else no residual compares, and the kept half stays as it was
            // more than half of the points are kept: every point is written to the next slot,
            // which moves on for a kept one, and the last slot gets the last kept point
            int count = 0, last = 0;
            for (int i = 0; i < len; i++) {
                put(std::min(count, half - 1), i);
                const bool keep = err[i] <= median;
                count += keep;
                last = keep ? i : last;
            }
            put(half - 1, last);
        }
        fit(RT, Cols{ha.data(), half}, Cols{hb.data(), half}, rigid);
    }
}

void lin_matmult(const float* A, const float* B, float* X) {
    for (int i = 0; i < 4; i++)
        for (int j = 0; j < 4; j++) {
            float acc = 0.0f;
            for (int k = 0; k < 4; k++) acc += A[i + 4 * k] * B[k + 4 * j];
            X[i + 4 * j] = acc;
        }
}

int lin_estimate_from_stats(float* X, const float* Xprev, const float* minval, const int* minind, int m1, int n1,
                            int o1, int g, float q, int hw, bool rigid, int* allcount_out, float* quantile_out) {
    const int sz1 = m1 * n1 * o1, len = 2 * hw + 1, stephw = (g - 1) / 2;
    const float* mv[2] = {minval, minval + sz1};
    const int* mi[2] = {minind, minind + sz1};
    int allcount = 0;
    for (int v = 0; v < 2; v++)
        for (int i = 0; i < sz1; i++) allcount += mv[v][i] < 1e19f;
    // quantile() of src/linearBCV.cpp:36-46 at 0.5*allcount/sz1/2 (double, then float)
    const float qf = (float)(0.5 * (double)allcount / (double)(float)sz1 / 2.0);
    const int qi = (int)((float)sz1 * std::min(std::max(qf, 0.01f), 0.99f));
    float med[2];
    std::vector<uint32_t> scratch;
    // cost volumes are non-negative, the exclusion value is 1e20
    for (int v = 0; v < 2; v++) med[v] = kth_smallest_nonneg(mv[v], sz1, qi, scratch);
    int valsz = 0;
    for (int i = 0; i < sz1; i++) valsz += (mv[0][i] < med[0]) + (mv[1][i] < med[1]);
    if (allcount_out) *allcount_out = allcount;
    if (quantile_out) *quantile_out = qf;
    // ties at the quantile (e.g. a constant image pair) can leave no point strictly
    // below it; the caller reports that instead of fitting
    if (valsz < kMinFitPoints) return valsz;
    std::vector<float> p1(4 * (size_t)valsz), p2(4 * (size_t)valsz);
    float* p1c[4] = {p1.data(), p1.data() + valsz, p1.data() + 2 * (size_t)valsz, p1.data() + 3 * (size_t)valsz};
    float* p2c[4] = {p2.data(), p2.data() + valsz, p2.data() + 2 * (size_t)valsz, p2.data() + 3 * (size_t)valsz};
    int cur = 0;
    for (int i = 0, i1 = 0, j1 = 0, k1 = 0; i < sz1; i++, i1++) {
        if (i1 == m1) {
            i1 = 0;
            if (++j1 == n1) {
                j1 = 0;
                k1++;
            }
        }
        const int cy = i1 * g + stephw, cx = j1 * g + stephw, cz = k1 * g + stephw;
        for (int v = 0; v < 2; v++) {
            if (!(mv[v][i] < med[v])) continue;
            // label l -> displacement ((l%len)-hw, (l/len%len)-hw, (l/len^2)-hw) * q in (y, x, z)
            const int l = mi[v][i];
            const float dy = (l % len - hw) * q, dx = ((l / len) % len - hw) * q, dz = (l / (len * len) - hw) * q;
            // direction 1: node -> node + d; direction 2: node + d -> node
            float** at = v == 0 ? p1c : p2c;
            float** bt = v == 0 ? p2c : p1c;
            at[0][cur] = (float)cy; at[1][cur] = (float)cx; at[2][cur] = (float)cz;
            bt[0][cur] = cy + dy; bt[1][cur] = cx + dx; bt[2][cur] = cz + dz;
            p1c[3][cur] = 1.0f;
            p2c[3][cur] = 1.0f;
            cur++;
        }
    }
    float X1[16];
    lin_affine_robust(X1, p1.data(), p2.data(), valsz, rigid);
    lin_matmult(X1, Xprev, X);
    return valsz;
}

}  // namespace deeds
