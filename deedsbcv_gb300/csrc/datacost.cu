// Hamming cost volume on sm_103a (replaces dataCostCL, src/dataCostD.h:108-210).
//
// cost[node][label] = alpha1 * sum over the node's sampled g^3 block of
//   popcount(F[p] ^ M[clamp(p + d(label))]),
// d(label) = (ly, lx, lz) * q - q*hw, label = ly + lx*len + lz*len^2.
//
// Main path (grid spacing 2..8; few labels an axis: datacost_popc.cu): the sums run on the tensor cores, as dot products
// of 64 four-bit floats (E2M1) per code whose terms are bit differences less a
// constant of the fixed code (tmem_st_moving, expand_fixed); a row's sums over its
// node's sampled columns accumulate exactly in the fp32 accumulators (multiples of
// 1/2; a pair gives at most 56, a slot sums min(q, G) rows of up to 16 columns: at most 7168).
//
// A label step of q pairs only rows y of one residue modulo q, so rows are taken
// by residue class: class r of a tile of tn nodes along y (one x, z) has the fixed
// rows r + q a and the moving rows r + q b, and y label ly pairs b = a + ly.  With
// a0 = floor(t G / q), node t's fixed rows of any class are a = a0 + s for slots
// s < SL = ceil((G + q - 1) / q) at most, and (t, s, b) stands for the label
// ly = b - a0 - s in every class.  One step of work = (P z offsets, x offset lx) is
//   D[(p, b)][(t, s)] += <moving rows of class r, fixed rows of class r>
// over the node's sampled columns and the q classes, M = 128 moving rows (P offsets
// x R rows) by N >= tn SL slots, all in the accumulators; a label's cost is the sum
// of its SL entries.
//  * three producer warpgroups (classes in turn): one thread per moving row loads
//    its codes (from a copy of the volume with its rows split by class, so that
//    loads are contiguous), expands them in registers and stores them to tensor
//    memory as operand A: a ring of twelve x columns, of which a step shares all but
//    one with the step before where q is 1;
//  * two warps (steps in turn) issue tcgen05.mma.kind::mxf4 with unit scales; operand
//    B = the fixed rows, expanded once per CTA into shared memory;
//  * two epilogue warpgroups (steps in turn; three where the window slides) move the
//    accumulators to shared memory and sum the slots.
//
// Bound: of a step's products len P T in 128 N are used, and an MMA costs max(15,
// N / 2) clocks per column with operand A in tensor memory (max(39, 32 + N / 4) from
// shared memory): 25-47 useful code pairs a clock and SM, where the integer pipe does
// 12 (four 32-bit POPCs per three pairs with a carry-save adder) and the kernel that
// used it reached 7.5.  Reached: 13-20 (the tensor pipe is busy 43 % of the time at
// grid 8): issuing an MMA takes ~32 clocks and each class ~320 for the hand-overs
// between the warps.  192x160x256, one direction, grids 8/7/6/5/4 of the default
// schedule: 1.89 / 1.37 / 1.30 / 1.56 / 1.37 ms, 7.5 ms in all (13.8 ms on the integer
// pipe); a 131x118x141 level of grid 5, radius 4, step 3: 0.65 -> 0.24 ms.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace deeds {

namespace {

// ---- tensor memory and block-scaled 4-bit MMA (one CTA)
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st8(uint32_t addr, const uint32_t (&w)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(addr), "r"(w[0]),
                 "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t addr, float (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
        "[%16];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]),
          "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
        : "r"(addr)
        : "memory");
}
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(p));
    return p;
}
// D[128][N] (+)= A[128][64] B[N][64]: A in tensor memory (lane = row, eight 4-bit
// elements per column word), B in shared memory
template <bool FIRST>  // FIRST: where `more` is 0 the product replaces D
__device__ __forceinline__ void mma_mxf4(uint32_t d, uint32_t a, uint32_t blo, uint32_t bhi, uint32_t idesc, uint32_t sfa,
                                         uint32_t sfb, uint32_t more) {
    asm volatile(
        "{\n .reg .pred p;\n .reg .b64 b;\n mov.b64 b, {%2, %3};\n setp.ne.u32 p, %7, 0;\n"
        " tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [%1], b, %4, [%5], [%6], p;\n}" ::"r"(d),
        "r"(a), "r"(blo), "r"(bhi), "r"(idesc), "r"(sfa), "r"(sfb), "r"(FIRST ? more : 1u)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void st_shared(uint32_t at, float v) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory");
}
// Wait for an mbarrier phase with the hardware's own short suspension (a suspend-time
// hint polls, which took a third of the issue slots here).
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// A wait is bounded by its number of tries (kCostTries, 3.7 us each: a second; the time a
// preempted context spends off the GPU does not count).
//
// A warp that gives up waits for nothing more: producers and epilogues leave their loops, an
// MMA warp goes through its remaining steps with a limit of 0, issuing what nobody will use
// (which also ends the producers' waits).  The warps' waits run side by side, so a CTA ends
// within three bounds of a wait (an epilogue's, then an MMA warp's for the accumulator, then
// for the MMAs in flight) and sets *err; a CTA that starts after that does nothing.  So a launch
// that fails ends within about three seconds, whatever its number of tiles.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t tries) {
    for (uint32_t i = 0; i < tries; i++)
        if (mbar_try(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// true if any of the `count` threads on named barrier `id` passes true
__device__ __forceinline__ bool bar_any(int id, int count, bool v) {
    uint32_t r;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.or.pred q, %2, %3, p;\n selp.u32 %0, 1, 0, q;\n}"
        : "=r"(r)
        : "r"((uint32_t)v), "r"(id), "r"(count)
        : "memory");
    return r != 0;
}

// A code's 64 bits as 4-bit floats, nibble by nibble of its two words.  Each moving
// bit is used where it stands in its nibble, as 0.5, 1, 2 (bits 0, 1, 2) or as a
// sign (bit 3), so that a word costs one logic operation; the fixed code supplies
// the factor that makes the product of bit m and bit f
//   m (1 - 2 f) = (m ^ f) - f        (bits 0, 1, 2: factors +-2, +-1, +-1/2)
//   -(1 - 2 m)(1 - 2 f) / 2 = (m ^ f) - 1/2   (bit 3: the sign times -+1/2)
// so a code pair's dot product is popcount(m ^ f) - fixed_term(f).
__device__ __forceinline__ void tmem_st_moving(uint32_t addr, uint64_t c) {
    asm volatile(
        "{\n .reg .b32 w<8>;\n"
        " and.b32 w0, %1, 0x11111111;\n and.b32 w1, %1, 0x22222222;\n and.b32 w2, %1, 0x44444444;\n"
        " lop3.b32 w3, %1, 0x88888888, 0x22222222, 0xea;\n"
        " and.b32 w4, %2, 0x11111111;\n and.b32 w5, %2, 0x22222222;\n and.b32 w6, %2, 0x44444444;\n"
        " lop3.b32 w7, %2, 0x88888888, 0x22222222, 0xea;\n"
        " tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {w0, w1, w2, w3, w4, w5, w6, w7};\n}" ::"r"(addr),
        "r"((uint32_t)c), "r"((uint32_t)(c >> 32))
        : "memory");
}
__device__ __forceinline__ void expand_fixed(uint64_t c, uint32_t (&w)[8]) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const uint32_t v = (uint32_t)(c >> (32 * h));
        w[4 * h + 0] = ((v << 3) & 0x88888888u) | 0x44444444u;
        w[4 * h + 1] = ((v << 2) & 0x88888888u) | 0x22222222u;
        w[4 * h + 2] = ((v << 1) & 0x88888888u) | 0x11111111u;
        w[4 * h + 3] = (v & 0x88888888u) ^ 0x99999999u;
    }
}
__device__ __forceinline__ int fixed_term(uint64_t c) { return __popcll(c & 0x7777777777777777ull) + 8; }

// Producer and epilogue warpgroups: a sliding window expands a quarter of the codes
// per step and finishes as many labels, so it has one more epilogue warpgroup.
constexpr int kGroups = 5;
constexpr int epi_groups(bool slide) { return slide ? 3 : 2; }
constexpr int kMmaWarp = 4 * kGroups;
constexpr int kCostThreads = (kMmaWarp + 2) * 32;
constexpr int kRingCols = 12;  // x columns of operand A in tensor memory
constexpr int kDCols = 96;     // columns of all accumulators: one per epilogue warpgroup
constexpr int kEntryPitch = 132;  // entries [slot][128 moving rows]: neighbouring nodes' slots start in different banks
constexpr uint32_t kColD = 384, kColS = 480;  // tensor memory columns: A ring | accumulators | scales

// How a level's labels are cut into tiles (cost_plan).
struct CostPlan {
    int tn, SL;  // nodes per tile along y, slots per node
    int N;       // tn SL rounded up to 16
    int P, R;    // z offsets per step, moving rows of each: P R <= 128
    int nly;     // y labels per chunk
    int tiles_y, groups, groups_per_cta, splits, chunks;
    int pitch;   // moving rows per class of the split copy
    double clocks;  // of a column of tiles: all labels of one (x, z), on one SM
};

// The moving codes with each line's rows split by residue modulo q: class r, entry
// b = row r + q b of the line padded by `pad` clamped rows in front.
__global__ void k_split_rows(const uint64_t* __restrict__ M, uint64_t* __restrict__ Ms, int m, int pad, int q, int pitch) {
    const int e = blockIdx.y * blockDim.x + threadIdx.x;
    if (e >= q * pitch) return;
    const int r = e / pitch, b = e - r * pitch;
    const int64_t line = blockIdx.x;  // n o of them: too many for another grid axis
    Ms[line * q * pitch + e] = __ldg(M + line * m + clampi(r + q * b - pad, 0, m - 1));
}

// Ms: the split copy (q > 1) or the volume itself (q == 1, pitch 0).  SLIDE: a label
// step of 1 with every sample taken, where a step's window moves by one x column.
template <int G, bool SLIDE>
__global__ void __launch_bounds__(kCostThreads, 1)
    k_data_cost_mma(const uint64_t* __restrict__ F, const uint64_t* __restrict__ Ms, float* __restrict__ cost, int m,
                    int n, int o, int len, int q, CostPlan pl, float alpha1, uint32_t epi_tries, int* __restrict__ err) {
    constexpr int S = G > 4 ? 2 : 1;  // x and z sampling stride (RAND_SAMPLES=1, src/dataCostD.h:141-155)
    constexpr int NX = (G + S - 1) / S, NZ = NX, NC = NX * NZ;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t b_full[4], b_done[8], b_acc[3], b_free[3], b_turn[2], b_drain[2];
    __shared__ uint32_t s_tmem;
    __shared__ int s_failed;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int len2 = len * len, len3 = len2 * len;
    const int m1 = m / G, n1 = n / G;
    constexpr int kEpiGroups = epi_groups(SLIDE), kProdGroups = kGroups - kEpiGroups;
    constexpr int kMaxN = kDCols / kEpiGroups;  // slots of a tile at most
    constexpr int USTEP = SLIDE ? 1 : NX;  // new x columns per tile
    // shared memory: B [class][column][2][N][16 B] | entries [epilogue warpgroups][N][kEntryPitch] | fixed terms [tn]
    const uint32_t col_bytes = (uint32_t)pl.N * 32u;
    float* entries = reinterpret_cast<float*>(smem_raw + (size_t)q * NC * col_bytes);
    int* s_term = reinterpret_cast<int*>(entries + kEpiGroups * pl.N * kEntryPitch);
    int b = blockIdx.x;
    const int ty = b % pl.tiles_y;
    b /= pl.tiles_y;
    const int nxn = b % n1, nzn = b / n1;
    const int g_first = blockIdx.y * pl.groups_per_cta;
    const int n_groups = min(pl.groups_per_cta, pl.groups - g_first);
    const int ly0 = blockIdx.z * pl.nly;
    const int n_ly = min(pl.nly, len - ly0);
    const int group_tiles = q * len;
    int n_tiles = n_groups * group_tiles, n_steps = n_groups * len;
    const int y_first = ty * pl.tn, y0 = y_first * G;
    const int pad = q * (len - 1) / 2;
    const int y0_q = y0 / q, y0_res = y0 - y0_q * q;

    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&s_tmem))
                     : "memory");
        if (lane == 0) {
            for (int i = 0; i < 4; i++) mbar_init(&b_full[i], 4);
            for (int i = 0; i < 8; i++) mbar_init(&b_done[i], 1);
            for (int i = 0; i < kEpiGroups; i++) {
                mbar_init(&b_acc[i], 1);
                mbar_init(&b_free[i], 4);
            }
            for (int i = 0; i < 2; i++) {
                mbar_init(&b_turn[i], 1);
                mbar_init(&b_drain[i], 1);
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    if (tid == 0) s_failed = *(volatile int*)err;  // a wait of an earlier CTA gave up: no further waits
    for (int e = tid; e < pl.tn; e += kCostThreads) s_term[e] = 0;
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, s_tmem, 0);
    if (s_failed) n_tiles = n_steps = 0;
    if (warp < 4) {  // unit scales (E8M0 127) in every byte of the scale columns
        const uint32_t one = 0x7f7f7f7fu;
        const uint32_t w[8] = {one, one, one, one, one, one, one, one};
        const uint32_t at = tmem + kColS + ((uint32_t)(warp * 32) << 16);
        tmem_st8(at, w);
        tmem_st8(at + 8, w);
        tmem_wait_st();
    }
    // operand B: slot (t, s) of class r holds the fixed row f = r + q (a0 + s) where it is
    // one of node t's, else zero
    for (int e = tid; e < q * NC * pl.N; e += kCostThreads) {
        const int rc = e / pl.N, a = e - rc * pl.N;
        const int r = rc / NC, c = rc - r * NC;
        const int t = a / pl.SL, f = r + q * (t * G / q + a - t * pl.SL), j = c % NX, k = c / NX;
        uint32_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (t < pl.tn && f >= t * G && f < t * G + G && y0 + f < m) {
            const uint64_t code = F[(y0 + f) + (int64_t)(nxn * G + j * S) * m + (int64_t)(nzn * G + k * S) * m * n];
            expand_fixed(code, w);
            atomicAdd(&s_term[t], fixed_term(code));
        }
        uint4* d = reinterpret_cast<uint4*>(smem_raw + (size_t)rc * col_bytes + a * 16);
        d[0] = make_uint4(w[0], w[1], w[2], w[3]);
        d[pl.N] = make_uint4(w[4], w[5], w[6], w[7]);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();

    const auto wait_done = [&](int t) { return mbar_wait(&b_done[t & 7], (uint32_t)((t >> 3) & 1), kCostTries); };
    const uint32_t quadrant = (uint32_t)((warp & 3) * 32) << 16;
    const int row = tid & 127;
    const int p = row / pl.R, yb = row - p * pl.R;  // this thread's z offset and moving row
    bool ok = true;
    if (warp < 4 * kProdGroups) {
        // ---- producers
        const int wg = warp >> 2;
        const uint32_t line = q > 1 ? (uint32_t)(q * pl.pitch) : (uint32_t)m;
        // a row's place in its line: entry y0 / q + ly0 + yb of a class, or the clamped row
        const uint32_t at = q > 1 ? (uint32_t)(ly0 + yb) : (uint32_t)clampi(y0 + ly0 + yb - pad, 0, m - 1);
        uint32_t zo[NZ];  // this thread's place in the volume less the x offset (below 2^32: cost_plan)
        uint64_t code[NX][NZ];
        // the tile to load next: class r, x offset lx of group gi; x = tile of the group
        int r = 0, lx = 0, gi = 0, x = 0, col = 0;  // col: its first ring column
        auto next = [&]() {
            if (++r == q) { r = 0; lx++; }
            col += USTEP;
            if (++x == group_tiles) { x = 0; lx = 0; gi++; col += NX - USTEP; }
            if (col >= kRingCols) col -= kRingCols;
        };
        for (int i = 0; i < wg; i++) next();
        int group_set = -1;
        auto load = [&]() {
            if (gi != group_set) {
                group_set = gi;
                const int lz = (g_first + gi) * pl.P + p;
#pragma unroll
                for (int k = 0; k < NZ; k++)
                    zo[k] = at + (uint32_t)clampi(nzn * G + k * S + lz * q - pad, 0, o - 1) * (uint32_t)n * line;
            }
            const int cls = y0_res + r >= q ? y0_res + r - q : y0_res + r;
            const uint32_t off = q > 1 ? (uint32_t)(cls * pl.pitch + y0_q + (y0_res + r >= q)) : 0u;
#pragma unroll
            for (int j = 0; j < NX; j++) {
                if (SLIDE && x > 0 && j < NX - 1) continue;  // the column is in the ring
                const uint64_t* src = Ms + ((uint32_t)clampi(nxn * G + j * S + lx * q - pad, 0, n - 1) * line + off);
#pragma unroll
                for (int k = 0; k < NZ; k++) code[j][k] = __ldg(src + zo[k]);
            }
        };
        if (wg < n_tiles) load();
        for (int t = wg; t < n_tiles; t += kProdGroups) {
            // the columns overwritten were last read by tile t - 3 or before: a tile
            // moves the ring by at most NX <= 4 of its 12 columns.  (A parity tells a phase
            // only from its neighbours: every tile's phase is waited for in turn, so the one
            // before it is over, and the next use of a barrier is tile t + 3 or later, which
            // cannot be issued before this tile is in place, so none is missed.)
            for (int d = kProdGroups + 2; d >= 3 && ok; d--)
                if (t >= d) ok = wait_done(t - d);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tmem_fence_after();
            int cj = col;
#pragma unroll
            for (int j = 0; j < NX; j++) {
                if (!SLIDE || x == 0 || j == NX - 1) {
                    const uint32_t to = tmem + quadrant + (uint32_t)(cj * NZ * 8);
#pragma unroll
                    for (int k = 0; k < NZ; k++) tmem_st_moving(to + k * 8, code[j][k]);
                }
                cj = cj + 1 == kRingCols ? 0 : cj + 1;
            }
            for (int i = 0; i < kProdGroups; i++) next();
            if (t + kProdGroups < n_tiles) load();
            tmem_wait_st();
            tmem_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&b_full[t & 3]);
        }
    } else if (warp < kMmaWarp) {
        // ---- epilogue: warpgroup e takes steps e, e + kEpiGroups, ... from accumulator e
        const int e = (warp >> 2) - kProdGroups;
        const uint32_t acc = tmem + kColD + (uint32_t)(e * kMaxN) + quadrant;
        float* const mine = entries + e * pl.N * kEntryPitch;
        const uint32_t at = smem_u32(mine) + 4u * (uint32_t)row;
        const int ny_here = min(pl.tn, m1 - y_first);
        // this thread's sums: kSums at most in registers, others recomputed
        constexpr int kSums = 5;
        const int outputs = pl.P * pl.tn * pl.nly;
        int s_at[kSums], s_out[kSums], s_k[kSums];  // first entry, cost entry (-1: none), fixed term
        auto sum_of = [&](int x, int& from, int& to, int& term) {
            const int a = x / pl.nly, ly = x - a * pl.nly;  // x = (pp tn + node) nly + ly
            const int pp = a / pl.tn, node = a - pp * pl.tn;
            from = node * pl.SL * kEntryPitch + pp * pl.R + node * G / q + ly;
            to = x < outputs && node < ny_here && ly < n_ly ? node * len3 + pp * len2 + ly : -1;
            term = x < outputs ? s_term[node] : 0;
        };
#pragma unroll
        for (int i = 0; i < kSums; i++) sum_of(row + i * 128, s_at[i], s_out[i], s_k[i]);
        float* const cost0 = cost + (int64_t)(y_first + nxn * m1 + nzn * m1 * n1) * len3 + ly0;
        int lx = e, gi = 0;
        while (lx >= len) { lx -= len; gi++; }
        for (int st = e; st < n_steps; st += kEpiGroups) {
            ok = __all_sync(0xffffffffu, mbar_wait(&b_acc[e], (uint32_t)((st / kEpiGroups) & 1), epi_tries));
            if (ok) {
                tmem_fence_after();
#pragma unroll
                for (int c = 0; c < kMaxN; c += 16) {
                    if (c >= pl.N) break;
                    float v[16];
                    tmem_ld16(acc + c, v);
                    tmem_wait_ld();
#pragma unroll
                    for (int u = 0; u < 16; u++) st_shared(at + 4 * (c + u) * kEntryPitch, v[u]);
                }
                tmem_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&b_free[e]);
            }
            if (bar_any(1 + e, 128, !ok)) { ok = false; break; }
            const int lz0 = (g_first + gi) * pl.P;
            float* ct = cost0 + lx * len + lz0 * len2;
            auto emit = [&](int from, int to, int term) {
                float sum = (float)term;  // popcount = the entries + the fixed terms, exact
                #pragma unroll
                for (int i = 0; i < G; i++)
                    if (i < pl.SL) sum += mine[from + i * (kEntryPitch + 1)];
                ct[to] = __fmul_rn(sum, alpha1);
            };
            const bool whole = lz0 + pl.P <= len;  // the last group may have fewer z offsets
            if (whole) {
#pragma unroll
                for (int i = 0; i < kSums; i++)
                    if (s_out[i] >= 0) emit(s_at[i], s_out[i], s_k[i]);
            }
            for (int x = row + (whole ? kSums * 128 : 0); x < outputs; x += 128) {
                int from, to, term;
                sum_of(x, from, to, term);
                if (to >= 0 && lz0 + to % len3 / len2 < len) emit(from, to, term);
            }
            __syncwarp();
            bar_any(1 + e, 128, false);  // the entries are read
            lx += kEpiGroups;
            while (lx >= len) { lx -= len; gi++; }
        }
    } else {
        // ---- MMA warps: warp e issues steps e, e + 2, ... into the accumulators in turn
        // (e a constant of each copy: the operands' arithmetic stays uniform)
        const auto issue_steps = [&](auto which) {
        constexpr int e = decltype(which)::value;
        const uint32_t el = elect_one();
        uint32_t limit = kCostTries;  // 0 after a wait that gave up
        // M = 128, N, E2M1 operands, E8M0 scales, K = 64
        const uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(pl.N >> 3) << 17) | (1u << 23) | (1u << 27);
        // B: K-major without swizzle: 8 x 16 B core matrices, 128 B apart along the
        // rows, N * 16 B apart along K
        const uint32_t blo0 = ((smem_u32(smem_raw) & 0x3ffffu) >> 4) | ((uint32_t)pl.N << 16);
        const uint32_t bhi = 8u | (1u << 14), sf = tmem + kColS;
        int x = 0, col = 0;  // the step's number in its group, its first ring column
        const auto next = [&]() {
            col += q * USTEP;
            if (++x == len) { x = 0; col += NX - USTEP; }
            col %= kRingCols;
        };
        if (e) next();
        for (int st = e; st < n_steps; st += 2) {
            // (A wait that gives up only sets the limit of the waits that follow to 0: with a branch, or
            // with the issue made to depend on it, the operands leave the uniform registers and the
            // issue stalls, 1.9 -> 3.4 ms at grid 8.)
            bool in = true;
            // the other warp has seen every tile of its step in place, and its accumulator
            // free (a parity says nothing about the phase before it)
            if (st >= 1) in = mbar_wait(&b_turn[1 - e], (uint32_t)(((st - 1) >> 1) & 1), limit);
            const int acc = st % kEpiGroups;
            if (st >= kEpiGroups) in = in && mbar_wait(&b_free[acc], (uint32_t)((st / kEpiGroups - 1) & 1), limit);
            const uint32_t d = tmem + kColD + (uint32_t)(acc * kMaxN);
            ok = ok && in;
            int cj = col;
            uint32_t blo = blo0;
            for (int r = 0; r < q; r++) {
                const int t = st * q + r;
                limit = ok ? limit : 0u;
                ok = mbar_wait(&b_full[t & 3], (uint32_t)((t >> 2) & 1), limit) && ok;
                if (r == q - 1 && lane == 0) mbar_arrive(&b_turn[e]);
                tmem_fence_after();
                if (el) {
#pragma unroll
                    for (int j = 0; j < NX; j++) {
                        int c = cj + j;
                        c = c >= kRingCols ? c - kRingCols : c;
                        const uint32_t a = tmem + (uint32_t)(c * NZ * 8);
#pragma unroll
                        for (int k = 0; k < NZ; k++) {
                            const uint32_t bl = blo + (uint32_t)(k * NX + j) * (col_bytes >> 4);
                            if (j + k == 0) mma_mxf4<true>(d, a, bl, bhi, idesc, sf, sf + 8, (uint32_t)r);
                            else mma_mxf4<false>(d, a + k * 8, bl, bhi, idesc, sf, sf + 8, 1u);
                        }
                    }
                    mma_commit(&b_done[t & 7]);
                    if (r == q - 1) mma_commit(&b_acc[acc]);
                }
                __syncwarp();
                cj += NX;
                cj = cj >= kRingCols ? cj - kRingCols : cj;
                blo += (uint32_t)NC * (col_bytes >> 4);
            }
            next();
            next();
        }
        // no MMA is in flight when the memory is given back (a commit covers all MMAs of the
        // thread that issued them)
        if (n_steps > e) {
            if (el) mma_commit(&b_drain[e]);
            __syncwarp();
            ok = mbar_wait(&b_drain[e], 0, kCostTries) && ok;
        }
        };
        if (warp == kMmaWarp) issue_steps(std::integral_constant<int, 0>{});
        else issue_steps(std::integral_constant<int, 1>{});
    }
    if (!ok) atomicCAS(err, 0, 3);
    __syncwarp();  // the lanes left their last waits one by one; barrier and release want them together
    tmem_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

// Generic path (any grid spacing): one CTA per node, clamped global reads.
__global__ void __launch_bounds__(256) k_data_cost(const uint64_t* __restrict__ F, const uint64_t* __restrict__ M,
                                                   float* __restrict__ cost, int m, int n, int o, int g, int hw,
                                                   int q, int sy, int sx, int sz, float alpha1) {
    extern __shared__ uint64_t s_f[];
    const int m1 = m / g, n1 = n / g;
    const int node = blockIdx.x;
    const int z = node / (m1 * n1), x = (node / m1) % n1, y = node % m1;
    const int len = 2 * hw + 1, len3 = len * len * len;
    const int pad = q * hw;
    const int64_t mn = (int64_t)m * n;
    const int ny = (g + sy - 1) / sy, nx = (g + sx - 1) / sx, nz = (g + sz - 1) / sz;
    const int ns = ny * nx * nz;
    const int y1 = y * g, x1 = x * g, z1 = z * g;
    for (int s = threadIdx.x; s < ns; s += blockDim.x) {
        const int si = s % ny, sj = (s / ny) % nx, sk = s / (ny * nx);
        s_f[s] = F[(y1 + si * sy) + (int64_t)(x1 + sj * sx) * m + (int64_t)(z1 + sk * sz) * mn];
    }
    __syncthreads();
    for (int l = threadIdx.x; l < len3; l += blockDim.x) {
        const int lz = l / (len * len), lx = (l / len) % len, ly = l % len;
        const int yb = y1 + ly * q - pad, xb = x1 + lx * q - pad, zb = z1 + lz * q - pad;
        int acc = 0;
        int s = 0;
        for (int k = 0; k < nz; k++) {
            const int64_t zo = (int64_t)clampi(zb + k * sz, 0, o - 1) * mn;
            for (int jj = 0; jj < nx; jj++) {
                const uint64_t* row = M + zo + (int64_t)clampi(xb + jj * sx, 0, n - 1) * m;
                for (int i = 0; i < ny; i++, s++) acc += __popcll(s_f[s] ^ __ldg(row + clampi(yb + i * sy, 0, m - 1)));
            }
        }
        cost[(int64_t)node * len3 + l] = __fmul_rn((float)acc, alpha1);
    }
}

constexpr int kMaxSmem = 200 * 1024;
size_t cost_smem(const CostPlan& c, int g, int q) {
    const int S = g > 4 ? 2 : 1, NX = (g + S - 1) / S;
    return (size_t)q * NX * NX * c.N * 32 + (size_t)epi_groups(q == 1 && g <= 4) * c.N * kEntryPitch * 4 + (size_t)c.tn * 4;
}

// The tile that makes a level cheapest, in clocks.  Measured per class: 33 per MMA
// (its issue; N / 2 above N = 64) and 320 for the hand-overs; with a sliding window
// the two issuing warps overlap.  A step's epilogue: 16 per slot, 270 per 128 sums.
// A CTA's start: 3500 and the fixed rows.
bool cost_plan(int m, int n, int o, int g, int len, int q, CostPlan& best) {
    if (g < 2 || g > 8 || len < 3 || q < 1 || q > 64) return false;
    const int S = g > 4 ? 2 : 1, NX = (g + S - 1) / S, NC = NX * NX;
    const int m1 = m / g, n1 = n / g, o1 = o / g;
    const int ustep = q == 1 && S == 1 ? 1 : NX;
    // y labels per chunk: all of them unless they alone exceed the 128 rows
    int chunks = 1;
    while ((len + chunks - 1) / chunks - 1 + (g + q - 1) / q > 128) chunks++;
    const int nly = (len + chunks - 1) / chunks;
    chunks = (len + nly - 1) / nly;
    double best_t = 1e300;
    for (int tn = 1; tn <= m1; tn++) {
        CostPlan c{};
        c.tiles_y = (m1 + tn - 1) / tn;
        if (tn > 1 && (m1 + tn - 2) / (tn - 1) == c.tiles_y) continue;  // fewer rows give the same tile count
        c.tn = tn;
        c.SL = (g + q - 1 + q - 1) / q;
        if (g % q == 0) c.SL = g / q;
        c.N = (tn * c.SL + 15) / 16 * 16;
        c.R = (tn - 1) * g / q + c.SL + nly - 1;
        c.nly = nly;
        c.chunks = chunks;
        if (c.N > kDCols / epi_groups(q == 1 && g <= 4) || c.R > 128) break;
        for (c.P = 1; c.P * c.R <= 128 && c.P <= len; c.P++) {
            c.groups = (len + c.P - 1) / c.P;
            if (c.P > 1 && c.groups == (len + c.P - 2) / (c.P - 1)) continue;
            if (cost_smem(c, g, q) > kMaxSmem) continue;
            const bool slide = q == 1 && g <= 4;
            const double rounds = (c.P * tn * nly + 127) / 128;
            const double mma = slide ? NC * 22.0 + 350.0 : q * (NC * 33.0 + 320.0);
            const double epi = (250.0 + 16.0 * c.N + 270.0 * rounds) / epi_groups(slide);
            const double start = 3500.0 + q * NC * c.N * 0.8;
            const double t = (std::max(mma, epi) * len * c.groups + start) * c.tiles_y;
            if (t < best_t) {
                best_t = c.clocks = t;
                best = c;
            }
        }
    }
    if (best_t == 1e300) return false;
    // rows per class: the last tile's rows (beyond the volume too) and the label reach
    best.pitch = q > 1 ? (best.tiles_y * best.tn * g + q - 1) / q + chunks * nly + 2 : 0;
    if ((uint64_t)std::max(m, q * best.pitch) * n * o >= (1ull << 32) || q * best.pitch > 128 * 65535) return false;
    // enough CTAs for several waves of one per SM
    const int64_t cols = (int64_t)best.tiles_y * n1 * o1 * chunks;
    int splits = 1;
    while (splits < best.groups && cols * splits < 8 * 152) splits++;
    best.groups_per_cta = (best.groups + splits - 1) / splits;
    best.splits = (best.groups + best.groups_per_cta - 1) / best.groups_per_cta;
    return true;
}

template <int G, bool SLIDE>
cudaError_t launch_mma(const uint64_t* d_F, const uint64_t* d_Ms, int m, int n, int o, int len, int q,
                       const CostPlan& pl, float alpha1, float* d_cost, int* d_err, uint32_t epi_tries, cudaStream_t s) {
    const size_t smem = cost_smem(pl, G, q);
    // the same limit on every call: other threads launch the kernel for other sizes
    cudaError_t e = cudaFuncSetAttribute(k_data_cost_mma<G, SLIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    if (e != cudaSuccess) return e;
    const dim3 grid((unsigned)(pl.tiles_y * (n / G) * (o / G)), (unsigned)pl.splits, (unsigned)pl.chunks);
    k_data_cost_mma<G, SLIDE>
        <<<grid, kCostThreads, smem, s>>>(d_F, d_Ms, d_cost, m, n, o, len, q, pl, alpha1, epi_tries, d_err);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace

namespace {
// Code pairs a call compares.
double cost_pairs(int m, int n, int o, int g, int len) {
    const int S = g > 4 ? 2 : 1, NX = (g + S - 1) / S;
    return (double)(m / g) * (n / g) * (o / g) * len * len * len * g * NX * NX;
}
// The integer kernel is the faster one for few labels an axis, where an MMA step has few
// columns of labels against a CTA's start and its classes' hand-overs, and at grid 2, whose
// steps have one or two live classes.  Measured at 192x160x256, integer pipe and tensor cores,
// each with its copy (the ratio differs little at 113x97x131 and 96x80x112):
//   3 and 5 labels, always: grid 4, 5 labels, step 1: 466 us, 830; grid 8, 5 labels, step 2:
//     156, 215;
//   7 labels: grid 5, step 2: 437, 715; grid 4, step 1: 1083, 1388.  Grids 4, 7 and 8 fill a step of
//     the tensor cores better at label steps of 3 to 8: grid 4, step 4: 1310, 952 (step 12:
//     1520, 3770);
//   grid 2 with steps above 1: 96x80x112, 11 labels, step 2: 0.66 of the time.
// With 9 labels the sums no longer stay in registers: grid 4, step 1: 5.2 ms, 1.39.
bool popc_faster(int g, int len, int q) {
    if (len == 7) return q < 3 || q > 8 || !(g == 4 || g == 7 || g == 8);
    return len < 7 || (g == 2 && q > 1);
}
// Large label steps leave most of a tile's classes almost empty, and one node's samples in
// registers' reach do better: the generic kernel compares 2 to 4 code pairs a clock and SM
// whatever the step (21x150x33, grid 5, 11 labels, step 12: 61 us, tensor cores 138;
// 96x80x112, grid 4, 9 labels, step 28: no tile, 0.63 ms).  A CTA takes 4000 clocks more
// than cost_plan's start.
bool generic_faster(int m, int n, int o, int g, int len, const CostPlan& pl) {
    const double sm_clocks = 152.0, us = 2070.0;
    const double columns = (double)(n / g) * (o / g) * pl.chunks;
    const double ctas = columns * pl.tiles_y * pl.splits;
    const double per_cta = pl.clocks / pl.tiles_y / pl.splits + 4000.0;
    const double mma = std::max(1.0, ctas / sm_clocks) * per_cta / us;
    return cost_pairs(m, n, o, g, len) / (2.2 * sm_clocks * us) + 10.0 < mma / 0.85;
}
}  // namespace

CostPath data_cost_path(int m, int n, int o, int g, int hw, int q) {
    CostPlan pl;
    const int len = 2 * hw + 1;
    if (popc_faster(g, len, q)) {
        // its padded copy must not outweigh the sums (a word costs as much as six pairs), or be
        // small (8 MB: 4 us)
        const size_t pad = data_cost_popc_count(m, n, o, g, hw, q);
        if (pad > 0 && (pad <= (1u << 20) || 4.0 * pad <= cost_pairs(m, n, o, g, len))) return CostPath::kPopc;
        // small steps do not fit only where an axis has more lines than a launch grid takes
        return q <= 8 && cost_plan(m, n, o, g, len, q, pl) ? CostPath::kMma : CostPath::kGeneric;
    }
    const bool mma = cost_plan(m, n, o, g, len, q, pl);
    return mma && (len == 7 || !generic_faster(m, n, o, g, len, pl)) ? CostPath::kMma : CostPath::kGeneric;
}

size_t data_cost_scratch_count(int m, int n, int o, int g, int hw, int q) {
    CostPlan pl;
    switch (data_cost_path(m, n, o, g, hw, q)) {
        case CostPath::kPopc: return data_cost_popc_count(m, n, o, g, hw, q);
        case CostPath::kMma: return cost_plan(m, n, o, g, 2 * hw + 1, q, pl) ? (size_t)pl.pitch * q * n * o : 0;
        default: return 0;
    }
}

cudaError_t launch_data_cost_mma(const uint64_t* d_F, const uint64_t* d_M, uint64_t* d_split, int m, int n, int o,
                                 int g, int hw, int q, float alpha1, float* d_cost, int* d_err, cudaStream_t s,
                                 uint32_t epi_tries) {
    CostPlan pl;
    const int len = 2 * hw + 1;
    if (!cost_plan(m, n, o, g, len, q, pl)) return cudaErrorInvalidValue;
    const uint64_t* d_Ms = d_M;
    if (q > 1) {
        k_split_rows<<<dim3(n * o, (q * pl.pitch + 127) / 128), 128, 0, s>>>(d_M, d_split, m, q * hw, q, pl.pitch);
        count_launches(1);
        if (const cudaError_t e = cudaGetLastError(); e != cudaSuccess) return e;
        d_Ms = d_split;
    }
#define DEEDS_MMA_ARGS d_F, d_Ms, m, n, o, len, q, pl, alpha1, d_cost, d_err, epi_tries, s
    switch (g) {
        case 2: return q == 1 ? launch_mma<2, true>(DEEDS_MMA_ARGS) : launch_mma<2, false>(DEEDS_MMA_ARGS);
        case 3: return q == 1 ? launch_mma<3, true>(DEEDS_MMA_ARGS) : launch_mma<3, false>(DEEDS_MMA_ARGS);
        case 4: return q == 1 ? launch_mma<4, true>(DEEDS_MMA_ARGS) : launch_mma<4, false>(DEEDS_MMA_ARGS);
        case 5: return launch_mma<5, false>(DEEDS_MMA_ARGS);
        case 6: return launch_mma<6, false>(DEEDS_MMA_ARGS);
        case 7: return launch_mma<7, false>(DEEDS_MMA_ARGS);
        default: return launch_mma<8, false>(DEEDS_MMA_ARGS);
    }
#undef DEEDS_MMA_ARGS
}

cudaError_t launch_data_cost(const uint64_t* d_F, const uint64_t* d_M, int m, int n, int o, int g, int hw, int q,
                             int sy, int sx, int sz, float alpha1, float* d_cost, cudaStream_t s) {
    const int sz1 = (m / g) * (n / g) * (o / g);
    const int ns = ((g + sy - 1) / sy) * ((g + sx - 1) / sx) * ((g + sz - 1) / sz);
    const size_t smem = (size_t)ns * sizeof(uint64_t);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_data_cost, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             std::max(kMaxSmem, (int)smem));  // as above: one limit for all
        if (e != cudaSuccess) return e;
    }
    const int len3 = (2 * hw + 1) * (2 * hw + 1) * (2 * hw + 1);
    const int threads = len3 >= 256 ? 256 : ((len3 + 31) / 32) * 32;
    k_data_cost<<<sz1, threads, smem, s>>>(d_F, d_M, d_cost, m, n, o, g, hw, q, sy, sx, sz, alpha1);
    count_launches(1);
    return cudaGetLastError();
}

namespace {
// Register-only throughput probe of the cost-volume inner operation
// (64-bit XOR, two 32-bit POPC, accumulate): 8 independent chains per thread.
__global__ void k_popc_probe(int iters, unsigned long long* sink) {
    // the cost volume's inner operation, register only: nine 64-bit samples per
    // iteration, each XORed with its own key, summed three at a time through the
    // carry-save adder (two 64-bit POPCs per three samples)
    uint64_t v[9];
    int acc[3] = {0, 0, 0};
#pragma unroll
    for (int j = 0; j < 9; j++) v[j] = 0x9E3779B97F4A7C15ull * (uint64_t)(threadIdx.x * 9 + j + 1) ^ (uint64_t)blockIdx.x;
    uint64_t k1 = (uint64_t)clock64(), k2 = k1 * 0x2545F4914F6CDD1Dull, k3 = k1 ^ 0xD1B54A32D192ED03ull;
    for (int it = 0; it < iters; it++) {
#pragma unroll
        for (int g = 0; g < 3; g++) {
            const uint64_t a = v[3 * g] ^ k1, b = v[3 * g + 1] ^ k2, x = v[3 * g + 2] ^ k3;
            const uint64_t sum = a ^ b ^ x, carry = (a & b) | (x & (a ^ b));
            acc[g] += __popcll(sum) + 2 * __popcll(carry);
        }
        k1 += 0x5851F42D4C957F2Dull;
        k2 ^= k1;
        k3 += k2;
    }
    const int t = acc[0] + acc[1] + acc[2];
    if (t == -1) sink[0] = (unsigned long long)t;  // never true; keeps the loop live
}
}  // namespace

cudaError_t launch_popc_probe(int blocks, int threads, int iters, unsigned long long* d_sink, cudaStream_t s) {
    k_popc_probe<<<blocks, threads, 0, s>>>(iters, d_sink);
    count_launches(1);
    return cudaGetLastError();
}

namespace {
// Self-test of the cost volume's bounded mbarrier wait: an mbarrier that expects
// one arrival which never comes; status = 1 if the wait gave up, 2 otherwise.
__global__ void k_selftest_mbar_wait(int* status) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        *status = mbar_wait(&bar, 0, kCostTries) ? 2 : 1;
    }
}
}  // namespace

cudaError_t launch_selftest_mbar_wait(int* status, cudaStream_t s) {
    k_selftest_mbar_wait<<<1, 32, 0, s>>>(status);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace deeds
