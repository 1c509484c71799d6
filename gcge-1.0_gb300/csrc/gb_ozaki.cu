// gb_ozaki.cu -- FP64-accurate dense contractions of the solver on the tcgen05
// tensor cores.
//
// GB300 runs FP64 at ~1.2 TFLOP/s (FP64 tensor MMA no faster) while its f16
// tensor cores run at ~2 PFLOP/s. The two dense contractions of the solver -- the
// Gram product V^T W and the linear combination X C -- therefore use an
// error-free splitting in the style of the Ozaki scheme (Ozaki, Ogita, Oishi,
// Rump, Numer. Algorithms 59, 2012), restated here:
//
//  * every FP64 entry is written against a power-of-two scale of its row or
//    column (gb_tc05.h: oz_bias) as seven balanced base-256 digits, each exact
//    in f16, with integer operations only;
//  * a product x y is sum_{p,q} d_p d'_q 2^(-8(p+q)) 2^(e + f - 10); the digit
//    pairs of levels p + q < 8 are kept (34 pairs; the dropped ones lie below
//    2^-57 of the scale product per term);
//  * all pairs of one level L = p + q share one FP32 accumulator in TMEM, which
//    stays an exact integer for up to OZ_EXACT_TERMS terms; it is drained at
//    most every OZ_EXACT_TERMS terms into exact int64 sums (levels 0-2 and the
//    lower ones) that are rounded once to FP64 (oz_to_double).
//
// Both kernels share one structure (tcgen05, 128 x 64 output tile per CTA):
//  * 16 warps, one CTA per SM; warps 0-14 split FP64 operands into f16 digit
//    planes in shared memory (two stages of K = 32, no-swizzle K-major core
//    matrices), lane 0 of warp 15 issues the digit-pair MMAs of a stage
//    (M = 128, K = 16, accumulators: 8 levels x N TMEM columns, N = 16 .. 64), and
//    all 16 warps drain TMEM (warp w: lanes 32 (w % 4) .. +31, columns 4 (w / 4)
//    .. +3 of every 16, so that a narrow output is shared by all of them);
//  * hand-offs through mbarriers: full[b] (stage b written, 480 arrivals),
//    empty[b] (MMAs of stage b done, tcgen05.commit), drained (TMEM read out,
//    512 arrivals), copied[b] (bulk copy of the pre-split planes of stage b);
//    every wait is bounded and reports a timeout through the context's device
//    error word;
//  * the next stage's FP64 values are on their way while the MMAs of the current one
//    run: registers in k_lincomb_tc; in k_gram_tc, whose sums fill the registers, a
//    lane's own slot of shared memory (cp.async, one group per core matrix, refilled as
//    soon as it has been read).
// k_lincomb_tc: Y = alpha X C + beta Y, M = 128 rows of X, K = columns of X,
//   per-row scales (of X equilibrated by the row scales of C), C split once per
//   call by k_lc_coef_split;
// k_gram_tc: V^T W, M = 128 columns of V, N = 64 columns of W, K = rows of a
//   row split, per-column scales from a pre-pass (k_col_exponent); the splits'
//   exact integer sums meet in atomics (any order, the same value) and the split
//   that comes last rounds them to FP64.
#include <cstdint>
#include <cuda_runtime.h>

#include "gb_internal.h"
#include "gb_launch.h"
#include "gb_tc05.h"

#define GB_PROF(ctx, cls, bytes, flops) \
    do { if ((ctx)->prof) gb_prof_begin((ctx), (cls), (bytes), (flops)); } while (0)

extern "C" int gb_gram_reduce_launch(gcge_gpu_ctx *ctx, int k1, int k2, int nsplit, const double *part,
                                     double *a_dev, int lda, int sym);

// ---------------------------------------------------------------- tile geometry
#define TC_M 128                                     // MMA M, TMEM lanes
#define TC_N 64                                      // columns of a tile (max), TMEM columns per level
#define TC_KS 32                                     // K per pipeline stage
#define TC_APLANE (TC_M * TC_KS * 2)                 // bytes of one f16 digit plane, A operand
#define TC_BPLANE (TC_N * TC_KS * 2)                 // and, at most, B operand
#define TC_STAGE (OZ_DIGITS * (TC_APLANE + TC_BPLANE))
#define TC_HDR 1024                                  // mbarriers, TMEM address, flags, scales
#define TC_WARPS 16
#define TC_THREADS (32 * TC_WARPS)
#define TC_SPLIT_WARPS (TC_WARPS - 1)
#define TC_SPLIT_THREADS (32 * TC_SPLIT_WARPS)
#define TC_ACORES (TC_M / 8 * TC_KS / 8)             // core matrices of the A operand per stage
#define TC_BCORES (TC_N / 8 * TC_KS / 8)
#define TC_COLS_PER_WARP (TC_N * 4 / TC_WARPS)       // output columns drained per warp (16)
#define TC_TMEM_COLS 512
#define TC_WAIT_NS 1000000000ull
// Core-matrix layout of one digit plane (no swizzle, K-major): the 8-row x
// 8-element core matrix (g, c) -- rows 8g..8g+7, K 8c..8c+7 of the stage --
// occupies bytes [(4g + c) 128, +128), row by row (16 bytes each). K-adjacent
// core matrices are 128 bytes apart, row-group-adjacent ones 512.
#define TC_LBO 128
#define TC_SBO 512
// stages per exact accumulation when the K range is longer than OZ_EXACT_TERMS
#define TC_CHUNK_STAGES (OZ_EXACT_TERMS / TC_KS)

// shared header of both kernels
struct tc_hdr {
    uint64_t bar[8];             // full[2], empty[2], drained, copied[2] (bulk copies of a stage), scales
    uint32_t tmem;
    int flag;                    // a bounded wait ran out in this CTA
};
static_assert(sizeof(tc_hdr) <= 80, "header overlaps the scale arrays");

__device__ __forceinline__ void tc_fail(tc_hdr *h, int *err)
{
    h->flag = 1;
    atomicExch(err, 1);
}

// CTA start: TMEM allocation (warp 0), mbarrier initialisation (thread 0)
__device__ __forceinline__ void tc_setup(tc_hdr *h)
{
    if ((threadIdx.x >> 5) == 0) tc_tmem_alloc(tc_smem_addr(&h->tmem), TC_TMEM_COLS);
    if (threadIdx.x == 0) {
        const uint32_t b = tc_smem_addr(h->bar);
        tc_mbar_init(b, TC_SPLIT_THREADS);
        tc_mbar_init(b + 8, TC_SPLIT_THREADS);
        tc_mbar_init(b + 16, 1);
        tc_mbar_init(b + 24, 1);
        tc_mbar_init(b + 32, TC_THREADS);
        tc_mbar_init(b + 40, 1);
        tc_mbar_init(b + 48, 1);
        tc_mbar_init(b + 56, TC_SPLIT_THREADS);
        h->flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
}

// the digit-pair MMAs of the stage whose planes begin at a0 (see tc_issue_stage)
template <int LEVELS, int N>
__device__ __forceinline__ void tc_issue_mmas(uint32_t a0, uint32_t tmem, bool first)
{
    constexpr int GROUP = 256 / N < OZ_DIGITS ? 256 / N : OZ_DIGITS;   // B digits of one MMA
    const uint32_t b0 = a0 + OZ_DIGITS * TC_APLANE;
#pragma unroll
    for (int ks = 0; ks < TC_KS / 16; ++ks) {
        const bool over = first && ks == 0;
#pragma unroll
        for (int p = 0; p < OZ_DIGITS; ++p) {
            const int qmax = (LEVELS - 1 - p < OZ_DIGITS - 1) ? LEVELS - 1 - p : OZ_DIGITS - 1;
            const uint64_t ad = tc_sdesc(a0 + p * TC_APLANE + ks * 256, TC_LBO, TC_SBO);
#pragma unroll
            for (int q0 = 0; q0 <= qmax; q0 += GROUP) {
                const int nq = qmax - q0 + 1 < GROUP ? qmax - q0 + 1 : GROUP;
                const bool begins = p == 1 && q0 + nq == OZ_DIGITS;    // its last pair begins level OZ_DIGITS
                const uint64_t bd = tc_sdesc(b0 + q0 * (N * TC_KS * 2) + ks * 256, TC_LBO, TC_SBO);
                if (begins && over) {
                    if (nq > 1) tc_mma_kf16(tmem + (p + q0) * N, ad, bd, tc_idesc_f16(TC_M, N * (nq - 1)), 1u);
                    tc_mma_kf16(tmem + OZ_DIGITS * N, ad,
                                tc_sdesc(b0 + (OZ_DIGITS - 1) * (N * TC_KS * 2) + ks * 256, TC_LBO, TC_SBO),
                                tc_idesc_f16(TC_M, N), 0u);
                } else {
                    tc_mma_kf16(tmem + (p + q0) * N, ad, bd, tc_idesc_f16(TC_M, N * nq), p == 0 && over ? 0u : 1u);
                }
            }
        }
    }
}

// MMA issue of stage s (lane 0 of the MMA warp): wait for the stage's planes
// (and, at the first stage of a chunk, for the previous chunk's drain), issue the
// digit pairs with p + q < LEVELS x TC_KS / 16 K steps, commit to empty[buf].
// The B digit planes of a stage (N rows, N a multiple of 16) lie back to back with the
// same 512-byte stride between 8-row groups, and level L of the accumulator is TMEM
// columns N L .. N L + N - 1, so the pairs (p, q0) .. (p, q0 + j - 1) are one MMA with
// N j <= 256 columns whose D starts at level p + q0: 11 MMAs per K step at N = 64 and
// 7 at N = 16 instead of 34, and each A plane is read from shared memory once per such group instead of once per pair. The first K
// step of a chunk overwrites: with p = 0, and the one level that begins with p = 1 by
// an MMA of its own. (With planes of 64 rows whatever N, and the first step pairwise, a
// stage's MMAs ended 2.2 us after its split at any N.)
// stall (test hook, GCGE_GPU_TestStallTensorWait): before the first stage the
// issuing thread waits for the first drain, an arrival that cannot come before
// the MMAs it would issue, so that bounded wait runs out and the CTA takes the
// timeout path (no MMA is issued; the other warps' waits run out in turn).
template <int LEVELS, bool COPIED>
__device__ __forceinline__ void tc_issue_stage(tc_hdr *h, uint32_t sbase, uint32_t tmem, int N, int s, int cs,
                                               int *commits, int *err, int stall)
{
    const int buf = s & 1;
    const uint32_t full = tc_smem_addr(h->bar) + 8 * buf, empty = tc_smem_addr(h->bar) + 16 + 8 * buf;
    const uint32_t drained = tc_smem_addr(h->bar) + 32, copied = tc_smem_addr(h->bar) + 40 + 8 * buf;
    if (stall && s == 0 && !tc_mbar_wait(drained, 0, TC_WAIT_NS)) {
        tc_fail(h, err);
        return;
    }
    bool ok = tc_mbar_wait(full, (s >> 1) & 1, TC_WAIT_NS);
    if (COPIED && ok) ok = tc_mbar_wait(copied, (s >> 1) & 1, TC_WAIT_NS);
    if (ok && cs == 0 && s > 0) ok = tc_mbar_wait(drained, (commits[2] - 1) & 1, TC_WAIT_NS);
    if (!ok || *(volatile int *)&h->flag) {
        tc_fail(h, err);
        return;
    }
    tc_fence_after_sync();
    const uint32_t a0 = sbase + buf * TC_STAGE;
    if (N == 16) tc_issue_mmas<LEVELS, 16>(a0, tmem, cs == 0);
    else if (N == 32) tc_issue_mmas<LEVELS, 32>(a0, tmem, cs == 0);
    else if (N == 48) tc_issue_mmas<LEVELS, 48>(a0, tmem, cs == 0);
    else tc_issue_mmas<LEVELS, 64>(a0, tmem, cs == 0);
    tc_mma_commit(empty);
    ++commits[buf];
}

// TMEM read-out of 4 columns x LEVELS levels for this thread's lane (row of the tile)
template <int LEVELS>
__device__ __forceinline__ void tc_load_levels4(uint32_t taddr, int N, uint32_t v[][4])
{
#pragma unroll
    for (int L = 0; L < LEVELS; ++L)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(v[L][0]), "=r"(v[L][1]), "=r"(v[L][2]), "=r"(v[L][3])
                     : "r"(taddr + L * N));
    tc_tmem_wait_ld();
#pragma unroll
    for (int L = 0; L < LEVELS; ++L) asm volatile("" : "+r"(v[L][0]), "+r"(v[L][1]), "+r"(v[L][2]), "+r"(v[L][3]));
}

// wait for the chunk's last MMAs before the drain
__device__ __forceinline__ bool tc_wait_chunk(tc_hdr *h, int s, int *err)
{
    const uint32_t empty = tc_smem_addr(h->bar) + 16 + 8 * (s & 1);
    if (!tc_mbar_wait(empty, (s >> 1) & 1, TC_WAIT_NS)) tc_fail(h, err);
    if (*(volatile int *)&h->flag) return false;
    tc_fence_after_sync();
    return true;
}

// copies: bulk copies issued per buffer by thread 0 (nullptr if none)
__device__ __forceinline__ void tc_release(tc_hdr *h, uint32_t tmem, int mma_warp, const int *commits,
                                           const int *copies)
{
    __syncthreads();
    if (*(volatile int *)&h->flag) {
        // after a timeout: wait (bounded) for the MMAs and copies still in flight
        if (mma_warp && (threadIdx.x & 31) == 0) {
            const uint32_t e = tc_smem_addr(h->bar) + 16;
            if (commits[0]) tc_mbar_wait(e, (commits[0] - 1) & 1, TC_WAIT_NS);
            if (commits[1]) tc_mbar_wait(e + 8, (commits[1] - 1) & 1, TC_WAIT_NS);
        }
        if (copies && threadIdx.x == 0) {
            const uint32_t c = tc_smem_addr(h->bar) + 40;
            if (copies[0]) tc_mbar_wait(c, (copies[0] - 1) & 1, TC_WAIT_NS);
            if (copies[1]) tc_mbar_wait(c + 8, (copies[1] - 1) & 1, TC_WAIT_NS);
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if ((threadIdx.x >> 5) == 0) {
        tc_fence_after_sync();
        tc_tmem_dealloc(tmem, TC_TMEM_COLS);
    }
}

// ---------------------------------------------------------------- Gram column scales
// exps[c] = smallest e with |X[r, c]| < 2^e for all rows (OZ_NO_EXP for an
// all-zero column; subnormal entries count as zero). exps must hold OZ_NO_EXP
// on entry. A warp reads whole rows over 256-column chunks, so each row's bytes stream
// once per chunk; each block reduces its warps and issues one atomic per column.
#define CE_COLS 256

// f(j, entry) for the entries of columns lane + 32 j < kc of the warp's rows (zeros past
// them), eight loads in flight: of one row when it has more than 128 columns, of eight when
// it has 32. (One row at a time, 110592 x 60 and x 20 kept two loads and one: 28.3 -> 16.1 us.)
template <int NJ, class F>
__device__ __forceinline__ void ce_walk(int n, int kc, const double *__restrict__ X, long ldx, long warp, long nw, F f)
{
    constexpr int U = CE_COLS / 32 / NJ;
    const int lane = threadIdx.x & 31;
    for (long r = warp; r < n; r += U * nw) {
        double v[U][NJ];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int j = 0; j < NJ; ++j)
                v[u][j] = r + u * nw < n && lane + 32 * j < kc ? __ldg(X + (r + u * nw) * ldx + lane + 32 * j) : 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int j = 0; j < NJ; ++j) f(j, v[u][j]);
    }
}
template <class F>
__device__ __forceinline__ void ce_rows(int n, int kc, const double *__restrict__ X, long ldx, long warp, long nw, F f)
{
    if (kc <= 32) ce_walk<1>(n, kc, X, ldx, warp, nw, f);
    else if (kc <= 64) ce_walk<2>(n, kc, X, ldx, warp, nw, f);
    else if (kc <= 128) ce_walk<4>(n, kc, X, ldx, warp, nw, f);
    else ce_walk<CE_COLS / 32>(n, kc, X, ldx, warp, nw, f);
}

// grid (blocks, 2): blockIdx.y = 0 the columns of V (exps[0:k1]), 1 those of W
// (exps[k1:]) -- one launch, so that the two short passes share the chip.
__global__ void __launch_bounds__(256)
k_col_exponent(int n, int k1, const double *__restrict__ V, long ldv, int k2, const double *__restrict__ W, long ldw,
               int *__restrict__ exps)
{
    GB_PDL();
    __shared__ int se[8][CE_COLS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int k = blockIdx.y ? k2 : k1;
    const double *X = blockIdx.y ? W : V;
    const long ldx = blockIdx.y ? ldw : ldv;
    if (blockIdx.y) exps += k1;
    const long warp = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long nw = ((long)gridDim.x * blockDim.x) >> 5;
    for (int c0 = 0; c0 < k; c0 += CE_COLS) {
        int e[CE_COLS / 32];
#pragma unroll
        for (int j = 0; j < CE_COLS / 32; ++j) e[j] = OZ_NO_EXP;
        ce_rows(n, min(CE_COLS, k - c0), X + c0, ldx, warp, nw,
                [&](int j, double x) { e[j] = max(e[j], oz_exponent(x)); });
#pragma unroll
        for (int j = 0; j < CE_COLS / 32; ++j) se[w][lane + 32 * j] = e[j];
        __syncthreads();
        for (int c = threadIdx.x; c < CE_COLS; c += blockDim.x) {
            int m = se[0][c];
#pragma unroll
            for (int q = 1; q < 8; ++q) m = max(m, se[q][c]);
            if (c0 + c < k && m > OZ_NO_EXP) atomicMax(exps + c0 + c, m);
        }
        __syncthreads();
    }
}

// start of a Gram: column exponents unset, tickets and integer sums zero (a grid of at most
// 65,536 threads, whatever their number)
__global__ void k_gram_init(int *__restrict__ exps, int cols, unsigned *__restrict__ ticket, int tiles,
                            ulonglong2 *__restrict__ sums, long total)
{
    GB_PDL();
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x, step = (long)gridDim.x * blockDim.x;
    for (long t = i; t < cols; t += step) exps[t] = OZ_NO_EXP;
    for (long t = i; t < tiles; t += step) ticket[t] = 0;
    for (long t = i; t < total; t += step) sums[t] = make_ulonglong2(0, 0);
}

// ---------------------------------------------------------------- Gram V^T W (tcgen05)
// core matrices a warp splits per stage: of V, and of W (dealt from the last warp down, so
// that no warp has the odd one of both)
#define GR_A ((TC_ACORES + TC_SPLIT_WARPS - 1) / TC_SPLIT_WARPS)
#define GR_B ((TC_BCORES + TC_SPLIT_WARPS - 1) / TC_SPLIT_WARPS)
#define GR_CORES_PER_WARP (GR_A + GR_B)
// Levels 0-7 (34 digit pairs, 8 x 64 TMEM columns), as the linear combination:
// the dropped pairs (level >= 8) add at most 2^-57.4 of the column-scale product
// 2^(e+f) per row, so over n rows the error stays below 2^-57.4 n 2^(e+f) even
// when every row drops the same amount (e.g. constant columns) -- far below the
// FP64 summation error of the same Gram. Levels 3-7 are summed in units of level 7
// (2^-56) and carried into the level 0-2 sum (units 2^-16) after every chunk, so
// neither int64 sum can overflow for the 2^20 rows a split may hold.
#define GR_LEVELS 8
#define GR_SMEM (2 * TC_STAGE + TC_HDR + 512 * (TC_ACORES + TC_BCORES))   // and a slot of 16 bytes a lane and core

// grid (tiles of mt <= 128 columns of V, ceil(k2 / 64), splits): V's columns are dealt
// evenly to the tiles, as the widest one sets the time (178 as 96 + 82: 0.83 of 128 +
// 50). A split's exact integer sum of the
// digit products of sum_r V[r, i] W[r, j] is (hi, lo), value
// (hi 2^40 + lo) 2^(e_i + f_j - 66). The splits add theirs to sums[i + j k1] by
// atomics -- integers, so the order does not show: |hi| < 2^28.2 a row, below 2^60
// over any n, and lo < 2^40 a split -- and the split that finishes last on a tile
// rounds the tile to FP64 once, a[i + j lda]: the correctly rounded value of the
// exact sum of the kept digit products, whatever the row split. (Partials per split
// summed by a second kernel took 16 to 32 us at 76 splits of 178 x 64, and their
// storage capped the splits of the allocation-free form at 46.)
// sym: tiles wholly below the diagonal are skipped, entries above it mirrored.
__global__ void __launch_bounds__(TC_THREADS, 1)
k_gram_tc(int n, int k1, int k2, const double *__restrict__ V, long ldv, const double *__restrict__ W, long ldw,
          const int *__restrict__ ev, const int *__restrict__ ew, unsigned long long *__restrict__ sums,
          unsigned *__restrict__ ticket, double *__restrict__ a, int lda, long rows_per_split, int mt, int sym,
          int *__restrict__ err, int stall)
{
    GB_PDL();
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    uint8_t *sm = tc_smem;
    const int i0 = blockIdx.x * mt, j0 = blockIdx.y * TC_N, iend = min(k1, i0 + mt);
    if (sym && i0 > j0 + TC_N - 1) return;
    if (*(volatile int *)err) return;                    // an earlier launch timed out: do nothing
    tc_hdr *h = (tc_hdr *)(sm + 2 * TC_STAGE);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long rb = (long)blockIdx.z * rows_per_split;
    const long re = min((long)n, rb + rows_per_split);
    const int nst = (int)((re - rb + TC_KS - 1) / TC_KS);
    const int N = min(TC_N, (k2 - j0 + 15) & ~15);
    const uint32_t sbase = tc_smem_addr(sm);
    const bool mma_warp = warp == TC_SPLIT_WARPS;
    const int quarter = warp & 3, col0 = (warp >> 2) * 4;    // drained: columns col0 .. +3 of every 16
    int commits[3] = {0, 0, 0};                          // empty[0], empty[1], drained chunks
    long long hi[TC_COLS_PER_WARP], lo[TC_COLS_PER_WARP];
#pragma unroll
    for (int q = 0; q < TC_COLS_PER_WARP; ++q) hi[q] = lo[q] = 0;

    // split-warp geometry: A cores (V) warp + 15 cc, B cores (W) 14 - warp + 15 cc, those that
    // hold columns; lane (i8, rp): column 8g + i8, rows 8c + 2 rp and 8c + 2 rp + 1.
    // Lanes past the last column read it again; their shift base leaves them no digits.
    const int i8 = lane & 7, rp = lane >> 3, rwarp = TC_SPLIT_WARPS - 1 - warp;
    const int cmaxV = iend - 1 - i0, cmaxW = min(TC_N, k2 - j0) - 1;
    const int ncA = 4 * (cmaxV / 8 + 1), ncB = 4 * (cmaxW / 8 + 1);
    // a core's copy of stage s: cc < GR_A of V, the others of W
    int off[GR_CORES_PER_WARP];                          // of the lane's entry from the stage's first row
#pragma unroll
    for (int cc = 0; cc < GR_CORES_PER_WARP; ++cc) {
        const bool isA = cc < GR_A;
        const int q = isA ? warp + TC_SPLIT_WARPS * cc : rwarp + TC_SPLIT_WARPS * (cc - GR_A);
        off[cc] = (8 * (q & 3) + 2 * rp) * (int)(isA ? ldv : ldw) + min(8 * (q >> 2) + i8, isA ? cmaxV : cmaxW);
    }
    auto copy_core = [&](int s, int cc) {
        const bool isA = cc < GR_A;
        const int q = isA ? warp + TC_SPLIT_WARPS * cc : rwarp + TC_SPLIT_WARPS * (cc - GR_A);
        const long r = rb + (long)s * TC_KS, ld = isA ? ldv : ldw;
        if (s < nst && q < (isA ? ncA : ncB)) {
            const double *src = (isA ? V + i0 : W + j0) + r * ld + off[cc];
            const uint32_t dst = sbase + 2 * TC_STAGE + TC_HDR + 512 * ((isA ? 0 : TC_ACORES) + q) + 16 * lane;
            if (r + TC_KS <= re) {
                tc_cp8(dst, src, 8);
                tc_cp8(dst + 8, src + ld, 8);
            } else {
                const long left = re - r - (8 * (q & 3) + 2 * rp);   // rows of this lane before the split's end
                tc_cp8(dst, left > 0 ? src : V, left > 0 ? 8 : 0);
                tc_cp8(dst + 8, left > 1 ? src + ld : V, left > 1 ? 8 : 0);
            }
        }
        tc_cp_commit();
    };
    if (!mma_warp) {
#pragma unroll
        for (int cc = 0; cc < GR_CORES_PER_WARP; ++cc) copy_core(0, cc);
    }
    // set-up while the first copies are on their way. (The digits of the padding -- core matrices
    // past the tile's columns -- are whatever is there: they reach only the sums of the padding.)
    tc_setup(h);
    int *sbs = (int *)(sm + 2 * TC_STAGE + 128);         // shift bases of the tile's columns of V, then of W
    for (int c = tid; c < TC_M + TC_N; c += TC_THREADS) {
        const int col = c < TC_M ? i0 + c : j0 + c - TC_M;
        sbs[c] = col < (c < TC_M ? iend : k2) ? (c < TC_M ? ev : ew)[col] + OZ_SHIFT0 : OZ_SHIFT_NONE;
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = h->tmem, trow = tmem + ((uint32_t)(quarter * 32) << 16) + col0;
    const int bplane = N * TC_KS * 2;

    // A chunk is drained after the stage that follows it has been split: the split runs while
    // the chunk's last MMAs do, and the next MMAs are ready to go when the drain ends.
    // (262144 x 178 x 64: 484 -> 445 us, 10000 x 30 x 10: 13.4 -> 10.1 us in the kernel, both
    // together with planes of the tile's width and two stages a split instead of four.)
    const uint8_t *raw = sm + 2 * TC_STAGE + TC_HDR + 16 * lane;
    for (int s = 0; s <= nst; ++s) {
        const int buf = s & 1, cs = s % TC_CHUNK_STAGES;
        if (s < nst && !mma_warp) {
            if (s >= 2 && !tc_mbar_wait(tc_smem_addr(h->bar) + 16 + 8 * buf, ((s >> 1) - 1) & 1, TC_WAIT_NS))
                tc_fail(h, err);
            uint8_t *A = sm + buf * TC_STAGE;
            uint8_t *B = A + OZ_DIGITS * TC_APLANE;
#pragma unroll
            for (int cc = 0; cc < GR_CORES_PER_WARP; ++cc) {
                const bool isA = cc < GR_A;
                const int q = isA ? warp + TC_SPLIT_WARPS * cc : rwarp + TC_SPLIT_WARPS * (cc - GR_A);
                tc_cp_wait<GR_CORES_PER_WARP - 1>();     // this core's copy, the oldest in flight
                if (q < (isA ? ncA : ncB)) {
                    const int sb = sbs[(isA ? 0 : TC_M) + 8 * (q >> 2) + i8];
                    const double2 xv = *reinterpret_cast<const double2 *>(raw + 512 * ((isA ? 0 : TC_ACORES) + q));
                    uint32_t d[OZ_DIGITS];
                    oz_pack(oz_bias(xv.x, sb), oz_bias(xv.y, sb), d);
                    uint32_t *dst = (uint32_t *)((isA ? A : B) + q * 128 + i8 * 16 + rp * 4);
                    const int pl = (isA ? TC_APLANE : bplane) / 4;
#pragma unroll
                    for (int p = 0; p < OZ_DIGITS; ++p) dst[p * pl] = d[p];
                }
                copy_core(s + 1, cc);
            }
            tc_fence_async_smem();
            tc_mbar_arrive(tc_smem_addr(h->bar) + 8 * buf);
        }
        if (s > 0 && (cs == 0 || s == nst)) {
            if (!tc_wait_chunk(h, s - 1, err)) break;
#pragma unroll
            for (int g4 = 0; g4 < TC_COLS_PER_WARP / 4; ++g4) {
                if (col0 + g4 * 16 < N) {
                    uint32_t v[GR_LEVELS][4];
                    tc_load_levels4<GR_LEVELS>(trow + g4 * 16, N, v);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        float lev[GR_LEVELS];
#pragma unroll
                        for (int L = 0; L < GR_LEVELS; ++L) lev[L] = __uint_as_float(v[L][q]);
                        long long a, b;
                        oz_levels_to_int(lev, a, b);
                        // lo < 2^40 before the chunk and a chunk's level 3-7 sum is < 2^56.1
                        const long long l = lo[g4 * 4 + q] + b;
                        hi[g4 * 4 + q] += a + (l >> 40);
                        lo[g4 * 4 + q] = l & ((1LL << 40) - 1);
                    }
                }
            }
            tc_fence_before_sync();
            tc_mbar_arrive(tc_smem_addr(h->bar) + 32);
            ++commits[2];
        }
        if (s < nst && mma_warp) {
            if (lane == 0) tc_issue_stage<GR_LEVELS, false>(h, sbase, tmem, N, s, cs, commits, err, stall);
            __syncwarp();
        }
        if (*(volatile int *)&h->flag) break;
    }

    tc_cp_wait<0>();
    __syncthreads();                                     // every wait of this CTA has ended: the flag is final
    if (!*(volatile int *)&h->flag) {
        const int i = i0 + quarter * 32 + lane;
        bool last = gridDim.z == 1;
        if (!last) {
#pragma unroll
            for (int q = 0; q < TC_COLS_PER_WARP; ++q) {
                const int j = j0 + col0 + (q >> 2) * 16 + (q & 3);
                if (i < iend && j < k2) {
                    unsigned long long *P = sums + 2 * (i + (long)j * k1);
                    atomicAdd(P, (unsigned long long)hi[q]);
                    atomicAdd(P + 1, (unsigned long long)lo[q]);
                }
            }
            __threadfence();
            __syncthreads();
            int *is_last = (int *)(sm + 2 * TC_STAGE + 80);
            if (tid == 0) *is_last = atomicAdd(ticket + blockIdx.y * gridDim.x + blockIdx.x, 1u) == gridDim.z - 1;
            __syncthreads();
            last = *is_last != 0;
            if (last) {
                __threadfence();
#pragma unroll
                for (int q = 0; q < TC_COLS_PER_WARP; ++q) {
                    const int j = j0 + col0 + (q >> 2) * 16 + (q & 3);
                    if (i < iend && j < k2) {
                        const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2 *>(sums) + i + (long)j * k1);
                        hi[q] = (long long)v.x;
                        lo[q] = (long long)v.y;
                    }
                }
            }
        }
        if (last) {
#pragma unroll 1
            for (int q = 0; q < TC_COLS_PER_WARP; ++q) {
                const int j = j0 + col0 + (q >> 2) * 16 + (q & 3);
                long long hq = 0, lq = 0;
#pragma unroll
                for (int u = 0; u < TC_COLS_PER_WARP; ++u)
                    if (u == q) {
                        hq = hi[u];
                        lq = lo[u];
                    }
                if (i < iend && j < k2 && !(sym && i > j)) {
                    const __int128 z = (__int128)hq * ((__int128)1 << 40) + lq;
                    const double s = z == 0 ? 0.0 : oz_i128_to_double(z, ev[i] + ew[j] - OZ_SCALE_OFFSET - 56);
                    a[i + (long)j * lda] = s;
                    if (sym && i != j) a[j + (long)i * lda] = s;
                }
            }
        }
    }
    tc_release(h, tmem, mma_warp, commits, nullptr);
}

// Row splits of the tensor-core Gram and the rows of each: about one CTA per SM, of two
// stages at least (one: the same to 1%; four: a 30 x 30 grid's solve 1% slower). int64 headroom: a row adds < 2^28.2 to the level 0-2 sum (units
// of 2^-16), so a split holds at most GR_MAX_ROWS rows (the level 3-7 sum is
// carried into it after every chunk).
#define GR_MAX_ROWS (1L << 20)
static int gram_tc_mt(int k1)
{
    const int ti = (k1 + TC_M - 1) / TC_M;
    return ((k1 + ti - 1) / ti + 7) / 8 * 8;
}
static long gram_tc_splits(int num_sms, int n, int k1, int k2, int sym, long *rps_out)
{
    const int ti = (k1 + TC_M - 1) / TC_M, tj = (k2 + TC_N - 1) / TC_N;
    int tiles = 0;
    for (int a = 0; a < ti; ++a)
        for (int b = 0; b < tj; ++b)
            if (!sym || a * gram_tc_mt(k1) <= b * TC_N + TC_N - 1) ++tiles;
    if (tiles < 1) tiles = 1;
    long nsplit = ((long)num_sms + tiles - 1) / tiles;
    const long max_split = (n + 2 * TC_KS - 1) / (2 * TC_KS);
    if (nsplit > max_split) nsplit = max_split;
    const long min_split = (n + GR_MAX_ROWS - 1) / GR_MAX_ROWS;
    if (nsplit < min_split) nsplit = min_split;
    if (nsplit < 1) nsplit = 1;
    const long rps = ((n + nsplit - 1) / nsplit + TC_KS - 1) / TC_KS * TC_KS;
    *rps_out = rps;
    nsplit = (n + rps - 1) / rps;
    return nsplit < 1 ? 1 : nsplit;
}

// a[i + j*lda] = sum_r V[r,i] W[r,j] to FP64 accuracy on the tensor cores.
// exps: device scratch of gb_gram_tc_ints(k1, k2) ints (column scales, tickets).
extern "C" size_t gb_gram_tc_ints(int k1, int k2)
{
    return (size_t)k1 + k2 + (size_t)((k1 + TC_M - 1) / TC_M) * ((k2 + TC_N - 1) / TC_N);
}
extern "C" int gb_gram_tc(gcge_gpu_ctx *ctx, int n, int k1, int k2, const double *V, long ldv, const double *W,
                          long ldw, double *a_dev, int lda, int sym, int *exps)
{
    if (k1 <= 0 || k2 <= 0) return GCGE_GPU_OK;
    if (n <= 0) return gb_gram_reduce_launch(ctx, k1, k2, 0, ctx->scratch, a_dev, lda, sym);   // zeros
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(k_gram_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, GR_SMEM) != cudaSuccess)
            return gb_fail(ctx, GCGE_GPU_ERR_CUDA);
        attr = true;
    }
    const int ti = (k1 + TC_M - 1) / TC_M, tj = (k2 + TC_N - 1) / TC_N;
    long rps = 0;
    const long nsplit = gram_tc_splits(ctx->num_sms, n, k1, k2, sym, &rps);
    const long total = (long)k1 * k2;
    int st = gb_scratch(ctx, (size_t)2 * total);
    if (st) return st;
    unsigned *ticket = (unsigned *)(exps + k1 + k2);
    const long cols = k1 + k2, most = total > cols ? total : cols;
    GB_LAUNCH(ctx, k_gram_init, (int)((most < 65536 ? most : 65536) + 255) / 256, 256, 0, exps, (int)cols, ticket,
              ti * tj, (ulonglong2 *)ctx->scratch, nsplit > 1 ? total : 0);
    GB_LAUNCH(ctx, k_col_exponent, dim3(ctx->num_sms * 4, 2), 256, 0, n, k1, V, ldv, k2, W, ldw, exps);
    dim3 grid(ti, tj, (unsigned)nsplit);
    GB_PROF(ctx, GB_K_GRAM, 8.0 * n * (k1 + k2), sym ? 1.0 * n * k1 * (k1 + 1) : 2.0 * n * k1 * k2);
    const int stall = ctx->tc_stall;
    ctx->tc_stall = 0;
    GB_LAUNCH(ctx, k_gram_tc, grid, TC_THREADS, GR_SMEM, n, k1, k2, V, ldv, W, ldw, exps, exps + k1,
              (unsigned long long *)ctx->scratch, ticket, a_dev, lda, rps, gram_tc_mt(k1), sym, ctx->dev_err,
              stall);
    return GCGE_GPU_OK;
}

// ---------------------------------------------------------------- Gram on fixed storage
// The allocation-free Gram on the tensor cores. What the FP64-pipe form took at
// 262,144 x (178, 64) was the FP64 pipe itself: 5.44 ms at 1.1 of 1.2 TFLOP/s.
//
// Column scales serve every row of a column: an entry x of a column with scale e (|x| < 2^e) is
// held to 2^(e - 54), so a small one keeps fewer bits than FP64 would, and a product of two
// such entries may be all that a sum consists of. The tensor form is therefore taken
// only where the data prove the bound of a plain FP64 sum, n 2^-53 sum |v w|, for every
// entry of the result. k_col_stats forms, beside a column's scale e, the number q of its
// nonzeros and the sum g of their gaps (e less the entry's exponent, |x| >= 2^(e - 1 - gap)).
// With q >= a n, g <= G n for every column of V that is not all zero and q' >= a' n,
// g' <= G' n for W's, at least s n = (a + a' - 1) n rows have both factors, and by the
// arithmetic-geometric mean over them
//   sum |v w| >= s n 2^(e + f - 2 - (G + G') / s).
// The digits' error, roundings of the entries at 2^-54 of their scales and dropped pairs at
// 2^-57.4, is at most 1.05 n 2^(e + f - 53), which lies below (n - 1) 2^-53 sum |v w| where
//   (G + G') / s <= log2((n - 1) s) - 2.1.
// GN_SPREAD caps the left side for large n: the digits' roundings are independent as a rule, and with
// a mean gap of 5 in both factors their sum over n rows stays near the FP64 form's own error (normal
// and smooth columns, n from 1,000 to 600,000: 0.4 to 0.02 of it). Otherwise, and where an
// entry is not finite or subnormal, the block that finishes last sets ctl->skip: the
// FP64-pipe kernel that follows then does the work, and nothing otherwise. A bounded wait
// that runs out sets skip as well.
#define GN_SPREAD 10.0f
struct gn_ctl {
    int skip;
    unsigned done;
    unsigned ticket[GB_GRAM_FIXED_COLS];                 // tiles <= k1 + k2
    int e[GB_GRAM_FIXED_COLS], cnt[GB_GRAM_FIXED_COLS];
    long long sum[GB_GRAM_FIXED_COLS];
};
extern "C" size_t gb_gram_fixed_ctl_bytes(void) { return sizeof(gn_ctl); }

__global__ void k_gn_init(gn_ctl *ctl, int cols, ulonglong2 *__restrict__ sums, long total)
{
    GB_PDL();
    const long c = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c == 0) {
        ctl->skip = 0;
        ctl->done = 0;
    }
    if (c < cols) {
        ctl->ticket[c] = 0;
        ctl->e[c] = OZ_NO_EXP;
        ctl->cnt[c] = 0;
        ctl->sum[c] = 0;
    }
    for (long t = c; t < total; t += (long)gridDim.x * blockDim.x) sums[t] = make_ulonglong2(0, 0);
}

// grid (blocks, 2): blockIdx.y = 0 the columns of V, 1 those of W; rows as k_col_exponent.
__global__ void __launch_bounds__(256)
k_col_stats(int n, int k1, const double *__restrict__ V, long ldv, int k2, const double *__restrict__ W, long ldw,
            gn_ctl *ctl)
{
    GB_PDL();
    __shared__ int se[8][CE_COLS], sc[8][CE_COLS], ss[8][CE_COLS];
    __shared__ int done, wide, fewest[2];                // of V and of W: the fewest nonzeros, the largest sum of gaps
    __shared__ unsigned long long gaps[2];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int k = blockIdx.y ? k2 : k1, off = blockIdx.y ? k1 : 0;
    const double *X = blockIdx.y ? W : V;
    const long ldx = blockIdx.y ? ldw : ldv;
    const long warp = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long nw = ((long)gridDim.x * blockDim.x) >> 5;
    for (int c0 = 0; c0 < k; c0 += CE_COLS) {
        int e[CE_COLS / 32], cnt[CE_COLS / 32], sum[CE_COLS / 32];   // a warp's rows: below 2^20
#pragma unroll
        for (int j = 0; j < CE_COLS / 32; ++j) {
            e[j] = OZ_NO_EXP;
            cnt[j] = 0;
            sum[j] = 0;
        }
        ce_rows(n, min(CE_COLS, k - c0), X + c0, ldx, warp, nw, [&](int j, double v) {
            // a subnormal entry has no digits: counted as not finite
            int x = oz_exponent(v);
            if (x == OZ_NO_EXP && (__double_as_longlong(v) << 1)) x = 1025;
            if (x != OZ_NO_EXP) {
                e[j] = max(e[j], x);
                ++cnt[j];
                sum[j] += x;
            }
        });
#pragma unroll
        for (int j = 0; j < CE_COLS / 32; ++j) {
            se[w][lane + 32 * j] = e[j];
            sc[w][lane + 32 * j] = cnt[j];
            ss[w][lane + 32 * j] = sum[j];
        }
        __syncthreads();
        for (int c = threadIdx.x; c < CE_COLS; c += blockDim.x) {
            int m = OZ_NO_EXP, q = 0;
            long long t = 0;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                m = max(m, se[u][c]);
                q += sc[u][c];
                t += ss[u][c];
            }
            if (c0 + c < k && m > OZ_NO_EXP) {
                atomicMax(&ctl->e[off + c0 + c], m);
                atomicAdd(&ctl->cnt[off + c0 + c], q);
                atomicAdd((unsigned long long *)&ctl->sum[off + c0 + c], (unsigned long long)t);
            }
        }
        __syncthreads();
    }
    __threadfence();
    if (threadIdx.x == 0) {
        done = atomicAdd(&ctl->done, 1u) == gridDim.x * 2 - 1;
        wide = 0;
        fewest[0] = fewest[1] = n;
        gaps[0] = gaps[1] = 0;
    }
    __syncthreads();
    if (!done) return;
    __threadfence();
    for (int c = threadIdx.x; c < k1 + k2; c += blockDim.x) {
        const int q = __ldcg(&ctl->cnt[c]), m = __ldcg(&ctl->e[c]), op = c >= k1;
        if (m > 1024) wide = 1;                            // e = 1025: not finite, or subnormal
        if (q && m <= 1024) {
            atomicMin(&fewest[op], q);
            atomicMax(&gaps[op], (unsigned long long)((long long)m * q - __ldcg(&ctl->sum[c])));
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const float both = (float)((long long)fewest[0] + fewest[1] - n);      // s n
        const float gap = (float)(gaps[0] + gaps[1]);                          // (G + G') n
        if (wide || !(both > 0.0f) || gap > both * fminf(GN_SPREAD, log2f(both) - 2.1f)) ctl->skip = 1;
    }
}

extern "C" int gb_gram_fixed_partials(cudaStream_t stream, int num_sms, int n, int k1, int k2, const double *V,
                                      long ldv, const double *W, long ldw, int sym, double *part, size_t part_cap,
                                      const int *run, int *st);
extern "C" int gb_gram_fixed_reduce(cudaStream_t stream, int num_sms, int k1, int k2, int nsplit, const double *part,
                                    double *a_dev, int lda, int sym, const int *run);

// Gram V^T W with caller-provided partials (part_cap doubles), control block and
// stream: no context, no allocation; part_cap >= 2 k1 k2. The tensor-core form where
// its estimate is the shorter one. Measured on the GB300: a CTA takes a stage of 32
// rows, its share of the column pass included, in 1.4 us for a few columns and 3.8 us for
// a full tile, and the form has 22 us of launches, scales and drain beside it, 36 for many
// outputs; the FP64 pipe takes 8.2 us for 32 rows of a 32 x 32 tile on each SM, 0.055 us
// a split to sum, and 8 us. Both sides, us, tensor cores / FP64 pipe: 3,500 rows, 3 x 3
// 25 / 22, 33 x 16 30 / 33, 64 x 64 42 / 42; 5,000 rows 26 / 34, 31 / 46, 45 / 64;
// 1,000 rows of 178 x 64 41 / 33, 2,000 43 / 58.
extern "C" long gb_gram_fixed_splits(int num_sms, int n, int k1, int k2, int sym, size_t part_cap, long *rps_out);
extern "C" int gb_gram_fixed(cudaStream_t stream, int num_sms, int n, int k1, int k2, const double *V, long ldv,
                             const double *W, long ldw, double *a_dev, int lda, int sym, double *part,
                             size_t part_cap, void *ctl_dev)
{
    gn_ctl *ctl = (gn_ctl *)ctl_dev;
    int st = GCGE_GPU_OK;
    const int *run = nullptr;
    if (k1 + k2 <= GB_GRAM_FIXED_COLS && ldv < GB_TC_MAX_LD && ldw < GB_TC_MAX_LD) {
        const int ti = (k1 + TC_M - 1) / TC_M, tj = (k2 + TC_N - 1) / TC_N;
        long rps = 0;
        const long nsplit = gram_tc_splits(num_sms, n, k1, k2, sym, &rps), total = (long)k1 * k2;
        const double waves = (double)(((long)ti * tj * nsplit + num_sms - 1) / num_sms);
        const double fill = (double)((k1 < TC_M ? k1 : TC_M) + (k2 < TC_N ? k2 : TC_N)) / (TC_M + TC_N);
        const double t_tc = 22.0 + 14.0 * (total < 8192 ? (double)total / 8192 : 1.0) +
                            waves * (double)(rps / TC_KS) * (1.35 + 2.5 * fill);
        long rps64 = 0;
        const long n64 = gb_gram_fixed_splits(num_sms, n, k1, k2, sym, part_cap, &rps64);
        const long b64 = n64 * ((k1 + 31) / 32) * ((k2 + 31) / 32);
        const double t_64 = 8.0 + 0.055 * (double)n64 +
                            8.2 * (double)(rps64 / 32) * (double)((b64 + num_sms - 1) / num_sms);
        if (t_tc < t_64) {
            if (cudaFuncSetAttribute(k_gram_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, GR_SMEM) != cudaSuccess)
                return GCGE_GPU_ERR_CUDA;
            const long most = total > k1 + k2 ? total : k1 + k2;
            gb_launch(stream, (int)((most < 65536 ? most : 65536) + 255) / 256, 256, 0, k_gn_init, ctl, k1 + k2,
                      (ulonglong2 *)part, nsplit > 1 ? total : 0L);
            gb_launch(stream, dim3(num_sms * 4, 2), 256, 0, k_col_stats, n, k1, V, ldv, k2, W, ldw, ctl);
            gb_launch(stream, dim3(ti, tj, (unsigned)nsplit), TC_THREADS, GR_SMEM, k_gram_tc,
                n, k1, k2, V, ldv, W, ldw, ctl->e, ctl->e + k1, (unsigned long long *)part, ctl->ticket, a_dev, lda,
                rps, gram_tc_mt(k1), sym, &ctl->skip, 0);
            if (cudaGetLastError() != cudaSuccess) return GCGE_GPU_ERR_CUDA;
            run = &ctl->skip;
        }
    }
    const int n64 = gb_gram_fixed_partials(stream, num_sms, n, k1, k2, V, ldv, W, ldw, sym, part, part_cap, run, &st);
    return st ? st : gb_gram_fixed_reduce(stream, num_sms, k1, k2, n64, part, a_dev, lda, sym, run);
}

// ---------------------------------------------------------------- linear combination (tcgen05)
#define LC_MAX_K 4096                                // inner dimension handled by the tensor-core path
#define LC_ER 8                                      // tiles whose row scales are kept
#define LC_HDR (80 + 4 * (LC_ER * TC_M + TC_N) + 48) // tc_hdr, er, ecs
#define LC_SMEM (2 * TC_STAGE + LC_HDR + 4 * LC_MAX_K)
#define LC_CORES_PER_WARP ((TC_ACORES + TC_SPLIT_WARPS - 1) / TC_SPLIT_WARPS)
#define LC_SCALE_LOADS 48                            // row-scale loads in flight per thread
// the largest of k_lincomb_tc's int offsets, a lane past the tile's cores among them (k_gram_tc's: 31 rows)
static_assert((8L * ((TC_SPLIT_WARPS * LC_CORES_PER_WARP - 1) >> 2) + 7) * GB_TC_MAX_LD + TC_KS <= 0x7fffffffL,
              "row strides of the tensor-core kernels");
// Levels 0-7 (34 digit pairs; 8 x 64 TMEM columns): the dropped pairs (level >= 8)
// lie below 2^-55 of the scale product per term; level 7 (weight 2^-56) needs no
// exactness, levels 0-6 stay exact for OZ_EXACT_TERMS terms.
#define LC_LEVELS 8

// Inner-dimension equilibration: X C = (X 2^g) (2^-g C) exactly for any integer
// g_i, so with g_i the exponent of row i of C (max_j |C[i, j]| < 2^g_i) the row
// scale of X 2^g measures |X[r, i]| |C[i, :]|, the size of each term's
// contribution, and the error of a row is relative to its largest term (as for
// an FP64 dot product) even when the columns of X differ widely in magnitude
// and C compensates (the triangular solve of a Cholesky QR).
//
// C (k1 x k2, column-major, only i <= j when upper) -> row scales g (all blocks
// compute them; block (0, 0) stores them), column scales F of 2^-g C (block
// (0, jt) stores its 64) and digit planes Bd[jt][stage][digit] of 2^-g C in
// the core-matrix layout (N = 16 .. 64 rows j, K = 32 entries i per stage).
// grid (stages, column tiles), 256 threads, k1 <= LC_MAX_K.
// One block or two at a solve's sizes, so only latency counts: each of the three passes over C
// has its loads in flight together, the first along C's columns (60 x 20: 8.2 -> 4.8 us;
// a call at 10000 x 178 x 64 90 -> 75 us).
__global__ void __launch_bounds__(256)
k_lc_coef_split(int k1, int k2, const double *__restrict__ C, int ldc, int upper, int nst, int *__restrict__ g_out,
                int *__restrict__ f_out, uint32_t *__restrict__ Bd)
{
    GB_PDL();
    __shared__ int gs[LC_MAX_K];
    __shared__ int fs[TC_N];
    const int s = blockIdx.x, jt = blockIdx.y, j0 = jt * TC_N;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // row exponents: lanes along the rows (contiguous in C), columns dealt to the warps
    for (int i = threadIdx.x; i < k1; i += 256) gs[i] = OZ_NO_EXP;
    __syncthreads();
    for (int i0 = 0; i0 < k1; i0 += 32) {
        const int i = i0 + lane;
        int e = OZ_NO_EXP;
#pragma unroll 4
        for (int j = (upper ? i0 : 0) + warp; j < k2; j += 8)
            if (i < k1 && (!upper || i <= j)) e = max(e, oz_exponent(C[i + (long)j * ldc]));
        if (e != OZ_NO_EXP) atomicMax(gs + i, e);
    }
    __syncthreads();
    if (s == 0 && jt == 0)
        for (int i = threadIdx.x; i < k1; i += 256) g_out[i] = gs[i];
    // column scales: a warp has columns warp, warp + 8, ..
    {
        int e[TC_N / 8];
#pragma unroll
        for (int cc = 0; cc < TC_N / 8; ++cc) e[cc] = OZ_NO_EXP;
        for (int i = lane; i < k1; i += 32) {
            const int g = gs[i];
            int ex[TC_N / 8];
#pragma unroll
            for (int cc = 0; cc < TC_N / 8; ++cc) {
                const int j = j0 + warp + 8 * cc;
                ex[cc] = j < k2 && (!upper || i <= j) ? oz_exponent(C[i + (long)j * ldc]) : OZ_NO_EXP;
            }
#pragma unroll
            for (int cc = 0; cc < TC_N / 8; ++cc)
                if (ex[cc] != OZ_NO_EXP) e[cc] = max(e[cc], ex[cc] - g);
        }
#pragma unroll
        for (int cc = 0; cc < TC_N / 8; ++cc) {
            const int jj = warp + 8 * cc, m = __reduce_max_sync(0xffffffffu, e[cc]);
            if (lane == 0) {
                fs[jj] = m;
                if (s == 0 && j0 + jj < k2) f_out[j0 + jj] = m;
            }
        }
    }
    __syncthreads();
    // planes of N rows back to back, each stage's at a fixed place
    uint32_t *out = Bd + (size_t)(jt * nst + s) * OZ_DIGITS * (TC_BPLANE / 4);
    const int N = min(TC_N, (k2 - j0 + 15) & ~15);
    const int n8 = lane >> 2, kp = lane & 3;
    double x[4][2];
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
        const int core = warp + 8 * cc, jj = (core >> 2) * 8 + n8, j = j0 + jj, i = s * TC_KS + (core & 3) * 8 + 2 * kp;
#pragma unroll
        for (int h = 0; h < 2; ++h)
            x[cc][h] = j < k2 && i + h < k1 && (!upper || i + h <= j) ? C[i + h + (long)j * ldc] : 0.0;
    }
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
        const int core = warp + 8 * cc, jj = (core >> 2) * 8 + n8, i = s * TC_KS + (core & 3) * 8 + 2 * kp;
        if (core >> 2 < N / 8) {
            uint32_t d[OZ_DIGITS];
            oz_pack(oz_bias(x[cc][0], i < k1 ? fs[jj] + gs[i] + OZ_SHIFT0 : OZ_SHIFT_NONE),
                    oz_bias(x[cc][1], i + 1 < k1 ? fs[jj] + gs[i + 1] + OZ_SHIFT0 : OZ_SHIFT_NONE), d);
#pragma unroll
            for (int q = 0; q < OZ_DIGITS; ++q) out[q * (N * TC_KS / 2) + (core * 128 + n8 * 16 + kp * 4) / 4] = d[q];
        }
    }
}

// Y[r, j0 + j] = alpha sum_i X[r, i] C[i, j0 + j] + beta Y[r, j0 + j];
// grid (P, column tiles) with P <= number of SMs, TC_THREADS threads, LC_SMEM
// dynamic shared memory. Persistent: CTA b walks the 128-row tiles b, b + P, ...
// with one TMEM allocation and one barrier set; the stage counter runs across
// tiles. While the K stages of a tile run, the split warps also load the next
// tile's entries of the same stage and fold their exponents into that tile's row
// scales (shared-memory atomicMax) one stage later, when the loads have landed,
// so only the first tile has a separate scale pass and every later tile's X is
// already in L2 when it is split. The drain
// writes Y directly. MULTI: the inner dimension is longer than one exact
// accumulation (k1 > OZ_EXACT_TERMS) and the drained chunks are summed in
// registers; the single-chunk form holds no FP64 accumulators while it splits.
template <bool MULTI>
__global__ void __launch_bounds__(TC_THREADS, 1)
k_lincomb_tc(int n, int k1, int k2, const double *__restrict__ X, long ldx, const uint4 *__restrict__ Bd,
             const int *__restrict__ g_in, const int *__restrict__ ec, double alpha, double beta,
             double *__restrict__ Y, long ldy, int nst, int *__restrict__ err, int stall)
{
    GB_PDL();
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    uint8_t *sm = tc_smem;
    if (*(volatile int *)err) return;                    // an earlier launch timed out: do nothing
    tc_hdr *h = (tc_hdr *)(sm + 2 * TC_STAGE);
    int *er = (int *)(sm + 2 * TC_STAGE + 80);           // [LC_ER][TC_M] row scales of X 2^g, tile by tile
    int *ecs = er + LC_ER * TC_M;                            // [TC_N] column scales of 2^-g C
    int *gs = (int *)(sm + 2 * TC_STAGE + LC_HDR);       // [k1] inner-dimension scales g
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int jt = blockIdx.y, j0 = jt * TC_N;
    const int N = min(TC_N, (k2 - j0 + 15) & ~15);
    const long ntiles = ((long)n + TC_M - 1) / TC_M;
    // one exact accumulation over all of K when it is short enough
    const int chunk_stages = k1 <= OZ_EXACT_TERMS ? nst : TC_CHUNK_STAGES;

    const bool mma_warp = warp == TC_SPLIT_WARPS;
    // split-warp geometry: core q = warp + 15 cc (A cores only); lane (r8, kp):
    // row 8g + r8, entries 8c + 2 kp and 8c + 2 kp + 1
    const int r8 = lane >> 2, kp = lane & 3;
    double xv[LC_CORES_PER_WARP][2];
    int off[LC_CORES_PER_WARP];                          // of the lane's entries from the stage's first one
#pragma unroll
    for (int cc = 0; cc < LC_CORES_PER_WARP; ++cc) {
        const int q = warp + TC_SPLIT_WARPS * cc;
        off[cc] = (8 * (q >> 2) + r8) * (int)ldx + 8 * (q & 3) + 2 * kp;
    }
    auto load_stage = [&](long row0, int s) {
        const double *Xs = X + row0 * ldx + s * TC_KS;
        if (row0 + TC_M <= n && (s + 1) * TC_KS <= k1) {
#pragma unroll
            for (int cc = 0; cc < LC_CORES_PER_WARP; ++cc)
                if (warp + TC_SPLIT_WARPS * cc < TC_ACORES) {
                    xv[cc][0] = Xs[off[cc]];
                    xv[cc][1] = Xs[off[cc] + 1];
                }
        } else {
#pragma unroll
            for (int cc = 0; cc < LC_CORES_PER_WARP; ++cc) {
                const int q = warp + TC_SPLIT_WARPS * cc, left = k1 - s * TC_KS - (8 * (q & 3) + 2 * kp);
                const bool in = q < TC_ACORES && row0 + 8 * (q >> 2) + r8 < n;
                xv[cc][0] = in && left > 0 ? Xs[off[cc]] : 0.0;
                xv[cc][1] = in && left > 1 ? Xs[off[cc] + 1] : 0.0;
            }
        }
    };
    // the first stage's values, on their way during the set-up and the scale pass
    if (!mma_warp) load_stage((long)blockIdx.x * TC_M, 0);

    tc_setup(h);
    // a zero row of C contributes nothing, nor do the entries past k1: no digits
    for (int i = tid; i < nst * TC_KS; i += TC_THREADS) {
        const int g = i < k1 ? g_in[i] : OZ_NO_EXP;
        gs[i] = g != OZ_NO_EXP ? g : -OZ_SHIFT_NONE;
    }
    if (tid < TC_N) ecs[tid] = j0 + tid < k2 ? ec[j0 + tid] : OZ_NO_EXP;
    for (int i = tid; i < (LC_ER - 1) * TC_M; i += TC_THREADS) er[TC_M + i] = OZ_NO_EXP;
    __syncthreads();
    // row scales of the first tile: 4 threads per row, up to LC_SCALE_LOADS
    // independent loads of the high words (sign, exponent) in flight per thread
    {
        const int rr = tid >> 2, t4 = tid & 3;
        const long r = (long)blockIdx.x * TC_M + rr;
        const bool rin = r < n;
        const unsigned *xh = reinterpret_cast<const unsigned *>(X + (rin ? r : 0) * ldx) + 1;
        int e = OZ_NO_EXP;
        for (int i0 = t4; i0 < k1; i0 += 4 * LC_SCALE_LOADS) {
            unsigned w[LC_SCALE_LOADS];
#pragma unroll
            for (int j = 0; j < LC_SCALE_LOADS; ++j) {
                const int i = i0 + 4 * j;
                w[j] = (rin && i < k1) ? __ldg(xh + 2 * (long)i) : 0u;
            }
#pragma unroll
            for (int j = 0; j < LC_SCALE_LOADS; ++j) {
                const int i = i0 + 4 * j;
                const int ex = (int)((w[j] >> 20) & 0x7ff);
                if (ex && i < k1) e = max(e, ex - 1022 + gs[i]);
            }
        }
        e = max(e, __shfl_xor_sync(0xffffffffu, e, 1));
        e = max(e, __shfl_xor_sync(0xffffffffu, e, 2));
        if (t4 == 0) er[rr] = e;
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = h->tmem, sbase = tc_smem_addr(sm);
    const int quarter = warp & 3, col0 = (warp >> 2) * 4;    // drained: columns col0 .. +3 of every 16
    const int my_row = quarter * 32 + lane;
    const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16) + col0;
    // alpha = +-1, beta = 0: the output is the drained value with its sign bit
    // flipped or not, an integer operation (the FP64 pipe runs at 1/64 rate)
    const bool plain = beta == 0.0 && (alpha == 1.0 || alpha == -1.0);
    const bool unit = beta == 1.0 && (alpha == 1.0 || alpha == -1.0);   // one FP64 addition: fma(1, y, +-v)
    const unsigned long long sflip = alpha == -1.0 ? 0x8000000000000000ull : 0ull;
    int commits[3] = {0, 0, 0};
    int copies[2] = {0, 0};                              // bulk copies per buffer (thread 0)

    unsigned pw[LC_CORES_PER_WARP][2];                   // high words of the next tile's entries, in flight
    auto load_words = [&](long row0, int s) {
        const double *Xs = X + row0 * ldx + s * TC_KS;
        const bool full = row0 + TC_M <= n && (s + 1) * TC_KS <= k1;
#pragma unroll
        for (int cc = 0; cc < LC_CORES_PER_WARP; ++cc) {
            const int q = warp + TC_SPLIT_WARPS * cc, left = k1 - s * TC_KS - (8 * (q & 3) + 2 * kp);
            const bool in = q < TC_ACORES && (full || row0 + 8 * (q >> 2) + r8 < n);
            const unsigned *xw = reinterpret_cast<const unsigned *>(Xs + off[cc]) + 1;
            pw[cc][0] = in && (full || left > 0) ? __ldg(xw) : 0u;
            pw[cc][1] = in && (full || left > 1) ? __ldg(xw + 2) : 0u;
        }
    };
    auto fold_words = [&](int *scales, int s) {          // into the scales of the words' tile
#pragma unroll
        for (int cc = 0; cc < LC_CORES_PER_WARP; ++cc) {
            const int q = warp + TC_SPLIT_WARPS * cc;
            if (q < TC_ACORES) {
                const int2 g = *reinterpret_cast<const int2 *>(gs + s * TC_KS + 8 * (q & 3) + 2 * kp);
                const int x0 = (int)((pw[cc][0] >> 20) & 0x7ff), x1 = (int)((pw[cc][1] >> 20) & 0x7ff);
                int e = max(x0 ? x0 + g.x : OZ_NO_EXP, x1 ? x1 + g.y : OZ_NO_EXP);
                e = max(e, __shfl_xor_sync(0xffffffffu, e, 1));
                e = max(e, __shfl_xor_sync(0xffffffffu, e, 2));
                if (kp == 0 && e > OZ_NO_EXP + 1022) atomicMax(scales + 8 * (q >> 2) + r8, e - 1022);
            }
        }
    };
    // Stages g of this CTA over all its tiles (lt: its tile, s: the stage in it). A chunk
    // is drained after the next stage has been split: the split of that one -- the next
    // tile's first, mostly -- runs while the chunk's last MMAs do, and the next MMAs are
    // ready to go when the drain ends.
    const int mytiles = (int)((ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x), total = mytiles * nst;
    const uint32_t scales_bar = tc_smem_addr(h->bar) + 56;
    double acc[MULTI ? TC_COLS_PER_WARP : 1];
    int s = 0, lt = 0, ps = 0, plt = 0;                  // this stage, the one before
    for (int g = 0; g <= total; ++g) {
        const int buf = g & 1;
        const long row0 = ((long)blockIdx.x + (long)lt * gridDim.x) * TC_M, nrow0 = row0 + (long)gridDim.x * TC_M;
        if (g < total && !mma_warp) {
            const bool has_next = lt + 1 < mytiles;
            if (g >= 2 && !tc_mbar_wait(tc_smem_addr(h->bar) + 16 + 8 * buf, ((g >> 1) - 1) & 1, TC_WAIT_NS))
                tc_fail(h, err);
            if (s == 0 && lt > 0) {
                // the tile's scales: the last words loaded for it, then every split lane's are in.
                // The slot cleared for the tile after the next held those of six tiles back: the
                // MMAs just waited for, of tile lt - 2 at the earliest, were issued after every
                // thread's drain of the tile before theirs.
                fold_words(er + lt % LC_ER * TC_M, nst - 1);
                if (tid < TC_M) er[(lt + 2) % LC_ER * TC_M + tid] = OZ_NO_EXP;
                tc_mbar_arrive(scales_bar);
                if (!tc_mbar_wait(scales_bar, (lt - 1) & 1, TC_WAIT_NS)) tc_fail(h, err);
            }
            const int *ert = er + lt % LC_ER * TC_M;
            uint8_t *A = sm + buf * TC_STAGE;
            uint8_t *B = A + OZ_DIGITS * TC_APLANE;
            // the pre-split C planes of this stage: one bulk copy, completing on copied[buf]
            if (tid == 0) {
                const uint32_t copied = tc_smem_addr(h->bar) + 40 + 8 * buf;
                tc_mbar_arrive_expect_tx(copied, OZ_DIGITS * N * TC_KS * 2);
                tc_bulk_g2s(tc_smem_addr(B), Bd + (size_t)(jt * nst + s) * (OZ_DIGITS * TC_BPLANE / 16),
                            OZ_DIGITS * N * TC_KS * 2, copied);
                ++copies[buf];
            }
#pragma unroll
            for (int cc = 0; cc < LC_CORES_PER_WARP; ++cc) {
                const int q = warp + TC_SPLIT_WARPS * cc;
                if (q < TC_ACORES) {
                    const int sb = ert[8 * (q >> 2) + r8] + OZ_SHIFT0;
                    const int2 gg = *reinterpret_cast<const int2 *>(gs + s * TC_KS + 8 * (q & 3) + 2 * kp);
                    uint32_t d[OZ_DIGITS];
                    oz_pack(oz_bias(xv[cc][0], sb - gg.x), oz_bias(xv[cc][1], sb - gg.y), d);
                    uint32_t *dst = (uint32_t *)(A + q * 128 + r8 * 16 + kp * 4);
#pragma unroll
                    for (int p = 0; p < OZ_DIGITS; ++p) dst[p * (TC_APLANE / 4)] = d[p];
                }
            }
            tc_fence_async_smem();
            tc_mbar_arrive(tc_smem_addr(h->bar) + 8 * buf);
            // in flight while the MMAs run: the next stage's values (or the next tile's first
            // ones), and the next tile's words of this stage; those of the stage before
            // have arrived and are folded first
            if (has_next && s > 0) fold_words(er + (lt + 1) % LC_ER * TC_M, s - 1);
            if (s + 1 < nst) load_stage(row0, s + 1);
            else if (has_next) load_stage(nrow0, 0);
            if (has_next) load_words(nrow0, s);
        }
        // ---- drain of the chunk that ended with the stage before
        if (g > 0 && (ps == nst - 1 || ps % chunk_stages == chunk_stages - 1)) {
            const bool first = ps < chunk_stages, last = ps == nst - 1;
            const long r = ((long)blockIdx.x + (long)plt * gridDim.x) * TC_M + my_row;
            double *y = Y + r * ldy + j0 + col0;
            const bool rin = r < n;
            double yv[TC_COLS_PER_WARP];                 // the old values, on their way while the MMAs end
            if (last && !plain) {
#pragma unroll
                for (int c = 0; c < TC_COLS_PER_WARP; ++c) {
                    const int j = 16 * (c >> 2) + (c & 3);
                    yv[c] = rin && j0 + col0 + j < k2 ? y[j] : 0.0;
                }
            }
            if (!tc_wait_chunk(h, g - 1, err)) break;
            const int my_e = er[plt % LC_ER * TC_M + my_row] - OZ_SCALE_OFFSET;
#pragma unroll
            for (int g4 = 0; g4 < TC_COLS_PER_WARP / 4; ++g4) {
                if (col0 + g4 * 16 < N) {
                    uint32_t v[LC_LEVELS][4];
                    tc_load_levels4<LC_LEVELS>(trow + g4 * 16, N, v);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        int lev[LC_LEVELS];
#pragma unroll
                        for (int L = 0; L < LC_LEVELS; ++L) lev[L] = __float2int_rn(__uint_as_float(v[L][q]));
                        double v2 = oz_levels_to_double(lev, my_e + ecs[col0 + g4 * 16 + q]);
                        if (MULTI) {
                            acc[g4 * 4 + q] = first ? v2 : acc[g4 * 4 + q] + v2;
                            v2 = acc[g4 * 4 + q];
                        }
                        if (last && rin && j0 + col0 + g4 * 16 + q < k2) {
                            const double sv = __longlong_as_double(__double_as_longlong(v2) ^ (long long)sflip);
                            const double yo = yv[g4 * 4 + q];
                            y[16 * g4 + q] = plain ? sv : unit ? yo + sv : fma(beta, yo, alpha * v2);
                        }
                    }
                }
            }
            tc_fence_before_sync();
            tc_mbar_arrive(tc_smem_addr(h->bar) + 32);
            ++commits[2];
        }
        if (g < total && mma_warp) {
            if (lane == 0) tc_issue_stage<LC_LEVELS, true>(h, sbase, tmem, N, g, s % chunk_stages, commits, err, stall);
            __syncwarp();
        }
        if (*(volatile int *)&h->flag) break;
        ps = s;
        plt = lt;
        if (++s == nst) {
            s = 0;
            ++lt;
        }
    }
    tc_release(h, tmem, mma_warp, commits, copies);
}

extern "C" int gb_lincomb_tc_ok(int k1, long ldx) { return k1 <= LC_MAX_K && ldx < GB_TC_MAX_LD; }
// Y may overlap X's columns (the same rows, the same leading dimension) when one
// column tile covers the output: a CTA reads every entry of its row tile before
// its drain writes that tile's rows, and walks only its own tiles (the
// next-tile prefetch and scale pass included)
extern "C" int gb_lincomb_tc_inplace_ok(int k1, int k2, long ldx) { return gb_lincomb_tc_ok(k1, ldx) && k2 <= TC_N; }

// Y = alpha X C + beta Y (C: k1 x k2 column-major on the device, upper: only
// i <= j of C is used) to FP64 accuracy on the tensor cores.
extern "C" int gb_lincomb_tc(gcge_gpu_ctx *ctx, int n, int k1, int k2, const double *X, long ldx, const double *C,
                             int ldc, double alpha, double beta, double *Y, long ldy, int upper)
{
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(k_lincomb_tc<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, LC_SMEM) !=
                cudaSuccess ||
            cudaFuncSetAttribute(k_lincomb_tc<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, LC_SMEM) !=
                cudaSuccess)
            return gb_fail(ctx, GCGE_GPU_ERR_CUDA);
        attr = true;
    }
    const int nst = (k1 + TC_KS - 1) / TC_KS, jtiles = (k2 + TC_N - 1) / TC_N;
    const size_t bd_bytes = (size_t)jtiles * nst * OZ_DIGITS * TC_BPLANE;
    int st = gb_ozbuf(ctx, bd_bytes);
    if (!st) st = gb_iscratch(ctx, (size_t)k1 + k2);
    if (st) return st;
    uint32_t *Bd = (uint32_t *)ctx->ozbuf;
    int *g = ctx->iscratch, *ec = ctx->iscratch + k1;
    GB_LAUNCH(ctx, k_lc_coef_split, dim3(nst, jtiles), 256, 0, k1, k2, C, ldc, upper, nst, g, ec, Bd);
    GB_PROF(ctx, GB_K_LINCOMB, 8.0 * n * k1 + (beta != 0.0 ? 16.0 : 8.0) * n * k2,
            upper ? 1.0 * n * k1 * (k2 + 1) : 2.0 * n * k1 * k2);
    const long ntiles = ((long)n + TC_M - 1) / TC_M;
    long P = ctx->num_sms / jtiles;
    if (P < 1) P = 1;
    if (P > ntiles) P = ntiles;
    const int stall = ctx->tc_stall;
    ctx->tc_stall = 0;
    if (k1 > OZ_EXACT_TERMS)
        GB_LAUNCH(ctx, k_lincomb_tc<true>, dim3((unsigned)P, jtiles), TC_THREADS, LC_SMEM, n, k1, k2, X, ldx,
                  (const uint4 *)Bd, g, ec, alpha, beta, Y, ldy, nst, ctx->dev_err, stall);
    else
        GB_LAUNCH(ctx, k_lincomb_tc<false>, dim3((unsigned)P, jtiles), TC_THREADS, LC_SMEM, n, k1, k2, X, ldx,
                  (const uint4 *)Bd, g, ec, alpha, beta, Y, ldy, nst, ctx->dev_err, stall);
    return GCGE_GPU_OK;
}
