// gb_bcg_persist.cu -- all FP64 rounds of a block-CG call in one cooperative launch.
//
// A round of GCGE_BCG (src/gcge_cg.c:200-294) is three passes over the block with a
// column-wise sum over all rows after two of them (p.w, then r.r). As separate
// launches (update of p, product, dot pass, column sums, alpha, update of x and r,
// column sums, beta) a round was eight kernels. Here the passes are phases of one
// persistent grid (every block resident, so that blocks may wait on one another) and
// the sums are formed inside the grid barrier (2.2 us, 4 to 6 with sums). A call that
// has no active column left ends there. Time of a round, us, separate launches -> here:
//   100 x 100 grid, k = 10: 52 -> 25 (latency)   30 x 30 grid, k = 6: 51 -> 20
//   7-point 64^3, k = 32: 371 -> 283             FEM 40^3, k = 20: 117 -> 96
//   FEM 64^3, k = 50: 1,001 -> 798 (4.1e8 FP64 multiply-adds: 0.85 of the pipe's 6e11 a second)
//   power-law graph of 100,000, k = 44: 674 -> 319 (rows past GB_LONG_ROW by a block)
// (Forming p where it is gathered, b p + r from two buffers, saves a barrier and a pass and
// costs a multiply-add more per entry and lane slot: 2 to 4% faster below 30 x 30 x 6, 5% slower
// at 100 x 100 x 10 and up to 36% beyond; that form is gone.)
//
// Mapping. A block owns slabs of 128 rows. In the vector phases a thread owns eight
// rows of a column, spaced by eight (a unit): its 16 or 32 loads are all in flight,
// and the eight products are one chain of fused multiply-adds, the association of
// the sums: chains of eight, two chains, eight row classes, slabs strided by 256
// and a tree. It does not depend on the grid, so results repeat bit for bit on any
// device. In the product L lanes own a row and Q columns each (column sl + L q of a
// chunk), the shape with the fewest idle slots: the FP64 pipe issues for idle lanes
// too. Only p crosses a barrier; x and r of an entry belong to one thread.
//
// Every wait is bounded (a.wait_ns); a block whose wait runs out sets the
// context's device error word and leaves, and so do the others in turn.
#include <cstdint>
#include <cuda_runtime.h>

#include "gb_bcg.h"
#include "gb_coop.h"
#include "gb_internal.h"
#include "gb_launch.h"

#define PB_THREADS 256
#define PB_WARPS (PB_THREADS / 32)
#define PB_SLAB 128
// partials (slabs x columns) up to which the block that arrives last sums them all;
// beyond, one block per column does (a trip more, but side by side)
#define PB_ONE_BLOCK_SUMS 1024

#define GB_PROF(ctx, cls, bytes, flops) \
    do { if ((ctx)->prof) gb_prof_begin((ctx), (cls), (bytes), (flops)); } while (0)

enum { PB_PLAIN, PB_INIT, PB_ALPHA, PB_BETA };

struct pb_args {
    int n, k, max_it, long_rows, nslab;
    int cw;                    // columns of an item (a slab's chunk of columns), at most L Q
    double rate;
    const int *rp, *ci;
    const double *val;
    double *R, *X, *P, *W;     // residual, solution, direction, A p
    long ldr, ldx, ld;         // of R, of X, of P and W
    const double *dinv;
    double *rho2, *err, *alpha, *beta;
    double *part;              // [column][slab]
    unsigned *bar;             // [0] arrivals, [1] columns' owners done, [2..3] generation and active columns
    int *dev_err;
    unsigned long long wait_ns;
};

// sqrt(|s|) / err >= rate (src/gcge_cg.c:286-294); far from the line, where rounding
// cannot matter, without the square root and the division (0.7 us of the barrier).
// Squares compare as the quotient does only for a positive rate: t2 keeps its sign.
__device__ __forceinline__ bool pb_active(double s, double err, double rate)
{
    const double m = fabs(s), t = rate * err, t2 = t * fabs(t);
    if (t2 > 1e-280 && t2 < 1e280) {
        if (m > 1.0000001 * t2 && m < 1e300) return true;
        if (m < 0.9999999 * t2) return false;
    }
    return sqrt(m) / err >= rate;
}

// column sums over the slabs' partials: slab b goes to entry b mod 256, the entries to
// a binary tree. One warp: lane l holds entries l + 32 j.
__device__ __forceinline__ double pb_sum_warp(const double *p, int nslab)
{
    const int lane = threadIdx.x & 31;
    double v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        v[j] = 0;
        for (int b = lane + 32 * j; b < nslab; b += 256) v[j] += __ldcg(p + b);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int j = 0; j < o; ++j)
            if (32 * (j + o) < nslab) v[j] += v[j + o];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[0] += __shfl_down_sync(0xffffffffu, v[0], o);
    return v[0];                                         // lane 0's
}

// the same by a block; the sum is thread 0's
__device__ __forceinline__ double pb_sum_block(const double *p, int nslab, double *sh)
{
    double s = 0;
    for (int b = threadIdx.x; b < nslab; b += PB_THREADS) s += __ldcg(p + b);
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = PB_THREADS / 2; o >= 32; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    s = 0;
    if (threadIdx.x < 32) {
        s = sh[threadIdx.x];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    }
    __syncthreads();
    return s;
}

// what follows from column c's sum: alpha, or beta and the new r.r (one thread)
__device__ __forceinline__ void pb_column(const pb_args &a, int op, int c, double s, double r1)
{
    if (op == PB_INIT) {
        a.rho2[c] = s;
        a.err[c] = sqrt(s);
    } else if (op == PB_ALPHA) {
        a.alpha[c] = r1 / s;
    } else {
        a.rho2[c] = s;
        a.beta[c] = s / r1;                              // the next round's beta (src/gcge_cg.c:219)
    }
}

// Grid barrier that forms the column sums of `ka` columns and what follows from them.
// gen: the generation so far, in thread 0. Returns the active columns, -1 when a wait
// ran out. The generation and the count travel in one 64-bit word, so that nobody
// reads the count in a second trip.
__device__ int pb_barrier(const pb_args &a, int op, int ka, double *sh, unsigned &gen)
{
    __shared__ int last, res;
    const unsigned G = gridDim.x;
    const bool one = op == PB_PLAIN || (long)a.nslab * ka <= PB_ONE_BLOCK_SUMS;
    const unsigned owners = min((unsigned)ka, G);
    __syncthreads();
    if (threadIdx.x == 0) {
        last = coop_arrive(a.bar) == G - 1;
        res = 0;
    }
    __syncthreads();
    bool release = one && last;
    int cnt = op == PB_INIT ? a.k : op == PB_BETA ? 0 : ka;
    if (release && op != PB_PLAIN) {
        // sums by warps, then the columns' divisions side by side
        for (int cb = 0; cb < a.k; cb += PB_THREADS) {
            const int c = cb + threadIdx.x, m = min(PB_THREADS, ka - cb);
            const double r1 = op != PB_INIT && c < a.k ? __ldcg(a.rho2 + c) : 0.0;
            const double e1 = op == PB_BETA && c < a.k ? __ldcg(a.err + c) : 0.0;
            for (int q = threadIdx.x >> 5; q < m; q += PB_WARPS) {
                const double s = pb_sum_warp(a.part + (size_t)(cb + q) * a.nslab, a.nslab);
                if ((threadIdx.x & 31) == 0) sh[q] = s;
            }
            __syncthreads();
            const double s = (int)threadIdx.x < m ? sh[threadIdx.x] : r1;
            if (op == PB_BETA) cnt += __syncthreads_count(c < a.k && pb_active(s, e1, a.rate));
            if ((int)threadIdx.x < m) pb_column(a, op, c, s, r1);
            __syncthreads();
        }
    } else if (!one && blockIdx.x < owners) {
        if (threadIdx.x == 0) {
            const unsigned long long t0 = coop_now();
            int spin = 0;
            while (coop_ld32(a.bar) != G)
                if ((++spin & 1023) == 0 && coop_now() - t0 > a.wait_ns) {
                    atomicExch(a.dev_err, 1);
                    res = -1;
                    break;
                }
        }
        __syncthreads();
        if (res < 0) return -1;
        for (int c = blockIdx.x; c < ka; c += G) {
            const double r1 = op != PB_INIT ? __ldcg(a.rho2 + c) : 0.0;
            const double s = pb_sum_block(a.part + (size_t)c * a.nslab, a.nslab, sh);
            if (threadIdx.x == 0) pb_column(a, op, c, s, r1);
        }
        __syncthreads();
        if (threadIdx.x == 0) last = coop_arrive(a.bar + 1) == owners - 1;
        __syncthreads();
        release = last;
        if (release && op == PB_BETA)
            for (int cb = 0; cb < a.k; cb += PB_THREADS) {
                const int c = cb + threadIdx.x;
                cnt += __syncthreads_count(c < a.k && pb_active(__ldcg(a.rho2 + c), __ldcg(a.err + c), a.rate));
            }
    }
    if (release) {
        if (threadIdx.x == 0) {
            *(volatile unsigned *)a.bar = 0;
            *(volatile unsigned *)(a.bar + 1) = 0;
            ++gen;
            res = cnt;
            coop_release(a.bar + 2, gen, (unsigned)cnt);
        }
    } else if (threadIdx.x == 0) {
        const unsigned long long t0 = coop_now();
        int spin = 0;
        unsigned long long v;
        while ((unsigned)((v = coop_ld64(a.bar + 2)) >> 32) == gen)
            if ((++spin & 1023) == 0 && coop_now() - t0 > a.wait_ns) {
                atomicExch(a.dev_err, 1);
                v = 0xffffffffull;
                break;
            }
        ++gen;
        res = (int)(unsigned)v;
    }
    __syncthreads();
    return res;
}

// unit u of a chunk of kc columns: column c, row class ty of eight, half h of the slab
#define PB_UNITS(u, kc) for (int u = threadIdx.x; u < 16 * (kc); u += PB_THREADS)
struct pb_unit {
    int c, row;                                          // column in the chunk, first row in the slab
    int slot;                                            // 8 h + ty
};
__device__ __forceinline__ pb_unit pb_decode(int u, int kc)
{
    pb_unit x;
    x.slot = u / kc;
    x.c = u - x.slot * kc;
    x.row = (x.slot & 7) + 64 * (x.slot >> 3);
    return x;
}

// the slab's partials of a chunk's columns from the units' chains red[slot][column]
template <int C>
__device__ __forceinline__ void pb_slab_partials(const pb_args &a, double (*red)[C], int c0, int kc, long slab)
{
    __syncthreads();
    for (int c = threadIdx.x; c < kc; c += PB_THREADS) {
        double t = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) t += red[q][c] + red[8 + q][c];
        a.part[(size_t)(c0 + c) * a.nslab + slab] = t;
    }
    __syncthreads();
}

// entries [beg, end) of a row in steps of `step` by a group of L lanes
template <int L, int Q>
__device__ __forceinline__ void pb_row(const pb_args &a, int beg, int end, int step, int sl, unsigned gmask,
                                       const int col[Q], double acc[Q])
{
    for (int base = beg; base < end; base += step) {
        const int e = base + sl;
        int j = 0;
        double v = 0;
        if (e < end) {
            j = __ldg(a.ci + e);
            v = __ldg(a.val + e);
        }
        const int m = min(L, end - base);
#pragma unroll 4
        for (int t = 0; t < m; ++t) {
            const int jj = __shfl_sync(gmask, j, t, L);
            const double vv = __shfl_sync(gmask, v, t, L);
            const double *p = a.P + (long)jj * a.ld;
#pragma unroll
            for (int q = 0; q < Q; ++q) acc[q] = fma(vv, p[col[q]], acc[q]);
        }
    }
}

// items: (slab, chunk of columns) pairs, the chunks of a slab side by side
#define PB_ITEMS(cols)                                                                \
    const unsigned nch = ((unsigned)(cols) + a.cw - 1) / a.cw, items = a.nslab * nch; \
    for (unsigned item = blockIdx.x; item < items; item += gridDim.x)
#define PB_ITEM(cols)                                 \
    const unsigned is = nch == 1 ? item : item / nch; \
    const long slab = is;                             \
    const int c0 = (int)((item - is * nch) * a.cw), kc = min(a.cw, (cols) - c0);

// MB blocks an SM (the registers for it): two for matrices without long rows where that takes no
// more waves of items than three do, see gb_bcg_persist64
template <int L, int Q, int MB>
__global__ void __launch_bounds__(PB_THREADS, MB)
k_bcg_persist(const pb_args a)
{
    GB_PDL();
    constexpr int RPB = PB_THREADS / L, C = L * Q;
    __shared__ double red[16][C];
    __shared__ double sh[PB_THREADS];
    __shared__ int lflag[MB == 3 ? RPB : 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sl = lane % L, slot = threadIdx.x / L;
    const unsigned gmask = (L == 32) ? 0xffffffffu : (((1u << L) - 1u) << ((lane / L) * L));
    const int n = a.n, k = a.k;
    if (*(volatile int *)a.dev_err) return;              // an earlier wait ran out: do nothing
    unsigned gen = threadIdx.x == 0 ? (unsigned)(coop_ld64(a.bar + 2) >> 32) : 0;

    // norms of the initial residual
    {
        PB_ITEMS(k)
        {
            PB_ITEM(k)
            PB_UNITS(u, kc)
            {
                const pb_unit x = pb_decode(u, kc);
                double run = 0;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const long r = slab * PB_SLAB + x.row + 8 * i;
                    if (r < n) {
                        const double v = a.R[r * a.ldr + c0 + x.c];
                        run = fma(v, a.dinv ? a.dinv[r] * v : v, run);
                    }
                }
                red[x.slot][x.c] = run;
            }
            pb_slab_partials<C>(a, red, c0, kc, slab);
        }
    }
    int ka = pb_barrier(a, PB_INIT, k, sh, gen);

    for (int it = 1; ka > 0 && it < a.max_it; ++it) {
        const bool first = it == 1;
        // p = z + beta p on the active columns (p = z first; z = r, or D^-1 r)
        {
            PB_ITEMS(ka)
            {
                PB_ITEM(ka)
                PB_UNITS(u, kc)
                {
                    const pb_unit x = pb_decode(u, kc);
                    const int c = c0 + x.c;
                    const double b = first ? 0.0 : __ldcg(a.beta + c);
                    double z[8], p[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const long r = slab * PB_SLAB + x.row + 8 * i;
                        z[i] = r < n ? a.R[r * a.ldr + c] : 0.0;
                        p[i] = r < n && !first ? a.P[r * a.ld + c] : 0.0;
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const long r = slab * PB_SLAB + x.row + 8 * i;
                        if (r < n) {
                            const double zz = a.dinv ? __dmul_rn(a.dinv[r], z[i]) : z[i];
                            a.P[r * a.ld + c] = first ? zz : fma(b, p[i], zz);
                        }
                    }
                }
            }
        }
        if (pb_barrier(a, PB_PLAIN, ka, sh, gen) < 0) return;
        // w = A p and the column sums of p.w
        {
            PB_ITEMS(ka)
            {
                PB_ITEM(ka)
                int col[Q];
#pragma unroll
                for (int q = 0; q < Q; ++q) col[q] = c0 + min(sl + L * q, kc - 1);   // idle slots: a column again
                for (int b = 0; b < PB_SLAB; b += RPB) {
                    const long r0 = slab * PB_SLAB + b, r = r0 + slot;
                    int beg = 0, end = 0;
                    if (r < n) {
                        beg = __ldg(a.rp + r);
                        end = __ldg(a.rp + r + 1);
                    }
                    double acc[Q];
#pragma unroll
                    for (int q = 0; q < Q; ++q) acc[q] = 0;
                    const bool lng = MB == 3 && a.long_rows && end - beg > GB_LONG_ROW;
                    if (!lng) pb_row<L, Q>(a, beg, end, L, sl, gmask, col, acc);
                    // rows longer than GB_LONG_ROW: all groups of the block on one row, the
                    // group sums added by shuffles and then warp by warp, in row order
                    if (MB == 3 && a.long_rows && __syncthreads_or(lng)) {
                        if (sl == 0) lflag[slot] = lng;
                        __syncthreads();
                        for (int q0 = 0; q0 < RPB; ++q0) {
                            if (!lflag[q0]) continue;
                            const int lb = __ldg(a.rp + r0 + q0), le = __ldg(a.rp + r0 + q0 + 1);
                            double la[Q];
#pragma unroll
                            for (int q = 0; q < Q; ++q) la[q] = 0;
                            pb_row<L, Q>(a, lb + slot * L, le, PB_THREADS, sl, gmask, col, la);
                            __syncwarp();
#pragma unroll
                            for (int q = 0; q < Q; ++q) {
#pragma unroll
                                for (int o = L; o < 32; o <<= 1) la[q] += __shfl_xor_sync(0xffffffffu, la[q], o);
                                if (lane < L) red[warp][sl + L * q] = la[q];
                            }
                            __syncthreads();
                            if (slot == q0) {
#pragma unroll
                                for (int q = 0; q < Q; ++q) {
                                    double t = 0;
#pragma unroll
                                    for (int w = 0; w < PB_WARPS; ++w) t += red[w][sl + L * q];
                                    acc[q] = t;
                                }
                            }
                            __syncthreads();
                        }
                    }
                    if (r < n) {
#pragma unroll
                        for (int q = 0; q < Q; ++q)
                            if (sl + L * q < kc) a.W[r * a.ld + c0 + sl + L * q] = acc[q];
                    }
                }
                __syncthreads();                         // the item's w is written
                PB_UNITS(u, kc)
                {
                    const pb_unit x = pb_decode(u, kc);
                    const int c = c0 + x.c;
                    double p[8], w[8], run = 0;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const long r = slab * PB_SLAB + x.row + 8 * i;
                        p[i] = r < n ? a.P[r * a.ld + c] : 0.0;
                        w[i] = r < n ? a.W[r * a.ld + c] : 0.0;
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (slab * PB_SLAB + x.row + 8 * i < n) run = fma(p[i], w[i], run);
                    red[x.slot][x.c] = run;
                }
                pb_slab_partials<C>(a, red, c0, kc, slab);
            }
        }
        if (pb_barrier(a, PB_ALPHA, ka, sh, gen) < 0) return;
        // x += alpha p, r -= alpha w and the column sums of r.z
        {
            PB_ITEMS(ka)
            {
                PB_ITEM(ka)
                PB_UNITS(u, kc)
                {
                    const pb_unit x = pb_decode(u, kc);
                    const int c = c0 + x.c;
                    const double al = __ldcg(a.alpha + c);
                    double xv[8], rv[8], p[8], w[8], run = 0;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const long r = slab * PB_SLAB + x.row + 8 * i;
                        const bool in = r < n;
                        p[i] = in ? a.P[r * a.ld + c] : 0.0;
                        w[i] = in ? a.W[r * a.ld + c] : 0.0;
                        xv[i] = in ? a.X[r * a.ldx + c] : 0.0;
                        rv[i] = in ? a.R[r * a.ldr + c] : 0.0;
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const long r = slab * PB_SLAB + x.row + 8 * i;
                        if (r < n) {
                            a.X[r * a.ldx + c] = fma(al, p[i], xv[i]);
                            const double rn = fma(-al, w[i], rv[i]);
                            a.R[r * a.ldr + c] = rn;
                            run = fma(rn, a.dinv ? a.dinv[r] * rn : rn, run);
                        }
                    }
                    red[x.slot][x.c] = run;
                }
                pb_slab_partials<C>(a, red, c0, kc, slab);
            }
        }
        ka = pb_barrier(a, PB_BETA, ka, sh, gen);
    }
}

// (L, Q) with the fewest idle lane slots for k columns (ties: the larger L)
static void pb_shape(int k, int maxq, int *Lo, int *Qo)
{
    double best = -1;
    for (int L = 16; L >= 4; L >>= 1) {
        int q = (k + L - 1) / L;
        if (q > maxq) q = maxq;
        const int cols = L * q, chunks = (k + cols - 1) / cols;
        const double eff = (double)k / ((double)chunks * cols);
        if (eff > best + 1e-12) {
            best = eff;
            *Lo = L;
            *Qo = q;
        }
    }
}

static const void *pb_kernel(int L, int Q, int mb)
{
#define PB_K4(LL, q, MB) (const void *)k_bcg_persist<LL, q, MB>, (const void *)k_bcg_persist<LL, q + 1, MB>, \
                         (const void *)k_bcg_persist<LL, q + 2, MB>, (const void *)k_bcg_persist<LL, q + 3, MB>
#define PB_K8(LL, MB) {PB_K4(LL, 1, MB), PB_K4(LL, 5, MB)}
    static const void *const tab[2][3][8] = {{PB_K8(4, 2), PB_K8(8, 2), PB_K8(16, 2)}, {PB_K8(4, 3), PB_K8(8, 3), PB_K8(16, 3)}};
#undef PB_K4
#undef PB_K8
    return tab[mb - 2][L == 4 ? 0 : L == 8 ? 1 : 2][Q - 1];
}

extern "C" int gb_bcg_persist64(gcge_gpu_ctx *ctx, const gcge_gpu_mat *A, const gb_bcg_args *b, const bcg_state *s,
                                double *R, long ldr, double *X, long ldx, double *P, double *W, long ld)
{
    pb_args a = {};
    a.n = b->n;
    a.k = b->k;
    a.max_it = b->max_it;
    a.rate = b->rate;
    a.nslab = (b->n + PB_SLAB - 1) / PB_SLAB;
    a.long_rows = A->max_row_nnz > GB_LONG_ROW;
    a.rp = A->rp;
    a.ci = A->ci;
    a.val = A->v;
    a.R = R;
    a.ldr = ldr;
    a.X = X;
    a.ldx = ldx;
    a.P = P;
    a.W = W;
    a.ld = ld;
    a.dinv = b->dinv;
    a.rho2 = s->rho2;
    a.err = s->err;
    a.alpha = s->alpha;
    a.beta = s->beta;
    a.part = s->part;
    a.bar = ctx->dev_bar;
    a.dev_err = ctx->dev_err;
    a.wait_ns = gb_coop_wait_ns(ctx);
    int L = 16, Q = 1, per_sm = 0;
    // Items of fewer columns where whole slabs would leave SMs without work: the chunk
    // count with the shortest busiest SM, an item costing its latencies (as much as
    // eight columns) and its lane slots.
    const long sms = ctx->num_sms;
    double best = 0;
    for (int chunks = 1; chunks <= 32 && chunks <= a.k; ++chunks) {
        int l = 16, q = 1, cw = (a.k + chunks - 1) / chunks;
        pb_shape(cw, 4, &l, &q);
        if (cw > l * q) continue;
        const double t = (double)((a.nslab * (long)((a.k + cw - 1) / cw) + sms - 1) / sms) * (8 + l * q);
        if (best == 0 || t < 0.95 * best) {
            best = t;
            a.cw = cw;
        }
    }
    if (best == 0 || (long)a.nslab >= 4 * sms) a.cw = a.k;
    pb_shape(a.cw, 8, &L, &Q);
    if (a.cw > L * Q) a.cw = L * Q;
    const long items = (long)a.nslab * ((a.k + a.cw - 1) / a.cw);
    // Three blocks an SM hide more of the gathers' latency, two have registers for all their loads in
    // flight (three spill 108 to 224 bytes) and leave a last item less often alone on its SM.
    // Two where that takes no more waves of items: 27-point 40^3, k = 64 (500 items) 336 -> 261 us
    // a round, eight separate kernels took 293; 7-point 40^3, k = 32 103 -> 82 (101); one wave either way 2
    // to 7%. One wave more and two lose: 27-point 36^3, k = 32 (365) 108 -> 126, 5-point 200^2, k = 24 46 ->
    // 57; from 12 items an SM on both are within 13%. Long rows keep three: 20,000-node
    // graph, k = 20 84 against 109 us.
    auto waves = [&](int b) { return (items + b * sms - 1) / (b * sms); };
    const int mb = !a.long_rows && waves(2) == waves(3) ? 2 : 3;
    const void *fn = pb_kernel(L, Q, mb);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, PB_THREADS, 0) != cudaSuccess || per_sm < 1)
        return gb_fail(ctx, GCGE_GPU_ERR_CUDA);
    long G = (long)ctx->num_sms * per_sm;
    if (G > items) G = items;
    const double nk = (double)a.n * a.k, rounds = a.max_it > 1 ? a.max_it - 1 : 0;
    GB_PROF(ctx, GB_K_SPMM64, rounds * (12.0 * A->nnz + 4.0 * (A->n + 1) + 88.0 * nk),
            rounds * (2.0 * A->nnz * a.k + 10.0 * nk));
    void *args[] = {&a};
    if (cudaLaunchCooperativeKernel(fn, dim3((unsigned)G), dim3(PB_THREADS), args, 0, ctx->stream) != cudaSuccess) {
        cudaGetLastError();
        return gb_fail(ctx, GCGE_GPU_ERR_CUDA);
    }
    ctx->launches++;
    ctx->spmm_launches += (long long)rounds;
    if (ctx->prof) gb_prof_end(ctx);
    return gb_check_launch(ctx);
}
