// gb_adjoint.cu -- reverse-mode (adjoint) kernels of the computed eigenpairs:
// gradients of a function of eigenpairs with respect to the stored entries of A
// and B. The reference has no differentiation; these entry points extend the C
// ABI for callers that need sensitivities of A x = lambda B x.
//
// For a B-orthonormal eigenpair (lambda, x) of the symmetric pencil and a
// perturbation of one stored entry (i, j):
//   d lambda / d A_ij =  x_i x_j,          d lambda / d B_ij = -lambda x_i x_j
// (Hellmann-Feynman). For a function L(x) of a simple eigenvector with gradient
// g = dL/dx, let mu solve (A - lambda B) mu = (I - B x x^T) g with x^T B mu = 0;
// then
//   dL / d A_ij = -mu_i x_j,   dL / d B_ij = lambda mu_i x_j - (g^T x / 2) x_i x_j.
// Both are sums of products U[i, t] V[j, t] over the sparsity pattern (an SDDMM),
// which GCGE_GPU_PatternGrad evaluates; GCGE_GPU_EigvecAdjoint computes mu.
#include "gb_coop.h"
#include "gb_internal.h"
#include "gb_launch.h"

#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include <stdlib.h>
#include <string.h>

#define AD_CUDA(ctx, call)                                                             \
    do {                                                                               \
        if ((call) != cudaSuccess) return gb_fail((ctx), GCGE_GPU_ERR_CUDA);           \
    } while (0)

#define PG_THREADS 256
#define PG_ROWS 64                      // most rows of a block
#define PG_CHUNK 2048                   // entries whose rows are listed at a time
#define PG_SMEM (44 * 1024)             // scaled U rows of a block (48 KB with the lists)
#define PG_MAX_R 768

// grad[e] = (acc ? grad[e] : 0) + sum_t s[t] U[i, t] V[j, t], e = (i, j) stored.
// A block owns a run of rows: their scaled U values in shared memory, and the row of
// every entry of the run beside them, so that the entries -- not the rows -- are dealt
// to the lanes, LPE consecutive lanes each, and every lane works whatever the
// row lengths (an FP64 instruction costs a warp 16 clocks for one lane as for 32: a warp
// per row with lanes over t and a shuffle tree per entry spent five adds of all lanes
// on each, 502 us for the 5-point 512^2 pattern with r = 20; here 71 us). LPE: two
// lanes read 16 consecutive bytes of a V row, four (r >= 32) a whole sector.
// Sums in a fixed order: the result does not depend on scheduling.
template <int LPE>
__global__ void __launch_bounds__(PG_THREADS)
k_pattern_grad(int n, const int *__restrict__ rp, const int *__restrict__ ci, const double *__restrict__ U,
               long ldu, const double *__restrict__ V, long ldv, int r, const double *__restrict__ s, int acc,
               double *__restrict__ grad, int rows)
{
    GB_PDL();
    extern __shared__ double us[];      // [rows][r | 1]
    __shared__ unsigned char row_of[PG_CHUNK];
    __shared__ int first[PG_ROWS + 1];
    const int ldus = r | 1;             // odd: the lanes' rows fall in different banks
    const long i0 = (long)blockIdx.x * rows;
    const int nr = (int)min((long)rows, n - i0);
    for (int t = threadIdx.x; t < nr * r; t += PG_THREADS) {
        const int i = t / r, q = t - i * r;
        us[i * ldus + q] = s[q] * U[(i0 + i) * ldu + q];
    }
    for (int i = threadIdx.x; i <= nr; i += PG_THREADS) first[i] = rp[i0 + i];
    __syncthreads();
    const int e0 = first[0], e1 = first[nr], sub = threadIdx.x % LPE;
    // the lanes of an entry: one k for all of them, but loops over t of unequal length
    const unsigned group = ((1u << LPE) - 1) << ((threadIdx.x & 31) & ~(LPE - 1));
    for (int base = e0; base < e1; base += PG_CHUNK) {
        const int cnt = min(PG_CHUNK, e1 - base);
        // four threads list a row's entries
        for (int i = threadIdx.x >> 2; i < nr; i += PG_THREADS / 4)
            for (int e = max(first[i], base) + (threadIdx.x & 3); e < min(first[i + 1], base + cnt); e += 4)
                row_of[e - base] = (unsigned char)i;
        __syncthreads();
        for (int k = threadIdx.x / LPE; k < cnt; k += PG_THREADS / LPE) {
            const double *vr = V + (long)__ldg(ci + base + k) * ldv;
            const double *ur = us + row_of[k] * ldus;
            double sum = 0.0;
#pragma unroll 4
            for (int t = sub; t < r; t += LPE) sum = fma(ur[t], __ldg(vr + t), sum);
#pragma unroll
            for (int o = 1; o < LPE; o <<= 1) sum += __shfl_xor_sync(group, sum, o, LPE);
            if (sub == 0) grad[base + k] = acc ? grad[base + k] + sum : sum;
        }
        __syncthreads();
    }
}

static int pg_launch(gcge_gpu_ctx *ctx, const gcge_gpu_mat *M, const double *U, long ldu, const double *V, long ldv,
                     int r, const double *s_dev, int acc, double *grad_dev)
{
    int rows = PG_SMEM / 8 / (r | 1);
    if (rows > PG_ROWS) rows = PG_ROWS;
    // few rows: a block for every SM
    if ((long)rows * ctx->num_sms > M->n) rows = (M->n + ctx->num_sms - 1) / ctx->num_sms;
    if (rows < 1) return gb_fail(ctx, GCGE_GPU_ERR_ARG);
    const int blocks = (int)(((long)M->n + rows - 1) / rows);
    const size_t smem = sizeof(double) * (size_t)rows * (r | 1);
    if (r < 4)
        GB_LAUNCH(ctx, k_pattern_grad<1>, blocks, PG_THREADS, smem, M->n, M->rp, M->ci, U, ldu, V, ldv, r, s_dev, acc,
                  grad_dev, rows);
    else if (r < 32)
        GB_LAUNCH(ctx, k_pattern_grad<2>, blocks, PG_THREADS, smem, M->n, M->rp, M->ci, U, ldu, V, ldv, r, s_dev, acc,
                  grad_dev, rows);
    else
        GB_LAUNCH(ctx, k_pattern_grad<4>, blocks, PG_THREADS, smem, M->n, M->rp, M->ci, U, ldu, V, ldv, r, s_dev, acc,
                  grad_dev, rows);
    return GCGE_GPU_OK;
}

static int mv_cols_ok(const gcge_gpu_mv *m, int c0, int k)
{
    return m && c0 >= 0 && k >= 0 && c0 + k <= m->ncols;
}

extern "C" int GCGE_GPU_PatternGrad(const gcge_gpu_mat *M, const gcge_gpu_mv *U, int u0, const gcge_gpu_mv *V,
                                    int v0, int r, const double *scale, int accumulate, double *grad)
{
    if (!M || !U || !V || !scale || !grad) return GCGE_GPU_ERR_ARG;
    gcge_gpu_ctx *ctx = M->ctx;
    if (r < 1 || !mv_cols_ok(U, u0, r) || !mv_cols_ok(V, v0, r) || U->n != M->n || V->n != M->n ||
        r > PG_MAX_R)
        return gb_fail(ctx, GCGE_GPU_ERR_ARG);
    if (M->nnz == 0) return GCGE_GPU_OK;
    double *g_dev = nullptr, *s_dev = nullptr;
    int st = GCGE_GPU_OK;
    if (gb_call_alloc(ctx, (void **)&g_dev, sizeof(double) * (size_t)M->nnz) ||
        gb_call_alloc(ctx, (void **)&s_dev, sizeof(double) * (size_t)r)) {
        st = gb_fail(ctx, GCGE_GPU_ERR_NOMEM);
        goto done;
    }
    if (cudaMemcpyAsync(s_dev, scale, sizeof(double) * r, cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess ||
        (accumulate && cudaMemcpyAsync(g_dev, grad, sizeof(double) * (size_t)M->nnz, cudaMemcpyHostToDevice,
                                       ctx->stream) != cudaSuccess)) {
        st = gb_fail(ctx, GCGE_GPU_ERR_CUDA);
        goto done;
    }
    st = pg_launch(ctx, M, U->d + u0, U->ld, V->d + v0, V->ld, r, s_dev, accumulate != 0, g_dev);
    if (st) goto done;
    if (cudaMemcpyAsync(grad, g_dev, sizeof(double) * (size_t)M->nnz, cudaMemcpyDeviceToHost, ctx->stream) !=
            cudaSuccess ||
        cudaStreamSynchronize(ctx->stream) != cudaSuccess)
        st = gb_fail(ctx, GCGE_GPU_ERR_CUDA);
done:
    cudaStreamSynchronize(ctx->stream);
    gb_call_free(ctx, g_dev);
    gb_call_free(ctx, s_dev);
    return st;
}

// ---------------------------------------------------------------- single-vector kernels
// The adjoint CG works on one n-vector at a time; these kernels are sized for
// that (the block kernels of the solver are not).
#define AV_THREADS 256
#define AV_BLOCKS_PER_SM 4

static int av_grid(gcge_gpu_ctx *ctx, long work)
{
    long g = (work + AV_THREADS - 1) / AV_THREADS, cap = (long)ctx->num_sms * AV_BLOCKS_PER_SM;
    if (g > cap) g = cap;
    return (int)(g < 1 ? 1 : g);
}

// y = a x + b y (b == 0: y = a x, y not read)
__global__ void k_av_axpby(long n, double a, const double *__restrict__ x, double b, double *__restrict__ y)
{
    GB_PDL();
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        y[i] = b == 0.0 ? a * x[i] : fma(a, x[i], b * y[i]);
}

// part[block] = sum over the block's grid-stride slice of x_i y_i (fixed order)
__global__ void __launch_bounds__(AV_THREADS)
k_av_dot_part(long n, const double *__restrict__ x, const double *__restrict__ y, double *__restrict__ part)
{
    GB_PDL();
    __shared__ double red[AV_THREADS / 32];
    double s = 0.0;
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        s = fma(x[i], y[i], s);
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < AV_THREADS / 32; ++w) t += red[w];
        part[blockIdx.x] = t;
    }
}

// out[0] = sum of nparts partials (one warp, fixed order)
__global__ void k_av_sum(int nparts, const double *__restrict__ part, double *__restrict__ out)
{
    GB_PDL();
    double s = 0.0;
    for (int i = threadIdx.x; i < nparts; i += 32) s += part[i];
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) out[0] = s;
}

// part[block][j] = sum over the block's rows of X[r, j] v[r], j < m <= 64: a warp
// per row, lanes over the columns (a row of X is contiguous)
__global__ void __launch_bounds__(AV_THREADS)
k_av_xtv_part(long n, int m, const double *__restrict__ X, long ldx, const double *__restrict__ v,
              double *__restrict__ part)
{
    GB_PDL();
    __shared__ double red[AV_THREADS / 32][64];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double s0 = 0.0, s1 = 0.0;
    const long nw = ((long)gridDim.x * AV_THREADS) >> 5;
    for (long r = ((long)blockIdx.x * AV_THREADS + threadIdx.x) >> 5; r < n; r += nw) {
        const double vr = v[r];
        const double *xr = X + r * ldx;
        if (lane < m) s0 = fma(xr[lane], vr, s0);
        if (lane + 32 < m) s1 = fma(xr[lane + 32], vr, s1);
    }
    red[w][lane] = s0;
    red[w][lane + 32] = s1;
    __syncthreads();
    for (int j = threadIdx.x; j < m; j += AV_THREADS) {
        double t = 0.0;
        for (int q = 0; q < AV_THREADS / 32; ++q) t += red[q][j];
        part[(long)blockIdx.x * m + j] = t;
    }
}

// c[j] = sum of the partials of column j (thread per column, fixed order)
__global__ void k_av_xtv_sum(int nparts, int m, const double *__restrict__ part, double *__restrict__ c)
{
    GB_PDL();
    const int j = threadIdx.x;
    if (j >= m) return;
    double t = 0.0;
    for (int b = 0; b < nparts; ++b) t += part[(long)b * m + j];
    c[j] = t;
}

// y = v - X c (thread per row, c in shared memory), m <= 64
__global__ void __launch_bounds__(AV_THREADS)
k_av_v_minus_xc(long n, int m, const double *__restrict__ X, long ldx, const double *__restrict__ c,
                const double *__restrict__ v, double *__restrict__ y)
{
    GB_PDL();
    __shared__ double cs[64];
    if (threadIdx.x < m) cs[threadIdx.x] = c[threadIdx.x];
    __syncthreads();
    for (long r = (long)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (long)gridDim.x * blockDim.x) {
        const double *xr = X + r * ldx;
        double s = 0.0;
        for (int j = 0; j < m; ++j) s = fma(xr[j], cs[j], s);
        y[r] = v[r] - s;
    }
}

// ---------------------------------------------------------------- adjoint solve
// Work of one adjoint solve, all device resident (n-vectors contiguous, ld 1).
struct ad_work {
    double *BX;        // B X (n x m, ld m) or NULL when B = I
    double *y, *r, *p, *q, *t, *u, *w;
    double *c;         // m coefficients
    double *dot;       // one scalar, or the iteration's state
    double *part;      // block partials (grid x max(m, 1))
    double *h_c;       // host copy of m coefficients
};

#define AD_SKINNY_M 64                  // widest X handled by the single-vector kernels

static int ad_axpby(gcge_gpu_ctx *ctx, int n, double a, const double *x, double b, double *y)
{
    GB_LAUNCH(ctx, k_av_axpby, av_grid(ctx, n), AV_THREADS, 0, (long)n, a, x, b, y);
    return GCGE_GPU_OK;
}

static int ad_dot(gcge_gpu_ctx *ctx, int n, const double *x, const double *y, ad_work *W, double *out)
{
    const int g = av_grid(ctx, n);
    GB_LAUNCH(ctx, k_av_dot_part, g, AV_THREADS, 0, (long)n, x, y, W->part);
    GB_LAUNCH(ctx, k_av_sum, 1, 32, 0, g, W->part, W->dot);
    AD_CUDA(ctx, cudaMemcpyAsync(out, W->dot, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    AD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (!isfinite(*out)) return gb_fail(ctx, GCGE_GPU_ERR_NONFINITE);
    return GCGE_GPU_OK;
}

// c = X^T v (m coefficients, device)
static int ad_xtv(gcge_gpu_ctx *ctx, int n, int m, const double *X, long ldx, const double *v, double *c, ad_work *W)
{
    if (m > AD_SKINNY_M) return gb_gram(ctx, n, m, 1, X, ldx, v, 1, c, m, 0);
    const int g = av_grid(ctx, (long)n * 32);
    GB_LAUNCH(ctx, k_av_xtv_part, g, AV_THREADS, 0, (long)n, m, X, ldx, v, W->part);
    GB_LAUNCH(ctx, k_av_xtv_sum, 1, 64, 0, g, m, W->part, c);
    return GCGE_GPU_OK;
}

// y = v - X c (y may be v)
static int ad_v_minus_xc(gcge_gpu_ctx *ctx, int n, int m, const double *X, long ldx, const double *c,
                         const double *v, double *y)
{
    if (m > AD_SKINNY_M) {
        int st = y != v ? ad_axpby(ctx, n, 1.0, v, 0.0, y) : GCGE_GPU_OK;
        return st ? st : gb_lincomb(ctx, n, m, 1, X, ldx, c, m, -1.0, 1.0, y, 1, 0);
    }
    GB_LAUNCH(ctx, k_av_v_minus_xc, av_grid(ctx, n), AV_THREADS, 0, (long)n, m, X, ldx, c, v, y);
    return GCGE_GPU_OK;
}

// dst = src - Xo (X^T Bsrc): the B-orthogonal projection onto the complement of
// X's columns (Xo = X, Bsrc = B src) or its transpose (Xo = B X, Bsrc = src)
static int ad_project(gcge_gpu_ctx *ctx, int n, int m, const double *X, long ldx, const double *Xo, long ldo,
                      const double *src, const double *Bsrc, double *dst, ad_work *W)
{
    int st = ad_xtv(ctx, n, m, X, ldx, Bsrc, W->c, W);
    return st ? st : ad_v_minus_xc(ctx, n, m, Xo, ldo, W->c, src, dst);
}

// q = P^T (A - lambda B) P p with P = I - X X^T B (t, u, w scratch)
static int ad_apply(gcge_gpu_ctx *ctx, const gcge_gpu_mat *A, const gcge_gpu_mat *B, int n, int m, const double *X,
                    long ldx, double lambda, const double *p, double *q, ad_work *W)
{
    int st;
    const double *BX = W->BX ? W->BX : X;
    const long ldbx = W->BX ? m : ldx;
    // t = P p
    if (B) {
        if ((st = gb_spmm(ctx, B, p, 1, W->w, 1, 1, 1.0, nullptr, 0.0, nullptr))) return st;
        if ((st = ad_project(ctx, n, m, X, ldx, X, ldx, p, W->w, W->t, W))) return st;
    } else if ((st = ad_project(ctx, n, m, X, ldx, X, ldx, p, p, W->t, W))) {
        return st;
    }
    // u = A t - lambda B t
    if ((st = gb_spmm(ctx, A, W->t, 1, W->u, 1, 1, 1.0, nullptr, 0.0, nullptr))) return st;
    if (B) {
        if ((st = gb_spmm(ctx, B, W->t, 1, W->w, 1, 1, 1.0, nullptr, 0.0, nullptr))) return st;
        if ((st = ad_axpby(ctx, n, -lambda, W->w, 1.0, W->u))) return st;
    } else if ((st = ad_axpby(ctx, n, -lambda, W->t, 1.0, W->u))) {
        return st;
    }
    // q = P^T u = u - B X (X^T u)
    return ad_project(ctx, n, m, X, ldx, BX, ldbx, W->u, W->u, q, W);
}

// ---------------------------------------------------------------- the CG iteration in one launch
// An iteration is a projection (X^T p, p - X c), a product, a second projection, a dot
// product, the updates and another dot. As launches that was fifteen kernels and two
// host synchronisations, 167 us on 16,384 unknowns with ten vectors, of which the
// arithmetic needs five. Here the phases are those of one cooperative grid and the
// sums are formed in its barriers (five an iteration, six with B): 28 us. A block owns
// tiles of 128 rows, a thread a row; for X^T v the lanes of a warp take columns
// instead (32 / lanes-for-m rows at once), as one FP64 instruction costs a warp the
// same 16 clocks for one lane as for 32.
#define AC_ROWS 128
#define AC_WARPS (AC_ROWS / 32)

// scalars of the iteration, written by the block that ends a barrier
struct ac_state {
    double rr, alpha, beta, bnorm;
    int it, status;
};
struct ac_args {
    int n, m, max_it, warp_rows;             // warp_rows: products by a warp per row (long rows)
    double lambda, tol;
    const int *arp, *aci, *brp, *bci;
    const double *av, *bv;                   // bv: NULL when B = I
    const double *X, *BX;
    long ldx, ldbx;
    double *y, *r, *p, *q, *t, *u;
    double *c, *part;                        // m sums; [m][grid] partials
    ac_state *s;
    unsigned *bar;
    int *dev_err;
    unsigned long long wait_ns;
};
enum { AC_PLAIN, AC_COEF, AC_PQ, AC_RR };

// grid barrier with ns column sums (fixed order) and what the op derives from them;
// the message is 1 to go on, 0 to stop; -1: a wait ran out
__device__ int ac_barrier(const ac_args &a, int op, int ns, unsigned &gen)
{
    __shared__ int last, res;
    __shared__ double sum0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, G = gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) last = coop_arrive(a.bar) == (unsigned)G - 1;
    __syncthreads();
    if (last) {
        for (int j = warp; j < ns; j += AC_WARPS) {
            double s = 0;
            for (int b = lane; b < G; b += 32) s += __ldcg(a.part + (size_t)j * G + b);
#pragma unroll
            for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) {
                if (op == AC_COEF) a.c[j] = s;
                else sum0 = s;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            ac_state *s = a.s;
            int go = 1;
            if (op == AC_PQ || op == AC_RR) {
                const double v = sum0, rr = __ldcg(&s->rr);
                if (!isfinite(v)) {
                    s->status = GCGE_GPU_ERR_NONFINITE;
                    go = 0;
                } else if (op == AC_PQ) {
                    if (v > 0) s->alpha = rr / v;
                    else go = 0;                         // left the SPD complement: stop
                } else {
                    const int it = __ldcg(&s->it) + 1;
                    s->beta = v / rr;
                    s->rr = v;
                    s->it = it;
                    go = sqrt(v) > a.tol * __ldcg(&s->bnorm) && it < a.max_it;
                }
            }
            *(volatile unsigned *)a.bar = 0;
            ++gen;
            res = go;
            coop_release(a.bar + 2, gen, (unsigned)go);
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

// row r of M v (one thread)
__device__ __forceinline__ double ac_row(const int *rp, const int *ci, const double *val, const double *v, long r)
{
    double s = 0;
    const int end = __ldg(rp + r + 1);
#pragma unroll 4
    for (int e = __ldg(rp + r); e < end; ++e) s = fma(__ldg(val + e), v[__ldg(ci + e)], s);
    return s;
}
// row r of M v by a warp
__device__ __forceinline__ double ac_row_warp(const int *rp, const int *ci, const double *val, const double *v, long r)
{
    double s = 0;
    const int end = __ldg(rp + r + 1);
    for (int e = __ldg(rp + r) + (threadIdx.x & 31); e < end; e += 32) s = fma(__ldg(val + e), v[__ldg(ci + e)], s);
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}
// M v for the tile's rows: this thread's row r0 + threadIdx.x (tile: scratch)
__device__ __forceinline__ double ac_product(const ac_args &a, const int *rp, const int *ci, const double *val,
                                             const double *v, long r0, double *tile)
{
    const long r = r0 + threadIdx.x;
    if (!a.warp_rows) return r < a.n ? ac_row(rp, ci, val, v, r) : 0.0;
    __syncthreads();
    for (int i = threadIdx.x >> 5; i < AC_ROWS; i += AC_WARPS) {
        const double s = r0 + i < a.n ? ac_row_warp(rp, ci, val, v, r0 + i) : 0.0;
        if ((threadIdx.x & 31) == 0) tile[i] = s;
    }
    __syncthreads();
    return tile[threadIdx.x];
}

// the tile's part of X^T v, v = this thread's value of row r0 + threadIdx.x: lane
// (sub, c) adds rows sub, sub + 32 / W, ... of the warp's 32 for columns c and c + 32
__device__ __forceinline__ void ac_xtv(const ac_args &a, double v, long r0, double *tile, int W, double acc[2])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = lane & (W - 1), sub = lane / W;
    __syncwarp();
    tile[threadIdx.x] = v;
    __syncwarp();
    const long rw = r0 + warp * 32;
    const double *vt = tile + warp * 32;
    const int step = 32 / W;
#pragma unroll 4
    for (int i = sub; i < 32; i += step) {
        const bool in = rw + i < a.n;
        const double *xr = a.X + (rw + i) * a.ldx;
        const double x0 = in && c < a.m ? xr[c] : 0.0;
        acc[0] = fma(x0, vt[i], acc[0]);
        if (a.m > 32) {
            const double x1 = in && c + 32 < a.m ? xr[c + 32] : 0.0;
            acc[1] = fma(x1, vt[i], acc[1]);
        }
    }
}

// the block's partials of X^T v from the lanes' sums
__device__ __forceinline__ void ac_xtv_part(const ac_args &a, double acc[2], int W, double (*red)[64])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 2; ++q)
        for (int o = W; o < 32; o <<= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
    red[warp][lane] = acc[0];
    red[warp][lane + 32] = acc[1];
    __syncthreads();
    for (int j = threadIdx.x; j < a.m; j += AC_ROWS) {
        double t = 0;
#pragma unroll
        for (int w = 0; w < AC_WARPS; ++w) t += red[w][j];
        a.part[(size_t)j * gridDim.x + blockIdx.x] = t;
    }
    __syncthreads();
}

__device__ __forceinline__ void ac_dot_part(const ac_args &a, double s, double (*red)[64])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) red[warp][0] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int w = 0; w < AC_WARPS; ++w) t += red[w][0];
        a.part[blockIdx.x] = t;
    }
    __syncthreads();
}

// v - sum_j M[r, j] c_j
__device__ __forceinline__ double ac_minus(const ac_args &a, const double *M, long ldm, long r, double v, const double *cs)
{
    const double *mr = M + r * ldm;
    double s = 0;
#pragma unroll 4
    for (int j = 0; j < a.m; ++j) s = fma(mr[j], cs[j], s);
    return v - s;
}

// CG on P^T (A - lambda B) P y = b, P = I - X X^T B, from y = 0 with r = p = b
__global__ void __launch_bounds__(AC_ROWS, 4)
k_adjoint_cg(const ac_args a)
{
    GB_PDL();
    __shared__ double red[AC_WARPS][64], tile[AC_ROWS], cs[64];
    const int n = a.n, m = a.m;
    const long stride = (long)gridDim.x * AC_ROWS, first = (long)blockIdx.x * AC_ROWS;
    if (*(volatile int *)a.dev_err) return;              // an earlier wait ran out: do nothing
    unsigned gen = threadIdx.x == 0 ? (unsigned)(coop_ld64(a.bar + 2) >> 32) : 0;
    int W = 1;
    while (W < m && W < 32) W <<= 1;
    double beta = 0;
    for (bool start = true;; start = false) {
        // p = r + beta p; c = X^T B p
        double acc[2] = {0, 0};
        for (long r0 = first; r0 < n; r0 += stride) {
            const long r = r0 + threadIdx.x;
            double p = 0;
            if (r < n) {
                p = a.p[r];
                if (!start) a.p[r] = p = fma(beta, p, a.r[r]);
            }
            if (!a.bv) ac_xtv(a, p, r0, tile, W, acc);
        }
        if (a.bv) {
            if (ac_barrier(a, AC_PLAIN, 0, gen) < 0) return;
            for (long r0 = first; r0 < n; r0 += stride)
                ac_xtv(a, ac_product(a, a.brp, a.bci, a.bv, a.p, r0, tile), r0, tile, W, acc);
        }
        ac_xtv_part(a, acc, W, red);
        if (ac_barrier(a, AC_COEF, m, gen) < 0) return;
        // t = P p
        for (int j = threadIdx.x; j < m; j += AC_ROWS) cs[j] = __ldcg(a.c + j);
        __syncthreads();
        for (long r0 = first; r0 < n; r0 += stride) {
            const long r = r0 + threadIdx.x;
            if (r < n) a.t[r] = ac_minus(a, a.X, a.ldx, r, a.p[r], cs);
        }
        if (ac_barrier(a, AC_PLAIN, 0, gen) < 0) return;
        // u = (A - lambda B) t; c = X^T u
        acc[0] = acc[1] = 0;
        for (long r0 = first; r0 < n; r0 += stride) {
            const long r = r0 + threadIdx.x;
            double u = ac_product(a, a.arp, a.aci, a.av, a.t, r0, tile);
            const double bt = a.bv ? ac_product(a, a.brp, a.bci, a.bv, a.t, r0, tile) : r < n ? a.t[r] : 0.0;
            u = fma(-a.lambda, bt, u);
            if (r < n) a.u[r] = u;
            else u = 0;
            ac_xtv(a, u, r0, tile, W, acc);
        }
        ac_xtv_part(a, acc, W, red);
        if (ac_barrier(a, AC_COEF, m, gen) < 0) return;
        // q = P^T u; p.q
        for (int j = threadIdx.x; j < m; j += AC_ROWS) cs[j] = __ldcg(a.c + j);
        __syncthreads();
        double s = 0;
        for (long r0 = first; r0 < n; r0 += stride) {
            const long r = r0 + threadIdx.x;
            if (r < n) {
                const double q = ac_minus(a, a.BX, a.ldbx, r, a.u[r], cs);
                a.q[r] = q;
                s = fma(a.p[r], q, s);
            }
        }
        ac_dot_part(a, s, red);
        if (ac_barrier(a, AC_PQ, 1, gen) <= 0) return;
        // y += alpha p, r -= alpha q; r.r
        const double alpha = __ldcg(&a.s->alpha);
        s = 0;
        for (long r0 = first; r0 < n; r0 += stride) {
            const long r = r0 + threadIdx.x;
            if (r < n) {
                a.y[r] = fma(alpha, a.p[r], a.y[r]);
                const double rn = fma(-alpha, a.q[r], a.r[r]);
                a.r[r] = rn;
                s = fma(rn, rn, s);
            }
        }
        ac_dot_part(a, s, red);
        if (ac_barrier(a, AC_RR, 1, gen) <= 0) return;
        beta = __ldcg(&a.s->beta);
    }
}

// the iteration from the right-hand side in W->r and W->p, y = 0, r.r = rr
static int ad_iterate(gcge_gpu_ctx *ctx, const gcge_gpu_mat *A, const gcge_gpu_mat *B, int n, int m, const double *X,
                      long ldx, const double *BX, long ldbx, double lambda, double rr, double tol, int max_it,
                      int *iters, ad_work *W)
{
    ac_state s = {rr, 0.0, 0.0, sqrt(rr), 0, GCGE_GPU_OK};
    AD_CUDA(ctx, cudaMemcpyAsync(W->dot, &s, sizeof(s), cudaMemcpyHostToDevice, ctx->stream));
    ac_args a = {};
    a.n = n;
    a.m = m;
    a.max_it = max_it;
    // a thread per row leaves a warp waiting for its longest one
    a.warp_rows = A->max_row_nnz > 64.0 || (B && B->max_row_nnz > 64.0);
    a.lambda = lambda;
    a.tol = tol;
    a.arp = A->rp;
    a.aci = A->ci;
    a.av = A->v;
    if (B) {
        a.brp = B->rp;
        a.bci = B->ci;
        a.bv = B->v;
    }
    a.X = X;
    a.ldx = ldx;
    a.BX = BX;
    a.ldbx = ldbx;
    a.y = W->y;
    a.r = W->r;
    a.p = W->p;
    a.q = W->q;
    a.t = W->t;
    a.u = W->u;
    a.c = W->c;
    a.part = W->part;
    a.s = (ac_state *)W->dot;
    a.bar = ctx->dev_bar;
    a.dev_err = ctx->dev_err;
    a.wait_ns = gb_coop_wait_ns(ctx);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_adjoint_cg, AC_ROWS, 0) != cudaSuccess || per_sm < 1)
        return gb_fail(ctx, GCGE_GPU_ERR_CUDA);
    if (per_sm > AV_BLOCKS_PER_SM) per_sm = AV_BLOCKS_PER_SM;   // the partials' room
    long G = (long)ctx->num_sms * per_sm, tiles = ((long)n + AC_ROWS - 1) / AC_ROWS;
    if (G > tiles) G = tiles;
    void *args[] = {&a};
    if (cudaLaunchCooperativeKernel(k_adjoint_cg, dim3((unsigned)G), dim3(AC_ROWS), args, 0, ctx->stream) != cudaSuccess) {
        cudaGetLastError();
        return gb_fail(ctx, GCGE_GPU_ERR_CUDA);
    }
    ctx->launches++;
    AD_CUDA(ctx, cudaMemcpyAsync(&s, W->dot, sizeof(s), cudaMemcpyDeviceToHost, ctx->stream));
    AD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    *iters = s.it;
    if (s.status) return gb_fail(ctx, s.status);
    return gb_check_device_error(ctx);
}

static int ad_solve(gcge_gpu_ctx *ctx, const gcge_gpu_mat *A, const gcge_gpu_mat *B, int n, int m, const double *X,
                    long ldx, const double *eval, int k, const double *g, long ldg, double *mu, long ldmu,
                    double cluster_tol, double tol, int max_it, int *iters, ad_work *W)
{
    int st;
    const double lambda = eval[k];
    const double *BX = X;
    long ldbx = ldx;
    if (B) {
        if ((st = gb_spmm(ctx, B, X, ldx, W->BX, m, m, 1.0, nullptr, 0.0, nullptr))) return st;
        BX = W->BX;
        ldbx = m;
    }
    // c = X^T g; explicit components a_j = c_j / (lambda_j - lambda) outside k's cluster
    if ((st = gb_axpby(ctx, n, 1, 1.0, g, ldg, 0.0, W->r, 1))) return st;   // r = g (contiguous)
    if ((st = ad_xtv(ctx, n, m, X, ldx, W->r, W->c, W))) return st;
    AD_CUDA(ctx, cudaMemcpyAsync(W->h_c, W->c, sizeof(double) * m, cudaMemcpyDeviceToHost, ctx->stream));
    AD_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    const double cscale = fmax(fabs(lambda), DBL_MIN);
    double *h_a = (double *)malloc(sizeof(double) * m);
    if (!h_a) return gb_fail(ctx, GCGE_GPU_ERR_NOMEM);
    for (int j = 0; j < m; ++j) {
        const double gap = eval[j] - lambda;
        h_a[j] = fabs(gap) <= cluster_tol * cscale ? 0.0 : -W->h_c[j] / gap;   // negated: v - X c form
    }
    double rr = 0, bnorm = 0;
    int it = 0;
    // b = P^T g = g - B X c (into r), the right-hand side of the projected system;
    // CG on P^T (A - lambda B) P y = b from y = 0
    st = ad_v_minus_xc(ctx, n, m, BX, ldbx, W->c, W->r, W->r);
    if (!st) st = gb_set_zero(ctx, W->y, (size_t)n);
    if (!st) st = ad_axpby(ctx, n, 1.0, W->r, 0.0, W->p);
    if (!st) st = ad_dot(ctx, n, W->r, W->r, W, &rr);
    bnorm = sqrt(rr);
    if (!st && m <= AD_SKINNY_M && bnorm > 0 && bnorm > tol * bnorm && max_it > 0)
        st = ad_iterate(ctx, A, B, n, m, X, ldx, BX, ldbx, lambda, rr, tol, max_it, &it, W);
    // more vectors than the single launch takes
    while (!st && m > AD_SKINNY_M && bnorm > 0 && sqrt(rr) > tol * bnorm && it < max_it) {
        double pq;
        if ((st = ad_apply(ctx, A, B, n, m, X, ldx, lambda, W->p, W->q, W))) break;
        if ((st = ad_dot(ctx, n, W->p, W->q, W, &pq))) break;
        if (!(pq > 0)) break;                               // left the SPD complement: stop
        const double alpha = rr / pq;
        if ((st = ad_axpby(ctx, n, alpha, W->p, 1.0, W->y))) break;
        if ((st = ad_axpby(ctx, n, -alpha, W->q, 1.0, W->r))) break;
        double rr2;
        if ((st = ad_dot(ctx, n, W->r, W->r, W, &rr2))) break;
        const double beta = rr2 / rr;
        rr = rr2;
        if ((st = ad_axpby(ctx, n, 1.0, W->r, beta, W->p))) break;
        ++it;
    }
    if (iters) *iters = it;
    // mu = P y + X a
    if (!st) {
        if (B) {
            if (!(st = gb_spmm(ctx, B, W->y, 1, W->w, 1, 1, 1.0, nullptr, 0.0, nullptr)))
                st = ad_project(ctx, n, m, X, ldx, X, ldx, W->y, W->w, W->t, W);
        } else {
            st = ad_project(ctx, n, m, X, ldx, X, ldx, W->y, W->y, W->t, W);
        }
    }
    if (!st && cudaMemcpyAsync(W->c, h_a, sizeof(double) * m, cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess)
        st = gb_fail(ctx, GCGE_GPU_ERR_CUDA);
    if (!st) st = ad_v_minus_xc(ctx, n, m, X, ldx, W->c, W->t, W->t);
    if (!st) st = gb_axpby(ctx, n, 1, 1.0, W->t, 1, 0.0, mu, ldmu);
    cudaStreamSynchronize(ctx->stream);
    free(h_a);
    return st;
}

extern "C" int GCGE_GPU_EigvecAdjoint(const gcge_gpu_mat *A, const gcge_gpu_mat *B, const gcge_gpu_mv *X, int m,
                                      const double *eval, int k, const gcge_gpu_mv *G, int g_col, gcge_gpu_mv *MU,
                                      int mu_col, double cluster_tol, double tol, int max_it, int *iters)
{
    if (!A || !X || !eval || !G || !MU) return GCGE_GPU_ERR_ARG;
    gcge_gpu_ctx *ctx = A->ctx;
    const int n = A->n;
    if (m < 1 || k < 0 || k >= m || !mv_cols_ok(X, 0, m) || !mv_cols_ok(G, g_col, 1) || !mv_cols_ok(MU, mu_col, 1) ||
        X->n != n || G->n != n || MU->n != n || (B && B->n != n) || !(cluster_tol >= 0) || !(tol > 0) ||
        max_it < 0)
        return gb_fail(ctx, GCGE_GPU_ERR_ARG);
    for (int j = 0; j < m; ++j)
        if (!isfinite(eval[j])) return gb_fail(ctx, GCGE_GPU_ERR_ARG);
    ad_work W;
    memset(&W, 0, sizeof(W));
    int st = GCGE_GPU_OK;
    double *base = nullptr;
    // sub-buffers start on 256-byte boundaries
    const size_t vn = ((size_t)n + 31) & ~(size_t)31, vm = ((size_t)m + 31) & ~(size_t)31;
    const size_t np = (((size_t)ctx->num_sms * AV_BLOCKS_PER_SM * (size_t)(m > 1 ? m : 1)) + 31) & ~(size_t)31;
    const size_t nv = 7 * vn + vm + 32 + np + (B ? (((size_t)n * m + 31) & ~(size_t)31) : 0);
    if (gb_call_alloc(ctx, (void **)&base, sizeof(double) * nv)) return gb_fail(ctx, GCGE_GPU_ERR_NOMEM);
    W.y = base;
    W.r = W.y + vn;
    W.p = W.r + vn;
    W.q = W.p + vn;
    W.t = W.q + vn;
    W.u = W.t + vn;
    W.w = W.u + vn;
    W.c = W.w + vn;
    W.dot = W.c + vm;
    W.part = W.dot + 32;
    W.BX = B ? W.part + np : nullptr;
    W.h_c = (double *)malloc(sizeof(double) * m);
    if (!W.h_c) {
        gb_call_free(ctx, base);
        return gb_fail(ctx, GCGE_GPU_ERR_NOMEM);
    }
    // the projections are n x m by one column: FP64-pipe Gram and combination
    // kernels (no tensor-core set-up per call)
    const int tc = ctx->tc;
    ctx->tc = 0;
    st = ad_solve(ctx, A, B, n, m, X->d, X->ld, eval, k, G->d + g_col, G->ld, MU->d + mu_col, MU->ld, cluster_tol,
                  tol, max_it, iters, &W);
    ctx->tc = tc;
    cudaStreamSynchronize(ctx->stream);
    gb_call_free(ctx, base);
    free(W.h_c);
    return st;
}
