// gb_dense.cu -- small dense FP64 linear algebra kept resident on the GPU.
//
// The projected (Rayleigh-Ritz) matrices and the orthogonalisation Gram blocks
// are at most a few hundred wide, so these kernels are latency bound; on GB300
// the FP64 pipe also runs ~1/58 of FP32, so they are written to keep the
// dependent-operation chains short and to run independent work (eigenvalues,
// eigenvectors, columns) on separate warps or blocks.
//
//  * gb_small_gemm: column-major C = alpha op(A) op(B) + beta C.
//  * gb_chol_deflate: Cholesky of a Gram matrix with deflation of (numerically)
//    dependent columns, and the inverse of the kept triangular factor -- the
//    building block of the Cholesky-QR orthonormalisation.
//  * gb_syevx: partial symmetric eigensolver with the structure of LAPACK's
//    dsyevx for a range of indices (the routine the reference calls in
//    GCGE_Default_DenseMatEigenSolver, src/gcge_ops.c:302-316): Householder
//    tridiagonalisation, bisection on Sturm counts (32-way multisection, four
//    rounds a pass), inverse iteration with reorthogonalisation inside clusters of close
//    eigenvalues, and back-transformation by the stored reflectors.
#include <cfloat>
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "gb_internal.h"
#include "gb_launch.h"

#define FULL 0xffffffffu

#define GB_PROF(ctx, cls, bytes, flops) \
    do { if ((ctx)->prof) gb_prof_begin((ctx), (cls), (bytes), (flops)); } while (0)

// ---------------------------------------------------------------- small GEMM
// C = alpha op(A) op(B) + beta C for the projected matrices (m, n, k of a few hundred
// at most). FP64 on GB300 is narrow (~2 FMA per clock per SM) and a dependent FP64
// chain costs ~40 ns per step, so the work is spread thin: an 8 x 8 tile of C per
// block, 256 threads = 64 outputs x 4 slices of the inner dimension, each slice
// accumulated in two interleaved chains (k / 8 dependent steps), the slices summed
// in a fixed order in shared memory.
#define SG_T 8
__global__ void __launch_bounds__(256)
k_small_gemm(char ta, char tb, int m, int n, int k, double alpha, const double *__restrict__ A, int lda,
             const double *__restrict__ B, int ldb, double beta, double *__restrict__ C, int ldc)
{
    GB_PDL();
    __shared__ double part[4][SG_T * SG_T];
    const int t = threadIdx.x, o = t & 63, sl = t >> 6;
    const int i = blockIdx.x * SG_T + (o & 7), j = blockIdx.y * SG_T + (o >> 3);
    double a0 = 0, a1 = 0;
    if (i < m && j < n) {
        const bool an = ta == 'N', bn = tb == 'N';
        int l = sl;
        for (; l + 4 < k; l += 8) {
            const double x0 = an ? A[i + (long)l * lda] : A[l + (long)i * lda];
            const double y0 = bn ? B[l + (long)j * ldb] : B[j + (long)l * ldb];
            const double x1 = an ? A[i + (long)(l + 4) * lda] : A[(l + 4) + (long)i * lda];
            const double y1 = bn ? B[(l + 4) + (long)j * ldb] : B[j + (long)(l + 4) * ldb];
            a0 = fma(x0, y0, a0);
            a1 = fma(x1, y1, a1);
        }
        if (l < k) {
            const double x0 = an ? A[i + (long)l * lda] : A[l + (long)i * lda];
            const double y0 = bn ? B[l + (long)j * ldb] : B[j + (long)l * ldb];
            a0 = fma(x0, y0, a0);
        }
    }
    part[sl][o] = a0 + a1;
    __syncthreads();
    if (sl == 0 && i < m && j < n) {
        const double acc = (part[0][o] + part[1][o]) + (part[2][o] + part[3][o]);
        double *c = C + i + (long)j * ldc;
        *c = beta == 0.0 ? alpha * acc : alpha * acc + beta * *c;
    }
}

extern "C" int gb_small_gemm(gcge_gpu_ctx *ctx, char ta, char tb, int m, int n, int k, double alpha,
                             const double *A, int lda, const double *B, int ldb, double beta, double *C, int ldc)
{
    if (m <= 0 || n <= 0) return GCGE_GPU_OK;
    dim3 grid((m + SG_T - 1) / SG_T, (n + SG_T - 1) / SG_T);
    GB_PROF(ctx, GB_K_DENSE, 8.0 * ((double)m * k + (double)k * n + (double)m * n), 2.0 * m * n * (double)k);
    GB_LAUNCH(ctx, k_small_gemm, grid, 256, 0, ta, tb, m, n, k > 0 ? k : 0, alpha, A, lda, B, ldb, beta, C, ldc);
    return GCGE_GPU_OK;
}

// ---------------------------------------------------------------- misc helpers
__global__ void k_set_zero(double *a, size_t count)
{
    GB_PDL();
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < count; t += (size_t)gridDim.x * blockDim.x)
        a[t] = 0.0;
}
extern "C" int gb_set_zero(gcge_gpu_ctx *ctx, double *a, size_t count)
{
    if (!count) return GCGE_GPU_OK;
    size_t g = (count + 255) / 256;
    if (g > 4096) g = 4096;
    GB_LAUNCH(ctx, k_set_zero, (int)g, 256, 0, a, count);
    return GCGE_GPU_OK;
}
extern "C" int gb_copy_d(gcge_gpu_ctx *ctx, double *dst, const double *src, size_t count)
{
    if (!count) return GCGE_GPU_OK;
    if (cudaMemcpyAsync(dst, src, count * sizeof(double), cudaMemcpyDeviceToDevice, ctx->stream) != cudaSuccess)
        return gb_fail(ctx, GCGE_GPU_ERR_CUDA);
    return GCGE_GPU_OK;
}
__global__ void k_set_diag(double *H, int ldh, int count, const double *vals)
{
    GB_PDL();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
        H[i + (long)i * ldh] = vals[i];
}
extern "C" int gb_set_diag_from(gcge_gpu_ctx *ctx, double *H, int ldh, int count, const double *vals)
{
    if (count <= 0) return GCGE_GPU_OK;
    GB_LAUNCH(ctx, k_set_diag, (count + 255) / 256, 256, 0, H, ldh, count, vals);
    return GCGE_GPU_OK;
}
// A-orthogonal mode: the projected eigenvalues nu of -V^T B V (ascending) are
// kept in nu and turned into lambda = -1/nu (ascending as well)
__global__ void k_neg_recip(int count, double *v, double *nu)
{
    GB_PDL();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const double x = v[i];
        nu[i] = x;
        v[i] = -1.0 / x;
    }
}
extern "C" int gb_neg_recip(gcge_gpu_ctx *ctx, int count, double *v, double *nu)
{
    if (count <= 0) return GCGE_GPU_OK;
    GB_LAUNCH(ctx, k_neg_recip, (count + 255) / 256, 256, 0, count, v, nu);
    return GCGE_GPU_OK;
}
// soft locking: H[0:s, w0:m] = H[w0:m, 0:s] = 0 (the W block decoupled from the s
// locked Ritz vectors); C[:, 0:s] = e_0 .. e_(s-1); C[0:s, s:iu] = 0
__global__ void k_soft_lock(double *H, int ldh, int m, int w0, int s, double *C, int ldc, int iu)
{
    GB_PDL();
    const long nh = (long)(m - w0) * s, nc = (long)m * s, nz = (long)(iu - s) * s;
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < nh + nc + nz; t += (long)gridDim.x * blockDim.x) {
        if (t < nh) {
            const int i = (int)(t % s), j = w0 + (int)(t / s);
            H[i + (long)j * ldh] = 0.0;
            H[j + (long)i * ldh] = 0.0;
        } else if (t < nh + nc) {
            const long u = t - nh;
            const int i = (int)(u % m), j = (int)(u / m);
            C[i + (long)j * ldc] = i == j ? 1.0 : 0.0;
        } else {
            const long u = t - nh - nc;
            const int i = (int)(u % s), j = s + (int)(u / s);
            C[i + (long)j * ldc] = 0.0;
        }
    }
}
extern "C" int gb_soft_lock(gcge_gpu_ctx *ctx, double *H, int ldh, int m, int w0, int s, double *C, int ldc, int iu)
{
    if (s <= 0) return GCGE_GPU_OK;
    GB_LAUNCH(ctx, k_soft_lock, ctx->num_sms, 256, 0, H, ldh, m, w0, s, C, ldc, iu);
    return GCGE_GPU_OK;
}
__global__ void k_sym_upper(double *H, int ldh, int m)
{
    GB_PDL();
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < (long)m * m; t += (long)gridDim.x * blockDim.x) {
        const int i = (int)(t % m), j = (int)(t / m);
        if (i > j) H[i + (long)j * ldh] = H[j + (long)i * ldh];
    }
}
extern "C" int gb_symmetrize_from_upper(gcge_gpu_ctx *ctx, double *H, int ldh, int m)
{
    if (m <= 1) return GCGE_GPU_OK;
    long t = (long)m * m;
    GB_LAUNCH(ctx, k_sym_upper, (int)((t + 255) / 256 > 2048 ? 2048 : (t + 255) / 256), 256, 0, H, ldh, m);
    return GCGE_GPU_OK;
}
__global__ void k_copy_block(int rows, int cols, const double *src, int lds, double *dst, int ldd)
{
    GB_PDL();
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < (long)rows * cols; t += (long)gridDim.x * blockDim.x) {
        const int i = (int)(t % rows), j = (int)(t / rows);
        dst[i + (long)j * ldd] = src[i + (long)j * lds];
    }
}
extern "C" int gb_copy_block(gcge_gpu_ctx *ctx, int rows, int cols, const double *src, int lds, double *dst,
                             int ldd)
{
    if (rows <= 0 || cols <= 0) return GCGE_GPU_OK;
    long t = (long)rows * cols;
    GB_LAUNCH(ctx, k_copy_block, (int)((t + 255) / 256 > 2048 ? 2048 : (t + 255) / 256), 256, 0, rows, cols, src,
              lds, dst, ldd);
    return GCGE_GPU_OK;
}
// ComputeP coefficient assembly (src/gcge_xpw.c:325-330): zero the p_ncols columns
// starting at p_start, then copy rows xx_nrows.. of column unlock[cp] into column
// p_start+cp.
__global__ void k_p_coef(double *coef, int ldc, int p_start, int p_ncols, int xx_nrows, const int *unlock)
{
    GB_PDL();
    const long total = (long)p_ncols * ldc;
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
        const int r = (int)(t % ldc), cp = (int)(t / ldc);
        double v = 0.0;
        if (r >= xx_nrows) v = coef[r + (long)unlock[cp] * ldc];
        coef[r + (long)(p_start + cp) * ldc] = v;
    }
}
extern "C" int gb_p_coef_assemble(gcge_gpu_ctx *ctx, double *coef, int ldc, int p_start, int p_ncols,
                                  int xx_nrows, const int *unlock_dev)
{
    if (p_ncols <= 0) return GCGE_GPU_OK;
    long t = (long)p_ncols * ldc;
    GB_LAUNCH(ctx, k_p_coef, (int)((t + 255) / 256), 256, 0, coef, ldc, p_start, p_ncols, xx_nrows, unlock_dev);
    return GCGE_GPU_OK;
}

// ---------------------------------------------------------------- Cholesky with deflation
// One block. S = G (upper used); for each column j in order: its remaining
// squared norm d = S[j,j] after removing the kept earlier columns; the column is
// dropped when d <= rel_tol * G[j,j] or sqrt(d) <= zero_tol (or not finite).
// Kept: R[j, j:] = S[j, j:] / sqrt(d), trailing update. Then U = R restricted to
// the kept rows/columns is inverted; T[K_q, p] = inv(U)[q, p] (zeros elsewhere).
//
// A step's pivot is a chain of a square root and a reciprocal (0.7 us of the FP64
// pipe's latency), so warp 0 updates the next row first and forms the next pivot while
// the other warps update the rest: one barrier a step. S and R share one array
// (a row is scaled in place), and T's columns go into the triangle below it, all in
// shared memory up to CD_SMEM_K columns (odd leading dimension: rows and columns
// free of bank conflicts); wider blocks use the caller's work array. (One thread's
// pivot, a reciprocal in all 512 threads, integer divisions for the indices and
// global arrays took 474 us on average of 64 and 114 columns; this form 170 and 437, 259 on that average.)
#define CD_THREADS 256
#define CD_SMEM_K 160

// n / b rounded as IEEE division, y = 1 / b correctly rounded: two corrections of n y by
// the exact remainder (Markstein, IBM J. Res. Dev. 34, 1990; with a quotient within
// one ulp and a correctly rounded reciprocal the second is exact), a chain of five
// operations. Operands of which the quotient could leave the range of normal numbers (|n| past 2^+-600, |b|
// past 2^+-300) take the division itself.
__device__ __forceinline__ double div_by(double n, double b, double y)
{
    const int en = __double2hiint(n) & 0x7ff00000, eb = __double2hiint(b) & 0x7ff00000;
    if (en < (423 << 20) || en > (1622 << 20) || eb < (723 << 20) || eb > (1322 << 20)) return n / b;
    double q = __dmul_rn(n, y);
    q = fma(fma(-b, q, n), y, q);
    return fma(fma(-b, q, n), y, q);
}

__global__ void __launch_bounds__(CD_THREADS)
k_chol_deflate(int k, const double *__restrict__ G, int ldg, double *__restrict__ T, int *kept_out,
               double zero_tol, double rel_tol, double *work, double *__restrict__ min_ratio)
{
    GB_PDL();
    extern __shared__ double cd_sm[];
    const int ld = k | 1;
    double *piv = cd_sm, *diag = piv + k, *rinv = diag + k;      // pivots d, G's diagonal, 1 / R[j, j]
    int *keep = (int *)(rinv + k), *pos = keep + k;
    double *A = work ? work : rinv + 2 * k;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = CD_THREADS / 32;
    for (int j = warp; j < k; j += nw)
        for (int i = lane; i <= j; i += 32) A[i + (long)j * ld] = G[i + (long)j * ldg];
    for (int j = tid; j < k; j += CD_THREADS) diag[j] = G[j + (long)j * ldg];
    __syncthreads();
    // pivot of row j (all lanes of a warp) and the row scaled into R
    auto pivot = [&](int j) {
        const double d = A[j + (long)j * ld], g = diag[j], r = sqrt(d);
        const bool ok = isfinite(d) && isfinite(g) && g > 0.0 && d > rel_tol * g && r > zero_tol;
        const double ri = 1.0 / r;
        __syncwarp();
        if (ok) {
            for (int m = j + 1 + lane; m < k; m += 32) A[j + (long)m * ld] *= ri;
            if (lane == 0) A[j + (long)j * ld] = r;
        }
        if (lane == 0) {
            piv[j] = d;
            rinv[j] = ri;
            keep[j] = ok;
        }
    };
    if (warp == 0) pivot(0);
    for (int j = 0; j + 1 < k; ++j) {
        __syncthreads();
        const bool kj = keep[j];
        if (warp == 0) {
            if (kj) {
                const double f = A[j + (long)(j + 1) * ld];
                for (int m = j + 1 + lane; m < k; m += 32) {
                    double *a = A + j + 1 + (long)m * ld;
                    *a = fma(-f, A[j + (long)m * ld], *a);
                }
                __syncwarp();
            }
            pivot(j + 1);
        } else if (kj) {
            for (int b = j + 1 + warp; b < k; b += nw - 1) {
                const double rb = A[j + (long)b * ld];
                for (int a = j + 2 + lane; a <= b; a += 32) {
                    double *t = A + a + (long)b * ld;
                    *t = fma(-A[j + (long)a * ld], rb, *t);
                }
            }
        }
    }
    __syncthreads();
    if (tid == 0) {
        int c = 0;
        for (int j = 0; j < k; ++j) { pos[j] = keep[j] ? c : -1; c += keep[j]; }
        *kept_out = c;
    }
    if (min_ratio && tid == 32) {
        double mr = 1.0;
        for (int j = 0; j < k; ++j)
            if (diag[j] > 0.0) mr = fmin(mr, piv[j] / diag[j]);
        *min_ratio = mr;
    }
    // column p of inv(U) for each kept column j (p = pos[j]):
    // x[p] = 1/U[p,p]; x[q] = -(sum_{l=q+1..p} U[q,l] x[l]) / U[q,q], walking kept
    // rows. x[l] of column jc is A[jc, l], zero for a dropped l. The sum is two chains (odd
    // and even l - q), one in each of two lanes, as the pipe takes as long for one
    // chain's instruction as for both; 16 columns a warp, a long and a short run of them
    // on every quarter of the SM.
    const int h = lane & 1, run = warp < 4 ? 7 - warp : warp - 4;
    const unsigned pair = 3u << (lane & 30);
    for (int j0 = (k - 1) / (16 * nw) * (16 * nw); j0 >= 0; j0 -= 16 * nw) {
        const int jc = j0 + 16 * run + (lane >> 1);
        if (jc >= k || !keep[jc]) continue;
        double *x = A + jc;
        for (int q = jc - 1; q >= 0; --q) {
            double s = 0, z = 0.0;
            if (keep[q]) {
                const double *u = A + q;
                int l = q + 1 + h;
                for (; l < jc; l += 2) s = fma(u[(long)l * ld], x[(long)l * ld], s);
                if (l == jc) s = fma(u[(long)jc * ld], rinv[jc], s);
                s += __shfl_xor_sync(pair, s, 1);
                z = div_by(-s, A[q + (long)q * ld], rinv[q]);
            }
            if (h == 0) x[(long)q * ld] = z;
            __syncwarp(pair);
        }
    }
    __syncthreads();
    const int kept = *(volatile int *)kept_out;
    for (int c = kept + warp; c < k; c += nw)                // columns past the kept ones
        for (int i = lane; i < k; i += 32) T[i + (long)c * k] = 0.0;
    for (int j = warp; j < k; j += nw) {
        if (!keep[j]) continue;
        double *t = T + (long)pos[j] * k;
        for (int i = lane; i < k; i += 32) t[i] = i < j ? A[j + (long)i * ld] : i == j ? rinv[j] : 0.0;
    }
}

static size_t cd_smem(int k, bool array)
{
    return sizeof(double) * (3 * (size_t)k + (array ? (size_t)k + (size_t)k * (k | 1) : 0)) + 2 * sizeof(int) * (size_t)k;
}

// work: at least k (k + 1) doubles
static int cd_launch(gcge_gpu_ctx *ctx, int k, const double *G, int ldg, double *T, int *kept_dev, double zero_tol,
                     double rel_tol, double *work, double *ratio_dev)
{
    // on either side of CD_SMEM_K (a wide block's pivots pass the default of 48 KB from 1,537 columns on):
    // 208 KB, the matrix of 160 columns or the pivots of 6,640
    if (cudaFuncSetAttribute(k_chol_deflate, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)cd_smem(CD_SMEM_K, true)) != cudaSuccess)
        return gb_fail(ctx, GCGE_GPU_ERR_CUDA);
    if (k <= CD_SMEM_K) work = nullptr;
    GB_LAUNCH(ctx, k_chol_deflate, 1, CD_THREADS, cd_smem(k, !work), k, G, ldg, T, kept_dev, zero_tol, rel_tol, work,
              ratio_dev);
    return GCGE_GPU_OK;
}

extern "C" int gb_chol_deflate(gcge_gpu_ctx *ctx, int k, const double *G, int ldg, double *T, int *kept_dev,
                               double zero_tol, double rel_tol, double *work)
{
    return k <= 0 ? GCGE_GPU_OK : cd_launch(ctx, k, G, ldg, T, kept_dev, zero_tol, rel_tol, work, nullptr);
}

// ---------------------------------------------------------------- eigensolver
// work layout (doubles): Aw[m*m] | d[m] | e[m] | tau[m] | Zt[m*m] | Zq[m*m] | G[m*m] | Tq[m*m] |
// cw[2*m*m] | 64 (the pivot ratio and kept count of the Cholesky-QR reorthogonalisation)
extern "C" size_t gb_syevx_work_doubles(int m)
{
    return (size_t)m * m * 7 + 3 * (size_t)m + 128;
}

// Householder reduction of the full symmetric H (lower reflectors, LAPACK dsytd2 "L").
__global__ void __launch_bounds__(1024)
k_tridiag(int m, const double *__restrict__ H, int ldh, double *__restrict__ Aw, double *__restrict__ d,
          double *__restrict__ e, double *__restrict__ tau)
{
    GB_PDL();
    extern __shared__ double sm[];
    double *v = sm;          // m
    double *w = sm + m;      // m
    __shared__ double red[32];
    __shared__ double s_alpha, s_beta, s_tau, s_K;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
    for (long t = tid; t < (long)m * m; t += nt) Aw[t] = H[(t % m) + (t / m) * (long)ldh];
    __syncthreads();
    for (int i = 0; i + 2 < m; ++i) {
        const int len = m - i - 1;
        double *col = Aw + (long)i * m + i + 1;           // x = Aw[i+1:m, i]
        // xn2 = ||x[1:]||^2
        double s = 0;
        for (int r = 1 + tid; r < len; r += nt) s = fma(col[r], col[r], s);
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
        if (lane == 0) red[wid] = s;
        __syncthreads();
        if (tid == 0) {
            double t = 0;
            for (int q = 0; q < nw; ++q) t += red[q];
            const double alpha = col[0];
            if (t == 0.0) {
                s_tau = 0.0;
                s_beta = alpha;
            } else {
                const double beta = -copysign(sqrt(alpha * alpha + t), alpha);
                s_tau = (beta - alpha) / beta;
                s_beta = beta;
                s_alpha = 1.0 / (alpha - beta);
            }
            d[i] = Aw[i + (long)i * m];
            e[i] = s_beta;
            tau[i] = s_tau;
        }
        __syncthreads();
        const double tv = s_tau;
        if (tv == 0.0) {
            for (int r = 1 + tid; r < len; r += nt) col[r] = 0.0;   // stored reflector is zero
            __syncthreads();
            continue;
        }
        const double sc = s_alpha;
        for (int r = tid; r < len; r += nt) {
            const double vr = (r == 0) ? 1.0 : col[r] * sc;
            v[r] = vr;
            if (r > 0) col[r] = vr;                            // keep v (unit lead implied)
        }
        __syncthreads();
        // p = tau * A22 v with A22 = Aw[i+1:, i+1:] held in its lower triangle:
        // warp per row r; A22[r, c] = Aw[r, c] for c <= r and Aw[c, r] for c > r.
        const double *A22 = Aw + (long)(i + 1) * m + (i + 1);
        for (int r = wid; r < len; r += nw) {
            double a0 = 0;
            for (int c = lane; c < len; c += 32) {
                const double a = (c <= r) ? A22[r + (long)c * m] : A22[c + (long)r * m];
                a0 = fma(a, v[c], a0);
            }
            for (int o = 16; o; o >>= 1) a0 += __shfl_xor_sync(FULL, a0, o);
            if (lane == 0) w[r] = tv * a0;
        }
        __syncthreads();
        // K = tau/2 * p.v
        s = 0;
        for (int r = tid; r < len; r += nt) s = fma(w[r], v[r], s);
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
        if (lane == 0) red[wid] = s;
        __syncthreads();
        if (tid == 0) {
            double t = 0;
            for (int q = 0; q < nw; ++q) t += red[q];
            s_K = 0.5 * tv * t;
        }
        __syncthreads();
        const double K = s_K;
        for (int r = tid; r < len; r += nt) w[r] = w[r] - K * v[r];
        __syncthreads();
        // lower triangle of A22 -= v w^T + w v^T: warp per column, lanes down the rows
        double *B22 = Aw + (long)(i + 1) * m + (i + 1);
        for (int c = wid; c < len; c += nw) {
            const double vc = v[c], wc = w[c];
            for (int r = c + lane; r < len; r += 32) B22[r + (long)c * m] -= v[r] * wc + w[r] * vc;
        }
        __syncthreads();
    }
    if (tid == 0) {
        if (m >= 2) {
            d[m - 2] = Aw[(m - 2) + (long)(m - 2) * m];
            e[m - 2] = Aw[(m - 1) + (long)(m - 2) * m];
            tau[m - 2] = 0.0;
        }
        d[m - 1] = Aw[(m - 1) + (long)(m - 1) * m];
        e[m - 1] = 0.0;
        tau[m - 1] = 0.0;
    }
}

// The same reduction with the lower triangle packed in shared memory (column c,
// rows c..m-1, at c m - c (c - 1) / 2), for m <= TD_SMEM_MAX_M: the row-wise half
// of the matrix-vector product then reads shared memory instead of global rows
// at a stride of m doubles, and the rank-2 update stays on chip. Same operations
// in the same order as k_tridiag; the reflectors are written back to Aw (columns
// i, rows i+1..) at the end for the back-transformation.
#define TD_SMEM_MAX_M 230
static size_t td_smem_bytes(int m) { return sizeof(double) * ((size_t)m * (m + 1) / 2 + 2 * (size_t)m); }

__global__ void __launch_bounds__(1024)
k_tridiag_smem(int m, const double *__restrict__ H, int ldh, double *__restrict__ Aw, double *__restrict__ d,
               double *__restrict__ e, double *__restrict__ tau)
{
    GB_PDL();
    extern __shared__ double sm[];
    double *L = sm;                                   // packed lower triangle
    double *v = sm + (size_t)m * (m + 1) / 2;         // m
    double *w = v + m;                                // m
    __shared__ double red[32];
    __shared__ double s_alpha, s_beta, s_tau, s_K;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
    auto off = [m](int c) { return (long)c * m - (long)c * (c - 1) / 2; };
    for (int c = wid; c < m; c += nw)
        for (int r = c + lane; r < m; r += 32) L[off(c) + (r - c)] = H[r + (long)c * ldh];
    __syncthreads();
    for (int i = 0; i + 2 < m; ++i) {
        const int len = m - i - 1;
        double *col = L + off(i) + 1;                 // x = A[i+1:m, i]
        double s = 0;
        for (int r = 1 + tid; r < len; r += nt) s = fma(col[r], col[r], s);
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
        if (lane == 0) red[wid] = s;
        __syncthreads();
        if (tid == 0) {
            double t = 0;
            for (int q = 0; q < nw; ++q) t += red[q];
            const double alpha = col[0];
            if (t == 0.0) {
                s_tau = 0.0;
                s_beta = alpha;
            } else {
                const double beta = -copysign(sqrt(alpha * alpha + t), alpha);
                s_tau = (beta - alpha) / beta;
                s_beta = beta;
                s_alpha = 1.0 / (alpha - beta);
            }
            d[i] = L[off(i)];
            e[i] = s_beta;
            tau[i] = s_tau;
        }
        __syncthreads();
        const double tv = s_tau;
        if (tv == 0.0) {
            for (int r = 1 + tid; r < len; r += nt) col[r] = 0.0;
            __syncthreads();
            continue;
        }
        const double sc = s_alpha;
        for (int r = tid; r < len; r += nt) {
            const double vr = (r == 0) ? 1.0 : col[r] * sc;
            v[r] = vr;
            if (r > 0) col[r] = vr;
        }
        __syncthreads();
        // p = tau * A22 v, A22 = A[i+1:, i+1:]: warp per row r, A22[r, c] from
        // column c (c <= r) or column r (c > r) of the packed triangle
        const int b = i + 1;
        for (int r = wid; r < len; r += nw) {
            double a0 = 0;
            for (int c = lane; c < len; c += 32) {
                const double a = (c <= r) ? L[off(b + c) + (r - c)] : L[off(b + r) + (c - r)];
                a0 = fma(a, v[c], a0);
            }
            for (int o = 16; o; o >>= 1) a0 += __shfl_xor_sync(FULL, a0, o);
            if (lane == 0) w[r] = tv * a0;
        }
        __syncthreads();
        s = 0;
        for (int r = tid; r < len; r += nt) s = fma(w[r], v[r], s);
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
        if (lane == 0) red[wid] = s;
        __syncthreads();
        if (tid == 0) {
            double t = 0;
            for (int q = 0; q < nw; ++q) t += red[q];
            s_K = 0.5 * tv * t;
        }
        __syncthreads();
        const double K = s_K;
        for (int r = tid; r < len; r += nt) w[r] = w[r] - K * v[r];
        __syncthreads();
        for (int c = wid; c < len; c += nw) {
            const double vc = v[c], wc = w[c];
            double *Lc = L + off(b + c);
            for (int r = c + lane; r < len; r += 32) Lc[r - c] -= v[r] * wc + w[r] * vc;
        }
        __syncthreads();
    }
    if (tid == 0) {
        if (m >= 2) {
            d[m - 2] = L[off(m - 2)];
            e[m - 2] = L[off(m - 2) + 1];
            tau[m - 2] = 0.0;
        }
        d[m - 1] = L[off(m - 1)];
        e[m - 1] = 0.0;
        tau[m - 1] = 0.0;
    }
    // reflectors (and the rest of the lower triangle) back to Aw for the back-transformation
    for (int c = wid; c < m; c += nw)
        for (int r = c + lane; r < m; r += 32) Aw[r + (long)c * m] = L[off(c) + (r - c)];
}

// The same reduction for m <= TS_MAX_M, with the matrix in full in shared memory and FP64
// instructions counted: one keeps its quarter of the SM busy for 64 clocks whatever the
// lanes that take part, so few of them, and on all four quarters. (A warp per row of
// p = A22 v -- an FMA per 32 columns, then the five additions of a shuffle tree -- and a
// warp per column of the update, lanes below the diagonal idle, spend most of
// theirs on idle lanes.)
//  * p = A22 v: a lane per row; of the 32 partial sums that are the lanes of that tree
//    a warp takes the eight of one residue mod 4 and the tree's first three levels,
//    and the row's thread the last two: 15 instructions a warp per 32 rows and columns.
//  * The update walks the lower triangle folded into a rectangle, and mirrors it.
//  * Warp 0 updates the next pivot column first and forms its reflector (a square root,
//    and both quotients as two lanes of one division) while the others update the rest.
// The same operations in the same order as k_tridiag with 256 threads. m = 33:
// 134 -> 94 us.
#define TS_MAX_M 127
#define TS_THREADS 512
static size_t ts_smem_bytes(int m) { return sizeof(double) * ((size_t)m * (m | 1) + 7 * (size_t)m); }

__global__ void __launch_bounds__(TS_THREADS)
k_tridiag_small(int m, const double *__restrict__ H, int ldh, double *__restrict__ Aw, double *__restrict__ d,
                double *__restrict__ e, double *__restrict__ tau)
{
    GB_PDL();
    extern __shared__ double sm[];
    const int ld = m | 1;
    double *A = sm, *vb = sm + (size_t)m * ld, *w = vb + 2 * m, *part = w + m;   // v of both parities, w, partials [4][m]
    __shared__ double s_tau[2], red[4];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = TS_THREADS >> 5;
    for (int c = wid; c < m; c += nw)
        for (int r = c + lane; r < m; r += 32) {
            const double h = H[r + (long)c * ldh];
            A[r + c * ld] = h;
            A[c + r * ld] = h;
        }
    __syncthreads();
    auto tree = [&](double s) {
#pragma unroll
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
        return s;
    };
    // reflector of column i (warp 0): v, tau, d, e
    auto reflector = [&](int i) {
        const int len = m - i - 1;
        double *col = A + i * ld + i + 1, *v = vb + (i & 1) * m;  // x = A[i+1:m, i]
        double t = 0;
        for (int r0 = 1; r0 < len; r0 += 32) {
            const double x = r0 + lane < len ? col[r0 + lane] : 0.0;
            t += tree(x * x);
        }
        const double alpha = col[0];
        double tv = 0.0, beta = alpha, sc = 0.0;
        if (t != 0.0) {
            beta = -copysign(sqrt(alpha * alpha + t), alpha);
            const double q = (lane ? 1.0 : beta - alpha) / (lane ? alpha - beta : beta);
            tv = __shfl_sync(FULL, q, 0);
            sc = __shfl_sync(FULL, q, 1);
        }
        if (lane == 0) {
            d[i] = A[i * ld + i];
            e[i] = beta;
            tau[i] = tv;
            s_tau[i & 1] = tv;
        }
        __syncwarp();
        for (int r = lane; r < len; r += 32) {
            const double vr = tv == 0.0 ? 0.0 : col[r] * sc;   // a zero reflector is stored as zeros
            if (r > 0) col[r] = vr;
            v[r] = r == 0 ? 1.0 : vr;
        }
    };
    if (wid == 0 && m > 2) reflector(0);
    for (int i = 0; i + 2 < m; ++i) {
        const int len = m - i - 1, b = i + 1;
        const double *v = vb + (i & 1) * m;
        double *A22 = A + b * ld + b;
        __syncthreads();
        const double tv = s_tau[i & 1];
        if (tv == 0.0) {                                   // uniform: nothing to apply
            if (wid == 0 && i + 3 < m) reflector(i + 1);
            continue;
        }
        // the partial sums of p = A22 v: (32 rows, residue) per warp
        for (int k = wid; k < 4 * ((len + 31) / 32); k += nw) {
            const int q = k & 3, r = 32 * (k >> 2) + lane;
            double P[8];
#pragma unroll
            for (int l = 0; l < 8; ++l) P[l] = 0;
            const double *a = A22 + min(r, len - 1);
            for (int c0 = q; c0 < len; c0 += 32) {
#pragma unroll
                for (int l = 0; l < 8; ++l)
                    if (c0 + 4 * l < len) P[l] = fma(a[(c0 + 4 * l) * ld], v[c0 + 4 * l], P[l]);
            }
#pragma unroll
            for (int o = 4; o; o >>= 1)
#pragma unroll
                for (int l = 0; l < o; ++l)
                    if (q + 4 * (l + o) < len) P[l] += P[l + o];
            if (r < len) part[q * m + r] = P[0];
        }
        __syncthreads();
        // p = tau times the rows' sums, K = tau / 2 p.v, w = p - K v: 32 rows a warp
        if (wid < 4) {
            const int r = 32 * wid + lane, n4 = min(4, (len + 31) / 32);
            double p = 0, x = 0;
            if (r < len) {
                p = tv * ((part[r] + part[2 * m + r]) + (part[m + r] + part[3 * m + r]));
                x = p * v[r];
            }
            if (32 * wid < len) {
                x = tree(x);
                if (lane == 0) red[wid] = x;
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
            double t = 0;
            for (int q = 0; q < n4; ++q) t += red[q];
            const double K = 0.5 * tv * t;
            if (r < len) w[r] = p - K * v[r];
        }
        __syncthreads();
        // A22 -= v w^T + w v^T
        auto update = [&](int r, int c) {
            const double vc = v[c], wc = w[c];
            double t = A22[r + c * ld];
            t -= v[r] * wc + w[r] * vc;
            A22[r + c * ld] = t;
            A22[c + r * ld] = t;
        };
        if (wid == 0) {
            for (int r = lane; r < len; r += 32) update(r, 0);
            __syncwarp();
            if (i + 3 < m) reflector(i + 1);
        } else {
            // columns 1 .. len - 1 (len - c entries each) as rows of width len: column 1 + y
            // and column len - 1 - y share one
            const int n1 = len - 1, rows = (n1 + 1) / 2, width = n1 + 1;
            int y = 0, xx = tid - 32;
            while (xx >= width) {
                xx -= width;
                ++y;
            }
            while (y < rows) {
                const int lc = n1 - y;                     // entries of column 1 + y
                if (xx < lc) update(1 + y + xx, 1 + y);
                else if (n1 - 1 - y != y) update(n1 - y + xx - lc, n1 - y);
                xx += TS_THREADS - 32;
                while (xx >= width) {
                    xx -= width;
                    ++y;
                }
            }
        }
    }
    __syncthreads();
    if (tid == 0) {
        if (m >= 2) {
            d[m - 2] = A[(m - 2) * ld + m - 2];
            e[m - 2] = A[(m - 2) * ld + m - 1];
            tau[m - 2] = 0.0;
        }
        d[m - 1] = A[(m - 1) * ld + m - 1];
        e[m - 1] = 0.0;
        tau[m - 1] = 0.0;
    }
    // reflectors (and the rest of the lower triangle) back to Aw for the back-transformation
    for (int c = wid; c < m; c += nw)
        for (int r = c + lane; r < m; r += 32) Aw[r + (long)c * m] = A[r + c * ld];
}

// 1/x by Newton-Raphson refinement of the hardware reciprocal approximation
// (rcp.approx.ftz.f64): two steps r <- r + r (1 - x r) square the relative error
// each time, leaving a few ulp. For the pivots of inverse iteration, whose
// iterate tolerates a slightly perturbed solve; an exact IEEE division costs
// several hundred cycles on this chain. Tiny or zero x take the exact division.
__device__ __forceinline__ double nr_recip(double x)
{
    if (!(fabs(x) >= DBL_MIN) || isinf(x)) return 1.0 / x;
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    double t = fma(-x, r, 1.0);
    r = fma(r, t, r);
    t = fma(-x, r, 1.0);
    return fma(r, t, r);
}

// ---------------------------------------------------------------- cluster tridiagonalisation
// The same reduction as k_tridiag (dsytd2 "L": reflectors in the columns of Aw,
// d, e, tau) spread over a thread-block cluster of TC CTAs, so that the FP64 work
// of the matrix-vector product and the rank-2 update runs on TC SMs. The lower
// triangle is dealt out by columns, cyclically: column c lives in CTA c mod TC,
// rows c..m-1, packed in that CTA's shared memory. Step i:
//   A  the owner of column i forms the reflector (v, tau, beta) and publishes v;
//   B  after a cluster barrier every CTA copies v (distributed shared memory) and
//      forms its partial of p = A22 v from its own columns (row sums over the
//      columns it holds left of the row, plus the column dots below the diagonal);
//   C  after a second barrier every CTA adds the TC partials in rank order (the
//      same sum everywhere), K = tau/2 p.v, w = tau p - K v, and updates its
//      columns: A22 -= v w^T + w v^T.
// Exchange buffers alternate by step parity; barriers are the hardware cluster
// barrier (no waits on flags). All control flow is uniform over the cluster.
#define TD_THREADS 512

__device__ __forceinline__ double td_block_sum(double s, double *red)
{
    // fixed-order tree over the warps of the block (red: >= 32 doubles)
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
    if (lane == 0) red[w] = s;
    __syncthreads();
    if (w == 0) {
        double t = lane < nw ? red[lane] : 0.0;
#pragma unroll
        for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(FULL, t, o);
        if (lane == 0) red[32] = t;
    }
    __syncthreads();
    const double r = red[32];
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(TD_THREADS)
k_tridiag_cluster(int m, const double *__restrict__ H, int ldh, double *__restrict__ Aw, double *__restrict__ d,
                  double *__restrict__ e, double *__restrict__ tau)
{
    GB_PDL();
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const int TC = (int)cl.num_blocks(), b = (int)cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = TD_THREADS >> 5;
    extern __shared__ double tsm[];
    __shared__ double red[33];
    __shared__ double s_tau, s_scale;
    const int ncol = b < m ? (m - 1 - b) / TC + 1 : 0;       // own columns b, b + TC, ...
    // layout: vbuf[2][m], pbuf[2][m], v[m], p[m], then the packed columns; offsets int[ncol+1] after
    double *vbuf = tsm, *pbuf = vbuf + 2 * (size_t)m, *v = pbuf + 2 * (size_t)m, *p = v + m, *A = p + m;
    long tot = 0;
    for (int l = 0; l < ncol; ++l) tot += m - (b + l * TC);
    int *off = (int *)(A + tot);
    if (tid == 0) {
        int o = 0;
        for (int l = 0; l < ncol; ++l) {
            off[l] = o;
            o += m - (b + l * TC);
        }
        off[ncol] = o;
    }
    __syncthreads();
    for (int l = 0; l < ncol; ++l) {
        const int c = b + l * TC;
        for (int r = c + tid; r < m; r += TD_THREADS) A[off[l] + (r - c)] = H[r + (long)c * ldh];
    }
    __syncthreads();
    for (int i = 0; i + 2 < m; ++i) {
        const int len = m - i - 1, par = i & 1, owner = i % TC;
        double *vb = vbuf + (size_t)par * m, *pb = pbuf + (size_t)par * m;
        // ---- A: the owner forms the reflector of column i
        if (b == owner) {
            const int l = i / TC;
            const double *col = A + off[l];               // rows i..m-1; x = rows i+1..
            double sq = 0;
            for (int r = 2 + tid; r <= len; r += TD_THREADS) sq = fma(col[r], col[r], sq);
            const double xn2 = td_block_sum(sq, red);
            if (tid == 0) {
                const double alpha = col[1];
                d[i] = col[0];
                if (xn2 == 0.0) {
                    s_tau = 0.0;
                    e[i] = alpha;
                    s_scale = 0.0;
                } else {
                    // the two quotients by Newton reciprocals (a few ulp): an IEEE
                    // division is several hundred cycles on this serial path
                    const double beta = -copysign(sqrt(alpha * alpha + xn2), alpha);
                    s_tau = (beta - alpha) * nr_recip(beta);
                    s_scale = nr_recip(alpha - beta);
                    e[i] = beta;
                }
                tau[i] = s_tau;
            }
            __syncthreads();
            const double sc = s_scale;
            for (int r = tid; r < len; r += TD_THREADS) {
                const double vr = r == 0 ? 1.0 : col[1 + r] * sc;
                vb[r] = vr;
                if (r > 0) Aw[(long)i * m + i + 1 + r] = vr;      // stored reflector (unit lead implied)
            }
            if (tid == 0) vb[m - 1] = s_tau;                    // tau rides along in the last slot
        }
        cl.sync();
        // ---- B: copy v and tau, partial p = A22 v over the own columns
        const double *vr_own = cl.map_shared_rank(vbuf + (size_t)par * m, owner);
        for (int r = tid; r < len; r += TD_THREADS) v[r] = vr_own[r];
        if (tid == 0) s_tau = vr_own[m - 1];
        __syncthreads();
        const double tv = s_tau;
        if (tv != 0.0) {
            int l0 = (i + 1 - b + TC - 1) / TC;                  // first own column >= i + 1
            if (i + 1 <= b) l0 = 0;
            // row sums: p_b[r] = sum over own columns c <= row of A[row, c] v[c]
            for (int r = tid; r < len; r += TD_THREADS) {
                const int row = i + 1 + r;
                double a0 = 0, a1 = 0;
                int l = l0;
                for (; l + 1 < ncol && b + (l + 1) * TC <= row; l += 2) {
                    const int c0 = b + l * TC, c1 = c0 + TC;
                    a0 = fma(A[off[l] + (row - c0)], v[c0 - i - 1], a0);
                    a1 = fma(A[off[l + 1] + (row - c1)], v[c1 - i - 1], a1);
                }
                if (l < ncol && b + l * TC <= row) {
                    const int c0 = b + l * TC;
                    a0 = fma(A[off[l] + (row - c0)], v[c0 - i - 1], a0);
                }
                pb[r] = a0 + a1;
            }
            __syncthreads();
            // column dots below the diagonal: p_b[c] += sum_{row > c} A[row, c] v[row]
            for (int l = l0 + wid; l < ncol; l += nw) {
                const int c = b + l * TC;
                const double *col = A + off[l];
                double s = 0;
                for (int rr = 1 + lane; rr < m - c; rr += 32) s = fma(col[rr], v[c + rr - i - 1], s);
#pragma unroll
                for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
                if (lane == 0) pb[c - i - 1] += s;
            }
        }
        cl.sync();
        // ---- C: p = tau * sum of the partials (rank order), K, w, rank-2 update
        if (tv != 0.0) {
            for (int r = tid; r < len; r += TD_THREADS) {
                // all TC remote loads issued before the sum (rank order kept)
                double t[16];
#pragma unroll
                for (int q = 0; q < 16; ++q) t[q] = q < TC ? cl.map_shared_rank(pbuf + (size_t)par * m, q)[r] : 0.0;
                double s = 0;
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    if (q < TC) s += t[q];
                p[r] = tv * s;
            }
            __syncthreads();
            double kv = 0;
            for (int r = tid; r < len; r += TD_THREADS) kv = fma(p[r], v[r], kv);
            const double K = 0.5 * tv * td_block_sum(kv, red);
            for (int r = tid; r < len; r += TD_THREADS) p[r] -= K * v[r];     // p now holds w
            __syncthreads();
            int l0 = (i + 1 - b + TC - 1) / TC;
            if (i + 1 <= b) l0 = 0;
            for (int l = l0; l < ncol; ++l) {
                const int c = b + l * TC, cc = c - i - 1;
                const double vc = v[cc], wc = p[cc];
                double *col = A + off[l];
                for (int rr = tid; rr < m - c; rr += TD_THREADS) {
                    const int rv = cc + rr;
                    col[rr] -= v[rv] * wc + p[rv] * vc;
                }
            }
        } else if (b == owner) {
            // zero reflector: nothing to apply; the stored column below the subdiagonal is zero
            for (int r = 1 + tid; r < len; r += TD_THREADS) Aw[(long)i * m + i + 1 + r] = 0.0;
        }
        __syncthreads();
    }
    // the last two diagonal entries and the last off-diagonal
    if (m >= 2 && b == (m - 2) % TC && tid == 0) {
        const double *col = A + off[(m - 2) / TC];
        d[m - 2] = col[0];
        e[m - 2] = col[1];
        tau[m - 2] = 0.0;
    }
    if (b == (m - 1) % TC && tid == 0) {
        d[m - 1] = A[off[(m - 1) / TC]];
        e[m - 1] = 0.0;
        tau[m - 1] = 0.0;
    }
    cl.sync();                                        // no CTA leaves while others may read its buffers
}

// shared memory of k_tridiag_cluster for m and a cluster of tc CTAs (CTA 0 holds the most)
static size_t td_cluster_smem(int m, int tc)
{
    const int ncol = (m - 1) / tc + 1;
    size_t tot = 0;
    for (int l = 0; l < ncol; ++l) tot += (size_t)(m - l * tc);
    return sizeof(double) * (6 * (size_t)m + tot) + sizeof(int) * (ncol + 1) + 16;
}

// cluster size for m, 0 if the single-SM kernel is to be used
// Each of the m - 2 steps carries dependent FP64 latency (reductions, the sqrt
// and reciprocals of the reflector, two cluster barriers, the gather of the
// partial products) whatever the number of SMs, so the cluster pays only where
// a step's arithmetic on one SM (3 len^2 / 2 FMAs at ~2 FP64 FMA per clock)
// outweighs that. With the partials' remote loads issued together and Newton
// reciprocals, 16 CTAs win from m = 128 on: the dsyevx-signature call at
// m = 178 (58 wanted pairs) takes 4.69 ms against 6.45 ms with the single-SM
// reduction (8 CTAs: 4.93 ms), at m = 130 3.23 against 3.94 ms (at m = 720
// one SM would need ~60 ms of FP64 issue per reduction).
static int td_cluster_size(gcge_gpu_ctx *ctx, int m)
{
    if (m < 128) return 0;
    static int cached_m = -1, cached_tc = 0;
    if (m == cached_m) {
        if (cached_tc &&
            cudaFuncSetAttribute(k_tridiag_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)td_cluster_smem(m, cached_tc)) != cudaSuccess)
            return 0;
        return cached_tc;
    }
    cached_m = m;
    cached_tc = 0;
    static int probed = 0, allow16 = 0;
    if (!probed) {
        probed = 1;
        if (cudaFuncSetAttribute(k_tridiag_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess)
            allow16 = 1;
        cudaGetLastError();
    }
    const int want = allow16 ? 16 : 8;
    for (int tc = want; tc >= 8; tc /= 2) {
        const size_t smem = td_cluster_smem(m, tc);
        if (smem > 200 * 1024) continue;
        if (cudaFuncSetAttribute(k_tridiag_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
            cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = tc;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(tc);
        cfg.blockDim = dim3(TD_THREADS);
        cfg.dynamicSmemBytes = smem;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int nclusters = 0;
        if (cudaOccupancyMaxActiveClusters(&nclusters, k_tridiag_cluster, &cfg) == cudaSuccess && nclusters > 0)
            return cached_tc = tc;
        cudaGetLastError();
    }
    (void)ctx;
    return 0;
}

static int td_cluster_launch(gcge_gpu_ctx *ctx, int tc, int m, const double *H, int ldh, double *Aw, double *d,
                             double *e, double *tau)
{
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = tc;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(tc);
    cfg.blockDim = dim3(TD_THREADS);
    cfg.dynamicSmemBytes = td_cluster_smem(m, tc);
    cfg.stream = ctx->stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, k_tridiag_cluster, m, H, ldh, Aw, d, e, tau) != cudaSuccess)
        return gb_fail(ctx, GCGE_GPU_ERR_CUDA);
    ctx->launches++;
    if (ctx->prof) gb_prof_end(ctx);
    return gb_check_launch(ctx);
}

// n / b on the path of the Sturm counts: the hardware reciprocal refined once (Newton-
// Raphson, about 2^-40), then the quotient corrected by its exact remainder, which
// leaves an error of 2^-80 before the one rounding -- the IEEE quotient but for values
// that close to the middle of two doubles. It falls as b grows, as IEEE's does: quotients of
// neighbouring divisors are 2^-53 apart or more before the rounding, which keeps their order.
// Five FP64 instructions; a quotient is most of a Sturm step, and each instruction takes
// a quarter of the SM for 64 clocks. Operands past 2^+-450, of which the
// quotient could leave the range of normal numbers, take the division itself.
__device__ __forceinline__ double sturm_div(double n, double b)
{
    const int en = __double2hiint(n) & 0x7ff00000, eb = __double2hiint(b) & 0x7ff00000;
    if (en < (573 << 20) || en > (1472 << 20) || eb < (573 << 20) || eb > (1472 << 20)) return n / b;
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
    r = fma(fma(-b, r, 1.0), r, r);
    const double q = __dmul_rn(n, r);
    return fma(fma(-b, q, n), r, q);
}

// x = m 2^e with |m| in [1, 2) (x normal): m, and e added to ex
__device__ __forceinline__ double take_exponent(double x, int &ex)
{
    const int hi = __double2hiint(x);
    ex += ((hi >> 20) & 0x7ff) - 1023;
    return __hiloint2double((hi & 0x800fffff) | 0x3ff00000, __double2loint(x));
}

// number of eigenvalues of the tridiagonal (d, e2 = e^2) smaller than x (the
// ratio form of the Sturm sequence with the pivmin guard; its count is monotone
// in x under IEEE arithmetic, which the bisection relies on inside clusters);
// det 2^ex: det(T - x I), the product of the ratios (off the chain of them)
__device__ __forceinline__ int sturm_count(int m, const double *d, const double *e2, double x, double pivmin,
                                           double &det, int &ex)
{
    double q = d[0] - x;
    if (fabs(q) < pivmin) q = -pivmin;
    int cnt = q < 0.0;
    ex = 0;
    det = take_exponent(q, ex);
    for (int i = 1; i < m; ++i) {
        q = (d[i] - x) - sturm_div(e2[i - 1], q);
        if (fabs(q) < pivmin) q = -pivmin;
        cnt += q < 0.0;
        det = take_exponent(__dmul_rn(det, take_exponent(q, ex)), ex);
    }
    return cnt;
}

// one block per wanted eigenvalue index j (il-1+block), 32-point multisection.
// guess (may be NULL): an estimate of each wanted eigenvalue (the previous
// Rayleigh-Ritz step's). Its first round counts at g -/+ |g| 2^-(3l+1), l = 0..15
// (lanes 0-15 below, 16-31 above); the closest points whose counts still bracket
// eigenvalue j become the interval, and the multisection goes on from there: a
// guess within relative d of the eigenvalue leaves a bracket of relative width
// ~16 d instead of the Gershgorin interval. The counts are monotone in x, so a
// wrong guess only loses that round.
//
// A warp's 32 counts keep its quarter of the SM's FP64 pipe busy, so a pass of four
// warps takes as long as one: warp L counts at the points of the L-th round from
// here, along the path that an estimate of the eigenvalue predicts (at first the guess,
// then the zero of det(T - x I) by inverse interpolation through the four points
// around its sign change; the last ratio alone says nothing where T all but splits).
// Rounds whose predicted interval turns out to be the actual one are done; the first
// always is. m = 33: 149 us (one round a pass, IEEE divisions) -> 92.
#define BI_WARPS 4
__global__ void __launch_bounds__(32 * BI_WARPS)
k_bisect(int m, const double *__restrict__ dg, const double *__restrict__ eg, int il, int iu,
         double *__restrict__ eval, int *info, const double *__restrict__ guess)
{
    GB_PDL();
    extern __shared__ double sm[];
    double *d = sm, *e2 = sm + m;
    __shared__ double px[BI_WARPS][32], pq[BI_WARPS][32], plo[BI_WARPS], phi[BI_WARPS];
    __shared__ unsigned pge[BI_WARPS];
    __shared__ int pe[BI_WARPS][32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int i = tid; i < m; i += blockDim.x) {
        d[i] = dg[i];
        e2[i] = (i < m - 1) ? eg[i] * eg[i] : 0.0;
    }
    __syncthreads();
    // Gershgorin interval and pivot floor, every warp for itself
    double gl = DBL_MAX, gu = -DBL_MAX, emax = 0;
    for (int i = lane; i < m; i += 32) {
        const double r = (i > 0 ? fabs(eg[i - 1]) : 0.0) + (i < m - 1 ? fabs(eg[i]) : 0.0);
        gl = fmin(gl, d[i] - r);
        gu = fmax(gu, d[i] + r);
        if (i < m - 1) emax = fmax(emax, e2[i]);
    }
    for (int o = 16; o; o >>= 1) {
        gl = fmin(gl, __shfl_xor_sync(FULL, gl, o));
        gu = fmax(gu, __shfl_xor_sync(FULL, gu, o));
        emax = fmax(emax, __shfl_xor_sync(FULL, emax, o));
    }
    const double bn = fmax(fabs(gl), fabs(gu));
    const double piv = DBL_MIN * fmax(1.0, emax);
    const double fudge = 2.0 * DBL_EPSILON * bn * m + 2.0 * piv;
    const int j = il + (int)blockIdx.x;                               // 1-based wanted index
    double lo = gl - fudge, hi = gu + fudge, est = 0.5 * (lo + hi), q;
    int ex;
    if (guess) {
        const double g = guess[j - il];
        if (isfinite(g) && g != 0.0) {                                // every warp the same counts
            const int l = lane & 15;
            const double del = ldexp(fabs(g), -(3 * l + 1));
            const double x = lane < 16 ? g - del : g + del;
            const int c = sturm_count(m, d, e2, x, piv, q, ex);
            const unsigned below = __ballot_sync(FULL, lane < 16 && c < j) & 0xffffu;
            const unsigned above = __ballot_sync(FULL, lane >= 16 && c >= j) >> 16;
            if (below) {
                const double xl = __shfl_sync(FULL, x, 31 - __clz(below));
                if (xl > lo) lo = xl;
            }
            if (above) {
                const double xh = __shfl_sync(FULL, x, 16 + (31 - __clz(above)));
                if (xh < hi) hi = xh;
            }
            est = g;
        }
    }
    // the round's next interval, given which of its points the eigenvalue lies below
    auto next = [&](unsigned ge, double x, double &a, double &b) {
        if (ge == 0u) {
            a = __shfl_sync(FULL, x, 31);
        } else {
            const int f = __ffs(ge) - 1;
            b = __shfl_sync(FULL, x, f);
            const double xm = __shfl_sync(FULL, x, f > 0 ? f - 1 : 0);
            if (f > 0) a = xm;
        }
    };
    auto narrow = [&](double a, double b) { return b - a <= 2.0 * DBL_EPSILON * fmax(fabs(a), fabs(b)) + piv; };
    bool more = true;
    for (int it = 0; it < 80 && more && !narrow(lo, hi);) {
        // this warp's round on the predicted path
        double a = lo, b = hi, x = 0;
        for (int L = 0;; ++L) {
            x = a + (b - a) * (double)(lane + 1) / 33.0;
            if (L == wid) break;
            next(__ballot_sync(FULL, x >= est), x, a, b);
        }
        const int c = sturm_count(m, d, e2, x, piv, q, ex);
        const unsigned ge = __ballot_sync(FULL, c >= j);
        px[wid][lane] = x;
        pq[wid][lane] = q;
        pe[wid][lane] = ex;
        if (lane == 0) {
            pge[wid] = ge;
            plo[wid] = a;
            phi[wid] = b;
        }
        __syncthreads();
        // the rounds that hold, in every warp
        int deep = 0;
        for (int L = 0; L < BI_WARPS && it < 80; ++L, ++it) {
            if (narrow(lo, hi)) {
                more = false;
                break;
            }
            if (plo[L] != lo || phi[L] != hi) break;                  // not this way: L >= 1
            double nlo = lo, nhi = hi;
            next(pge[L], px[L][lane], nlo, nhi);
            deep = L;
            if (nlo == lo && nhi == hi) {                             // no representable progress
                more = false;
                break;
            }
            lo = nlo;
            hi = nhi;
        }
        // the next estimate: inverse interpolation of the determinant around its sign change
        if (more) {
            const unsigned g = pge[deep];
            const int f = g ? __ffs(g) - 1 : 32, f0 = min(max(f - 2, 0), 28);
            double X[4], Q[4];
            const int e0 = max(pe[deep][f0], pe[deep][f0 + 3]);       // a common scale, near enough
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                X[t] = px[deep][f0 + t];
                Q[t] = ldexp(pq[deep][f0 + t], max(-1000, min(1000, pe[deep][f0 + t] - e0)));
            }
            est = 0.5 * (lo + hi);
            const bool down = Q[0] > Q[1] && Q[1] > Q[2] && Q[2] > Q[3] && Q[0] > 0.0 && Q[3] < 0.0;
            const bool up = Q[0] < Q[1] && Q[1] < Q[2] && Q[2] < Q[3] && Q[0] < 0.0 && Q[3] > 0.0;
            if (down || up) {
#pragma unroll
                for (int s = 1; s < 4; ++s)
#pragma unroll
                    for (int t = 0; t + s < 4; ++t) X[t] = X[t] + (X[t + 1] - X[t]) * (Q[t] / (Q[t] - Q[t + s]));
                if (X[0] > lo && X[0] < hi) est = X[0];
            }
        }
        __syncthreads();                                              // before the points are overwritten
    }
    if (tid == 0) {
        const double ev = 0.5 * (lo + hi);
        eval[j - il] = ev;
        if (!isfinite(ev)) atomicExch(info, 1);
    }
}

// start vectors of inverse iteration, hashed
__device__ __forceinline__ double start_value(int j, int i)
{
    unsigned long long z = (unsigned long long)(j + 1) * 0x9E3779B97F4A7C15ULL ^ (unsigned long long)(i + 7) * 0xD1B54A32D192ED03ULL;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    z ^= z >> 31;
    return (double)(z >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

__global__ void k_recip_probe(int n, const double *__restrict__ x, double *__restrict__ r)
{
    GB_PDL();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) r[i] = nr_recip(x[i]);
}
__global__ void k_div_probe(int n, int kind, const double *__restrict__ x, const double *__restrict__ y,
                            double *__restrict__ q)
{
    GB_PDL();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) q[i] = kind ? sturm_div(x[i], y[i]) : div_by(x[i], y[i], 1.0 / y[i]);
}

// Internal checks of nr_recip and of the two divisions (not part of the public interface), on
// the current device: r[i] = nr_recip(x[i]); q[i] = div_by (kind 0) or sturm_div (kind 1) of
// x[i] and y[i], for n host values.
static int probe(int n, const double *x_host, const double *y_host, int kind, double *r_host)
{
    if (n <= 0 || !x_host || !r_host) return GCGE_GPU_ERR_ARG;
    const size_t bytes = sizeof(double) * n;
    double *dx = nullptr, *dy = nullptr, *dr = nullptr;
    int st = GCGE_GPU_OK;
    if (cudaMalloc(&dx, bytes) != cudaSuccess || cudaMalloc(&dr, bytes) != cudaSuccess ||
        cudaMemcpy(dx, x_host, bytes, cudaMemcpyHostToDevice) != cudaSuccess ||
        (y_host && (cudaMalloc(&dy, bytes) != cudaSuccess ||
                    cudaMemcpy(dy, y_host, bytes, cudaMemcpyHostToDevice) != cudaSuccess)))
        st = GCGE_GPU_ERR_CUDA;
    if (!st) {
        if (y_host) k_div_probe<<<(n + 255) / 256, 256>>>(n, kind, dx, dy, dr);
        else k_recip_probe<<<(n + 255) / 256, 256>>>(n, dx, dr);
        if (cudaGetLastError() != cudaSuccess || cudaMemcpy(r_host, dr, bytes, cudaMemcpyDeviceToHost) != cudaSuccess)
            st = GCGE_GPU_ERR_CUDA;
    }
    cudaFree(dx);
    cudaFree(dy);
    cudaFree(dr);
    return st;
}
extern "C" int gb_recip_check(int n, const double *x_host, double *r_host) { return probe(n, x_host, nullptr, 0, r_host); }
extern "C" int gb_div_check(int kind, int n, const double *x_host, const double *y_host, double *q_host)
{
    return y_host ? probe(n, x_host, y_host, kind, q_host) : GCGE_GPU_ERR_ARG;
}

// inverse iteration: a block of one warp per wanted eigenvalue, so that the chains
// spread over the SMs (the FP64 pipe of an SM is narrow); LU of T - lambda I with
// partial pivoting (dgttrf layout) and three solves from a hashed start vector, the
// working arrays in shared memory. Lane 0 walks the recurrences, with the next
// elements in registers; what has no recurrence (set-up, pivots' reciprocals, start
// vector, maxima, scalings) is done by all lanes. (All by one lane: 71 us for 13
// vectors of 30, here 34.)
__global__ void __launch_bounds__(32)
k_invit(int m, const double *__restrict__ d, const double *__restrict__ e, int nev,
        const double *__restrict__ eval, double *__restrict__ Zt, int ldz)
{
    GB_PDL();
    extern __shared__ double ism[];
    const int lane = threadIdx.x, j = blockIdx.x;
    double *dl = ism, *dd = dl + m, *du = dd + m, *du2 = du + m, *inv = du2 + m, *z = inv + m;
    int *ip = (int *)(z + m);
    double tnorm = 0;
    for (int i = lane; i < m; i += 32)
        tnorm = fmax(tnorm, fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < m - 1 ? fabs(e[i]) : 0.0));
    for (int o = 16; o; o >>= 1) tnorm = fmax(tnorm, __shfl_xor_sync(FULL, tnorm, o));
    // perturb a shift that repeats the previous one (dstein: separate close shifts)
    double lam = eval[j];
    const double pert = 10.0 * DBL_EPSILON * fmax(fabs(lam), tnorm * 1e-3);
    if (j > 0 && lam - eval[j - 1] < pert) {
        int k = j;
        while (k > 0 && eval[k] - eval[k - 1] < pert) --k;
        lam = eval[k] + (double)(j - k) * pert;
    }
    for (int i = lane; i < m; i += 32) {
        dd[i] = d[i] - lam;
        const double ei = i < m - 1 ? e[i] : 0.0;
        dl[i] = ei;
        du[i] = ei;
        du2[i] = 0.0;
        ip[i] = i;
        z[i] = start_value(j, i);
    }
    __syncwarp();
    if (lane == 0) {
        double di = dd[0], ui = du[0];                   // row i of the partly reduced matrix
        for (int i = 0; i + 1 < m; ++i) {
            const double li = dl[i], dn = dd[i + 1], un = du[i + 1];
            if (fabs(di) >= fabs(li)) {
                dd[i] = di;
                du[i] = ui;
                double f = 0.0, t = dn;
                if (di != 0.0) {
                    f = li * nr_recip(di);
                    t -= f * ui;
                }
                dl[i] = f;
                di = t;
                ui = un;
            } else {
                const double f = di * nr_recip(li);
                dd[i] = li;
                dl[i] = f;
                du[i] = dn;
                di = ui - f * dn;
                ui = un;
                if (i + 2 < m) {
                    du2[i] = un;
                    ui = -f * un;
                }
                ip[i] = i + 1;
            }
        }
        dd[m - 1] = di;
    }
    __syncwarp();
    const double tiny = DBL_EPSILON * fmax(tnorm, DBL_MIN);
    for (int i = lane; i < m; i += 32) {
        double di = dd[i];
        if (fabs(di) < tiny) di = copysign(tiny, di == 0.0 ? 1.0 : di);
        inv[i] = nr_recip(di);
    }
    __syncwarp();
    for (int iter = 0; iter < 3; ++iter) {
        // solve L U x = z (dgttrs, no transpose)
        if (lane == 0) {
            double zi = z[0];
            for (int i = 0; i + 1 < m; ++i) {
                const double f = dl[i], zn = z[i + 1];
                if (ip[i] == i) {
                    z[i] = zi;
                    zi = zn - f * zi;
                } else {
                    z[i] = zn;
                    zi = zi - f * zn;
                }
            }
            double z1 = zi * inv[m - 1], z2 = 0.0;       // z[i + 1], z[i + 2]
            z[m - 1] = z1;
            if (m >= 2) {
                z2 = z1;
                z1 = (z[m - 2] - du[m - 2] * z2) * inv[m - 2];
                z[m - 2] = z1;
            }
            for (int i = m - 3; i >= 0; --i) {
                const double t = (z[i] - du[i] * z1 - du2[i] * z2) * inv[i];
                z[i] = t;
                z2 = z1;
                z1 = t;
            }
        }
        __syncwarp();
        double mx = 0;
        for (int i = lane; i < m; i += 32) mx = fmax(mx, fabs(z[i]));
        for (int o = 16; o; o >>= 1) mx = fmax(mx, __shfl_xor_sync(FULL, mx, o));
        const double sc = mx > 0 ? 1.0 / mx : 1.0;
        for (int i = lane; i < m; i += 32) z[i] *= sc;
        __syncwarp();
    }
    double nn = 0;                                       // every lane the same chain
    for (int i = 0; i < m; ++i) nn = fma(z[i], z[i], nn);
    const double sc = 1.0 / sqrt(nn);
    double *zo = Zt + (size_t)j * ldz;
    for (int i = lane; i < m; i += 32) zo[i] = z[i] * sc;
}

// reorthogonalise inside clusters (gap <= 1e-3 ||T||_1, as dstein) by two
// classical Gram-Schmidt passes, then normalise; a block per cluster (the b-th run of
// close eigenvalues to block b), vectors in order; with SMEM the cluster's vectors are
// worked on in shared memory. m <= 1024: a thread per row, and eight warps at least: the
// products with the earlier vectors, four to a warp and one tree of additions for the four,
// keep all quarters of the SM at their FP64. (Two warps at m = 60, a tree per product: 185
// us for 25 vectors in one cluster, now 104. All vectors in one block of
// 1,024 threads spent 2.3 us on each, mostly barriers and a serial sum of 32 warps, although
// most of them belong to no cluster: 73 us for 13 vectors of 30, here 12.)
template <bool SMEM>
__global__ void __launch_bounds__(1024)
k_cluster_orth(int m, const double *__restrict__ d, const double *__restrict__ e, int nev,
               const double *__restrict__ eval, double *__restrict__ Zg, int ldz)
{
    GB_PDL();
    extern __shared__ double zsm[];
    __shared__ double coef[1024];
    __shared__ double red[32];
    __shared__ unsigned starts[32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
    // ||T||: the largest row sum
    double tn = 0;
    for (int i = tid; i < m; i += blockDim.x)
        tn = fmax(tn, fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < m - 1 ? fabs(e[i]) : 0.0));
    for (int o = 16; o; o >>= 1) tn = fmax(tn, __shfl_xor_sync(FULL, tn, o));
    if (lane == 0) red[wid] = tn;
    __syncthreads();
    for (int q = 0; q < nw; ++q) tn = fmax(tn, red[q]);
    const double ortol = 1e-3 * tn;
    // the b-th run of eigenvalues: [first, end)
    int first = -1, end = nev, seen = 0;
    for (int j0 = 0; j0 < nev && first < 0; j0 += 1024) {
        __syncthreads();
        for (int w = wid; w < 32; w += nw) {
            const int j = j0 + 32 * w + lane;
            const unsigned b = __ballot_sync(FULL, j < nev && (j == 0 || eval[j] - eval[j - 1] > ortol));
            if (lane == 0) starts[w] = b;
        }
        __syncthreads();
        for (int w = 0; w < 32 && first < 0; ++w) {
            unsigned b = starts[w];
            const int c = __popc(b);
            if (seen + c > (int)blockIdx.x) {
                for (int q = blockIdx.x - seen; q > 0; --q) b &= b - 1;
                first = j0 + 32 * w + __ffs(b) - 1;
            }
            seen += c;
        }
    }
    if (first < 0) return;                               // fewer runs than blocks
    for (int j = first + 1; j < nev; ++j)
        if (eval[j] - eval[j - 1] > ortol) {
            end = j;
            break;
        }
    double *Zt = Zg + (size_t)first * ldz;
    long ld = ldz;
    if (SMEM) {
        for (int c = wid; c < end - first; c += nw)
            for (int r = lane; r < m; r += 32) zsm[(size_t)c * m + r] = Zt[(size_t)c * ldz + r];
        Zt = zsm;
        ld = m;
    }
    __syncthreads();
    for (int np = 0; np < end - first; ++np) {
        double *zj = Zt + (size_t)np * ld;
        if (np > 0) {
            for (int pass = 0; pass < 2; ++pass) {
                for (int q = wid; q < np; q += 4 * nw) {
                    // four vectors a warp: lanes with bits 4 and 3 equal to (u & 1, u >> 1) end with
                    // vector u's sum, the halves added in the order of a butterfly of its own
                    double s[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const double *zi = Zt + (size_t)min(q + u * nw, np - 1) * ld;
                        s[u] = 0;
                        if (q + u * nw < np)
                            for (int r = lane; r < m; r += 32) s[u] = fma(zi[r], zj[r], s[u]);
                    }
                    const bool b4 = lane & 16, b3 = lane & 8;
                    const double t0 = (b4 ? s[1] : s[0]) + __shfl_xor_sync(FULL, b4 ? s[0] : s[1], 16);
                    const double t1 = (b4 ? s[3] : s[2]) + __shfl_xor_sync(FULL, b4 ? s[2] : s[3], 16);
                    double t = (b3 ? t1 : t0) + __shfl_xor_sync(FULL, b3 ? t0 : t1, 8);
#pragma unroll
                    for (int o = 4; o; o >>= 1) t += __shfl_xor_sync(FULL, t, o);
                    const int c = q + ((b4 ? 1 : 0) + (b3 ? 2 : 0)) * nw;
                    if ((lane & 7) == 0 && c < np && c < 1024) coef[c] = t;
                }
                __syncthreads();
                for (int r = tid; r < m; r += blockDim.x) {
                    double acc = zj[r];
                    for (int q = 0; q < np && q < 1024; ++q) acc -= coef[q] * Zt[(size_t)q * ld + r];
                    zj[r] = acc;
                }
                __syncthreads();
            }
        }
        double s = 0;
        for (int r = tid; r < m; r += blockDim.x) s = fma(zj[r], zj[r], s);
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
        if (lane == 0) red[wid] = s;
        __syncthreads();
        if (tid == 0) {
            double t = 0;
            for (int q = 0; q < nw; ++q) t += red[q];
            red[0] = t > 0 ? 1.0 / sqrt(t) : 1.0;
        }
        __syncthreads();
        const double inv = red[0];
        for (int r = tid; r < m; r += blockDim.x) zj[r] *= inv;
        __syncthreads();
    }
    if (SMEM) {
        double *Zo = Zg + (size_t)first * ldz;
        for (int c = wid; c < end - first; c += nw)
            for (int r = lane; r < m; r += 32) Zo[(size_t)c * ldz + r] = zsm[(size_t)c * m + r];
    }
}

// Z = Q Zt with Q = H_0 H_1 ... H_{m-3}; a block of one warp per column (its FP64
// chain alone on an SM), reflectors in reverse. The vector stays in shared memory and
// the next BT_AHEAD reflectors are on their way there (with both in global memory a step
// waited for two trips to L2: 33 us for 13 vectors of 30, here 22). A non-finite result
// sets info.
#define BT_AHEAD 4
__device__ __forceinline__ void bt_fetch(double *slot, const double *v, int i, int m)
{
    for (int r = i + 2 + (int)threadIdx.x; r < m; r += 32)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(slot + r)),
                     "l"(v + r)
                     : "memory");
}
__global__ void __launch_bounds__(32)
k_backtransform(int m, const double *__restrict__ Aw, const double *__restrict__ tau, int nev,
                const double *__restrict__ Zt, int ldzt, double *__restrict__ Z, int ldz, int *info)
{
    GB_PDL();
    extern __shared__ double bsm[];                      // z, then BT_AHEAD + 1 reflectors
    const int lane = threadIdx.x, c = blockIdx.x;
    double *z = bsm, *ring = bsm + m;
    const double *zt = Zt + (size_t)c * ldzt;
    for (int q = 0; q < BT_AHEAD; ++q) {
        const int i = m - 3 - q;
        if (i >= 0) bt_fetch(ring + (size_t)q * m, Aw + (size_t)i * m, i, m);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int r = lane; r < m; r += 32) z[r] = zt[r];
    __syncwarp();
    int slot = 0, fill = BT_AHEAD;
    for (int i = m - 3; i >= 0; --i) {
        const int ahead = i - BT_AHEAD;
        if (ahead >= 0) bt_fetch(ring + (size_t)fill * m, Aw + (size_t)ahead * m, ahead, m);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const double t = tau[i];
        asm volatile("cp.async.wait_group %0;" ::"n"(BT_AHEAD) : "memory");
        __syncwarp();
        const double *v = ring + (size_t)slot * m;       // v[i+1] = 1, v[i+2:] stored
        if (t != 0.0) {
            double s = 0;
            for (int r = i + 1 + lane; r < m; r += 32) s = fma(r == i + 1 ? 1.0 : v[r], z[r], s);
            for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
            const double f = t * s;
            for (int r = i + 1 + lane; r < m; r += 32) z[r] -= f * (r == i + 1 ? 1.0 : v[r]);
        }
        __syncwarp();
        slot = slot == BT_AHEAD ? 0 : slot + 1;
        fill = fill == BT_AHEAD ? 0 : fill + 1;
    }
    bool bad = false;
    for (int r = lane; r < m; r += 32) {
        bad |= !isfinite(z[r]);
        Z[r + (size_t)c * ldz] = z[r];
    }
    if (bad) atomicExch(info, 2);
}

// Reorthogonalisation of many inverse-iteration vectors by Cholesky-QR.
// k_cluster_orth orthogonalises each vector against the earlier members of its
// cluster (eigenvalues closer than 1e-3 ||T||, dstein's criterion) by modified
// Gram-Schmidt in one thread block; when ||T|| is large against the wanted
// eigenvalues (a graph pencil: projected spectrum to ~2e3, wanted ones below 1)
// every wanted vector falls in one cluster, and that block does O(nev^2 m) FP64
// work alone. Gram-Schmidt over all vectors in index order is the Q factor of
// Z = Q R, which Cholesky-QR computes with parallel small GEMMs: G = Z^T Z,
// R^T R = G, Z <- Z R^-1. Inverse-iteration vectors are nearly orthonormal, so
// one pass leaves them orthonormal to rounding when every pivot keeps at least
// half of its column's norm squared (condition number of Z below ~1.5); a second
// pass repairs the first one's rounding otherwise. Vectors of well-separated
// eigenvalues are already orthogonal to O(eps ||T|| / gap), so the mixing
// outside the clusters is of that order. A pivot below 1e-10 of its column's
// norm (nearly dependent vectors) keeps the vectors as they were and the caller
// falls back to k_cluster_orth. (m = 720, nev = 208, one GB300: 33 ms per
// dsyevx-signature call against 44.5 ms with k_cluster_orth, both passes run.)
#define CQ_MIN_NEV 96
static int cholqr_reorth(gcge_gpu_ctx *ctx, int m, int nev, double *Zt, double *ext, int *done)
{
    double *Zq = ext, *G = Zq + (size_t)m * m, *Tq = G + (size_t)m * m, *cw = Tq + (size_t)m * m;
    double *ratio_dev = cw + 2 * (size_t)m * m;
    int *kept_dev = (int *)(ratio_dev + 8);
    *done = 0;
    for (int pass = 0; pass < 2; ++pass) {
        double *src = pass == 0 ? Zt : Zq, *dst = pass == 0 ? Zq : Zt;
        int st = gb_small_gemm(ctx, 'T', 'N', nev, nev, m, 1.0, src, m, src, m, 0.0, G, nev);
        if (st) return st;
        if ((st = cd_launch(ctx, nev, G, nev, Tq, kept_dev, 0.0, 1e-10, cw, ratio_dev))) return st;
        struct { int kept; int pad; double ratio; } h = {0, 0, 0.0};
        if (cudaMemcpyAsync(&h.kept, kept_dev, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream) != cudaSuccess ||
            cudaMemcpyAsync(&h.ratio, ratio_dev, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream) != cudaSuccess ||
            cudaStreamSynchronize(ctx->stream) != cudaSuccess)
            return gb_fail(ctx, GCGE_GPU_ERR_CUDA);
        if (h.kept != nev) {
            // nearly dependent vectors: leave them (the second pass' input is copied back)
            if (pass == 1 && (st = gb_copy_block(ctx, m, nev, Zq, m, Zt, m))) return st;
            return GCGE_GPU_OK;
        }
        if ((st = gb_small_gemm(ctx, 'N', 'N', m, nev, nev, 1.0, src, m, Tq, nev, 0.0, dst, m))) return st;
        if (pass == 0 && h.ratio >= 0.5) {
            if ((st = gb_copy_block(ctx, m, nev, Zq, m, Zt, m))) return st;
            break;
        }
    }
    *done = 1;
    return GCGE_GPU_OK;
}

// largest matrix: 52 bytes of shared memory a row in k_invit, 48 in k_backtransform, 16 in k_tridiag (below
// the default of 48 KB) and k_bisect (above it with its 2.6 KB of static arrays)
#define SY_MAX_M 3000
static size_t bi_smem(int m) { return 2 * sizeof(double) * (size_t)m; }

extern "C" int gb_syevx_guess(gcge_gpu_ctx *ctx, int m, const double *H, int ldh, int il, int iu, double *eval,
                              double *Z, int ldz, double *work, int *info_dev, const double *guess);
extern "C" int gb_syevx(gcge_gpu_ctx *ctx, int m, const double *H, int ldh, int il, int iu, double *eval,
                        double *Z, int ldz, double *work, int *info_dev)
{
    return gb_syevx_guess(ctx, m, H, ldh, il, iu, eval, Z, ldz, work, info_dev, nullptr);
}

extern "C" int gb_syevx_guess(gcge_gpu_ctx *ctx, int m, const double *H, int ldh, int il, int iu, double *eval,
                              double *Z, int ldz, double *work, int *info_dev, const double *guess)
{
    if (m <= 0 || il < 1 || iu > m || il > iu) return gb_fail(ctx, GCGE_GPU_ERR_ARG);
    if (m > SY_MAX_M) return gb_fail(ctx, GCGE_GPU_ERR_ARG);
    const int nev = iu - il + 1;
    double *Aw = work, *d = Aw + (size_t)m * m, *e = d + m, *tau = e + m, *Zt = tau + m;
    if (cudaMemsetAsync(info_dev, 0, sizeof(int), ctx->stream) != cudaSuccess) return gb_fail(ctx, GCGE_GPU_ERR_CUDA);
    const int tthreads = m >= 512 ? 1024 : (m >= 128 ? 512 : 256);
    GB_PROF(ctx, GB_K_EIG, 8.0 * m * m, 4.0 / 3.0 * m * (double)m * m);
    const int tc = td_cluster_size(ctx, m);
    if (tc) {
        int st = td_cluster_launch(ctx, tc, m, H, ldh, Aw, d, e, tau);
        if (st) return st;
    } else {
        static bool td_attr = false;
        if (!td_attr) {
            if (cudaFuncSetAttribute(k_tridiag_smem, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)td_smem_bytes(TD_SMEM_MAX_M)) != cudaSuccess ||
                cudaFuncSetAttribute(k_tridiag_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)ts_smem_bytes(TS_MAX_M)) != cudaSuccess)
                return gb_fail(ctx, GCGE_GPU_ERR_CUDA);
            td_attr = true;
        }
        if (m <= TS_MAX_M)
            GB_LAUNCH(ctx, k_tridiag_small, 1, TS_THREADS, ts_smem_bytes(m), m, H, ldh, Aw, d, e, tau);
        else if (m <= TD_SMEM_MAX_M)
            GB_LAUNCH(ctx, k_tridiag_smem, 1, tthreads, td_smem_bytes(m), m, H, ldh, Aw, d, e, tau);
        else
            GB_LAUNCH(ctx, k_tridiag, 1, tthreads, 2 * m * sizeof(double), m, H, ldh, Aw, d, e, tau);
    }
    // the 48 KB default covers static and dynamic shared memory together: these kernels are
    // opened once to the most they can ask for (k_bisect 48 KB at m = 3000, k_invit 156 KB,
    // k_backtransform 144 KB, k_cluster_orth<true> 160 KB)
    static bool attrs = false;
    if (!attrs) {
        if (cudaFuncSetAttribute(k_bisect, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bi_smem(SY_MAX_M)) != cudaSuccess ||
            cudaFuncSetAttribute(k_invit, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024) != cudaSuccess ||
            cudaFuncSetAttribute(k_cluster_orth<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024) !=
                cudaSuccess ||
            cudaFuncSetAttribute(k_backtransform, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024) != cudaSuccess)
            return gb_fail(ctx, GCGE_GPU_ERR_CUDA);
        attrs = true;
    }
    GB_PROF(ctx, GB_K_EIG, 0.0, 0.0);
    GB_LAUNCH(ctx, k_bisect, nev, 32 * BI_WARPS, bi_smem(m), m, d, e, il, iu, eval, info_dev, guess);
    GB_PROF(ctx, GB_K_EIG, 0.0, 0.0);
    const size_t ismem = (size_t)m * (6 * sizeof(double) + sizeof(int));
    GB_LAUNCH(ctx, k_invit, nev, 32, ismem, m, d, e, nev, eval, Zt, m);
    GB_PROF(ctx, GB_K_EIG, 0.0, 0.0);
    int reorth_done = 0;
    if (nev >= CQ_MIN_NEV) {
        const int st = cholqr_reorth(ctx, m, nev, Zt, Zt + (size_t)m * m, &reorth_done);
        if (st) return st;
    }
    const size_t osmem = sizeof(double) * (size_t)m * nev;
    const int othreads = m > 1024 ? 1024 : m > 256 ? (m + 31) / 32 * 32 : 256;
    if (reorth_done) {
        // the vectors are orthonormal: Cholesky-QR over all of them
    } else if (osmem <= 160 * 1024) {
        GB_LAUNCH(ctx, k_cluster_orth<true>, nev, othreads, osmem, m, d, e, nev, eval, Zt, m);
    } else {
        GB_LAUNCH(ctx, k_cluster_orth<false>, nev, othreads, 0, m, d, e, nev, eval, Zt, m);
    }
    GB_PROF(ctx, GB_K_EIG, 0.0, 0.0);
    GB_LAUNCH(ctx, k_backtransform, nev, 32, sizeof(double) * (size_t)m * (BT_AHEAD + 2), m, Aw, tau, nev, Zt, m, Z, ldz,
              info_dev);
    return GCGE_GPU_OK;
}
