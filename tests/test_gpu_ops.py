"""Per-operation parity of the CUDA path (through the C ABI) against the oracle.

Each GCGE_OPS multivector member is compared with the oracle's restatement of
the reference default (src/gcge_ops.c:115-300) or CSR backend
(app/csr/gcge_app_csr.c:297-378) on seeded inputs. Tolerances: 1e-13 relative
(FP64 arithmetic in a different order, fused multiply-adds).
"""
import numpy as np
import pytest

import gcge_gb300 as G
import pyoracle
from gcge_gb300 import problems as P

pytestmark = pytest.mark.gpu
RTOL = 1e-13


@pytest.fixture(scope="module")
def ctx():
    c = G.Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def oracle():
    return pyoracle.Oracle()


def rel(a, b):
    return np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300)


def cols_to_oracle(X):
    return np.ascontiguousarray(np.asarray(X).T)


@pytest.mark.parametrize("maker,k", [(lambda: P.laplace2d(37, 23)[0], 1), (lambda: P.laplace2d(37, 23)[0], 7),
                                     (lambda: P.fem_q1_cube(9)[0], 64), (lambda: P.fem_q1_cube(9)[1], 65),
                                     (lambda: P.powerlaw_graph(3000, seed=5, dmax=300)[0], 33)])
@pytest.mark.parametrize("sx,sy", [(2, 4), (1, 3)])      # (1, 3): column ranges off the 16-byte grid
def test_matdotmultivec(ctx, oracle, maker, k, sx, sy):
    A = maker()
    rng = np.random.default_rng(1)
    X = rng.standard_normal((A.n, k + 3))
    dA = ctx.matrix(A)
    x = ctx.multivec(A.n, k + 3, X)
    y = ctx.multivec(A.n, k + 5)
    G.mat_dot_multivec(dA, x, y, (sx, sy), (sx + k, sy + k))
    got = y.download()[:, sy:sy + k]
    ref = oracle.matmultivec(A, cols_to_oracle(X[:, sx:sx + k])).T
    assert rel(got, ref) < RTOL


@pytest.mark.parametrize("a,b", [(0.0, 2.5), (1.0, 0.0), (-3.0, 0.0), (2.0, -0.5), (0.0, 0.0)])
def test_axpby_special_cases(ctx, oracle, a, b):
    rng = np.random.default_rng(2)
    n = 1001
    X, Y = rng.standard_normal((n, 9)), rng.standard_normal((n, 9))
    x, y = ctx.multivec(n, 9, X), ctx.multivec(n, 9, Y)
    G.multivec_axpby(a, x, b, y, (1, 3), (7, 9))
    got = y.download()
    ref = Y.copy()
    for j in range(6):
        ref[:, 3 + j] = oracle.axpby(a, X[:, 1 + j], b, Y[:, 3 + j])
    assert np.array_equal(got[:, :3], Y[:, :3])
    assert rel(got, ref) < RTOL


@pytest.mark.parametrize("n,k1,k2,lda", [(5000, 13, 9, 20), (20000, 70, 40, 70), (333, 1, 1, 1), (4097, 33, 65, 40)])
def test_linear_comb(ctx, oracle, n, k1, k2, lda):
    rng = np.random.default_rng(3)
    X = rng.standard_normal((n, k1))
    coef = rng.standard_normal(lda * k2)
    x, y = ctx.multivec(n, k1, X), ctx.multivec(n, k2 + 2)
    G.multivec_linear_comb(x, y, (0, 2), (k1, 2 + k2), coef, lda)
    got = y.download()[:, 2:]
    ref = oracle.lincomb(cols_to_oracle(X), coef, k2, lda).T
    assert rel(got, ref) < RTOL


@pytest.mark.parametrize("sym", [False, True])
@pytest.mark.parametrize("n,k1,k2,lda", [(10000, 17, 17, 30), (300000, 64, 64, 64), (777, 40, 40, 45)])
def test_inner_prod(ctx, oracle, sym, n, k1, k2, lda):
    rng = np.random.default_rng(4)
    V, W = rng.standard_normal((n, k1 + 1)), rng.standard_normal((n, k2))
    if sym:
        W = V[:, 1:1 + k2] * 0.5 + W * 1e-3
    v, w = ctx.multivec(n, k1 + 1, V), ctx.multivec(n, k2, W)
    got = G.multivec_inner_prod(v, w, (1, 0), (1 + k1, k2), lda, sym=sym, out=np.full(lda * k2, 7.0))
    ref = np.full(lda * k2, 7.0)
    ref_o = oracle.innerprod(cols_to_oracle(V[:, 1:1 + k1]), cols_to_oracle(W), lda, sym)
    for j in range(k2):
        ref[j * lda:j * lda + k1] = ref_o[j * lda:j * lda + k1]
    np.testing.assert_allclose(got, ref, rtol=1e-12, atol=1e-12 * np.max(np.abs(ref)))


def test_swap(ctx):
    rng = np.random.default_rng(5)
    n = 999
    X, Y = rng.standard_normal((n, 6)), rng.standard_normal((n, 5))
    x, y = ctx.multivec(n, 6, X), ctx.multivec(n, 5, Y)
    G.multivec_swap(x, y, (1, 2), (4, 5))
    gx, gy = x.download(), y.download()
    assert np.array_equal(gx[:, 1:4], Y[:, 2:5]) and np.array_equal(gy[:, 2:5], X[:, 1:4])
    assert np.array_equal(gx[:, [0, 4, 5]], X[:, [0, 4, 5]])


@pytest.mark.parametrize("k,max_it", [(8, 20), (13, 7)])
def test_bcg_fp64_matches_oracle(ctx, oracle, k, max_it):
    """FP64 block CG follows GCGE_BCG's iteration (including its active-column rule)."""
    A, _ = P.laplace2d(40, 30)
    rng = np.random.default_rng(6)
    R0, W0 = rng.standard_normal((A.n, k)), rng.standard_normal((A.n, k)) * 0.1
    dA = ctx.matrix(A)
    r, w = ctx.multivec(A.n, k, R0), ctx.multivec(A.n, k + 1)
    w.upload(W0, 1)
    G.bcg(dA, r, 0, w, 1, k, cg_max_it=max_it, cg_rate=1e-2, precision=0)
    Xo, Ro = oracle.bcg(A, cols_to_oracle(R0), cols_to_oracle(W0), max_it, 1e-2)
    assert rel(w.download()[:, 1:], Xo.T) < 1e-9
    assert rel(r.download(), Ro.T) < 1e-7


def test_bcg_fp32_close_to_fp64(ctx):
    A, _ = P.laplace2d(40, 30)
    rng = np.random.default_rng(7)
    k = 10
    R0 = rng.standard_normal((A.n, k))
    dA = ctx.matrix(A, keep_fp32=True)
    out = []
    for prec in (0, 1):
        r, w = ctx.multivec(A.n, k, R0), ctx.multivec(A.n, k)
        G.bcg(dA, r, 0, w, 0, k, cg_max_it=20, cg_rate=1e-2, precision=prec)
        out.append((w.download(), r.download()))
    # 19 rounds shrink every residual; the FP32 defect-correction iterate tracks the FP64 one
    Asp = A.to_scipy()
    res = []
    for Wsol, _ in out:
        r = np.linalg.norm(R0 - Asp @ Wsol, axis=0) / np.linalg.norm(R0, axis=0)
        assert np.all(r < 0.5)
        res.append(r)
    assert np.max(np.abs(res[1] - res[0])) < 1e-3
    assert rel(out[1][0], out[0][0]) < 1e-3


@pytest.mark.parametrize("k,max_it,rate", [(2, 8, 1e-2), (4, 10, 1e-2), (7, 10, 1e-2), (10, 10, 1e-2),
                                            (10, 5, 1e-1), (20, 8, 1e-2), (40, 8, 1e-2), (70, 6, 1e-1)])
def test_bcg_fp32_tracks_fp64_while_columns_deactivate(ctx, k, max_it, rate):
    """Columns of very different difficulty leave the active range at different
    rounds; the FP32 rounds' per-block partials must stay aligned with the column
    sums over the full column range, so the FP32 iterate keeps FP32 accuracy."""
    A, _ = P.laplace2d(40, 30)
    Asp = A.to_scipy()
    rng = np.random.default_rng(100 + k)
    R0 = rng.standard_normal((A.n, k)) * np.logspace(0, -3, k)
    R0[:, ::3] = Asp @ rng.standard_normal((A.n, (k + 2) // 3))
    dA = ctx.matrix(A, keep_fp32=True)
    out = []
    for prec in (0, 1):
        r, w = ctx.multivec(A.n, k, R0), ctx.multivec(A.n, k)
        G.bcg(dA, r, 0, w, 0, k, cg_max_it=max_it, cg_rate=rate, precision=prec)
        out.append(w.download())
    assert np.all(np.isfinite(out[1]))
    assert rel(out[1], out[0]) < 1e-4


@pytest.mark.parametrize("k", [3, 8, 16, 30, 64, 100, 200])
def test_bcg_fp32_long_rows(ctx, k):
    """A power-law graph whose hub rows exceed the long-row length: those rows go
    to the block-per-row SpMM launch, the rest to the grid-stride one; the FP32
    iterate tracks the FP64 one and repeats bit for bit (fixed-order sums). The
    shift keeps the condition number near 25, so that FP32 rounding, amplified by
    the rounds roughly in proportion to it, stays far below the bound, while a
    wrong sum over a hub row would not."""
    A, _ = P.powerlaw_graph(n=20000, seed=11, shift=100.0)
    assert int(np.sum(np.diff(A.rowptr) > 64)) > 100
    rng = np.random.default_rng(200 + k)
    R0 = rng.standard_normal((A.n, k))
    dA = ctx.matrix(A, keep_fp32=True)
    out = []
    for prec in (0, 1, 1):
        r, w = ctx.multivec(A.n, k, R0), ctx.multivec(A.n, k)
        G.bcg(dA, r, 0, w, 0, k, cg_max_it=12, cg_rate=1e-30, precision=prec)
        out.append(w.download())
    assert np.all(np.isfinite(out[1]))
    assert rel(out[1], out[0]) < 1e-4
    assert np.array_equal(out[1], out[2])


@pytest.mark.parametrize("k", [33, 40, 64])
def test_bcg_fp32_fem_cube(ctx, k):
    """Q1 cube stiffness (27 entries per row) at the solver's block widths: the
    FP32 iterate tracks the FP64 one and repeats bit for bit; new values of the
    same structure scale the result exactly (2 A: half the iterate)."""
    A, _ = P.fem_q1_cube(24)
    rng = np.random.default_rng(300 + k)
    R0 = rng.standard_normal((A.n, k))
    dA = ctx.matrix(A, keep_fp32=True)
    out = []
    for prec in (0, 1, 1):
        r, w = ctx.multivec(A.n, k, R0), ctx.multivec(A.n, k)
        G.bcg(dA, r, 0, w, 0, k, cg_max_it=12, cg_rate=1e-30, precision=prec)
        out.append(w.download())
    assert np.all(np.isfinite(out[1]))
    assert rel(out[1], out[0]) < 1e-4
    assert np.array_equal(out[1], out[2])
    # new values, same structure: 2 A
    dA.set_values(2.0 * A.val)
    r, w = ctx.multivec(A.n, k, R0), ctx.multivec(A.n, k)
    G.bcg(dA, r, 0, w, 0, k, cg_max_it=12, cg_rate=1e-30, precision=1)
    assert rel(2.0 * w.download(), out[1]) < 1e-5


def test_newton_reciprocal_of_inverse_iteration(ctx):
    """The reciprocal used for the pivots of inverse iteration (hardware
    approximation refined by two Newton-Raphson steps) is within 2 ulp of the
    IEEE quotient 1/x over the normal range; zero, infinities and subnormal
    inputs take the exact division."""
    import ctypes as C
    lib = G.load()
    rng = np.random.default_rng(12)
    x = np.concatenate([rng.uniform(1.0, 2.0, 4000) * np.exp2(rng.integers(-1020, 1020, 4000)),
                        -rng.uniform(1.0, 2.0, 1000) * np.exp2(rng.integers(-60, 60, 1000)),
                        [1.0, -1.0, 3.0, 2.0 ** -1022, 2.0 ** 1023, 0.0, -0.0, np.inf, -np.inf, 5e-324, 1e-310]])
    r = np.zeros_like(x)
    lib.gb_recip_check.restype = C.c_int
    assert lib.gb_recip_check(len(x), x.ctypes.data_as(C.c_void_p), r.ctypes.data_as(C.c_void_p)) == 0
    with np.errstate(divide="ignore", over="ignore"):
        ref = 1.0 / x
    normal = np.isfinite(ref) & (np.abs(x) >= 2.0 ** -1022) & np.isfinite(x) & (np.abs(ref) >= 2.0 ** -1022)
    ulp = np.spacing(np.abs(ref[normal]))
    assert np.max(np.abs(r[normal] - ref[normal]) / ulp) <= 2.0
    special = ~normal
    assert np.array_equal(r[special], ref[special]) or np.allclose(r[special], ref[special], rtol=1e-15, equal_nan=True)


@pytest.mark.parametrize("w_orth_type", [None, "cbgs", "scbgs", "bgs"])
@pytest.mark.parametrize("use_b", [False, True])
def test_orthonormalize(ctx, use_b, w_orth_type):
    """B-orthonormalisation of W against B-orthonormal V, every w_orth_type variant:
    orthonormal to 1e-12, the dependent column dropped, the inputs in the span."""
    Aa, Bb = P.fem_q1_cube(12)
    B = Bb if use_b else None
    n = Aa.n
    rng = np.random.default_rng(8)
    k0, k = 9, 12
    V = rng.standard_normal((n, k0 + k))
    V[:, k0 + 5] = V[:, k0 + 2] * 2 - V[:, 3]          # dependent on earlier columns
    Bs = B.to_scipy() if B is not None else None
    # make the first k0 columns B-orthonormal on the host
    Q = V[:, :k0].copy()
    M = Q.T @ (Bs @ Q if Bs is not None else Q)
    L = np.linalg.cholesky(M)
    V[:, :k0] = np.linalg.solve(L, Q.T).T
    v = ctx.multivec(n, k0 + k, V)
    dB = ctx.matrix(B) if B is not None else None
    end = G.orthonormalize(v, k0, k0 + k, dB, w_orth_type=w_orth_type)
    assert end == k0 + k - 1                             # the dependent column was deflated
    Q = v.download()[:, :end]
    BQ = Bs @ Q if Bs is not None else Q
    assert np.max(np.abs(Q.T @ BQ - np.eye(end))) < 1e-12
    # span of the kept columns contains the independent inputs
    keep = [c for c in range(k0 + k) if c != k0 + 5]
    coeffs = Q.T @ (Bs @ V[:, keep] if Bs is not None else V[:, keep])
    resid = V[:, keep] - Q @ coeffs
    assert np.max(np.abs(resid)) / np.max(np.abs(V)) < 1e-10


def test_matrix_csr_validation(ctx):
    A, _ = P.laplace2d(5, 5)
    bad = P.CSR(A.rowptr.copy(), A.col.copy(), A.val.copy())
    bad.col[3] = 999
    with pytest.raises(G.GcgeGpuError) as e:
        ctx.matrix(bad)
    assert e.value.status == 4
    bad2 = P.CSR(A.rowptr.copy(), A.col.copy(), A.val.copy())
    bad2.rowptr[4] = bad2.rowptr[5] + 1
    with pytest.raises(G.GcgeGpuError):
        ctx.matrix(bad2)
    bad3 = P.CSR(A.rowptr.copy(), A.col.copy(), A.val.copy())
    bad3.col[-1] = -1                                   # checked on the device after the upload
    with pytest.raises(G.GcgeGpuError) as e:
        ctx.matrix(bad3)
    assert e.value.status == 4
    dA = ctx.matrix(A)                                  # a valid matrix after the rejected ones
    assert dA.n == A.n


def test_range_checks(ctx):
    x, y = ctx.multivec(100, 4), ctx.multivec(100, 4)
    with pytest.raises(G.GcgeGpuError):
        G.multivec_axpby(1.0, x, 0.0, y, (0, 2), (3, 5))


def _block_cg(A, R0, W0, rounds, rate):
    """GCGE_BCG's iteration in numpy: the first `count` columns are iterated, count taken
    over all columns after each round."""
    x, r = W0.copy(), R0 - A @ W0
    rho = np.sum(r * r, axis=0)
    err, p, act = np.sqrt(rho), np.zeros_like(r), r.shape[1]
    beta = np.zeros(r.shape[1])
    for _ in range(rounds):
        if act == 0:
            break
        a = slice(0, act)
        p[:, a] = r[:, a] + beta[a] * p[:, a]
        w = A @ p[:, a]
        alpha = rho[a] / np.sum(p[:, a] * w, axis=0)
        x[:, a] += alpha * p[:, a]
        r[:, a] -= alpha * w
        new = np.sum(r[:, a] ** 2, axis=0)
        beta[a], rho[a] = new / rho[a], new
        act = int(np.sum(np.sqrt(rho) / err >= rate))
    return x, r


@pytest.mark.parametrize("shape,k,rounds,rate", [
    ((1, 1), 1, 2, 1e-3), ((16, 8), 3, 6, 1e-2), ((43, 3), 17, 6, 1e-2), ((30, 30), 150, 5, 1e-2),
    ((100, 100), 10, 8, 1e-3), ((200, 200), 5, 8, 1e-2), ((120, 90), 131, 4, 1e-30), ((300, 280), 33, 5, 1e-30),
    ("graph", 6, 8, 1e-2), ("graph", 40, 4, 1e-30)])
def test_bcg_fp64_on_the_sides_of_its_forms(ctx, shape, k, rounds, rate):
    """One launch for all rounds: fewer rows than a slab, a slab and a row, more columns than
    a chunk, sums by one block and by a block per column, p formed where it is gathered or
    in a pass, rows past the long-row length, columns that leave the active range. The
    matrices have condition numbers of at most 25, so rounding grows by little over
    a few rounds: 1e-11 is four orders above it and far below any wrong term."""
    if shape == "graph":
        A, _ = P.powerlaw_graph(n=9000, seed=12, shift=100.0)
        assert int(np.sum(np.diff(A.rowptr) > 64)) > 20
    else:
        A, _ = P.laplace2d(*shape)
        A = P.CSR.from_scipy(A.to_scipy() + 4.0 * __import__("scipy.sparse").sparse.identity(A.n))
    rng = np.random.default_rng(k)
    R0 = rng.standard_normal((A.n, k)) * np.logspace(0, -3, k)
    R0[:, ::3] = A.to_scipy() @ rng.standard_normal((A.n, (k + 2) // 3))
    W0 = 0.1 * rng.standard_normal((A.n, k))
    dA = ctx.matrix(A)
    out = []
    for _ in range(2):
        r, w = ctx.multivec(A.n, k + 1), ctx.multivec(A.n, k + 3)
        r.upload(R0, 1)
        w.upload(W0, 3)
        G.bcg(dA, r, 1, w, 3, k, cg_max_it=rounds + 1, cg_rate=rate, precision=0)
        out.append((w.download(3, k), r.download(1, k)))
    x, res = _block_cg(A.to_scipy(), R0, W0, rounds, rate)
    assert rel(out[0][0], x) < 1e-11
    assert np.linalg.norm(out[0][1] - res) < 1e-11 * np.linalg.norm(R0)
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("shape,k", [((1, 1), 1), ((43, 3), 3), ((30, 30), 4), ((91, 77), 5), ((91, 77), 13), ((120, 90), 20),
                                     ((300, 280), 33), ((300, 280), 64), ((91, 77), 65), ((91, 77), 130), ((60, 50), 256)])
def test_bcg_mixed_precision_widths(ctx, shape, k):
    """Every width of the FP32 rounds' kernels, a part of a float4 group and of a block of
    column sums included. Condition numbers are at most 25 and nothing leaves the active range:
    six rounds with rows of five entries lose a few hundred units of 2^-24 of the correction
    at most, 2e-5; 1e-4 is above that and far below any wrong term. Twice the same bits."""
    A, _ = P.laplace2d(*shape)
    A = P.CSR.from_scipy(A.to_scipy() + 4.0 * __import__("scipy.sparse").sparse.identity(A.n))
    rng = np.random.default_rng(k)
    R0, W0 = rng.standard_normal((A.n, k)), 0.1 * rng.standard_normal((A.n, k))
    dA = ctx.matrix(A, keep_fp32=True)
    out = []
    for _ in range(2):
        r, w = ctx.multivec(A.n, k, R0), ctx.multivec(A.n, k, W0)
        G.bcg(dA, r, 0, w, 0, k, cg_max_it=7, cg_rate=1e-30, precision=1)
        out.append(w.download())
    x, _ = _block_cg(A.to_scipy(), R0, W0, 6, 1e-30)
    assert np.linalg.norm(out[0] - x) < 1e-4 * np.linalg.norm(x - W0)
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("n,k,dep", [(400, 1, 0), (400, 33, 4), (900, 129, 7), (900, 160, 0), (900, 161, 5), (2500, 250, 9)])
def test_orthonormalize_widths(ctx, n, k, dep):
    """Blocks at the sides of the Cholesky's forms (a warp's columns, all of a block's, the
    widest in shared memory and the first past it), with columns that repeat others: the
    kept ones are orthonormal to a few roundings a row and span the rest."""
    rng = np.random.default_rng(k)
    W0 = rng.standard_normal((n, k))
    for i in range(dep):
        W0[:, k - 1 - 2 * i] = W0[:, i] * 2.0 - W0[:, i + 1]
    w = ctx.multivec(n, k, W0)
    end = G.orthonormalize(w, 0, k)
    assert end == k - dep
    Q = w.download(0, end)
    assert np.max(np.abs(Q.T @ Q - np.eye(end))) < 1e-13
    assert np.linalg.norm(W0 - Q @ (Q.T @ W0)) < 1e-11 * np.linalg.norm(W0)


def test_orthonormalize_wide_block_first_in_a_process():
    """1,600 columns as a process' first block: no earlier, narrower call has raised a limit."""
    import subprocess
    import sys
    code = """
import numpy as np, sys
sys.path[:0] = %r
import gcge_gb300 as G
with G.Context(0) as c:
    n, k = 2000, 1600
    V = np.random.default_rng(2).standard_normal((n, k))
    v = c.multivec(n, k, V)
    assert G.orthonormalize(v, 0, k) == k
    Q = v.download()
assert np.max(np.abs(Q.T @ Q - np.eye(k))) < 1e-11
"""
    r = subprocess.run([sys.executable, "-c", code % sys.path], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]


def test_bcg_fp64_negative_rate_drops_no_column(ctx):
    """cg_rate <= 0: ||r|| / ||r0|| >= cg_rate always holds, so every column runs all rounds, the
    same for 0 and below it."""
    A, _ = P.laplace2d(43, 31)
    dA = ctx.matrix(A)
    R = np.random.default_rng(31).standard_normal((A.n, 9))
    out = []
    for rate in (0.0, -1.0, -1e-3):
        r, w = ctx.multivec(A.n, 9, R), ctx.multivec(A.n, 9)
        G.bcg(dA, r, 0, w, 0, 9, cg_max_it=40, cg_rate=rate)
        out.append(w.download())
    assert np.linalg.norm(A.to_scipy() @ out[0] - R) < 0.5 * np.linalg.norm(R)
    assert np.array_equal(out[1], out[0]) and np.array_equal(out[2], out[0])


def _quotients(kind, num, den):
    import ctypes as C
    lib = G.load()
    num, den = np.ascontiguousarray(num), np.ascontiguousarray(den)
    q = np.zeros_like(num)
    lib.gb_div_check.restype = C.c_int
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert lib.gb_div_check(kind, len(num), p(num), p(den), p(q)) == 0
    with np.errstate(all="ignore"):
        return q, num / den


def _division_operands(rng, count):
    """Significands at random and at both ends, exponents over the whole range and around every
    power that either division's own range ends at; zeros, infinities, NaN and subnormals."""
    sig = np.where(rng.random(count) < 0.2, rng.choice([1.0, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 1.5], count),
                   rng.uniform(1.0, 2.0, count))
    ex = np.where(rng.random(count) < 0.5, rng.integers(-60, 61, count),
                  np.where(rng.random(count) < 0.5, rng.integers(-1022, 1024, count),
                           rng.choice([-900, -700, -600, -450, -300, 300, 450, 600, 700, 900], count) +
                           rng.integers(-2, 3, count)))
    x = rng.choice([-1.0, 1.0], count) * np.ldexp(sig, ex)
    x[:64] = rng.choice([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -1e-310, 2.0 ** -1022, 1.7e308], 64)
    return x


def test_quotient_by_a_known_reciprocal(ctx):
    """The Cholesky inverse divides by a pivot whose reciprocal it has: IEEE division, bit for bit."""
    rng = np.random.default_rng(41)
    q, ref = _quotients(0, _division_operands(rng, 1 << 21), rng.permutation(_division_operands(rng, 1 << 21)))
    assert np.array_equal(q, ref, equal_nan=True)


def test_quotient_of_the_sturm_counts(ctx):
    """The division of the Sturm counts: its value before the one rounding is within 2^-78 of the quotient, so it is
    IEEE division but where the quotient lies that close to the middle of two doubles; and never
    decreasing as the divisor falls through neighbouring doubles, which the bisection relies on."""
    from fractions import Fraction
    rng = np.random.default_rng(42)
    num, den = _division_operands(rng, 1 << 21), rng.permutation(_division_operands(rng, 1 << 21))
    q, ref = _quotients(1, num, den)
    bad = np.flatnonzero(~((q == ref) | (np.isnan(q) & np.isnan(ref))))
    # 2^-25 of random significands are expected there; of the chosen ones 1 / (2 - 2^-52) lies 2^-106 from a middle
    assert np.sum(np.abs(np.frexp(den[bad])[0]) != 1.0 - 2.0 ** -53) <= 16
    for i in bad:
        mid = (Fraction(float(q[i])) + Fraction(float(ref[i]))) / 2
        ex = Fraction(float(num[i])) / Fraction(float(den[i]))
        assert abs(ex / mid - 1) <= Fraction(1, 2 ** 78)
    for e in (0, -40, 449, 450, 451, -449, -450, -451):
        n1 = float(np.ldexp(rng.uniform(1.0, 2.0), e))
        d = np.ldexp(2.0 - np.arange(1 << 16) * 2.0 ** -52, e // 3)   # falls, and passes a power of two
        d = np.concatenate([d, np.ldexp(1.0 + np.arange(1 << 15, -(1 << 15), -1) * 2.0 ** -53, e)])
        for part in (d[:1 << 16], d[1 << 16:]):
            q, _ = _quotients(1, np.full(len(part), n1), part)
            assert np.all(np.diff(q) >= 0)


@pytest.mark.parametrize("op", ["bcg", "grad", "adjoint", "widths"])
def test_large_workspaces_go_back_after_the_call(op):
    """Single calls' workspaces are kept for later ones up to 256 MiB in all: after a call that needs
    more, or calls of growing widths, the device has the rest of its memory again (other buffers of
    the calls: within 300 MiB)."""
    torch = pytest.importorskip("torch")
    with G.Context(0) as c:
        A, _ = P.laplace2d(1200, 1000)
        n = A.n
        if op == "bcg":
            dA, x, y = c.matrix(A), c.multivec(n, 64), c.multivec(n, 64)
            run = lambda: G.bcg(dA, x, 0, y, 0, 64, cg_max_it=2)  # noqa: E731
        elif op == "widths":
            dA, x, y = c.matrix(A), c.multivec(n, 12), c.multivec(n, 12)
            run = lambda: [G.bcg(dA, x, 0, y, 0, k, cg_max_it=2) for k in (4, 8, 12)]  # noqa: E731
        elif op == "grad":
            import scipy.sparse as sp
            M = P.CSR.from_scipy(sp.csr_matrix(sp.diags([np.ones(n)] * 41, range(41), shape=(n, n))))
            dA, x = c.matrix(M), c.multivec(n, 2)
            run = lambda: G.pattern_grad(dA, x, 0, x, 0, 1, [1.0], M.nnz)  # noqa: E731
        else:
            dA, x, y = c.matrix(A), c.multivec(n, 40), c.multivec(n, 2)
            dB = c.matrix(P.CSR(np.arange(n + 1), np.arange(n), np.ones(n)))
            run = lambda: G.eigvec_adjoint(dA, dB, x, 40, np.arange(40.0), 0, y, 0, y, 1, max_it=1)  # noqa: E731
        c.sync()
        before = torch.cuda.mem_get_info()[0]
        run()
        c.sync()
        assert before - torch.cuda.mem_get_info()[0] <= 300 << 20


@pytest.mark.parametrize("items,k", [(152, 2), (304, 3), (305, 3), (456, 2), (457, 5), (608, 1), (609, 2), (304, 33), (500, 9)])
def test_bcg_fp64_two_or_three_blocks_an_sm(ctx, items, k):
    """Row slabs on either side of where two blocks an SM take a wave more than three (304 and 608 slabs of
    128 rows on 152 SMs), the last slab of one row: as test_bcg_fp64_on_the_sides_of_its_forms."""
    test_bcg_fp64_on_the_sides_of_its_forms(ctx, (128 * (items - 1) + 1, 1), k, 4, 1e-30)
