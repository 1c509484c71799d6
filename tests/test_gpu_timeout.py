"""The failure path of the kernels that wait, made to run on purpose: the tensor-core
kernels, and those with barriers of their own grid (at the end).

Every mbarrier wait of the tcgen05 Gram and linear-combination kernels is
bounded (1 s of %globaltimer). GCGE_GPU_TestStallTensorWait makes the next
tensor-core launch's MMA-issuing thread wait for an arrival that cannot come,
so that wait runs out: the kernel must return (no hang), report
GCGE_GPU_ERR_TIMEOUT through GCGE_GPU_Synchronize, leave later tensor-core
launches on that context without effect, and free its TMEM, so that a fresh
context on the same GPU computes correct results afterwards. No fault, trap or
endless loop is involved: the only change is one wait that nothing satisfies."""
import time

import numpy as np
import pytest

import gcge_gb300 as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op", ["lincomb", "gram"])
def test_bounded_tensor_wait_runs_out_and_recovers(op):
    rng = np.random.default_rng(11)
    n, k1, k2 = 262144, 64, 48
    X = rng.standard_normal((n, k1))
    W = rng.standard_normal((n, k2))
    Cm = np.asfortranarray(rng.standard_normal((k1, k2)))
    exact_lc = X @ Cm
    exact_gram = X.T @ W

    def run(ctx, sentinel=False):
        mx, mw = ctx.multivec(n, k1, X), ctx.multivec(n, k2, W)
        Y = ctx.multivec(n, k2, np.full((n, k2), np.nan) if sentinel else None)
        if op == "lincomb":
            G.multivec_linear_comb(mx, Y, (0, 0), (k1, k2), Cm.ravel(order="F"), k1)
            return Y.download()
        a = np.full(k1 * k2, np.nan)
        ctx.lib.GCGE_GPU_MultiVecInnerProd(mx.h, mw.h, a.ctypes.data, b"nonsym", G._ints(0, 0), G._ints(k1, k2), k1)
        return a.reshape(k2, k1).T

    ctx = G.Context(0)
    try:
        assert ctx.lib.GCGE_GPU_TestStallTensorWait(ctx.h, 1) == 0
        t0 = time.time()
        try:
            run(ctx)
        except G.GcgeGpuError as e:                   # the call may already see the status
            assert e.status == G.ERR_TIMEOUT
        st = ctx.lib.GCGE_GPU_Synchronize(ctx.h)
        elapsed = time.time() - t0
        assert st == G.ERR_TIMEOUT, st
        assert elapsed < 30.0, elapsed               # bounded: a few 1 s waits, not a hang
        # later tensor-core launches on the failed context do no work
        if op == "lincomb":
            try:
                out = run(ctx, sentinel=True)
                assert np.all(np.isnan(out))
            except G.GcgeGpuError as e:
                assert e.status == G.ERR_TIMEOUT
        assert ctx.lib.GCGE_GPU_Synchronize(ctx.h) == G.ERR_TIMEOUT
    finally:
        ctx.close()
    # TMEM was released: a fresh context on the same GPU runs the tensor-core kernels
    ctx2 = G.Context(0)
    try:
        out = run(ctx2)
        assert ctx2.lib.GCGE_GPU_Synchronize(ctx2.h) == 0
    finally:
        ctx2.close()
    ref = exact_lc if op == "lincomb" else exact_gram
    assert np.max(np.abs(out - ref)) <= 1e-13 * np.max(np.abs(ref))


@pytest.mark.parametrize("op,n,k", [("bcg", 900, 1), ("bcg", 30000, 40), ("hook", 1600, 1), ("adjoint", 2500, 5)])
def test_bounded_grid_wait_runs_out_and_is_reported(op, n, k):
    """One block, sums by the last block to arrive, sums by a block a column: the stalled call
    returns GCGE_GPU_ERR_TIMEOUT, and so does the next on that context; a fresh context solves."""
    import ctypes as C

    from gcge_gb300 import problems as P
    A, _ = P.laplace2d(50, n // 50)
    rhs = np.random.default_rng(5).standard_normal((n, k))
    x = np.linalg.qr(np.random.default_rng(6).standard_normal((n, k)))[0]

    def run(ctx):
        dA, b, y = ctx.matrix(A), ctx.multivec(n, k, rhs), ctx.multivec(n, k)
        if op == "bcg":
            st = ctx.lib.GCGE_GPU_BCG(dA.h, b.h, 0, y.h, 0, k, 2000, 1e-10, 0)
        elif op == "adjoint":
            ev, xd = np.arange(1.0, k + 1), ctx.multivec(n, k, x)
            st = ctx.lib.GCGE_GPU_EigvecAdjoint(dA.h, None, xd.h, k, ev.ctypes.data, 0, b.h, 0, y.h, 0,
                                                1e-10, 1e-10, 50, None)
        else:
            from test_gpu_ops_table import OpsTable, mv_create, mv_download, mv_upload
            tab = OpsTable()
            assert ctx.lib.GCGE_GPU_SetOps(ctx.h, C.byref(tab)) == 0
            assert ctx.lib.GCGE_GPU_OpsSetLinearSolver(C.byref(tab), 1, 2000, 1e-10) == 0
            h = mv_create(ctx, tab, dA, 2)
            mv_upload(ctx, h, np.hstack([rhs, 0 * rhs]))
            C.CFUNCTYPE(None, *4 * [C.c_void_p])(tab.LinearSolver)(dA.h, h[0], h[1], C.cast(C.byref(tab), C.c_void_p))
            st = ctx.last_error()
            out = mv_download(ctx, h, 2, n)[:, 1:]
            tab.MultiVecDestroy(C.byref(h), 2, None)
            assert ctx.lib.GCGE_GPU_OpsSetLinearSolver(C.byref(tab), 0, 20, 1e-2) == 0
            return st, out
        return st, y.download()

    with G.Context(0) as ctx:
        assert ctx.lib.GCGE_GPU_TestStallGridWait(ctx.h, 1) == 0
        t0 = time.time()
        assert run(ctx)[0] == G.ERR_TIMEOUT
        assert time.time() - t0 < 10.0
        assert run(ctx)[0] == G.ERR_TIMEOUT
        assert ctx.lib.GCGE_GPU_Synchronize(ctx.h) == G.ERR_TIMEOUT
    with G.Context(0) as ctx:
        st, out = run(ctx)
        assert st == 0
        if op != "adjoint":
            assert np.linalg.norm(A.to_scipy() @ out - rhs) <= 1e-6 * np.linalg.norm(rhs)
