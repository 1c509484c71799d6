"""Workloads of the GCGE CSR eigensolver on one GPU, as a program that uses the package runs them.

A case is a dict of plain values; its "kind" names the call that the program makes:

* ``solve``      ``Context.solve``: matrices resident on the device, eigenpairs returned to the host.
* ``solve_host`` ``Context.solve_host``: CSR arrays and results in host memory (upload, solve, download).
* ``project``    a Rayleigh-Ritz projection, H = V^T (A W): ``mat_dot_multivec`` and ``multivec_inner_prod``.
* ``gram``       ``GCGE_GPU_InnerProdNoAlloc`` on the caller's own device memory and stream.
* ``cg``         ``bcg``: block CG as the linear solver of an outer iteration of the caller's.
* ``orth``       ``orthonormalize``: B-orthonormal block against a basis that is B-orthonormal already.
* ``grad``       ``pattern_grad``: the gradient of a sum of eigenvalues on the matrix's entries.
* ``adjoint``    ``eigvec_adjoint``: the adjoint of a functional of one eigenvector.
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gcge-1.0_gb300"))
import gcge_gb300 as G  # noqa: E402
from gcge_gb300 import problems as P  # noqa: E402

# the sides of the brick: far enough from equal that no two of its low modes coincide
SIDES = (1.0, 1.14, 1.235)
PROBLEMS = ("plane", "brick", "cells", "graph")


def listed():
    return [
        # the first program that anyone runs: a 2-D operator on 900 unknowns, six modes
        {"name": "solve_plane30", "kind": "solve", "problem": "plane", "size": 30, "nev": 6, "block": 6, "precision": 0, "tol": 1e-10},
        # the small configuration: a 100 x 100 grid, ten modes, plain FP64
        {"name": "solve_plane100", "kind": "solve", "problem": "plane", "size": 100, "nev": 10, "block": 10, "precision": 0, "tol": 1e-10},
        # a FEM pencil of middle size handed over and returned in host memory, plain FP64
        {"name": "host_brick40", "kind": "solve_host", "problem": "brick", "size": 40, "nev": 20, "block": 20, "precision": 0, "tol": 1e-10},
        # the headline configuration: Q1 FEM on 96^3 elements of a brick, 50 modes, block 64, mixed precision
        {"name": "solve_brick96", "kind": "solve", "problem": "brick", "size": 96, "nev": 50, "block": 64, "precision": 1, "tol": 1e-10},
        # heterogeneous diffusion on 3-D cells with a lumped mass, mixed precision
        {"name": "solve_cells48", "kind": "solve", "problem": "cells", "size": 48, "nev": 20, "block": 28, "precision": 1, "tol": 1e-10},
        # one Rayleigh-Ritz projection of a caller's own outer iteration, at the headline's widths
        {"name": "project_brick64", "kind": "project", "problem": "brick", "size": 64, "k1": 178, "k2": 64},
        # a Gram block in memory of the caller's pool
        {"name": "gram_262144", "kind": "gram", "n": 262144, "k1": 178, "k2": 64},
        # block CG for 32 right-hand sides, plain FP64
        {"name": "cg_cells64", "kind": "cg", "problem": "cells", "size": 64, "k": 32, "rounds": 20},
        # the same on the Laplacian of a power-law graph, rows of four entries to hundreds
        {"name": "cg_graph100k", "kind": "cg", "problem": "graph", "size": 100000, "k": 44, "rounds": 15},
        # a block of 64 new directions against a basis of 114
        {"name": "orth_brick64", "kind": "orth", "problem": "brick", "size": 64, "k1": 114, "k2": 64},
        # the gradient of the sum of the 20 smallest eigenvalues on a 512 x 512 grid
        {"name": "grad_plane512", "kind": "grad", "problem": "plane", "size": 512, "k": 20},
        # the adjoint of a functional of the lowest mode, with the modes that the solve left
        {"name": "adjoint_plane128", "kind": "adjoint", "problem": "plane", "size": 128, "k": 10},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, problem, lo, hi):
    """A size of `problem` with about lo to hi unknowns."""
    n = _log(rng, lo, hi)
    if problem == "graph":
        return n
    return int(round(n ** (0.5 if problem == "plane" else 1 / 3))) + (1 if problem == "brick" else 0)


def draw(rng):
    kind = rng.choice(("solve", "solve", "solve_host", "project", "gram", "cg", "orth", "grad", "adjoint"))
    problem = rng.choice(PROBLEMS)
    if kind in ("solve", "solve_host") and problem == "graph":
        problem = "brick"  # a graph's low modes lie so close together that the tolerance does not tell them apart
    if kind in ("solve", "solve_host"):
        nev = _log(rng, 4, 32)
        hi = {"plane": 12000, "brick": 250000, "cells": 110000}[problem]
        return {"kind": kind, "problem": problem, "size": _size(rng, problem, 900, hi), "nev": nev, "block": nev + rng.choice((0, 0, nev // 4)),
                "precision": rng.choice((0, 0, 1, 1, 2)), "tol": 1e-10}
    if kind == "gram":
        return {"kind": kind, "n": _log(rng, 1000, 600000), "k1": _log(rng, 3, 256), "k2": _log(rng, 3, 128)}
    if kind == "project":
        return {"kind": kind, "problem": problem, "size": _size(rng, problem, 1000, 250000), "k1": _log(rng, 8, 200), "k2": _log(rng, 4, 80)}
    if kind == "cg":
        return {"kind": kind, "problem": problem, "size": _size(rng, problem, 1000, 250000), "k": _log(rng, 2, 64), "rounds": rng.randint(5, 25)}
    if kind == "orth":
        return {"kind": kind, "problem": problem, "size": _size(rng, problem, 1000, 250000), "k1": _log(rng, 6, 130), "k2": _log(rng, 4, 70)}
    if kind == "grad":
        return {"kind": kind, "problem": problem, "size": _size(rng, problem, 1000, 250000), "k": _log(rng, 1, 100)}
    return {"kind": kind, "problem": "plane", "size": rng.randint(30, 130), "k": rng.randint(4, 12)}


# ---- inputs


def _axis(ne, d, seed):
    """1-D linear-element stiffness and mass on ne unequal intervals of [0, SIDES[d]], ends fixed: their three diagonals."""
    h = np.random.default_rng([seed, d]).uniform(0.95, 1.05, ne)
    h *= SIDES[d] / h.sum()
    a, b = h[:-1], h[1:]
    K = np.stack([-1 / a, 1 / a + 1 / b, -1 / b])
    M = np.stack([a / 6, (a + b) / 3, b / 6])
    return K, M


def _tensor_csr(N, terms):
    """The CSR matrix sum_t X_t (x) Y_t (x) Z_t of tridiagonal factors on N^3 unknowns (27 entries a row inside)."""
    i = np.arange(N)
    ok = np.stack([i > 0, i >= 0, i < N - 1], 1)
    keep = ok[:, None, None, :, None, None] & ok[None, :, None, None, :, None] & ok[None, None, :, None, None, :]
    val = sum(x.T[:, None, None, :, None, None] * y.T[None, :, None, None, :, None] * z.T[None, None, :, None, None, :] for x, y, z in terms)
    d = np.arange(-1, 2)
    row = (i[:, None, None] * N + i[None, :, None]) * N + i[None, None, :]
    off = (d[:, None, None] * N + d[None, :, None]) * N + d[None, None, :]
    col = (row[..., None, None, None] + off).astype(np.int32)
    rp = np.concatenate([[0], np.cumsum(keep.reshape(N ** 3, 27).sum(1))])
    return P.CSR(rp, col[keep], val[keep])


def _brick(ne, seed):
    (Kx, Mx), (Ky, My), (Kz, Mz) = (_axis(ne, d, seed) for d in range(3))
    A = _tensor_csr(ne - 1, [(Kx, My, Mz), (Mx, Ky, Mz), (Mx, My, Kz)])
    B = _tensor_csr(ne - 1, [(Mx, My, Mz)])
    return A, B


def _pencil(problem, size, seed):
    if problem == "plane":
        return P.varcoef2d(size, seed=seed)
    if problem == "cells":
        return P.varcoef3d(size, seed=seed)
    if problem == "graph":
        return P.powerlaw_graph(size, seed=seed)
    return _brick(size, seed)


@functools.lru_cache(maxsize=1)
def _context():
    return G.Context(0)


def _tall(n, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(n, k, generator=g, device="cuda", dtype=torch.float64)


def _smooth(n, k, seed):
    """Columns like the modes of a solve: oscillations along the rows of growing frequency, and noise well below them."""
    t = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n
    f = torch.arange(1, k + 1, device="cuda", dtype=torch.float64)
    return torch.sin(math.pi * t[:, None] * f) * math.sqrt(2.0 / n) + 1e-3 / math.sqrt(n) * _tall(n, k, seed)


def _pinned(k, n):
    return torch.empty(k, n, dtype=torch.float64, pin_memory=True)


def _download(mv, col, k, out):
    """Columns col .. col + k of a multivector into the caller's page-locked buffer."""
    if mv.lib.GCGE_GPU_MultiVecDownload(mv.h, col, k, ctypes.c_void_p(out.data_ptr())):
        raise RuntimeError("GCGE_GPU_MultiVecDownload")
    return out


def prepare(case, seed):
    c = dict(case)
    s = {"case": c}
    kind = c["kind"]
    if kind == "gram":
        s["V"], s["W"] = _smooth(c["n"], c["k1"], 2 * seed), _tall(c["n"], c["k2"], 2 * seed + 1)
        s["a"] = torch.zeros(c["k2"], c["k1"], device="cuda", dtype=torch.float64)
        return s
    ctx = s["ctx"] = _context()
    A, B = _pencil(c["problem"], c["size"], seed)
    n = A.n
    if kind == "solve_host":
        s["A"], s["B"] = A, B
    elif kind != "orth":
        s["A"] = ctx.matrix(A, keep_fp32=kind == "solve" and c["precision"] > 0)
    if kind in ("solve", "solve_host"):
        s["params"] = ctx.params(nev=c["nev"], block_size=c["block"], precision=c["precision"], ev_tol=c["tol"], conv_type="BR",
                                 ev_max_it=500, seed=seed + 1)
        if kind == "solve":
            s["B"] = ctx.matrix(B) if B is not None else None
            s["X"] = ctx.multivec(n, c["nev"])
    elif kind == "project":
        s["V"] = ctx.multivec(n, c["k1"], _smooth(n, c["k1"], 2 * seed).cpu().numpy())
        s["W"] = ctx.multivec(n, c["k2"], _tall(n, c["k2"], 2 * seed + 1).cpu().numpy())
        s["AW"] = ctx.multivec(n, c["k2"])
    elif kind == "cg":
        k = c["k"]
        s["b"] = ctx.multivec(n, k, _tall(n, k, seed).cpu().numpy())
        s["x0"] = ctx.multivec(n, k, _smooth(n, k, seed + 1).cpu().numpy())
        s["r"], s["x"], s["out"] = ctx.multivec(n, k), ctx.multivec(n, k), _pinned(k, n)
    elif kind == "orth":
        k1, k2 = c["k1"], c["k2"]
        s["B"] = ctx.matrix(B) if B is not None else None
        s["V"] = ctx.multivec(n, k1 + k2, _smooth(n, k1 + k2, seed).cpu().numpy())
        if G.orthonormalize(s["V"], 0, k1, s["B"]) != k1:
            raise RuntimeError("the basis lost a column")
        s["W"] = ctx.multivec(n, k2, (_smooth(n, k2, 2 * seed) + _tall(n, k2, 2 * seed + 1)).cpu().numpy())
        s["out"] = _pinned(k2, n)
    elif kind == "grad":
        s["X"] = ctx.multivec(n, c["k"], _smooth(n, c["k"], seed).cpu().numpy())
        s["scale"], s["nnz"] = np.linspace(1.0, 2.0, c["k"]), A.nnz
    else:
        k = c["k"]
        p = ctx.params(nev=k, block_size=k, ev_tol=1e-11, conv_type="BR", ev_max_it=500, seed=seed + 1)
        s["X"] = ctx.multivec(n, k)
        s["eval"], X, _ = ctx.solve(s["A"], None, p, evec=s["X"])
        w = np.random.default_rng([seed, 9]).uniform(0.0, 1.0, n)
        s["G"] = ctx.multivec(n, 1, 2.0 * w * X[:, 0])
        s["MU"] = ctx.multivec(n, 1)
    return s


# ---- one pass


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "gram":
        V, W, a = s["V"], s["W"], s["a"]
        st = G.load().GCGE_GPU_InnerProdNoAlloc(c["n"], c["k1"], c["k2"], V.data_ptr(), V.stride(0), W.data_ptr(), W.stride(0),
                                                a.data_ptr(), c["k1"], 0, torch.cuda.current_stream().cuda_stream)
        if st:
            raise RuntimeError("GCGE_GPU_InnerProdNoAlloc: status %d" % st)
        return a
    ctx = s["ctx"]
    if kind == "solve":
        ev, X, _ = ctx.solve(s["A"], s["B"], s["params"], evec=s["X"])
        return {"eval": ev, "evec": X}
    if kind == "solve_host":
        ev, X, _ = ctx.solve_host(s["A"], s["B"], s["params"])
        return {"eval": ev, "evec": X}
    if kind == "project":
        k1, k2 = c["k1"], c["k2"]
        G.mat_dot_multivec(s["A"], s["W"], s["AW"], (0, 0), (k2, k2))
        return G.multivec_inner_prod(s["V"], s["AW"], (0, 0), (k1, k2), k1)
    if kind == "cg":
        k = c["k"]
        G.multivec_axpby(1.0, s["b"], 0.0, s["r"], (0, 0), (k, k))
        G.multivec_axpby(1.0, s["x0"], 0.0, s["x"], (0, 0), (k, k))
        G.bcg(s["A"], s["r"], 0, s["x"], 0, k, cg_max_it=c["rounds"] + 1, cg_rate=1e-6)
        return _download(s["x"], 0, k, s["out"])
    if kind == "orth":
        k1, k2 = c["k1"], c["k2"]
        G.multivec_axpby(1.0, s["W"], 0.0, s["V"], (0, k1), (k2, k1 + k2))
        end = G.orthonormalize(s["V"], k1, k1 + k2, s["B"])
        return {"end": end, "block": _download(s["V"], k1, k2, s["out"])}
    if kind == "grad":
        return G.pattern_grad(s["A"], s["X"], 0, s["X"], 0, c["k"], s["scale"], s["nnz"])
    G.eigvec_adjoint(s["A"], None, s["X"], c["k"], s["eval"], 0, s["G"], 0, s["MU"], 0, tol=1e-12)
    return {"mu": s["MU"].download(0, 1)}


# ---- what a pass cannot do without


def _counts(problem, size):
    """(unknowns, entries of A, entries of B) of a problem, the graph's entries by its mean degree."""
    if problem == "graph":
        return size, int(11.2 * size), size
    if problem == "plane":
        return size ** 2, 5 * size ** 2, 0
    if problem == "cells":
        return size ** 3, 7 * size ** 3, size ** 3
    return (size - 1) ** 3, (3 * (size - 1) - 2) ** 3, (3 * (size - 1) - 2) ** 3


def work(case):
    c = case
    kind = c["kind"]
    if kind == "gram":
        return {"bytes": 8.0 * (c["n"] * (c["k1"] + c["k2"]) + c["k1"] * c["k2"]), "flops": 2.0 * c["n"] * c["k1"] * c["k2"]}
    n, za, zb = _counts(c["problem"], c["size"])
    a, b = 12.0 * za + 4.0 * n, 12.0 * zb + 4.0 * n
    if kind in ("solve", "solve_host"):
        # ten outer iterations are the least that any of these takes; each reads A and B for the
        # block and its residual, takes a few inner steps and recombines the basis once
        nev, k = c["nev"], c["block"]
        m = nev + 2 * k
        v = 4.0 if c["precision"] else 8.0
        it, steps = 10, 4
        per = 2 * (a + b) + steps * (a + 6 * v * n * k) + 8.0 * n * (3 * m + 4 * k)
        fl = 4.0 * (za + zb) * k + steps * (2.0 * za * k + 10.0 * n * k) + 6.0 * n * m * k
        return {"bytes": it * per + 8.0 * n * nev, "flops": it * fl}
    if kind == "project":
        return {"bytes": a + 8.0 * n * (c["k1"] + c["k2"]) + 8.0 * c["k1"] * c["k2"], "flops": 2.0 * za * c["k2"] + 2.0 * n * c["k1"] * c["k2"]}
    if kind == "cg":
        # every step takes in the matrix once, and each of x, r, p and A p of the block once
        return {"bytes": c["rounds"] * (a + 8.0 * 7 * n * c["k"]) + 16.0 * n * c["k"], "flops": c["rounds"] * (2.0 * za + 12.0 * n) * c["k"]}
    if kind == "orth":
        k1, k2 = c["k1"], c["k2"]
        return {"bytes": b + 8.0 * n * (k1 + 2 * k2), "flops": 2.0 * zb * k2 + 4.0 * n * k1 * k2 + 4.0 * n * k2 * k2}
    if kind == "grad":
        return {"bytes": 12.0 * za + 8.0 * n * c["k"], "flops": 2.0 * za * c["k"]}
    it = c["size"]
    return {"bytes": it * (a + 8.0 * n * (6 + 2 * c["k"])), "flops": it * (2.0 * za + 4.0 * n * c["k"] + 10.0 * n)}


# ---- the same in plain 64 bits


def _dense(A):
    r = np.repeat(np.arange(A.n), np.diff(A.rowptr))
    D = torch.zeros(A.n, A.n, dtype=torch.float64, device="cuda")
    D.index_put_((torch.from_numpy(r).cuda(), torch.from_numpy(A.col).long().cuda()), torch.from_numpy(A.val).cuda(), accumulate=True)
    return D


def _apply(A, X):
    """A X on the device, by runs of rows' entries."""
    if A is None:
        return X
    r = torch.from_numpy(np.repeat(np.arange(A.n), np.diff(A.rowptr))).cuda()
    col, val = torch.from_numpy(A.col).long().cuda(), torch.from_numpy(A.val).cuda()
    Y = torch.zeros_like(X)
    step = max(1, (1 << 27) // X.shape[1])
    for e in range(0, A.nnz, step):
        f = min(A.nnz, e + step)
        Y.index_add_(0, r[e:f], val[e:f, None] * X[col[e:f]])
    return Y


def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind == "gram":
        return _tall(c["n"], c["k2"], 2 * seed + 1).T @ _smooth(c["n"], c["k1"], 2 * seed)
    if kind in ("cg", "adjoint"):
        return None
    if kind in ("solve", "solve_host") and c["problem"] == "brick":
        mu = []
        for d in range(3):
            K, M = (np.diag(t[1]) + np.diag(t[2][:-1], 1) + np.diag(t[0][1:], -1) for t in _axis(c["size"], d, seed))
            L = np.linalg.inv(np.linalg.cholesky(M))
            mu.append(np.linalg.eigvalsh(L @ K @ L.T)[: c["nev"] + 2])
        s = (mu[0][:, None, None] + mu[1][None, :, None] + mu[2][None, None, :]).ravel()
        return {"eval": np.sort(s)[: c["nev"]], "evec": None}
    A, B = _pencil(c["problem"], c["size"], seed)
    if kind in ("solve", "solve_host"):
        if A.n > 6000:
            return None
        D = _dense(A)
        if B is not None:
            w = 1.0 / torch.sqrt(torch.from_numpy(B.val).cuda())
            D = w[:, None] * D * w
        return {"eval": torch.linalg.eigvalsh(D)[: c["nev"]].cpu().numpy(), "evec": None}
    if kind == "project":
        H = _apply(A, _tall(A.n, c["k2"], 2 * seed + 1)).T @ _smooth(A.n, c["k1"], 2 * seed)
        return H.reshape(-1).cpu().numpy()
    if kind == "grad":
        X = _smooth(A.n, c["k"], seed)
        XS = X * torch.linspace(1.0, 2.0, c["k"], dtype=torch.float64, device="cuda")
        r = torch.from_numpy(np.repeat(np.arange(A.n), np.diff(A.rowptr))).cuda()
        col = torch.from_numpy(A.col).long().cuda()
        return (XS[r] * X[col]).sum(1).cpu().numpy()
    # orth: the basis, then W off it, each by Cholesky twice
    k1, k2 = c["k1"], c["k2"]

    def chol(Q):
        for _ in range(2):
            R = torch.linalg.cholesky(Q.T @ _apply(B, Q)).T
            Q = torch.linalg.solve_triangular(R, Q, upper=True, left=False)
        return Q

    V = chol(_smooth(A.n, k1 + k2, seed)[:, :k1].contiguous())
    W = _smooth(A.n, k2, 2 * seed) + _tall(A.n, k2, 2 * seed + 1)
    for _ in range(2):
        W = W - V @ (V.T @ _apply(B, W))
    return {"end": None, "block": chol(W).T.cpu()}
