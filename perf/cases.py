"""The workloads a user of the framework runs, as cases that can be timed and compared.

Every case is a sparse system on a tensor grid, taken through the public calls: ``ParTree`` (``partition``,
``assemble``, ``factorize``), the preconditioner apply, ``dist_gmres`` and ``block_gmres``.  The fields of a case:

  op         "solve":   assemble + factorize + GMRES on a host right-hand side (the driver's whole run after the
                        ordering, and what a time step with new values repeats)
             "oneshot": assemble + factorize + one direct solve (the driver's first check, tight tolerances)
             "gmres":   GMRES for a new right-hand side on a factorized tree
             "apply":   one preconditioner apply on a device vector (what an outer Krylov method of the user calls)
             "block":   assemble + factorize + block GMRES on several right-hand sides
  matrix     "lapl" (2d+1-point Laplacian), "diff" (lognormal diffusion), "conv" (2D upwinded convection-diffusion)
  n, d       grid edge and dimension (n^d unknowns); levels: depth of the nested dissection
  tol, skip  sparsification tolerance; levels without sparsification at the bottom
  mixed      float factors with FP64 Krylov loop and pivoting (the FP64 method otherwise)
  learned    ranks from the shipped rank model (the column-pivoted QR of every interface otherwise)
  rtol, nrhs GMRES tolerance, right-hand sides

Inputs (coefficient field, right-hand side) are made from the seed.  The tree with its ordering is what a program
keeps between solves; factors are made inside the pass except where the case is about a factorized tree.
"""
import math

import numpy as np
import torch

from pspaqr_public_b200 import ParTree, dist_gmres, scale_columns
from pspaqr_public_b200.tree import block_gmres, load_rank_model


def _levels(n, d):
    """Leaves of about 128 unknowns: 6 levels at 64^2, 9 at 32^3, 12 at 64^3, 14 at 1024^2."""
    return max(3, int(round(math.log2(n ** d / 128.0))) + 1)


def _case(op, matrix, n, d, tol=1e-2, mixed=False, learned=False, skip=0, rtol=1e-12, nrhs=1, name=None):
    c = dict(op=op, matrix=matrix, n=n, d=d, levels=_levels(n, d), tol=tol, skip=skip, mixed=mixed, learned=learned,
             rtol=rtol, nrhs=nrhs)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: one apply of a small 2D preconditioner, all launch latency
        _case("apply", "lapl", 64, 2, name="apply_lapl2d_64"),
        # a small 2D solve, everything in it, to the driver's GMRES tolerance
        _case("solve", "lapl", 64, 2, name="solve_lapl2d_64"),
        # odd edge, nonsymmetric, the lowest levels not sparsified: a ragged mid-size 2D problem
        _case("solve", "conv", 187, 2, skip=1, name="solve_conv2d_187_skip1"),
        # odd 3D edge, plain FP64
        _case("solve", "diff", 25, 3, name="solve_diff3d_25"),
        # tight tolerance: large kept ranks, used as a direct solver
        _case("oneshot", "diff", 32, 3, tol=1e-3, name="oneshot_diff3d_32_t1e-3"),
        # odd 3D edge, mixed precision with the pivoted QR of every interface
        _case("solve", "diff", 45, 3, mixed=True, name="solve_diff3d_45_mixed"),
        # 16 right-hand sides as one block on a large nonsymmetric 2D problem, mixed precision, learned ranks
        _case("block", "conv", 384, 2, mixed=True, learned=True, nrhs=16, name="block_conv2d_384_mixed_learned"),
        # the apply of a large FP64 factorization, memory-bound
        _case("apply", "diff", 48, 3, name="apply_diff3d_48"),
        # new right-hand side on kept float factors
        _case("gmres", "diff", 48, 3, mixed=True, learned=True, name="gmres_diff3d_48_mixed_learned"),
        # the benchmark's workload: mixed precision, learned ranks
        _case("solve", "diff", 64, 3, mixed=True, learned=True, name="solve_diff3d_64_mixed_learned"),
        # the plain FP64 method at the benchmark's size: the largest run
        _case("solve", "lapl", 64, 3, name="solve_lapl3d_64"),
    ]


def draw(rng):
    op = rng.choice(["solve", "solve", "solve", "oneshot", "gmres", "apply", "block"])
    d = rng.choice([2, 3])
    lo, hi = (33, 400) if d == 2 else (12, 52)
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    matrix = rng.choice(["lapl", "diff", "conv"] if d == 2 else ["lapl", "diff"])
    mixed = op in ("block", "gmres") or (op == "solve" and rng.random() < 0.5)
    learned = mixed and rng.random() < 0.7
    tol = rng.choice([1e-2, 1e-2, 1e-3])
    if tol < 1e-2 and d == 3:  # ranks grow with the tolerance
        n = min(n, 40)
    nrhs = rng.choice([2, 5, 16]) if op == "block" else 1
    return _case(op, matrix, n, d, tol=tol, mixed=mixed, learned=learned, skip=rng.choice([0, 0, 1]), nrhs=nrhs)


# ------------------------------------------------------------------ inputs
def _field(n, d, seed, corr=8.0):
    """exp of a unit-variance Gaussian random field with correlation length corr (circulant embedding on 2n)."""
    M = 2 * n
    ax = np.minimum(np.arange(M), M - np.arange(M)).astype(np.float64) ** 2
    r2 = sum(ax.reshape([M if i == k else 1 for i in range(d)]) for k in range(d))
    S = np.maximum(np.fft.rfftn(np.exp(-r2 / (2.0 * corr ** 2))).real, 0.0)
    xi = np.random.default_rng(seed).standard_normal((M,) * d)
    g = np.fft.irfftn(np.sqrt(S) * np.fft.rfftn(xi), s=(M,) * d, axes=range(d))[(slice(0, n),) * d]
    return np.exp((g - g.mean()) / g.std())


def _stencil(case, seed):
    """(diag, [(up, dn)] per axis): up[i] = A(i, i + stride), dn[i] = A(i + stride, i), grid-shaped, 0 at the end."""
    n, d = case["n"], case["d"]
    shape = (n,) * d
    diag = np.zeros(shape)
    arms = []
    cut = lambda ax, s: tuple(s if a == ax else slice(None) for a in range(d))  # noqa: E731
    if case["matrix"] == "conv":  # -eps Lap u + w.grad u, first-order upwinding, unit rotating vortex
        eps, h = 1e-2, 1.0 / (n + 1)
        x, y = np.meshgrid((np.arange(n) + 1) * h - 0.5, (np.arange(n) + 1) * h - 0.5, indexing="ij")
        r = np.maximum(np.hypot(x, y), 1e-300)
        diag += 4.0 * eps / h ** 2
        for ax, w in ((0, -y / r), (1, x / r)):
            diag += np.abs(w) / h
            up, dn = np.zeros(shape), np.zeros(shape)
            up[cut(ax, slice(0, -1))] = (-eps / h ** 2 + np.minimum(w, 0.0) / h)[cut(ax, slice(0, -1))]
            dn[cut(ax, slice(0, -1))] = (-eps / h ** 2 - np.maximum(w, 0.0) / h)[cut(ax, slice(1, None))]
            arms.append((up, dn))
        return diag, arms
    k = _field(n, d, seed) if case["matrix"] == "diff" else np.ones(shape)
    for ax in range(d):  # harmonic-mean faces; a face to the boundary takes the cell's own coefficient
        lo, hi = k[cut(ax, slice(0, -1))], k[cut(ax, slice(1, None))]
        f = 2.0 * lo * hi / (lo + hi)
        up = np.zeros(shape)
        up[cut(ax, slice(0, -1))] = -f
        diag[cut(ax, slice(0, -1))] += f
        diag[cut(ax, slice(1, None))] += f
        diag[cut(ax, slice(0, 1))] += k[cut(ax, slice(0, 1))]
        diag[cut(ax, slice(-1, None))] += k[cut(ax, slice(-1, None))]
        arms.append((up, up))
    return diag, arms


def _csc(case, diag, arms):
    """Sorted CSC arrays of the stencil."""
    n, d = case["n"], case["d"]
    N = n ** d
    strides = [n ** (d - 1 - ax) for ax in range(d)]
    offs, cols = [], []
    for ax, s in enumerate(strides):  # rows j - s, largest stride first
        v = np.zeros(N)
        v[s:] = arms[ax][0].ravel()[:-s]
        offs.append(-s)
        cols.append(v)
    offs.append(0)
    cols.append(diag.ravel())
    for ax in reversed(range(d)):
        offs.append(strides[ax])
        cols.append(arms[ax][1].ravel())
    V = np.stack(cols, axis=1)
    mask = V != 0.0
    rows = np.arange(N)[:, None] + np.array(offs)[None, :]
    colptr = np.concatenate([[0], np.cumsum(mask.sum(axis=1))])
    return colptr.astype(np.int32), rows[mask].astype(np.int32), V[mask]


def _rhs(case, seed):
    N = case["n"] ** case["d"]
    return np.random.default_rng(seed + 7919).standard_normal((case["nrhs"], N))


_streams = []


def _stream():
    """One of eight side streams: the handle's stream captures graphs, so the default stream will not do."""
    if not _streams:
        _streams.extend(torch.cuda.Stream() for _ in range(8))
    _streams.append(_streams.pop(0))
    return _streams[0]


def prepare(case, seed):
    colptr, rowidx, vals = _csc(case, *_stencil(case, seed))
    t = ParTree(case["levels"], case["skip"])
    t.set_tol(case["tol"])
    t.set_coords_tensor(case["n"], case["d"])
    stream = _stream()
    t.set_stream(stream.cuda_stream)
    t.partition((colptr, rowidx, scale_columns(colptr, vals)))
    t.set_precision(32 if case["mixed"] else 64)
    if case["learned"]:
        t.set_rank_model(load_rank_model())
    b = _rhs(case, seed)
    state = {"case": case, "tree": t, "stream": stream, "b": b}
    if case["op"] in ("gmres", "apply"):
        t.assemble()
        t.factorize()
    if case["op"] == "apply":
        state["b"] = torch.from_numpy(b[0]).cuda()
        state["x"] = torch.empty_like(state["b"])
        torch.cuda.synchronize()
    return state


def run(state):
    case, t, b = state["case"], state["tree"], state["b"]
    op = case["op"]
    if op == "apply":  # x <- M^-1 b, in the tree's order, on the tree's stream
        with torch.cuda.stream(state["stream"]):
            x = state["x"].copy_(b)
            t.solve_inplace_device(x.data_ptr())
        return x
    if op != "gmres":
        t.assemble()
        t.factorize()
    if op == "oneshot":
        return t.solve(b[0])
    if op == "block":
        B = np.empty(b.shape)
        for r in range(b.shape[0]):
            t.distribute_x(b[r], B[r])
        block_gmres(t, B.T, iters=60, tol=case["rtol"])
        return np.stack([t.extract_x(B[r]) for r in range(b.shape[0])])
    x = np.empty(b.shape[1])
    t.distribute_x(b[0], x)
    dist_gmres(None, x, t, iters=100, tol=case["rtol"], verb=False)
    return t.extract_x(x)


def work(case):
    """Bytes: matrix (values, indices), right-hand sides and solutions once; a kept factorization is an input of the
    ops that use it and is read once per apply.  Flops: 2 m n k of the dense block operations, from the counts of
    factorizations of this family (they grow a little faster than the number of unknowns, and with the kept ranks)."""
    n, d, N = case["n"], case["d"], case["n"] ** case["d"]
    nnz = (2 * d + 1) * N
    size = 4 if case["mixed"] else 8
    log = math.log2(max(N, 256) / 128.0)
    # stored factor entries and flops per unknown (2D, 3D at tol 1e-2; tighter tolerances keep more)
    more = 1.0 + 0.35 * max(0.0, -math.log10(case["tol"]) - 2.0)
    entries = N * ((120.0 + 12.0 * log) if d == 2 else 75.0 * log) * more
    fac = N * ((1.5e4 + 1.0e3 * log) if d == 2 else 1.0e4 * log ** 2) * more ** 2
    io = 12.0 * nnz + 16.0 * N * case["nrhs"]
    if case["op"] == "apply":
        return {"bytes": size * entries + 16.0 * N, "flops": 2.0 * entries}
    its = 1 if case["op"] == "oneshot" else 6
    sweeps = its * case["nrhs"]
    if case["op"] == "gmres":
        return {"bytes": its * (size * entries + 12.0 * nnz) + 16.0 * N, "flops": sweeps * 2.0 * (entries + nnz)}
    return {"bytes": io + size * entries, "flops": fac + sweeps * 2.0 * (entries + nnz)}


def exact(case, seed):
    """The solution of the column-scaled system in 64 bits: block elimination over the grid's first axis with dense
    inverses, refined against the stencil.  An apply of the preconditioner and a one-shot solve at a tolerance have
    no such value."""
    if case["op"] in ("apply", "oneshot"):
        return None
    n, d = case["n"], case["d"]
    B = n ** (d - 1)
    dev = "cuda"
    diag, arms = _stencil(case, seed)
    up = [torch.from_numpy(np.ascontiguousarray(a[0])).to(dev) for a in arms]
    dn = [torch.from_numpy(np.ascontiguousarray(a[1])).to(dev) for a in arms]
    D = torch.from_numpy(diag).to(dev)

    def matvec(x):  # x: (nrhs, grid)
        y = D * x
        for ax in range(d):
            lo, m = x.narrow(ax + 1, 0, n - 1), n - 1
            hi = x.narrow(ax + 1, 1, m)
            y.narrow(ax + 1, 0, m).add_(up[ax].narrow(ax, 0, m) * hi)
            y.narrow(ax + 1, 1, m).add_(dn[ax].narrow(ax, 0, m) * lo)
        return y

    inner = (n,) * (d - 1)
    index = torch.arange(B, device=dev).reshape(inner)
    inv = []
    for k in range(n):
        S = torch.zeros(B, B, dtype=torch.float64, device=dev)
        S[index.reshape(-1), index.reshape(-1)] = D[k].reshape(-1)
        for ax in range(1, d):
            lo = index.narrow(ax - 1, 0, n - 1).reshape(-1)
            hi = index.narrow(ax - 1, 1, n - 1).reshape(-1)
            S[lo, hi] = up[ax][k].narrow(ax - 1, 0, n - 1).reshape(-1)
            S[hi, lo] = dn[ax][k].narrow(ax - 1, 0, n - 1).reshape(-1)
        if k:
            S -= dn[0][k - 1].reshape(-1, 1) * inv[-1] * up[0][k - 1].reshape(1, -1)
        inv.append(torch.linalg.inv(S))

    def solve(f):  # f: (nrhs, grid)
        f = f.reshape(f.shape[0], n, B)
        y = [f[:, 0]]
        for k in range(1, n):
            y.append(f[:, k] - dn[0][k - 1].reshape(-1) * (y[-1] @ inv[k - 1].T))
        x = [None] * n
        x[n - 1] = y[n - 1] @ inv[n - 1].T
        for k in range(n - 2, -1, -1):
            x[k] = (y[k] - up[0][k].reshape(-1) * x[k + 1]) @ inv[k].T
        return torch.stack(x, dim=1).reshape((f.shape[0],) + (n,) * d)

    b = torch.from_numpy(_rhs(case, seed)).to(dev).reshape((case["nrhs"],) + (n,) * d)
    x = solve(b)
    for _ in range(2):
        x += solve(b - matvec(x))
    norm2 = D ** 2  # columns scaled to norm 10: the unknowns of the scaled system are x * norm / 10
    for ax in range(d):
        m = n - 1
        norm2.narrow(ax, 1, m).add_(up[ax].narrow(ax, 0, m) ** 2)
        norm2.narrow(ax, 0, m).add_(dn[ax].narrow(ax, 0, m) ** 2)
    x = (x * norm2.sqrt() / 10.0).reshape(case["nrhs"], -1).cpu().numpy()
    return x if case["op"] == "block" else x[0]
