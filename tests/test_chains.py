"""Distributed panel QR of an elimination chain (kernels.cu dist_qr, dense.cuh panel_qr): reflectors, T factors and R
against the input, over part widths, cluster sizes and row counts at the edges of the 8-column parts, of the 32-column
panels and of the widest panel that fits in shared memory."""
import ctypes as C

import numpy as np
import pytest

NB = 32


def chain(S, Bs, cs, pipe, bits):
    from pspaqr_public_b200.tree import lib

    n = S.shape[0]
    s = np.array(S, order="F")
    b = np.concatenate([B.ravel(order="F") for B in Bs]) if Bs else np.zeros(0)
    rows = np.array([B.shape[0] for B in Bs], np.int32)
    T = np.zeros((len(Bs) + 1) * NB * n)
    p = lambda a, t: a.ctypes.data_as(C.POINTER(t))
    rc = lib().spq_debug_chain(p(s, C.c_double), n, p(b, C.c_double), p(rows, C.c_int), len(Bs), cs, pipe, bits,
                               p(T, C.c_double))
    assert rc == 0
    out, at = [], 0
    for B in Bs:
        out.append(b[at:at + B.size].reshape(B.shape, order="F"))
        at += B.size
    return s, out, T.reshape(len(Bs) + 1, n, NB).transpose(0, 2, 1)


def left_q(V, T, X):
    """Q X for the panels' block reflectors I - V T V^T (V with its unit part in place)."""
    n = V.shape[1]
    for j0 in range((n - 1) // NB * NB, -1, -NB):
        v, t = V[:, j0:j0 + NB], np.triu(T[: min(NB, n - j0), j0:j0 + NB])
        X = X - v @ (t @ (v.T @ X))
    return X


SHAPES = [  # n, rows of the blocks
    (1, [1]), (5, []), (8, [3, 1]), (9, [40]), (31, [7, 33]), (32, [64]), (33, [129, 16]), (40, [800]), (40, [1500]),
    (24, [3000]), (70, [65, 20, 1]), (164, [180, 5]), (300, [257]),
]


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("cs,pipe", [(1, 0), (4, 0), (8, 0), (1, 1), (4, 1)])
@pytest.mark.parametrize("n,rows", SHAPES)
def test_chain_is_a_qr(n, rows, cs, pipe, bits):
    rng = np.random.default_rng(n + sum(rows))
    f = np.float64 if bits == 64 else np.float32
    S = rng.standard_normal((n, n)).astype(f).astype(np.float64)
    Bs = [rng.standard_normal((m, n)).astype(f).astype(np.float64) for m in rows]
    s, bs, T = chain(S, Bs, cs, pipe, bits)
    u = np.finfo(f).eps / 2
    R, off = np.triu(s), np.cumsum([0] + rows)
    X = np.vstack([R] + [np.zeros_like(B) for B in Bs])
    # undo the steps from the last to the first: the input comes back
    for i in range(len(Bs) - 1, -1, -1):
        a, b = n + off[i], n + off[i + 1]
        V = np.vstack([np.eye(n), bs[i]])
        Y = left_q(V, T[i + 1], np.vstack([X[:n], X[a:b]]))
        X[:n], X[a:b] = Y[:n], Y[n:]
    X[:n] = left_q(np.tril(s, -1) + np.eye(n), T[0], X[:n])
    A = np.vstack([S] + Bs)
    # Householder QR is backward stable by columns with a constant of at most (rows of the reflector) x (columns) u
    # for each step (Higham, Accuracy and Stability, Theorem 19.4); random rounding stays far below
    bound = u * n * (n + sum(n + m for m in rows)) + 32 * u
    err = np.linalg.norm(X - A, axis=0) / np.linalg.norm(A, axis=0)
    assert err.max() <= bound, (err.max(), bound)
    # every block reflector is orthogonal: T + T^T = T^T (V^T V) T
    for i, V in [(0, np.tril(s, -1) + np.eye(n))] + [(i + 1, np.vstack([np.eye(n), b])) for i, b in enumerate(bs)]:
        for j0 in range(0, n, NB):
            v, t = V[:, j0:j0 + NB], np.triu(T[i][: min(NB, n - j0), j0:j0 + NB])
            assert np.abs(t + t.T - t.T @ (v.T @ v) @ t).max() <= 8 * u * NB * (len(v) + NB), (i, j0)
