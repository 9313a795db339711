"""Pivot selection of the column-pivoted QR (pivot.cu) against dlaqp2 with the tie rule (util.cpp:830-851, the same
restatement as the oracle's geqp3_trunc), on matrices whose pivots are decided by more than rounding."""
import ctypes as C

import numpy as np
import pytest


def pivots(A, tol, rtol):
    """dlaqp2: largest partial norm, first position within rtol of it, stop at |R(i,i)| / |R(0,0)| < tol."""
    A = A.copy()
    m, w = A.shape
    at = np.arange(w)
    vn = np.linalg.norm(A, axis=0)
    r00 = 0.0
    for i in range(min(m, w)):
        p = i + int(np.argmax(vn[i:] >= vn[i:].max() * (1.0 - rtol)))
        A[:, [i, p]], at[[i, p]], vn[[i, p]] = A[:, [p, i]], at[[p, i]], vn[[p, i]]
        if i == 0:
            r00 = vn[0]
        elif not (r00 > 0 and vn[i] / r00 >= tol):
            return at[:i]
        if vn[i] > 0:
            q = A[:, i] / vn[i]
            for _ in range(2):
                A[:, i + 1:] -= np.outer(q, q @ A[:, i + 1:])
        vn[i + 1:] = np.linalg.norm(A[:, i + 1:], axis=0)
    return at[:min(m, w)]


def matrix(kind, m, w, seed):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((m, w))
    if kind == "decay":  # norms over four decades, few directions strong
        A = np.linalg.qr(rng.standard_normal((m, m)))[0] @ (np.logspace(0, -4, m)[:, None] * A)
        A *= 10.0 ** (-2.0 * rng.random(w))
    elif kind == "ties":  # every norm equal: entries of one vector permuted, then repeated columns with signs
        v = rng.standard_normal(m)
        A = np.stack([rng.permutation(v) for _ in range(w)], axis=1)
        A[:, w // 2:] = -A[:, : w - w // 2]
    elif kind == "lowrank":  # exact rank deficiency, zero columns
        A = rng.standard_normal((m, max(1, m // 3))) @ rng.standard_normal((max(1, m // 3), w))
        A[:, ::7] = 0.0
    return A


SHAPES = [
    # m, w: edges of the 8-row and 8-column blocks, the panel width (128), the lane split (128 rows), long rows
    (1, 1), (1, 40), (2, 3), (7, 9), (8, 8), (9, 129), (16, 500), (31, 64), (33, 1000), (64, 127), (65, 2051),
    (128, 300), (129, 700), (140, 40), (301, 1203),
]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["random", "decay", "ties", "lowrank"])
@pytest.mark.parametrize("m,w", SHAPES)
def test_pivots_match_dlaqp2(kind, m, w):
    from pspaqr_public_b200.tree import lib

    f = lib().spq_debug_pivots
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_int, C.c_longlong, C.c_double, C.c_double, C.c_void_p,
                  C.c_void_p]
    A = matrix(kind, m, w, 3 * m + w)
    tol = 1e-2 if kind != "decay" else 1e-3
    want = pivots(A, tol, 1e-6)
    # clusters, both layouts, and shared-memory limits that force narrow panels and the panel in global memory
    for cs, cm, limit in ((1, 1, 0), (1, 0, 0), (2, 1, 0), (8, 0, 0), (1, 1, 60000), (4, 1, 24000), (2, 0, 9000)):
        buf = np.ascontiguousarray(A.T if cm else A)
        colat, rank = np.full(min(m, w), -1, np.int32), np.zeros(1, np.int32)
        rc = f(buf.ctypes.data, m, w, cm, cs, limit, tol, 1e-6, colat.ctypes.data, rank.ctypes.data)
        if rc == -12 and limit:
            continue  # the bounds of that many columns do not fit under the limit
        assert rc == 0
        assert rank[0] == len(want), (cs, cm, limit)
        assert np.array_equal(colat[: rank[0]], want), (cs, cm, limit)
