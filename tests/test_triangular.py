"""Triangular solves with explicit inverses of the 32 x 32 diagonal blocks (solve.cu by_inverse, dense.cuh mma_trsm_right)
on well and ill conditioned blocks: their residuals are those of a substitution, whatever the block's condition.

A substitution leaves |R x - b| <= gamma_n |R| |x| (Higham, Accuracy and Stability, Theorem 8.5).  Tested by norms and
block row by block row, with (n + 32) u for gamma_n, and twice that for the correction's own rounding.  Blocks with
|R_JJ| |R_JJ^{-1}| <= 256 (Frobenius) are solved by the inverse alone, whose residual is up to that factor larger."""
import ctypes as C

import numpy as np
import pytest

NB = 32
KINDS = ["mild", "refined", "substituted", "mixed"]


def upper(n, kind, seed, f):
    """Diagonal blocks with a chain -g above their diagonal: entries of the inverse reach g^31.  Only the second block,
    or the second and the fifth, are ill conditioned, so that the errors of a float solve stay in a float's range."""
    rng = np.random.default_rng(seed)
    R = np.triu(rng.standard_normal((n, n)), 1) * (0.05 / np.sqrt(n))
    bad = {"mild": {}, "refined": {1: 1.4}, "substituted": {1: 1.8}, "mixed": {1: 1.3, 4: 1.8}}[kind]
    if n <= NB:
        bad = {0: bad.get(1, 0.2)}
    for j in range(1, n):
        if j % NB:
            R[j - 1, j] = -bad.get(j // NB, 0.2)
    return (R + np.diag(rng.choice([-1.0, 1.0], n))).astype(f).astype(np.float64)


def check(R, x, b, u, first=0):
    """Residuals of R x = b (columns), block row by block row; the first block has NB - first rows."""
    n = len(R)
    res = (R.astype(np.longdouble) @ x.astype(np.longdouble) - b).astype(np.float64)
    for c in range(-first, n, NB):
        c, e = max(c, 0), min(n, c + NB)
        D = R[c:e, c:e]
        k = np.linalg.norm(D) * np.linalg.norm(np.linalg.inv(D))
        factor = max(2.0, k) if k <= 256.0 else 2.0
        for r in range(x.shape[1]):
            bound = (n + NB) * u * factor * np.linalg.norm(R[c:e]) * np.linalg.norm(x[c:, r])
            assert np.linalg.norm(res[c:e, r]) <= bound, (c, r, k, np.linalg.norm(res[c:e, r]) / bound)


# n, row limit: one and several blocks, remainders, two / eight / sixteen warps with panels of 32, 16 and 8 columns,
# panels in global memory
SHAPES = [(1, 0), (2, 0), (31, 0), (32, 0), (33, 0), (64, 0), (100, 0), (200, 0), (300, 0), (1000, 0), (90, 10)]


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,rows", SHAPES)
def test_sweep_solve_is_backward_stable(n, rows, kind, bits):
    from pspaqr_public_b200.tree import lib

    f = np.float64 if bits == 64 else np.float32
    R = upper(n, kind, n, f)
    p = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    for k in (1, 5):
        # right-hand sides of moderate solutions: products with the inverse cancel
        b = (R @ np.random.default_rng(k).standard_normal((n, k))).astype(f).astype(np.float64)
        x = np.array(b, order="F")
        assert lib().spq_debug_upper(p(np.asfortranarray(R)), n, p(x), k, bits, rows) == 0
        check(R, x, b, np.finfo(f).eps / 2)


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,m", [(1, 1), (31, 5), (32, 64), (33, 65), (100, 130), (300, 70)])
def test_column_scaling_is_backward_stable(n, m, kind, bits):
    from pspaqr_public_b200.tree import lib

    f = np.float64 if bits == 64 else np.float32
    R = upper(n, kind, n, f)
    p = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    b = (np.random.default_rng(m).standard_normal((m, n)) @ R).astype(f).astype(np.float64)
    x = np.array(b, order="F")
    assert lib().spq_debug_scale_cols(p(np.asfortranarray(R)), n, p(x), m, bits) == 0
    # X R = B is the transposed system with the order of the blocks reversed
    check(R[::-1, ::-1].T, x.T[::-1], b.T[::-1], np.finfo(f).eps / 2, NB - 1 - (n - 1) % NB)
