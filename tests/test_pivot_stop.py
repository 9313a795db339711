"""Stop of the pivot selection (pivot.cu): dlaqp2's |R(i,i)| / |R(0,0)| < tol keeps every column at tolerances of zero and
below, and stops at an exactly zero norm at every positive one, those whose square is zero in double precision among
them.  With a wide tie rule the column that stops it can be the first position within pivot_rtol of a larger norm."""
import ctypes as C

import numpy as np
import pytest
from test_pivots import matrix, pivots


def select(A, cs, cm, limit, tol, rtol):
    from pspaqr_public_b200.tree import lib

    f = lib().spq_debug_pivots
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_int, C.c_longlong, C.c_double, C.c_double, C.c_void_p,
                  C.c_void_p]
    m, w = A.shape
    buf = np.ascontiguousarray(A.T if cm else A)
    colat, rank = np.full(min(m, w), -1, np.int32), np.zeros(1, np.int32)
    assert f(buf.ctypes.data, m, w, cm, cs, limit, tol, rtol, colat.ctypes.data, rank.ctypes.data) == 0
    return colat[:rank[0]]


@pytest.mark.gpu
@pytest.mark.parametrize("tol,rank", [(1e-2, 4), (1e-150, 4), (1e-200, 4), (5e-324, 4), (0.0, 9), (-1.0, 9)])
def test_stop_at_zero_norms(tol, rank):
    m, w = 9, 40
    for scale in (1.0, 1e-12):
        A = np.zeros((m, w))  # four columns along the axes, exactly zero norms after them
        for k, c in enumerate((17, 3, 30, 8)):
            A[2 * k, c] = scale * (4 - k)
        for cs, cm in ((1, 1), (1, 0), (4, 1)):
            got = select(A, cs, cm, 0, tol, 1e-6)
            assert len(got) == rank, (scale, cs, cm)
            assert got[:4].tolist() == [17, 3, 30, 8]


@pytest.mark.gpu
@pytest.mark.parametrize("rtol", [1e-3, 0.1, 0.5, 0.9])
@pytest.mark.parametrize("kind,m,w", [("random", 128, 300), ("decay", 31, 64), ("decay", 33, 400), ("decay", 65, 2051)])
def test_stop_by_a_column_within_the_tie_rule(kind, m, w, rtol):
    A = matrix(kind, m, w, m + w)
    for tol in (1e-1, 1e-2, 1e-4):
        want = pivots(A, tol, rtol)
        for cs, cm, limit in ((1, 1, 0), (1, 0, 0), (4, 1, 0), (1, 1, 60000)):
            assert np.array_equal(select(A, cs, cm, limit, tol, rtol), want), (tol, cs, cm, limit)
