"""Stop of the pivot selection (pivot.cu) at the ends of the tolerance's range: dlaqp2's |R(i,i)| / |R(0,0)| < tol keeps
every column at tolerances of zero and below, and stops at an exactly zero norm at every positive one, those whose square
is zero in double precision among them."""
import ctypes as C

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("tol,rank", [(1e-2, 4), (1e-150, 4), (1e-200, 4), (5e-324, 4), (0.0, 9), (-1.0, 9)])
def test_stop_at_zero_norms(tol, rank):
    from pspaqr_public_b200.tree import lib

    f = lib().spq_debug_pivots
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_int, C.c_longlong, C.c_double, C.c_double, C.c_void_p,
                  C.c_void_p]
    m, w = 9, 40
    for scale in (1.0, 1e-12):
        A = np.zeros((m, w))  # four columns along the axes, exactly zero norms after them
        for k, c in enumerate((17, 3, 30, 8)):
            A[2 * k, c] = scale * (4 - k)
        for cs, cm in ((1, 1), (1, 0), (4, 1)):
            buf = np.ascontiguousarray(A.T if cm else A)
            colat, got = np.full(m, -1, np.int32), np.zeros(1, np.int32)
            assert f(buf.ctypes.data, m, w, cm, cs, 0, tol, 1e-6, colat.ctypes.data, got.ctypes.data) == 0
            assert got[0] == rank, (scale, cs, cm)
            assert colat[:4].tolist() == [17, 3, 30, 8]
