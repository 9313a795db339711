"""Clusters and blocks without rows or columns: as many levels as the unknowns allow, unknowns without neighbours (their
interfaces keep rank 0) and disconnected parts, with the trailing updates as whole tasks and as pipelines of ops."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

from pspaqr_public_b200 import ParTree
from pspaqr_public_b200 import matrices as M

pytestmark = pytest.mark.gpu


def _matrix(kind, n):
    cp, ri, v = M.laplacian(n, 2)
    A = sp.csc_matrix((v, ri, cp), shape=(n * n, n * n)).tolil()
    x, y = np.divmod(np.arange(n * n), n)
    part = {"deep": 0 * x, "split": (x >= n // 2).astype(int),
            "isolated": np.where((x < n // 2) & (y < n // 2), np.arange(n * n) + 1, 0),
            "diagonal": np.arange(n * n)}[kind]
    A = A.tocoo()
    keep = part[A.row] == part[A.col]
    A = sp.csc_matrix((A.data[keep], (A.row[keep], A.col[keep])), shape=A.shape)
    A.sort_indices()
    return A


@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("kind,n,L", [("deep", 4, 4), ("deep", 5, 5), ("split", 12, 6), ("isolated", 12, 6),
                                      ("isolated", 21, 7), ("diagonal", 8, 5)])
def test_empty_blocks(kind, n, L, bits):
    from pspaqr_public_b200.tree import lib

    A = _matrix(kind, n)
    b = np.random.default_rng(n).standard_normal(n * n)
    want = spl.spsolve(A, b)
    got = []
    for tasks in (0, 1 << 30):
        t = ParTree(L, 0)
        t.set_tol(1e-12)
        t.set_precision(bits)
        t.set_tensor_cores(0)
        t.set_coords_tensor(n, 2)
        assert lib().spq_debug_update_pipe(t._h, tasks) == 0
        t.partition((A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data))
        t.assemble()
        t.factorize()
        got.append(t.solve(b.copy()))
    assert np.array_equal(got[0], got[1])
    # a direct solve: condition (below n^2) times unknowns times the factors' rounding
    u = np.finfo(np.float64 if bits == 64 else np.float32).eps / 2
    assert np.linalg.norm(got[0] - want) <= n ** 2 * n ** 2 * u * np.linalg.norm(want)
