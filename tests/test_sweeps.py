"""The preconditioner apply's panel chains (solve.cu): one vector against the CPU oracle over the shapes of the kernels
(two, eight and sixteen warps, pipelined and whole interiors, panels in shared and in global memory), and blocks of
right-hand sides against single applies.

Tolerances: FP64 factors agree with the oracle's to 1e-10 and an apply is backward stable, so 1e-9 as for the apply
tests of the parity suite.  A block apply runs the same chains on the same factors in another order of summation:
512 eps of the norm (eps of the factors' precision; chains of a few hundred rows)."""
import ctypes as C

import numpy as np
import pytest

from oracle.oracle import OracleTree, random_reference
from pspaqr_public_b200 import ParTree, scale_columns
from pspaqr_public_b200 import matrices as M

pytestmark = pytest.mark.gpu


def _tree(kind, n, d, L, tol, bits, skip=0, rows=0):
    from pspaqr_public_b200.tree import lib

    A = {"lapl": M.laplacian, "diff": M.diffusion_lognormal, "conv": lambda n, d: M.convection_diffusion_2d(n)}[kind](n, d)
    t = ParTree(L, skip)
    t.set_tol(tol)
    t.set_precision(bits)
    t.set_coords_tensor(n, d)
    assert lib().spq_debug_sweep_rows(t._h, rows) == 0
    t.partition((A[0], A[1], scale_columns(A[0], A[2])))
    t.assemble()
    t.factorize()
    return t, A


CASES = [
    # kind, n, d, levels, tol, skip, row limit: leaves of one unknown row up, long interfaces (skip, tight tolerance),
    # limits that put every panel, or only the long ones, in global memory
    ("lapl", 9, 2, 3, 1e-2, 0, 0),
    ("conv", 37, 2, 5, 1e-2, 0, 0),
    ("conv", 65, 2, 3, 1e-2, 1, 0),
    ("diff", 15, 3, 5, 1e-3, 0, 0),
    ("diff", 20, 3, 4, 1e-3, 1, 0),
    ("lapl", 24, 3, 7, 1e-2, 0, 0),
    ("diff", 15, 3, 5, 1e-3, 0, 40),
    ("conv", 37, 2, 5, 1e-2, 0, 1),
]


@pytest.mark.parametrize("kind,n,d,L,tol,skip,rows", CASES)
def test_apply_matches_oracle(kind, n, d, L, tol, skip, rows):
    t, A = _tree(kind, n, d, L, tol, 64, skip, rows)
    o = OracleTree(L, skip, tol, 4)
    o.set_matrix(*A)
    o.set_coords_tensor(n, d)
    o.partition()
    o.assemble()
    o.factorize()
    b = random_reference(n ** d, 5)
    x, y = t.solve_inplace(b.copy()), o.solve_inplace(b)
    assert np.linalg.norm(x - y) <= 1e-9 * np.linalg.norm(y)


@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("nrhs", [1, 2, 8, 9, 17])
@pytest.mark.parametrize("kind,n,d,L,tol,skip,rows", [CASES[1], CASES[4], CASES[6]])
def test_block_apply_matches_single_applies(kind, n, d, L, tol, skip, rows, nrhs, bits):
    import torch
    from pspaqr_public_b200.tree import lib

    t, _ = _tree(kind, n, d, L, tol, bits, skip, rows)
    N = n ** d
    B = np.stack([random_reference(N, 7 + r) for r in range(nrhs)])
    X = torch.from_numpy(B.copy()).cuda()
    torch.cuda.synchronize()
    assert lib().spq_solve_block_device(t._h, C.c_void_p(X.data_ptr()), nrhs, N) == 0
    torch.cuda.synchronize()
    X = X.cpu().numpy()
    eps = np.finfo(np.float64 if bits == 64 else np.float32).eps
    for r in range(nrhs):
        y = t.solve_inplace(B[r].copy())
        assert np.linalg.norm(X[r] - y) <= 512 * eps * np.linalg.norm(y), r
