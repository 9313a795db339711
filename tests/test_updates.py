"""Trailing updates as a pipeline of ops (kernels.cu k_update_pipe) against one CTA for each task's whole list: every
block sees the same operations in the same order, so that the factors, and with them an apply, are equal bit for bit."""
import numpy as np
import pytest

from oracle.oracle import random_reference
from pspaqr_public_b200 import ParTree, scale_columns
from pspaqr_public_b200 import matrices as M

pytestmark = pytest.mark.gpu


def _apply(A, n, d, L, skip, bits, tasks):
    from pspaqr_public_b200.tree import lib

    t = ParTree(L, skip)
    t.set_tol(1e-2)
    t.set_precision(bits)
    t.set_tensor_cores(0)
    t.set_coords_tensor(n, d)
    assert lib().spq_debug_update_pipe(t._h, tasks) == 0
    t.partition((A[0], A[1], scale_columns(A[0], A[2])))
    out = []
    for _ in range(2):  # the second time from the stored plan
        t.assemble()
        t.factorize()
        out.append(t.solve_inplace(random_reference(n ** d, 3)))
    assert np.array_equal(out[0], out[1])
    return out[0]


@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("kind,n,d,L,skip", [
    # one interior a column and several that share lower blocks, single-panel ops, ops of many panels (skip, wide
    # leaves), chunks of 64 columns with a remainder
    ("conv", 9, 2, 2, 0), ("conv", 37, 2, 5, 0), ("conv", 65, 2, 3, 1), ("diff", 15, 3, 5, 0), ("diff", 22, 3, 4, 1),
])
def test_pipelined_updates_are_bit_identical(kind, n, d, L, skip, bits):
    A = M.diffusion_lognormal(n, d) if kind == "diff" else M.convection_diffusion_2d(n)
    whole = _apply(A, n, d, L, skip, bits, 0)
    for tasks in (30, 1 << 30):  # upper levels only, every level
        assert np.array_equal(_apply(A, n, d, L, skip, bits, tasks), whole)
