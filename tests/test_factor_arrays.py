"""Factor arrays as the introspection returns them: the block factors T are upper triangular panel by panel (LAPACK's
geqrt layout with zeros below), whatever their memory held before."""
import numpy as np
import pytest

from pspaqr_public_b200 import ParTree, scale_columns
from pspaqr_public_b200 import matrices as M

NB = 32


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [64, 32])
def test_t_factors_are_zero_below_their_diagonals(bits):
    A = M.convection_diffusion_2d(48)
    t = ParTree(5, 0)
    t.set_coords_tensor(48, 2)
    t.set_precision(bits)
    t.set_tensor_cores(0)
    t.partition((A[0], A[1], scale_columns(A[0], A[2])))
    for tol in (1e-1, 1e-8, 1e-2):  # other kept ranks, so that the arrays move over older ones
        t.set_tol(tol)
        t.assemble()
        t.factorize()
    seen = 0
    for c in range(t.num_clusters()):
        for which in (0, 1, 3):
            T = t.factor(c, which)
            for j0 in range(0, 0 if T is None else T.shape[1], NB):
                kb = min(NB, T.shape[1] - j0)
                assert not np.tril(T[:kb, j0:j0 + kb], -1).any(), (c, which, j0)
                seen += 1
    assert seen > 50
