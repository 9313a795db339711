"""Waits of the factorization's pipelines (kernels.cu chain_wait): bounded by lack of progress, not by their length; one
that runs out ends the factorization with -12, and the tree is usable again after it."""
import pytest

from pspaqr_public_b200 import ParTree, SpqError, dist_gmres, random_reference, scale_columns
from pspaqr_public_b200 import matrices as M

pytestmark = pytest.mark.gpu
SPIN = 2_000_000_000


def _tree(n, tol, bits):
    from pspaqr_public_b200.tree import lib

    A = M.diffusion_lognormal(n, 3)
    t = ParTree(8, 0)
    t.set_tol(tol)
    t.set_precision(bits)
    t.set_tensor_cores(0)
    t.set_coords_tensor(n, 3)
    t.partition((A[0], A[1], scale_columns(A[0], A[2])))
    return t, lambda chains, updates: lib().spq_debug_factor_spin(t._h, chains, updates)


@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("chains,updates", [(0, SPIN), (SPIN, 0)])
def test_wait_that_runs_out_is_reported(chains, updates, bits):
    t, spin = _tree(24, 1e-2, bits)
    assert spin(chains, updates) == 0
    t.assemble()
    with pytest.raises(SpqError) as e:
        t.factorize()
    assert e.value.status == -12 and "pipeline" in str(e.value)
    assert spin(SPIN, SPIN) == 0
    t.assemble()
    t.factorize()
    assert dist_gmres(None, random_reference(24 ** 3, 3), t, 100, 1e-10)[1] < 1e-9


def test_long_wait_with_progress_is_not_cut_off():
    """The last updates of a level wait for most of its milliseconds, 0.1 ms without progress is the limit here."""
    t, spin = _tree(32, 1e-3, 64)
    assert spin(SPIN, 200_000) == 0
    t.assemble()
    t.factorize()
    assert t.level_times()[:, list(ParTree.LEVEL_PHASES).index("updates")].max() > 0.3
    assert dist_gmres(None, random_reference(32 ** 3, 3), t, 100, 1e-10)[1] < 1e-9
