"""GPU: the coarsest grid's explicit inverse at the edges of its 64-wide blocks
(one block, an exact number of blocks, one row over, fixed dofs in the padding's
place), through a two-grid cycle against the oracle's Cholesky solve: 1e-10, the
tolerance of the cycle tests.  A matrix that is not positive definite is still
reported as a breakdown.
"""
import numpy as np
import pytest

from oracle import fem, gmg
from tosp import problems as P

pytestmark = pytest.mark.gpu


# coarsest systems of 24, 54, 126, 192 = 3 x 64, 585, 375, 576 = 9 x 64 and 900 dofs
@pytest.mark.parametrize("dims", [(2, 2, 2), (4, 4, 2), (12, 4, 2), (6, 6, 6), (24, 4, 8), (8, 8, 8), (10, 14, 6),
                                  (8, 8, 22)])
def test_inverse(tosp_mod, dims):
    pb = P.cantilever(*dims)
    dens = np.random.default_rng(dims[0]).uniform(0.1, 1, pb.nelem)
    s = tosp_mod.Solver(pb, tosp_mod.default_mg(ngrids=2, cycle=0, omega=0.5), opfilter=0)
    s.SetupGMG(dens)
    ks = fem.elem_stiff_gqmr(1, 1, 1, pb.nu, 1)
    K = fem.global_stiff_matrix(*dims, ks, dens, 3.0, 1e-9, pb.freedofs)
    H = gmg.setup_gmg(K, *dims, pb.freedofs, 2, 0.5)
    r = np.random.default_rng(2).standard_normal(pb.freedofs.size)
    z = gmg.precondition(H, r, 0, 1, 1)
    assert np.abs(s.MGCycle(r) - z).max() <= 1e-10 * np.abs(z).max()
    s.close()


def test_indefinite(tosp_mod):
    pb = P.cantilever(8, 8, 8)
    s = tosp_mod.Solver(pb, tosp_mod.default_mg(ngrids=2, cycle=0, omega=0.5), opfilter=0)
    with pytest.raises(tosp_mod.TospError) as e:
        s.SetupGMG(np.full(pb.nelem, -1.0))
    assert e.value.code == tosp_mod.TOSP_ERR_BREAKDOWN
    s.close()
