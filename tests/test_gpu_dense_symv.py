"""GPU: the coarse solve from the lower tiles alone (inverses above 64 MB), for every
remainder of the block count by the tiles of a block and with a padded last block,
through a two-grid cycle against the oracle's Cholesky solve.  FP64: 1e-10, the
tolerance of the cycle tests.  FP32 vectors: 1e-3, their rounding (6e-8) times a
condition number of the coarsest matrix below 1e4 (solid mesh, whose factors BF16
holds exactly).
"""
import numpy as np
import pytest

from oracle import fem, gmg
from tosp import problems as P

pytestmark = pytest.mark.gpu


# 2970, 3168, 3267 and 3630 dofs: 47, 50, 52 and 57 blocks
@pytest.mark.parametrize("dims", [(16, 18, 20), (14, 22, 20), (20, 20, 16), (20, 20, 18)])
@pytest.mark.parametrize("mixed", [0, 1])
def test_symv(tosp_mod, dims, mixed):
    pb = P.cantilever(*dims)
    dens = np.ones(pb.nelem) if mixed else np.random.default_rng(dims[0]).uniform(0.1, 1, pb.nelem)
    mg = tosp_mod.default_mg(ngrids=2, cycle=0, omega=0.5, flexible=mixed)
    s = tosp_mod.Solver(pb, mg, precision=tosp_mod.PREC_MIXED if mixed else tosp_mod.PREC_FP64, opfilter=0)
    s.SetupGMG(dens)
    ks = fem.elem_stiff_gqmr(1, 1, 1, pb.nu, 1)
    K = fem.global_stiff_matrix(*dims, ks, dens, 3.0, 1e-9, pb.freedofs)
    H = gmg.setup_gmg(K, *dims, pb.freedofs, 2, 0.5)
    r = np.random.default_rng(2).standard_normal(pb.freedofs.size)
    z = gmg.precondition(H, r, 0, 1, 1)
    y = s.MGCycle(r)
    assert np.abs(y - z).max() <= (1e-3 if mixed else 1e-10) * np.abs(z).max()
    assert np.array_equal(y, s.MGCycle(r))     # a fixed order of sums
    s.close()
