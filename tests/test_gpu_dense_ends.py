"""GPU: the two-ended sweep of the coarsest matrix where its schedule changes
(by the number of 64-wide blocks and the band, both from the coarse grid): no
pair of independent pivots, one, several; tiles that both pivots touch and none;
a last block that is nearly all padding.  Through a two-grid cycle against the
oracle's Cholesky solve: 1e-10, the tolerance of the cycle tests.
"""
import numpy as np
import pytest

from oracle import fem, gmg
from tosp import problems as P

pytestmark = pytest.mark.gpu


# blocks / block band of the coarsest system: 2 / 1, 3 / 1, 26 / 1, 29 / 1, 7 / 3, 16 / 9, 12 / 4, 24 / 9
@pytest.mark.parametrize("dims", [(6, 4, 4), (4, 4, 12), (4, 4, 118), (2, 4, 198), (12, 12, 4), (24, 24, 2), (12, 16, 6),
                                  (24, 24, 4)])
def test_ends(tosp_mod, dims):
    pb = P.cantilever(*dims)
    dens = np.random.default_rng(dims[2]).uniform(0.1, 1, pb.nelem)
    s = tosp_mod.Solver(pb, tosp_mod.default_mg(ngrids=2, cycle=0, omega=0.5), opfilter=0)
    ks = fem.elem_stiff_gqmr(1, 1, 1, pb.nu, 1)
    K = fem.global_stiff_matrix(*dims, ks, dens, 3.0, 1e-9, pb.freedofs)
    H = gmg.setup_gmg(K, *dims, pb.freedofs, 2, 0.5)
    r = np.random.default_rng(2).standard_normal(pb.freedofs.size)
    z = gmg.precondition(H, r, 0, 1, 1)
    for _ in range(2):
        s.SetupGMG(dens)
        assert np.abs(s.MGCycle(r) - z).max() <= 1e-10 * np.abs(z).max()
    s.close()
