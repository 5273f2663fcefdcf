"""GPU: the small levels' stencil products (a warp per node, a lane per value) and
the coarse solve's row pairs at their edges, through cycles against the oracle's:
1e-10, the tolerance of the cycle tests.

* grids one element thick, node counts that are no multiple of a block's eight,
  every position of a node at the faces, one to three sweeps;
* coarsest systems just below and above a chunk of 512 columns and above the
  2048 of one pass, odd row counts;
* the persistent cycle, which applies the same stencils.
"""
import numpy as np
import pytest

from oracle import fem, gmg
from tosp import problems as P

pytestmark = pytest.mark.gpu


def check(tosp_mod, dims, ngrids, cycle, sweeps, **kw):
    pb = P.cantilever(*dims)
    dens = np.random.default_rng(sum(dims)).uniform(0.1, 1, pb.nelem)
    mg = tosp_mod.default_mg(ngrids=ngrids, cycle=cycle, omega=0.5, smoothiter1=sweeps[0], smoothiter2=sweeps[1], **kw)
    s = tosp_mod.Solver(pb, mg, opfilter=0)
    s.SetupGMG(dens)
    ks = fem.elem_stiff_gqmr(1, 1, 1, pb.nu, 1)
    K = fem.global_stiff_matrix(*dims, ks, dens, 3.0, 1e-9, pb.freedofs)
    H = gmg.setup_gmg(K, *dims, pb.freedofs, ngrids, 0.5)
    r = np.random.default_rng(2).standard_normal(pb.freedofs.size)
    z = gmg.precondition(H, r, cycle, *sweeps)
    for _ in range(2):
        assert np.abs(s.MGCycle(r) - z).max() <= 1e-10 * np.abs(z).max()
    s.close()


@pytest.mark.parametrize("small", [0, 100000])
@pytest.mark.parametrize("cycle,sweeps", [(0, (1, 1)), (1, (2, 3))])
@pytest.mark.parametrize("dims", [(4, 4, 4), (8, 4, 12), (4, 20, 8), (36, 4, 4), (12, 16, 20)])
def test_stencils(tosp_mod, dims, cycle, sweeps, small):
    check(tosp_mod, dims, 3, cycle, sweeps, small_cycle_max=small)


# 510, 513, 1014, 2058 and 2535 dofs
@pytest.mark.parametrize("dims", [(32, 8, 2), (36, 4, 4), (24, 24, 2), (12, 12, 26), (24, 24, 8)])
def test_rows(tosp_mod, dims):
    check(tosp_mod, dims, 2, 0, (1, 1))
