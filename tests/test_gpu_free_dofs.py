"""GPU: free-dof vectors to and from full-length ones, through KelemProd on free
sets of every kind: lengths at the edges of a block's 1024 dofs, all dofs free, one
free dof, random sets, and a change of the set on the same handle.  Against the
oracle's element loop within 1e-13 of max |y| (as the product's own test), from
host and from device memory alike.
"""
import numpy as np
import pytest
import torch

from oracle import fem
from tosp import problems as P

pytestmark = pytest.mark.gpu


# 1020, 1026, 2046, 24 and 3 075 dofs
@pytest.mark.parametrize("dims", [(1, 9, 16), (1, 8, 18), (1, 10, 30), (1, 1, 1), (4, 4, 40)])
def test_free_sets(tosp_mod, dims):
    pb = P.cantilever(*dims)
    rng = np.random.default_rng(sum(dims))
    ndof = 3 * pb.nnodes
    dens = rng.uniform(0.1, 1, pb.nelem)
    mg = tosp_mod.default_mg(ngrids=2, cycle=0, omega=0.5, opchol=1)
    s = tosp_mod.Solver(pb, mg, opfilter=0)
    ks = fem.elem_stiff_gqmr(1, 1, 1, pb.nu, 1)
    w = fem.simp(dens, 3.0, 1e-9)
    some = np.sort(rng.choice(ndof, ndof // 2, replace=False))
    for free in (pb.freedofs, np.arange(ndof), some, np.array([ndof - 1]), np.array([0]), np.arange(0, ndof, 2)):
        s.SetFreedofs(free)
        s.SetupGMG(dens)
        x = rng.standard_normal(free.size)
        full = np.zeros(ndof)
        full[free] = x
        y = fem.kelem_prod_full(*dims, ks, w, full, 1)[free]
        got = s.KelemProd(x)
        assert np.abs(got - y).max() <= 1e-13 * max(np.abs(y).max(), 1e-300)
        xd = torch.tensor(x, device="cuda")
        yd = torch.full_like(xd, np.nan)
        assert tosp_mod._lib.tosp_kelem_prod(s.h, xd.data_ptr(), yd.data_ptr(), free.size) == 0
        assert np.array_equal(yd.cpu().numpy(), got)
    s.close()
