"""GPU: coarse operators from moments of the SIMP factors against the oracle's
P'AP, through the cycle (1e-10, the tolerance of the cycle tests): supports whose
fixed dofs have fixed parents (moments), and supports that do not (masked triple
products), small levels as stencils and (warp_stencil_max -1) as modal products,
MR factors 1, 2, 3, elements that are no cubes; switching supports on one handle.
"""
import numpy as np
import pytest

from oracle import fem, gmg
from tosp import problems as P

pytestmark = pytest.mark.gpu

DIMS = (16, 8, 12)


def problem(kind):
    pb = P.cantilever(*DIMS)
    pb.el, pb.eh, pb.ew = 0.7, 1.3, 1.0
    x0 = np.zeros(3 * pb.nnodes, bool)
    node = np.arange(pb.nnodes)
    y, x, z = node % pb.ny, node // pb.ny % pb.nx, node // (pb.ny * pb.nx)
    if kind == "face":
        m = x == 0
    elif kind == "edge":                       # two bottom edges
        m = (y == 0) & ((x == 0) | (x == pb.nx - 1))
    elif kind == "odd":                        # part of the face, up to an odd node
        m = (x == 0) & (y <= 3)
    else:                                      # a face and a node inside, at odd coordinates
        m = (x == 0) | ((x == 5) & (y == 3) & (z == 7))
    for c in range(3):
        x0[3 * node[m] + c] = True
    pb.freedofs = np.nonzero(~x0)[0].astype(np.int64)
    pb.f = np.random.default_rng(3).standard_normal(pb.freedofs.size)
    return pb


def oracle(pb, n, dens, cycle):
    ks = fem.elem_stiff_gqmr(pb.el, pb.eh, pb.ew, pb.nu, n)
    K = fem.global_stiff_matrix(*DIMS, ks, dens, 3.0, 1e-9, pb.freedofs)
    H = gmg.setup_gmg(K, *DIMS, pb.freedofs, 3, 0.5)
    r = np.random.default_rng(5).standard_normal(pb.freedofs.size)
    return r, gmg.precondition(H, r, cycle, 2, 1)


@pytest.mark.parametrize("kind", ["face", "edge", "odd", "inside"])
@pytest.mark.parametrize("wsm", [0, -1])
@pytest.mark.parametrize("n,cycle", [(1, 0), (2, 1), (3, 0), (1, 2)])
def test_cycle(tosp_mod, kind, wsm, n, cycle):
    pb = problem(kind)
    dens = np.random.default_rng(n).uniform(0.1, 1, pb.nelem * n ** 3)
    mg = tosp_mod.default_mg(ngrids=3, cycle=cycle, omega=0.5, smoothiter1=2, smoothiter2=1, warp_stencil_max=wsm)
    s = tosp_mod.Solver(pb, mg, mr_n=n, opfilter=0)
    s.SetupGMG(dens)
    r, z = oracle(pb, n, dens, cycle)
    assert np.abs(s.MGCycle(r) - z).max() <= 1e-10 * np.abs(z).max()
    s.close()


@pytest.mark.parametrize("wsm", [0, -1])
@pytest.mark.parametrize("prec,cg", [(0, 0), (1, 1)])
def test_switching_supports(tosp_mod, wsm, prec, cg):
    a, b = problem("face"), problem("inside")
    dens = np.random.default_rng(1).uniform(0.3, 1, a.nelem * 8)
    mg = tosp_mod.default_mg(ngrids=3, cycle=0, omega=0.5, warp_stencil_max=wsm, flexible=1, cg_product=cg)
    s = tosp_mod.Solver(a, mg, precision=prec, mr_n=2, opfilter=0)
    for pb in (a, b, a):
        s.SetFreedofs(pb.freedofs)
        s.SetupGMG(dens)
        u, it, rr, rc = s.SolveMG(np.zeros(pb.freedofs.size), pb.f)
        one = tosp_mod.Solver(pb, mg, precision=prec, mr_n=2, opfilter=0)
        one.SetupGMG(dens)
        v, it1, rr1, rc1 = one.SolveMG(np.zeros(pb.freedofs.size), pb.f)
        assert rc == rc1 == 0 and it == it1 and rr <= 1e-8
        assert np.abs(u - v).max() <= 1e-12 * np.abs(v).max()
        one.close()
    s.close()
