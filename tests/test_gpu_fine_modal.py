"""GPU: the marching modal product of the finest level at the edges of its
tiles and chunks, and what it does with K x (sweeps, residual, dots).

* Products against the oracle's element loop (I/WOK/KelemProd.m) on meshes of
  one element a direction, one element more or less than a tile or a chunk, and
  on elements that are no cubes: FP64 within 1e-13 of max |y| (about 40 sums of
  rounding 1.1e-16 each), FP32 within 2e-6 (the same with 6e-8).
* Cycles with zero to three sweeps on either side, V, W and FMV, against the
  oracle's cycle to 1e-10: the sweeps ping-pong between two buffers, an even or
  an odd number of times.
* Two solves on one handle give the same iterates when the first iteration is
  launched and the others replay captured ones.
"""
import numpy as np
import pytest

from oracle import fem, gmg
from tosp import problems as P

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


DIMS = [(1, 1, 1), (1, 2, 40), (2, 64, 1), (3, 65, 2), (40, 1, 1), (9, 7, 8), (15, 16, 17), (31, 14, 5), (30, 8, 33)]


@pytest.mark.parametrize("n", [1, 2, 3])
@pytest.mark.parametrize("dims", DIMS)
def test_product(tosp_mod, dims, n):
    pb = P.cantilever(*dims)
    pb.el, pb.eh, pb.ew = 0.7, 1.3, 1.0
    rng = np.random.default_rng(sum(dims) + n)
    dens = rng.uniform(0.001, 1, pb.nelem * n ** 3)
    cg = 1 if n * dims[1] % 2 == 0 else 0
    mg = tosp_mod.default_mg(ngrids=2, cycle=0, omega=0.5, opchol=1, flexible=1, cg_product=cg)
    s = tosp_mod.Solver(pb, mg, precision=tosp_mod.PREC_MIXED, mr_n=n, opfilter=0)
    s.SetupGMG(dens)
    ks = fem.elem_stiff_gqmr(pb.el, pb.eh, pb.ew, pb.nu, n)
    x = rng.standard_normal(pb.freedofs.size)
    full = np.zeros(3 * pb.nnodes)
    full[pb.freedofs] = x
    w = fem.simp(dens, 3.0, 1e-9)

    def oracle(wd, v):
        return fem.kelem_prod_full(*dims, ks, wd, v, n)[pb.freedofs]

    assert rel(s.KelemProd(x), oracle(w, full)) <= 1e-13
    f32 = full.astype(np.float32).astype(float)
    m, e = np.frexp(w)
    assert rel(s.KelemProdMixed(x), oracle(np.ldexp(np.round(m * 256) / 256, e), f32)) <= 2e-6
    if cg:
        assert rel(s.KelemProdCG32(x), oracle(w.astype(np.float32).astype(float), f32)) <= 2e-6
    s.close()


@pytest.mark.parametrize("sweeps", [(1, 1), (2, 1), (1, 2), (3, 3), (2, 0), (0, 2)])
@pytest.mark.parametrize("cycle", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 2])
def test_sweeps(tosp_mod, n, cycle, sweeps):
    pb = P.cantilever(16, 8, 12)
    dens = np.random.default_rng(n).uniform(0.2, 1, pb.nelem * n ** 3)
    mg = tosp_mod.default_mg(ngrids=3, cycle=cycle, omega=0.5, smoothiter1=sweeps[0], smoothiter2=sweeps[1])
    s = tosp_mod.Solver(pb, mg, mr_n=n, opfilter=0)
    s.SetupGMG(dens)
    ks = fem.elem_stiff_gqmr(1, 1, 1, pb.nu, n)
    K = fem.global_stiff_matrix(pb.nelx, pb.nely, pb.nelz, ks, dens, 3.0, 1e-9, pb.freedofs)
    H = gmg.setup_gmg(K, pb.nelx, pb.nely, pb.nelz, pb.freedofs, 3, 0.5)
    r = np.random.default_rng(9).standard_normal(pb.freedofs.size)
    z = gmg.precondition(H, r, cycle, *sweeps)
    assert rel(s.MGCycle(r), z) <= 1e-10
    assert rel(s.MGCycle(r), z) <= 1e-10       # the buffers are back where they were
    s.close()


@pytest.mark.parametrize("prec,cg", [(0, 0), (1, 0), (1, 1)])
@pytest.mark.parametrize("sweeps", [(1, 1), (2, 1), (2, 2), (1, 0)])
def test_solve_twice(tosp_mod, prec, cg, sweeps):
    pb = P.cantilever(24, 12, 12)
    dens = np.random.default_rng(4).uniform(0.3, 1, pb.nelem * 8)
    mg = tosp_mod.default_mg(ngrids=3, cycle=0, omega=0.5, smoothiter1=sweeps[0], smoothiter2=sweeps[1],
                             flexible=1, cg_product=cg)
    s = tosp_mod.Solver(pb, mg, precision=prec, mr_n=2, opfilter=0)
    s.SetupGMG(dens)
    x0 = np.zeros(pb.freedofs.size)
    u, it, rr, rc = s.SolveMG(x0, pb.f)
    v, it2, rr2, rc2 = s.SolveMG(x0, pb.f)
    assert rc == rc2 == 0 and it == it2 and rr <= 1e-8
    assert rel(u, v) <= 1e-14                   # no atomics: the same sums in the same order
    s.close()
