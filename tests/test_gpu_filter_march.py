"""GPU: the marching density filter (cubic cells, radius up to three cells) and
the modal sensitivities against the oracle at the edges of their tiles, with
fixed elements, for every compiled radius and one that falls back to the tile
kernel.  1e-13 of the largest value: sums of at most 123 positive terms, or
quadratic forms of 24 values, in FP64.
"""
import numpy as np
import pytest

from oracle import fem, filt
from tosp import problems as P

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("opfilter", [1, 2])
@pytest.mark.parametrize("radius", [1.0, 1.45, 1.75, 2.0, 2.3, 2.5, 2.9, 3.0, 3.5])
@pytest.mark.parametrize("dims", [(1, 1, 1), (9, 33, 3), (7, 31, 20), (8, 32, 5), (17, 65, 2)])
def test_filter(tosp_mod, dims, radius, opfilter):
    pb = P.cantilever(*dims)
    rng = np.random.default_rng(sum(dims))
    nd = pb.nelem
    fixed = np.unique(rng.integers(0, nd, max(1, nd // 7)))
    s = tosp_mod.Solver(pb, tosp_mod.default_mg(), opfilter=opfilter, rmin=radius, fixed_dens=fixed)
    W, w = filt.elem_neighborhood(*dims, 1, 1, 1, radius, opfilter, fixed)
    x = rng.uniform(0, 1, nd)
    assert rel(s.ApplyFilter(x), filt.apply_filter(x, W, w, opfilter, False)) <= 1e-13
    assert rel(s.ApplyFilter(x, trans=True), filt.apply_filter(x, W, w, opfilter, True)) <= 1e-13
    s.close()


def test_non_finite_stays_within_the_radius(tosp_mod):
    """A NaN or an infinity reaches the elements within the radius, no others."""
    pb = P.cantilever(12, 40, 9)
    s = tosp_mod.Solver(pb, tosp_mod.default_mg(), opfilter=1, rmin=2.0)
    W, _ = filt.elem_neighborhood(12, 40, 9, 1, 1, 1, 2.0, 1)
    x = np.random.default_rng(0).uniform(0, 1, pb.nelem)
    at = (4 * 12 + 6) * 40 + 31
    for bad in (np.nan, np.inf):
        x[at] = bad
        for trans in (False, True):
            y = s.ApplyFilter(x, trans=trans)
            assert np.array_equal(~np.isfinite(y), np.asarray(W[:, [at]].todense()).ravel() != 0)
    s.close()


@pytest.mark.parametrize("n", [1, 2, 3])
@pytest.mark.parametrize("dims", [(1, 1, 1), (5, 33, 3), (9, 14, 2)])
def test_grad(tosp_mod, dims, n):
    pb = P.cantilever(*dims)
    pb.el, pb.eh, pb.ew = 0.7, 1.3, 1.0
    rng = np.random.default_rng(n)
    dens = rng.uniform(0.01, 1, pb.nelem * n ** 3)
    free = np.unique(rng.integers(0, pb.nelem, max(1, 3 * pb.nelem // 4)))
    s = tosp_mod.Solver(pb, tosp_mod.default_mg(ngrids=2, opchol=1), mr_n=n, opfilter=0, free_dens_g=free)
    s.SetupGMG(dens)
    u = rng.standard_normal(3 * pb.nnodes)
    ks = fem.elem_stiff_gqmr(pb.el, pb.eh, pb.ew, pb.nu, n)
    _, g0 = filt.grad(*dims, ks, u, dens, 3.0, 1e-9, None, None, 0, free)
    assert rel(s.Grad(u, return_unfiltered=True)[1], g0) <= 1e-13
    s.close()
