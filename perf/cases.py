"""The calls that a user of this library has it do, as measurable cases.

A topology-optimisation program calls, per design, the filter, ``SetupGMG`` +
``SolveMG`` (the equilibrium solve) and ``Grad``; the matrix-free operator
``KelemProd`` is also called by itself (residual checks, a host's own Krylov
loop), and a service runs many independent solves through ``Server``.  The
cases take these entry points over the meshes of this repository's workloads
(``tosp.workloads``, the SLP loops and the serving stream of ``bench.py``) and
the small and ragged meshes of its tests, with device pointers through the C
ABI (``include/tosp.h``) or with host arrays through ``tosp.Solver``.

The inspection entry points (``KelemProdMixed``, ``KelemProdCG32``,
``MGCycle``, ``time_operator``) are no cases: a program has no use for them,
and the kernels behind them run inside every mixed solve.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("topopt-slp-3d_b200"))

import tosp  # noqa: E402
from tosp import problems  # noqa: E402

EMIN, PENAL = 1e-9, 3.0


def listed():
    return [
        # One operator product on the smallest test mesh: launch latency and
        # the call's own overhead.
        dict(name="product_16x8x8", kind="product", nelx=16, nely=8, nelz=8, n=1),
        # The operator on a ragged mesh (no multiple of any tile, n * nely
        # odd) with 27 density cells per element.
        dict(name="product_75x35x27_mr3", kind="product", nelx=75, nely=35, nelz=27, n=3),
        # The operator at the size of the headline benchmark.
        dict(name="product_192x96x96_mr2", kind="product", nelx=192, nely=96, nelz=96, n=2),
        # The density filter of the headline benchmark (radius 2 cells, 14.2 M cells).
        dict(name="filter_192x96x96_mr2", kind="filter", nelx=192, nely=96, nelz=96, n=2, cells=2.0, trans=False,
             opfilter=1),
        # Sensitivities and transposed filter of the MR-3 SLP loop (13.8 M cells).
        dict(name="grad_160x80x40_mr3", kind="grad", nelx=160, nely=80, nelz=40, n=3, cells=2.5, opfilter=1),
        # One iteration of the 48 x 24 x 24 SLP loop as its driver runs it: host
        # arrays, FP64, an early (nearly uniform) design.
        dict(name="slp_48x24x24_host", kind="step", nelx=48, nely=24, nelz=24, n=1, problem="cantilever",
             density="early", precision="fp64", cg_product=0, cycle=0, omega=0.6, ngrids=3, cells=1.5, io="host",
             its=25),
        # Equilibrium solve + sensitivities of the 96 x 48 x 48 MR-2 workload, FP64.
        dict(name="step_96x48x48_mr2_fp64", kind="step", nelx=96, nely=48, nelz=48, n=2, problem="cantilever",
             density="uniform", precision="fp64", cg_product=0, cycle=0, omega=0.5, ngrids=4, cells=2.0, io="device",
             its=19),
        # The headline benchmark's step in FP64 and in mixed precision.
        dict(name="step_192x96x96_mr2_fp64", kind="step", nelx=192, nely=96, nelz=96, n=2, problem="cantilever",
             density="grf", precision="fp64", cg_product=0, cycle=0, omega=0.5, ngrids=5, cells=2.0, io="device",
             its=110),
        dict(name="step_192x96x96_mr2_mixed", kind="step", nelx=192, nely=96, nelz=96, n=2, problem="cantilever",
             density="grf", precision="mixed", cg_product=1, cycle=0, omega=0.5, ngrids=5, cells=2.0, io="device",
             its=120),
        # The MR-3 bridge of the large SLP loop: mixed precision, V-cycle (the
        # W-cycle's mixed solve breaks down on some random designs of this size).
        dict(name="step_160x80x40_mr3_mixed", kind="step", nelx=160, nely=80, nelz=40, n=3, problem="bridge",
             density="grf", precision="mixed", cg_product=1, cycle=0, omega=0.5, ngrids=4, cells=2.5, io="device",
             its=120),
        # A mesh of the serving stream by itself, by the defaults of the
        # reference: FP64, W-cycle, one density cell per element.
        dict(name="step_64x32x32_fp64_w", kind="step", nelx=64, nely=32, nelz=32, n=1, problem="torsion",
             density="grf", corr=4.0, precision="fp64", cg_product=0, cycle=1, omega=0.5, ngrids=4, cells=1.5,
             io="device", its=20),
        # The serving loop: eight requests in flight at once, of two shapes and
        # two kinds of support, mixed precision.  (No bridges and no W-cycle:
        # with those some random designs are re-run in FP64, which makes the
        # time a matter of the seed.)
        dict(name="serve_8x32x16x16", kind="serve", nelx=32, nely=16, nelz=16, requests=8, ngrids=3, its=30),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["product", "product", "filter", "grad", "step", "step", "step", "step"])
    n = rng.choice([1, 2, 3])
    if kind != "step":
        # any size, odd ones among them, up to the headline workload's
        # 1.8 M elements and 14 M density cells
        while True:
            c = dict(kind=kind, nelx=_log(rng, 8, 192), nely=_log(rng, 4, 96), nelz=_log(rng, 4, 96), n=n)
            if _nelem(c) * n ** 3 <= 14_200_000:
                break
        if kind == "filter":
            c.update(cells=rng.choice([1.5, 2.0, 2.5]), trans=rng.random() < 0.5, opfilter=rng.choice([1, 1, 2]))
        if kind == "grad":
            c.update(cells=rng.choice([1.5, 2.0, 2.5]), opfilter=1)
        return c
    # meshes that take at least three grids, with a coarsest grid of 4 or more
    # elements a direction, as the level rule leaves it
    mixed = rng.random() < 0.6
    while True:
        g = rng.choice([3, 4])
        m = 2 ** (g - 1)
        c = dict(kind=kind, nelx=m * rng.randint(6, 24), nely=m * rng.randint(4, 12), nelz=m * rng.randint(4, 12), n=n)
        coarse = 3 * (c["nelx"] // m + 1) * (c["nely"] // m + 1) * (c["nelz"] // m + 1)
        if _nelem(c) <= (130_000 if n == 3 else 530_000) and coarse <= 4000:
            break
    # mixed solves of random bridges, and with the W-cycle, break down or
    # stall on some designs, which a program then hands to FP64
    problem = rng.choice(["cantilever", "torsion"] if mixed else ["cantilever", "bridge", "torsion"])
    w = rng.random() < 0.5 and not mixed
    c.update(problem=problem, density="grf", corr=rng.choice([8.0, 4.0 * n]),
             precision="mixed" if mixed else "fp64", cg_product=rng.choice([0, 1, 1]) if mixed else 0,
             cycle=1 if w else 0, omega=0.5, ngrids=g, cells=rng.choice([1.5, 2.0]),
             io=rng.choice(["device", "device", "host"]), its=30 if w else 60)
    return c


# ---- sizes and minimal work ---------------------------------------------------

def _nelem(c):
    return c["nelx"] * c["nely"] * c["nelz"]


def _ndof(c):
    return 3 * (c["nelx"] + 1) * (c["nely"] + 1) * (c["nelz"] + 1)


def _taps(c):
    return len(_filter_offsets(c["n"], c["cells"], c["opfilter"]))


def work(case):
    """Bytes: inputs read once and outputs written once; a solve's CG vectors
    and factors once per iteration (x, r, d, q, s: ten passes of 8 bytes, and
    the factors for the CG's product and two finest sweeps of the cycle).
    Operations: one dense 24 x 24 element product per operator application,
    three applications per iteration."""
    ne, nd = _nelem(case), _ndof(case)
    if case["kind"] == "serve":
        per = [work(dict(kind="step", nelx=case["nelx"], nely=case["nely"], nelz=case["nelz"], n=r["n"], cells=1.5,
                         opfilter=1, precision="mixed", its=case["its"])) for r in _requests(case)]
        return {"bytes": sum(w["bytes"] for w in per), "flops": sum(w["flops"] for w in per)}
    ns = ne * case["n"] ** 3
    if case["kind"] == "product":
        return {"bytes": 16.0 * nd + 8.0 * ns, "flops": 1152.0 * ne}
    if case["kind"] == "filter":
        return {"bytes": 24.0 * ns, "flops": 2.0 * ns * _taps(case)}
    if case["kind"] == "grad":
        return {"bytes": 8.0 * nd + 24.0 * ns, "flops": 1152.0 * ne + 2.0 * ns * _taps(case)}
    cyc = 4 if case["precision"] == "mixed" else 8
    per_it = 80.0 * nd + 4 * cyc * nd + (8.0 + cyc) * ns
    return {"bytes": case["its"] * per_it + 24.0 * ns + 24.0 * nd, "flops": case["its"] * 3 * 1152.0 * ne}


# ---- inputs ---------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))


def _uniform(count, gen, lo, hi):
    return lo + (hi - lo) * torch.rand(count, generator=gen, dtype=torch.float64, device="cuda")


def _grf(c, gen):
    """Gaussian random field of correlation length c["corr"] cells, mapped to
    [0, 1] by the normal CDF, projected (Heaviside, beta 4) and scaled to
    [0.001, 1]: the design fields of the benchmark (8 cells) and serving
    workloads (4 elements)."""
    n, corr = c["n"], c.get("corr", 8.0)
    shape = (c["nelz"] * n, c["nelx"] * n, c["nely"] * n)
    f = torch.fft.rfftn(torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda"))
    k = [torch.fft.fftfreq(s, dtype=torch.float64, device="cuda") for s in shape[:2]]
    k.append(torch.fft.rfftfreq(shape[2], dtype=torch.float64, device="cuda"))
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    v = torch.fft.irfftn(f * torch.exp(-2.0 * (math.pi * corr) ** 2 * k2), s=shape)
    v = torch.special.ndtr((v - v.mean()) / v.std())
    v = (math.tanh(2.0) + torch.tanh(4.0 * (v - 0.5))) / (2.0 * math.tanh(2.0))
    return (0.001 + 0.999 * v).reshape(-1).contiguous()


def _density(c, gen):
    ns = _nelem(c) * c["n"] ** 3
    kind = c.get("density", "grf")
    if kind == "early":            # the first steps of an SLP loop at volume fraction 0.3
        return _uniform(ns, gen, 0.25, 0.35)
    if kind == "uniform":          # i.i.d. densities, filtered
        return _filtered(c, _uniform(ns, gen, 0.001, 1.0), c["cells"], 1, False)
    return _grf(c, gen)


def _requests(c):
    return [dict(n=1 + i % 2, problem=("cantilever", "torsion")[i // 2 % 2]) for i in range(c["requests"])]


def _mg(c, precision):
    # FP64 solves to the default tolerance; mixed solves, which may stop an
    # iteration earlier or later from run to run, a digit further, so that
    # their results can be compared
    return tosp.default_mg(ngrids=c["ngrids"], cycle=c["cycle"], omega=c["omega"],
                           tolMG=1e-9 if precision == "mixed" else 1e-8, maxiterMG=1000,
                           flexible=1 if precision == "mixed" else 0, cg_product=c["cg_product"])


def _solver(c, pb):
    p = c.get("precision", "fp64")
    mg = _mg(c, p) if c["kind"] == "step" else tosp.default_mg(ngrids=2, opchol=1)
    return tosp.Solver(pb, mg, precision=tosp.PREC_MIXED if p == "mixed" else tosp.PREC_FP64, mr_n=c["n"], p=PENAL,
                       emin=EMIN, opfilter=c.get("opfilter", 1), rmin=c.get("cells", 1.5) / c["n"])


def prepare(case, seed):
    gen = _generator(seed)
    s = dict(case=case)
    if case["kind"] == "serve":
        s["server"] = tosp.Server(max_slots=case["requests"], hbm_budget_bytes=32 << 30)
        s["items"] = []
        for r in _requests(case):
            pb = getattr(problems, r["problem"])(case["nelx"], case["nely"], case["nelz"])
            c = dict(case, n=r["n"], corr=4.0 * r["n"], cycle=0, omega=0.5, cg_product=1)
            kw = dict(mg=_mg(c, "mixed"), precision=tosp.PREC_MIXED, mr_n=r["n"], p=PENAL, emin=EMIN, opfilter=1,
                      rmin=1.5 / r["n"])
            s["items"].append((pb, _grf(c, gen).cpu().numpy(), kw))
        for pb, _, kw in s["items"]:      # one idle handle per request
            s["server"].prepare(pb, count=1, **kw)
        return s
    pb = getattr(problems, case.get("problem", "cantilever"))(case["nelx"], case["nely"], case["nelz"])
    s["pb"] = pb
    s["solver"] = _solver(case, pb)
    nfree, ns = s["solver"].nfree, s["solver"].ndens
    x = _density(case, gen)
    if case["kind"] == "product":
        _handover()
        s["solver"].SetupGMG(x)
        s["x"] = torch.randn(nfree, generator=gen, dtype=torch.float64, device="cuda")
        s["y"] = torch.empty_like(s["x"])
    elif case["kind"] == "filter":
        s["x"] = x
        s["y"] = torch.empty_like(x)
    elif case["kind"] == "grad":
        _handover()
        s["solver"].SetupGMG(x)
        s["u"] = torch.randn(3 * pb.nnodes, generator=gen, dtype=torch.float64, device="cuda")
        s["g"] = torch.empty(ns, dtype=torch.float64, device="cuda")
    elif case["io"] == "host":
        s["x"] = x.cpu().numpy()
    else:
        s["x"] = x
        s["f"] = torch.tensor(pb.f, device="cuda")
        s["free"] = torch.tensor(pb.freedofs, device="cuda")
        s["u"] = torch.zeros(nfree, dtype=torch.float64, device="cuda")
        s["ufull"] = torch.zeros(3 * pb.nnodes, dtype=torch.float64, device="cuda")
        s["g"] = torch.empty(ns, dtype=torch.float64, device="cuda")
    return s


# ---- one pass ---------------------------------------------------------------------

def _ok(solver, rc):
    if rc < 0:
        raise tosp.TospError(rc, tosp._lib.tosp_last_error(solver.h).decode())


def _handover():
    """The library works on its handle's own stream: what torch has queued for
    its arguments has to be there before the call."""
    torch.cuda.current_stream().synchronize()


def run(state):
    case, lib = state["case"], tosp._lib
    if case["kind"] == "serve":
        srv = state["server"]
        ids = [srv.submit(pb, x, **kw) for pb, x, kw in state["items"]]
        out = []
        for rid in ids:
            srv.wait(rid)
            u, g, _ = srv.result(rid)
            out.append((u, g))
        return out
    s = state["solver"]
    if case["kind"] == "product":
        _ok(s, lib.tosp_kelem_prod(s.h, state["x"].data_ptr(), state["y"].data_ptr(), s.nfree))
        return state["y"]
    if case["kind"] == "filter":
        _ok(s, lib.tosp_apply_filter(s.h, state["x"].data_ptr(), state["y"].data_ptr(), s.ndens,
                                     1 if case["trans"] else 0))
        return state["y"]
    if case["kind"] == "grad":
        _ok(s, lib.tosp_grad(s.h, state["u"].data_ptr(), s.nfull, state["g"].data_ptr(), None, s.ndens))
        return state["g"]
    pb = state["pb"]
    if case["io"] == "host":
        s.SetupGMG(state["x"])
        u, _, _, _ = s.SolveMG(np.zeros(s.nfree), pb.f)
        full = np.zeros(3 * pb.nnodes)
        full[pb.freedofs] = u
        return {"u": u, "g": s.Grad(full)}
    s.SetupGMG(state["x"])
    u, full = state["u"].zero_(), state["ufull"]
    _handover()
    it, rr = ctypes.c_int32(), ctypes.c_double()
    _ok(s, lib.tosp_solve_mg(s.h, u.data_ptr(), state["f"].data_ptr(), s.nfree, ctypes.byref(it), ctypes.byref(rr)))
    full.index_copy_(0, state["free"], u)
    _handover()
    _ok(s, lib.tosp_grad(s.h, full.data_ptr(), s.nfull, state["g"].data_ptr(), None, s.ndens))
    return {"u": u, "g": state["g"]}


# ---- the same in 64 bits, in plain torch -----------------------------------------

def _filter_offsets(n, cells, opfilter):
    """(dx, dy, dz, weight) of the cells within the radius `cells` / n of a mesh
    of 1 / n cells, by the reference's rule (I/ElemNeighborhood.m:93-122):
    Gaussian of standard deviation radius / 3, or hat.  A constant factor of
    the weights cancels."""
    r, h, out = cells / n, 1.0 / n, []
    for kz in range(int(math.floor(r / h)) + 1):
        z2 = (kz * h) ** 2
        for ix in range(int(math.floor(math.sqrt(r * r - z2) / h)) + 1):
            x2 = (ix * h) ** 2
            for jy in range(int(math.floor(math.sqrt(r * r - z2 - x2) / h)) + 1):
                d2 = z2 + x2 + (jy * h) ** 2
                w = math.exp(-d2 / (2.0 * (r / 3.0) ** 2)) if opfilter == 1 else (r - math.sqrt(d2)) / r
                out += [(dx, dy, dz, w) for dx in {ix, -ix} for dy in {jy, -jy} for dz in {kz, -kz}]
    return out


def _filtered(c, x, cells, opfilter, trans):
    n = c["n"]
    shape = (c["nelz"] * n, c["nelx"] * n, c["nely"] * n)

    def gather(a):
        out = torch.zeros_like(a)
        for dx, dy, dz, w in _filter_offsets(n, cells, opfilter):
            cut = [(slice(max(0, -d), min(m, m - d)), slice(max(0, d), min(m, m + d)))
                   for d, m in zip((dz, dx, dy), shape)]
            if all(t.stop > t.start for t, _ in cut):
                out[tuple(t for t, _ in cut)] += w * a[tuple(f for _, f in cut)]
        return out

    a = x.reshape(shape)
    ws = gather(torch.ones_like(a))
    return (gather(a / ws) if trans else gather(a) / ws).reshape(-1)


class _Fem:
    """Element blocks by Gauss quadrature over the n^3 cells of a unit hex8
    element, the operator and the sensitivities, element by element."""

    def __init__(self, c, pb):
        n, nu = c["n"], pb.nu
        self.n, self.pb = n, pb
        sgn = np.array([[dx, dy, dz] for dz in (-1, 1) for dx in (-1, 1) for dy in (-1, 1)], float)
        D = np.zeros((6, 6))
        D[:3, :3] = nu
        D[range(3), range(3)] = 1 - nu
        D[range(3, 6), range(3, 6)] = (1 - 2 * nu) / 2
        D /= (1 + nu) * (1 - 2 * nu)
        blocks = []
        for cz in range(n):
            for cx in range(n):
                for cy in range(n):
                    K = np.zeros((24, 24))
                    for q in range(8):
                        g = np.array([(q & 1) * 2 - 1, (q >> 1 & 1) * 2 - 1, (q >> 2) * 2 - 1]) / math.sqrt(3.0)
                        p = (2.0 * np.array([cx, cy, cz]) + 1 + g) / n - 1
                        f = 1 + sgn * p
                        B = np.zeros((6, 24))
                        d = np.stack([sgn[:, 0] * f[:, 1] * f[:, 2], sgn[:, 1] * f[:, 0] * f[:, 2],
                                      sgn[:, 2] * f[:, 0] * f[:, 1]]) / 4.0
                        for a in range(3):
                            B[a, a::3] = d[a]
                        B[3, 0::3], B[3, 1::3] = d[1], d[0]
                        B[4, 1::3], B[4, 2::3] = d[2], d[1]
                        B[5, 0::3], B[5, 2::3] = d[2], d[0]
                        K += B.T @ D @ B / (8.0 * n ** 3)
                    blocks.append(K)
        self.ke = torch.tensor(np.stack(blocks), device="cuda")
        ez, ex, ey = torch.meshgrid(*(torch.arange(m, device="cuda") for m in (pb.nelz, pb.nelx, pb.nely)),
                                    indexing="ij")
        base = ((ez * pb.nx + ex) * pb.ny + ey).reshape(-1, 1)
        off = torch.tensor([(dz * pb.nx + dx) * pb.ny + dy for dz in (0, 1) for dx in (0, 1) for dy in (0, 1)],
                           device="cuda")
        self.dofs = (3 * (base + off)[:, :, None] + torch.arange(3, device="cuda")).reshape(-1, 24)
        self.free = torch.tensor(pb.freedofs, device="cuda")

    def cells(self, x):
        """Per-cell values as (element, cell), cells y fastest, then x, then z."""
        p, n = self.pb, self.n
        return x.reshape(p.nelz, n, p.nelx, n, p.nely, n).permute(0, 2, 4, 1, 3, 5).reshape(-1, n ** 3)

    def uncells(self, v):
        p, n = self.pb, self.n
        return v.reshape(p.nelz, p.nelx, p.nely, n, n, n).permute(0, 3, 1, 4, 2, 5).reshape(-1)

    def full(self, v):
        out = torch.zeros(3 * self.pb.nnodes, dtype=torch.float64, device="cuda")
        out[self.free] = v
        return out

    def product(self, w, v):
        ue = self.full(v)[self.dofs]
        ye = torch.zeros_like(ue)
        for s in range(self.n ** 3):
            ye += w[:, s:s + 1] * (ue @ self.ke[s])
        out = torch.zeros(3 * self.pb.nnodes, dtype=torch.float64, device="cuda")
        return out.index_add_(0, self.dofs.reshape(-1), ye.reshape(-1))[self.free]

    def solve(self, w, f, most):
        """Conjugate gradients with the inverse diagonal to 1e-13; None if it is
        not there after `most` iterations."""
        d = torch.zeros(3 * self.pb.nnodes, dtype=torch.float64, device="cuda")
        d.index_add_(0, self.dofs.reshape(-1), (w @ torch.diagonal(self.ke, dim1=1, dim2=2)).reshape(-1))
        m = 1.0 / d[self.free]
        x, r = torch.zeros_like(f), f.clone()
        p = z = m * r
        rz, end = r @ z, 1e-13 * float(f.norm())
        for k in range(most):
            q = self.product(w, p)
            a = rz / (p @ q)
            x, r = x + a * p, r - a * q
            if k % 50 == 49 and float(r.norm()) <= end:
                return x
            z = m * r
            rz, old = r @ z, rz
            p = z + (rz / old) * p
        return None

    def grad(self, x, ufull):
        ue = ufull[self.dofs]
        q = torch.stack([((ue @ self.ke[s]) * ue).sum(1) for s in range(self.n ** 3)], 1)
        return -PENAL * x ** (PENAL - 1) * (1.0 - EMIN) * self.uncells(q)


def _simp(x):
    return EMIN + (1.0 - EMIN) * x ** PENAL


def _exact_step(c, pb, x, cells):
    # an ill-conditioned design needs thousands of iterations of this plain
    # method: only small meshes are within reach
    if _nelem(c) * c["n"] ** 3 > 300_000:
        return None
    fem = _Fem(c, pb)
    u = fem.solve(fem.cells(_simp(x)), torch.tensor(pb.f, device="cuda"), 6000)
    if u is None:
        return None
    return u, _filtered(c, fem.grad(x, fem.full(u)), cells, 1, True)


def exact(case, seed):
    gen = _generator(seed)
    if case["kind"] == "serve":
        out = []
        for r in _requests(case):
            c = dict(case, n=r["n"], corr=4.0 * r["n"])
            pb = getattr(problems, r["problem"])(case["nelx"], case["nely"], case["nelz"])
            out.append(_exact_step(c, pb, _grf(c, gen), 1.5) or (None, None))
        return out
    pb = getattr(problems, case.get("problem", "cantilever"))(case["nelx"], case["nely"], case["nelz"])
    x = _density(case, gen)
    if case["kind"] == "filter":
        return _filtered(case, x, case["cells"], case["opfilter"], case["trans"])
    if case["kind"] == "product":
        fem = _Fem(case, pb)
        v = torch.randn(len(pb.freedofs), generator=gen, dtype=torch.float64, device="cuda")
        return fem.product(fem.cells(_simp(x)), v)
    if case["kind"] == "grad":
        u = torch.randn(3 * pb.nnodes, generator=gen, dtype=torch.float64, device="cuda")
        return _filtered(case, _Fem(case, pb).grad(x, u), case["cells"], case["opfilter"], True)
    got = _exact_step(case, pb, x, case["cells"])
    return None if got is None else {"u": got[0], "g": got[1]}
