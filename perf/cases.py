"""Measured workloads of the solver library, each through its public entry points.

The listed cases are what a program that uses the library has it do: apply an
operator it assembled itself, run a V-cycle as its own preconditioner, solve
with MG-PCG on uniform grids (latency-bound small ones to operators far larger
than L2), many right-hand sides on an adaptive quadtree, unstructured
triangles (one mesh and an uneven batch), the adjoint gradient on tetrahedra,
and the step of a loop whose diffusivity changes every time (new operator, new
hierarchy, one solve).  `draw` gives further cases of the same ranges.

Every case is a dict with a "kind" and that kind's plain parameters.
`prepare` builds what the program holds between calls (mesh, operators,
hierarchy, device vectors), `run` makes one pass.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multigrid-ldg_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import mgldg  # noqa: E402

DEV = "cuda:0"
MAXIT = 400
PRECISION = {"fp64": mgldg.PREC_FP64, "mixed": mgldg.PREC_MIXED, "mixed16": mgldg.PREC_MIXED_F16}
SMOOTHER = {"jacobi": mgldg.RELAX_JACOBI, "gs": mgldg.RELAX_GAUSS_SEIDEL}


def listed():
    return [
        # a user's own small P2-triangle operator applied once: the smallest call, launch latency
        dict(name="spmv p2 1021 rows", kind="spmv", b=6, rows=1021, lo=4, hi=10, alpha=1.0, beta=0.0),
        # residual r = b - A x with a user's Q3 operator larger than L2, FP64
        dict(name="residual q3 20011 rows", kind="spmv", b=16, rows=20011, lo=3, hi=7, alpha=-1.0, beta=1.0),
        # one V-cycle of the reference's default method (FP64 Gauss-Seidel V(3,3), whole
        # hierarchy, one-element Cholesky) as the preconditioner of a caller's own Krylov loop
        dict(name="vcycle 64x64 q2 gs", kind="vcycle", n=64, P=3, tau=1.0, smoother="gs", omega=0.8, pre=3, post=3,
             coarse="cholesky", mean=1),
        # the reference's method on the benchmark's small grid: latency of a whole small solve (without
        # the coarse mean projection, which does not suit Dirichlet data on a truncated hierarchy)
        dict(name="pcg 32x32 q2 fp64 gs", kind="pcg", n=32, P=3, tau=1.0, precision="fp64", smoother="gs", omega=0.8,
             pre=2, post=2, mean=0, tol=1e-10),
        # plain FP64 solve of an ordinary size with block Jacobi
        dict(name="pcg 128x128 q3 fp64 jacobi", kind="pcg", n=128, P=4, tau=1.0, precision="fp64", smoother="jacobi",
             omega=0.7, pre=2, post=2, mean=0, tol=1e-10),
        # mixed precision with the reference's smoother
        dict(name="pcg 256x256 q3 mixed gs", kind="pcg", n=256, P=4, tau=1.0, precision="mixed", smoother="gs",
             omega=0.8, pre=2, post=2, mean=0, tol=1e-10),
        # the benchmark's large uniform grid: 4.2 million unknowns, mixed precision, block Jacobi
        dict(name="pcg 512x512 q3 mixed jacobi", kind="pcg", n=512, P=4, tau=1.0, precision="mixed",
             smoother="jacobi", omega=0.7, pre=2, post=2, mean=0, tol=1e-10),
        # many right-hand sides on an adaptive quadtree (hanging faces)
        dict(name="pcg quadtree q2 64 rhs", kind="batched", base=5, extra=6, npts=4, point_seed=3000, P=3, k=64,
             precision="mixed", tol=1e-10),
        # one unstructured triangle mesh, P2
        dict(name="pcg disk p2 h0.006", kind="disk", h=0.006, P=3, precision="mixed", tol=1e-10),
        # an uneven batch of unstructured meshes solved together
        dict(name="pcg 14 disks p2", kind="disks", nseg=14, hlo=0.012, hhi=0.04, mesh_seed=4000, P=3,
             precision="mixed", tol=1e-10),
        # loss gradient with respect to a per-element diffusivity on tetrahedra: forward and adjoint solves
        dict(name="adjoint ball p2 h0.065", kind="adjoint", h=0.065, P=3, precision="mixed", tol=1e-10),
        # a loop whose diffusivity changes every step: operator, hierarchy, one solve
        dict(name="kappa step 64x64 q2", kind="kappa", n=64, P=3, tau=1.0, precision="mixed", smoother="jacobi",
             omega=0.7, pre=2, post=2, mean=0, tol=1e-10),
    ]


def _log_uniform(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(["spmv", "vcycle", "pcg", "pcg", "pcg", "batched", "disk", "disks", "adjoint", "kappa"])
    tol = rng.choice([1e-8, 1e-10])
    if kind == "spmv":
        b = rng.choice([3, 4, 6, 9, 10, 16, 25])
        lo = rng.randint(2, 5)
        rows = int(_log_uniform(rng, 300, 20000 * 256.0 / max(256, b * b)))
        alpha, beta = rng.choice([(1.0, 0.0), (-1.0, 1.0), (0.5, -2.0)])
        return dict(kind=kind, b=b, rows=rows, lo=lo, hi=lo + rng.randint(1, 4), alpha=alpha, beta=beta)
    tau = round(_log_uniform(rng, 0.6, 2.5), 3)
    smoother = rng.choice(["jacobi", "gs"])
    omega = round(rng.uniform(0.6, 0.7) if smoother == "jacobi" else rng.uniform(0.75, 0.95), 3)
    if kind == "vcycle":
        return dict(kind=kind, n=rng.choice([8, 16, 32, 64]), P=rng.choice([2, 3, 4]), tau=tau, smoother=smoother,
                    omega=omega, pre=rng.randint(1, 3), post=rng.randint(1, 3), coarse=rng.choice(["cholesky", "dense"]),
                    mean=rng.choice([0, 1]))
    if kind in ("pcg", "kappa"):
        n, P = rng.choice([8, 16, 32, 64] + ([128, 256] if kind == "pcg" else [])), rng.choice([2, 3, 4])
        pre = rng.randint(1, 3)
        return dict(kind=kind, n=n, P=P, tau=tau, precision=rng.choice(["fp64", "mixed", "mixed16"]),
                    smoother=smoother, omega=omega, pre=pre, post=pre, mean=0, tol=tol)
    precision = rng.choice(["fp64", "mixed", "mixed"])
    if kind == "batched":
        return dict(kind=kind, base=rng.choice([4, 5]), extra=rng.randint(1, 5), npts=rng.randint(1, 5),
                    point_seed=rng.randint(1, 10000), P=rng.choice([2, 3, 4]), k=rng.randint(2, 40),
                    precision=precision, tol=tol)
    if kind == "disk":
        P = rng.choice([2, 3, 4])
        return dict(kind=kind, h=round(_log_uniform(rng, 0.006 * P / 2, 0.06), 5), P=P, precision=precision, tol=tol)
    if kind == "disks":
        lo = round(_log_uniform(rng, 0.015, 0.04), 4)
        return dict(kind=kind, nseg=rng.randint(2, 11), hlo=lo, hhi=round(lo * rng.uniform(1.2, 3.0), 4),
                    mesh_seed=rng.randint(1, 10000), P=rng.choice([2, 3]), precision=precision, tol=tol)
    return dict(kind="adjoint", h=round(_log_uniform(rng, 0.07, 0.2), 4), P=rng.choice([2, 3]), precision=precision,
                tol=tol)


# ------------------------------------------------------------------ helpers --
_ctx = None


def _context():
    """The program's one context and its stream as torch sees it."""
    global _ctx
    if _ctx is None:
        ctx = mgldg.Context(0)
        _ctx = (ctx, torch.cuda.ExternalStream(ctx.stream))
    return _ctx


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _spmv_pattern(case):
    """Row pointers and sorted columns: lo..hi blocks per row, the diagonal one among them, the
    others within a band as in a space-filling element order."""
    rng = np.random.default_rng(17 + case["rows"])
    n, lo, hi = case["rows"], case["lo"], case["hi"]
    deg = np.minimum(rng.integers(lo, hi + 1, n), n)
    off = rng.integers(1, 1 + max(4, min(n - 1, 400)), (n, hi))
    cols, rp = [], np.zeros(n + 1, np.int64)
    keys = np.concatenate([np.arange(n)[:, None], (np.arange(n)[:, None] + off[:, 1:]) % n], axis=1)
    keep = np.arange(hi)[None, :] < deg[:, None]
    for s in range(0, n, 4096):
        for r in range(s, min(n, s + 4096)):
            c = np.unique(keys[r][keep[r]])
            cols.append(c)
            rp[r + 1] = rp[r] + len(c)
    return rp.astype(np.int32), np.concatenate(cols).astype(np.int32)


def _spmv_values(case, nnzb, seed):
    g = torch.Generator().manual_seed(seed)
    b, n = case["b"], case["rows"] * case["b"]
    v = torch.randn(nnzb * b * b, generator=g, dtype=torch.float64) / b
    x = torch.randn(n, generator=g, dtype=torch.float64)
    y = torch.randn(n, generator=g, dtype=torch.float64)
    return v, x, y


def _reference_element(P):
    """Gauss-Lobatto nodes on [0,1], mass matrix and differentiation matrix of the Lagrange basis."""
    leg = np.polynomial.legendre.Legendre.basis(P - 1)
    nodes = np.concatenate([[-1.0], np.sort(leg.deriv().roots().real), [1.0]]) * 0.5 + 0.5
    V = np.polynomial.legendre.legvander(2 * nodes - 1, P - 1)
    qx, qw = np.polynomial.legendre.leggauss(P + 1)
    phi = np.polynomial.legendre.legvander(qx, P - 1) @ np.linalg.inv(V)
    mass = phi.T @ (0.5 * qw[:, None] * phi)
    dV = np.stack([2 * np.polynomial.legendre.Legendre.basis(k).deriv()(2 * nodes - 1) for k in range(P)], axis=1)
    return nodes, mass, dV @ np.linalg.inv(V)


def _morton(n):
    """Grid positions of the elements in depth-first quadtree order: (ix, iy) per element."""
    e = np.arange(n * n, dtype=np.int64)
    ix, iy = np.zeros_like(e), np.zeros_like(e)
    for bit in range(n.bit_length() - 1):
        ix |= ((e >> (2 * bit + 1)) & 1) << bit
        iy |= ((e >> (2 * bit)) & 1) << bit
    return ix, iy


def _to_grid(u, n, P):
    """Element-major vector -> matrix over (x node, y node)."""
    ix, iy = (torch.from_numpy(a).to(u.device) for a in _morton(n))
    U = torch.zeros(n, n, P, P, dtype=u.dtype, device=u.device)
    U[ix, iy] = u.reshape(n * n, P, P)
    return U.permute(0, 2, 1, 3).reshape(n * P, n * P)


def _from_grid(U, n, P):
    ix, iy = (torch.from_numpy(a).to(U.device) for a in _morton(n))
    return U.reshape(n, P, n, P).permute(0, 2, 1, 3)[ix, iy].reshape(-1)


def _uniform_rhs(n, P, seed):
    """b = M f, f a sum of eight Gaussian bumps, on the n x n grid (element-major, on the GPU)."""
    rng = np.random.default_rng(seed)
    c, w, a = rng.random((8, 2)), rng.uniform(0.05, 0.2, 8), rng.standard_normal(8)
    nodes, mass, _ = _reference_element(P)
    z = torch.from_numpy(((np.arange(n)[:, None] + nodes[None, :]) / n).ravel()).to(DEV)
    F = torch.zeros(n * P, n * P, dtype=torch.float64, device=DEV)
    for k in range(8):
        gx, gy = (torch.exp(-((z - c[k, d]) ** 2) / (2 * w[k] ** 2)) for d in range(2))
        F += a[k] * gx[:, None] * gy[None, :]
    m = torch.from_numpy(mass / n).to(DEV)
    F = torch.einsum("ab,xbyd,cd->xayc", m, F.reshape(n, P, n, P), m)
    ix, iy = (torch.from_numpy(i).to(DEV) for i in _morton(n))
    return F.permute(0, 2, 1, 3)[ix, iy].reshape(-1).contiguous()


def _kappa(points, seed, corr=0.2, sigma=0.5, nfeat=64):
    """Log-normal diffusivity at the given points (random Fourier features)."""
    rng = np.random.default_rng(seed)
    w = rng.standard_normal((nfeat, points.shape[1])) / corr
    ph = rng.uniform(0, 2 * np.pi, nfeat)
    a = rng.standard_normal(nfeat) * sigma * np.sqrt(2.0 / nfeat)
    return np.exp(np.cos(points @ w.T + ph) @ a)


def _coarse_levels(prob, most=4096):
    """Agglomeration levels to keep so that the coarsest one fits the dense solve."""
    n = prob.ne * prob.npl
    for l in range(len(prob.T)):
        if n <= most:
            return l + 1
        n = (int(prob.partition(l).max()) + 1) * prob.T[l].info()[3]
    return len(prob.T) + 1


def _uniform_params(case):
    p = dict(npre=case["pre"], npost=case["post"], relaxation=SMOOTHER[case["smoother"]], omega=case["omega"],
             mean_project=case["mean"], precision=PRECISION[case.get("precision", "fp64")])
    if case.get("coarse", "dense") == "dense":
        # down to the 4 x 4 grid, inverted densely
        p.update(solver=mgldg.COARSE_DENSE, max_levels=max(2, case["n"].bit_length() - 2))
    return p


def _jacobi_params(case, levels, **kw):
    return dict(npre=2, npost=2, solver=mgldg.COARSE_DENSE, max_levels=levels, mean_project=0,
                relaxation=mgldg.RELAX_JACOBI, omega=0.7, precision=PRECISION[case["precision"]], **kw)


def _gaussian_rhs(ctx, prob, seed, out):
    ctx.check(mgldg.lib().mgldg_problem_rhs_gaussian_dev(ctx.h, prob.h, seed, _ptr(out)), "rhs")
    ctx.sync()


def _zeros(*shape):
    return torch.zeros(*shape, dtype=torch.float64, device=DEV)


# ------------------------------------------------------------------ prepare --
def prepare(case, seed):
    ctx, stream = _context()
    kind = case["kind"]
    s = dict(case=case, ctx=ctx, stream=stream)
    if kind == "spmv":
        rp, ci = _spmv_pattern(case)
        v, x, y = _spmv_values(case, len(ci), seed)
        s["A"] = mgldg.SparseBlockMatrix.from_csr(ctx, case["rows"], case["rows"], case["b"], case["b"], rp, ci,
                                                  v.numpy())
        s["x"], s["y0"] = x.to(DEV), y.to(DEV)
        s["y"] = torch.empty_like(s["y0"])
    elif kind in ("vcycle", "pcg", "kappa"):
        n, P = case["n"], case["P"]
        s["prob"] = prob = mgldg.CartesianProblem(ctx, P, n, tau0=case["tau"] * n, tauD=case["tau"] * n)
        s["b"] = _uniform_rhs(n, P, seed)
        s["x"] = torch.zeros_like(s["b"])
        if kind == "kappa":
            s["kappa"] = _uniform_kappa(n, seed)
        else:
            s["mg"] = mgldg.Multigrid(ctx, prob.ops, prob.T, **_uniform_params(case))
    elif kind == "batched":
        pts = mgldg.seeded_points(case["point_seed"], case["npts"])
        qt = mgldg.Quadtree.points(pts, case["base"], case["extra"], radius=0.5, balance=True)
        s["prob"] = prob = mgldg.CartesianProblem(ctx, case["P"], quadtree=qt, tau0=1.0, tauD=1.0, tau_per_face=True)
        s["mg"] = mgldg.Multigrid(ctx, prob.ops, prob.T, **_jacobi_params(case, max(2, prob.nlevels - 3)))
        k = case["k"]
        s["B"], tmp = _zeros(prob.ndof, k), _zeros(prob.ndof)
        for c in range(k):
            _gaussian_rhs(ctx, prob, 1000 * seed + c + 1, tmp)
            s["B"][:, c] = tmp
            torch.cuda.synchronize()
        s["X"] = torch.zeros_like(s["B"])
    elif kind in ("disk", "disks"):
        if kind == "disk":
            h, mesh, off = case["h"], mgldg.disk_mesh(case["h"]), None
        else:
            hs = np.random.default_rng(case["mesh_seed"]).uniform(case["hlo"], case["hhi"], case["nseg"])
            pts, tri, off = mgldg.mesh_union([mgldg.disk_mesh(float(v)) for v in hs])
            h, mesh = float(hs.min()), (pts, tri)
        s["prob"] = prob = mgldg.CartesianProblem(ctx, case["P"], mesh=mesh, tau0=1 / h, tauD=1 / h, agg_levels=12,
                                                  agg_seed=4000)
        s["mg"] = mgldg.Multigrid(ctx, prob.ops, prob.T, **_jacobi_params(case, _coarse_levels(prob)))
        s["b"], tmp = _zeros(prob.ndof), _zeros(prob.ndof)
        if kind == "disk":
            _gaussian_rhs(ctx, prob, seed + 1, s["b"])
        else:
            s["off"] = off = (off * prob.npl).astype(np.int64)
            for i in range(case["nseg"]):
                _gaussian_rhs(ctx, prob, 1000 * seed + i + 1, tmp)
                s["b"][off[i]:off[i + 1]] = tmp[off[i]:off[i + 1]]
                torch.cuda.synchronize()
        s["x"] = torch.zeros_like(s["b"])
    else:
        pts, tets = mgldg.ball_mesh(case["h"])
        h = case["h"]
        s["prob"] = prob = mgldg.CartesianProblem(ctx, case["P"], mesh=(pts, tets), tau0=1 / h, tauD=1 / h,
                                                  agg_levels=12, agg_seed=5000)
        prob.ops.construct_laplacian_kappa(_kappa(pts[tets].mean(axis=1), seed))
        s["mg"] = mgldg.Multigrid(ctx, prob.ops, prob.T,
                                  **_jacobi_params(case, _coarse_levels(prob), restriction=mgldg.RESTRICT_RAT))
        s["b"], s["u_obs"] = _zeros(prob.ndof), _zeros(prob.ndof)
        _gaussian_rhs(ctx, prob, seed + 1, s["b"])
        # the observation: the solution of a second forcing
        tmp, it = _zeros(prob.ndof), C.c_int()
        _gaussian_rhs(ctx, prob, seed + 2, tmp)
        ctx.check(mgldg.lib().mgldg_pcg_dev(ctx.h, s["mg"].h, prob.ops.A.h, _ptr(tmp), _ptr(s["u_obs"]), 1e-12, MAXIT,
                                            C.byref(it), np.zeros(MAXIT)), "pcg")
        s["u"], s["lam"], s["dk"] = _zeros(prob.ndof), _zeros(prob.ndof), _zeros(prob.ne)
    torch.cuda.synchronize()
    return s


def _uniform_kappa(n, seed):
    ix, iy = _morton(n)
    return _kappa(np.stack([(ix + 0.5) / n, (iy + 0.5) / n], axis=1), seed)


# ---------------------------------------------------------------------- run --
def run(s):
    case, ctx, L = s["case"], s["ctx"], mgldg.lib()
    kind = case["kind"]
    if kind == "spmv":
        if case["beta"] != 0:
            with torch.cuda.stream(s["stream"]):
                s["y"].copy_(s["y0"])
        ctx.check(L.mgldg_bsr_mv_dev(ctx.h, case["alpha"], s["A"].h, _ptr(s["x"]), case["beta"], _ptr(s["y"])), "mv")
        return s["y"]
    if kind == "vcycle":
        with torch.cuda.stream(s["stream"]):
            s["x"].zero_()
        ctx.check(L.mgldg_mg_vcycle_dev(ctx.h, s["mg"].h, _ptr(s["b"]), _ptr(s["x"])), "vcycle")
        return s["x"]
    if kind in ("pcg", "disk", "kappa"):
        ops, mg = s["prob"].ops, s.get("mg")
        if kind == "kappa":
            ops.construct_laplacian_kappa(s["kappa"])
            mg = mgldg.Multigrid(ctx, ops, s["prob"].T, **_uniform_params(case))
        with torch.cuda.stream(s["stream"]):
            s["x"].zero_()
        it, hist = C.c_int(), np.zeros(MAXIT)
        ctx.check(L.mgldg_pcg_dev(ctx.h, mg.h, ops.A.h, _ptr(s["b"]), _ptr(s["x"]), case["tol"], MAXIT, C.byref(it),
                                  hist), "pcg")
        return {"x": s["x"], "iterations": it.value}
    if kind == "batched":
        k = case["k"]
        with torch.cuda.stream(s["stream"]):
            s["X"].zero_()
        its, hist = np.zeros(k, np.int32), np.zeros(MAXIT * k)
        ctx.check(L.mgldg_pcg_batched_dev(ctx.h, s["mg"].h, s["prob"].ops.A.h, k, _ptr(s["B"]), _ptr(s["X"]),
                                          case["tol"], MAXIT, its, hist), "pcg_batched")
        return {"X": s["X"], "iterations": its}
    if kind == "disks":
        nseg = case["nseg"]
        with torch.cuda.stream(s["stream"]):
            s["x"].zero_()
        its, hist = np.zeros(nseg, np.int32), np.zeros(MAXIT * nseg)
        ctx.check(L.mgldg_pcg_segmented_dev(ctx.h, s["mg"].h, s["prob"].ops.A.h, nseg,
                                            s["off"].ctypes.data_as(C.POINTER(C.c_int64)), _ptr(s["b"]), _ptr(s["x"]),
                                            case["tol"], MAXIT, its, hist), "pcg_segmented")
        return {"x": s["x"], "iterations": its}
    with torch.cuda.stream(s["stream"]):
        s["u"].zero_()
        s["lam"].zero_()
    loss, its = C.c_double(), (C.c_int * 2)()
    ctx.check(L.mgldg_adjoint_l2_dev(ctx.h, s["mg"].h, s["prob"].ops.h, _ptr(s["b"]), _ptr(s["u_obs"]), case["tol"],
                                     MAXIT, _ptr(s["u"]), _ptr(s["lam"]), _ptr(s["dk"]), C.byref(loss), its), "adjoint")
    return {"u": s["u"], "dL_db": s["lam"], "dL_dkappa": s["dk"], "loss": loss.value,
            "iterations": [its[0], its[1]]}


# --------------------------------------------------------------------- work --
def _stencil(case):
    """(block rows, block size, stored blocks, values of the solution) of a case's finest operator."""
    kind = case["kind"]
    if kind == "spmv":
        rows, b, nnzb = case["rows"], case["b"], len(_spmv_pattern(case)[1])
        return rows, b, nnzb
    if kind in ("vcycle", "pcg", "kappa"):
        n = case["n"]
        return n * n, case["P"] ** 2, 5 * n * n - 4 * n
    if kind == "batched":
        # the base grid plus about 3/4 * pi * 0.25 * 4^base * 3 cells per point and extra level, before balancing
        ne = 4 ** case["base"] * (1 + 0.15 * case["npts"] * case["extra"])
        return ne, case["P"] ** 2, 5.5 * ne
    P = case["P"]
    if kind == "disk":
        ne = 2 * math.pi / case["h"] ** 2
    elif kind == "disks":
        hs = np.random.default_rng(case["mesh_seed"]).uniform(case["hlo"], case["hhi"], case["nseg"])
        ne = float((2 * math.pi / hs ** 2).sum())
    else:
        return 11.5 / case["h"] ** 3, P * (P + 1) * (P + 2) // 6, 11 * 11.5 / case["h"] ** 3
    return ne, P * (P + 1) // 2, 8 * ne


# typical MG-PCG iterations to 1e-10 (per solve)
_ITERATIONS = {"pcg": 20, "kappa": 22, "batched": 23, "disk": 36, "disks": 36, "adjoint": 100}


def work(case):
    """The operator's values (64 bits), right-hand sides and results once; the block products of one
    pass: per V-cycle pre + post sweeps and a residual on every level (4/3 of the finest level's), and
    one outer product per iteration."""
    rows, b, nnzb = _stencil(case)
    kind, n, a = case["kind"], rows * b, 8.0 * nnzb * b * b
    if kind == "spmv":
        return {"bytes": a + 8.0 * n * (3 if case["beta"] != 0 else 2), "flops": 2.0 * nnzb * b * b}
    k = case.get("k", 1)
    sweeps = case.get("pre", 2) + case.get("post", 2) + 1
    product = 2.0 * nnzb * b * b * k
    if kind == "vcycle":
        return {"bytes": a + 16.0 * n, "flops": product * sweeps * 4 / 3}
    it = _ITERATIONS[kind] * (0.8 if case["tol"] > 1e-9 else 1.0)
    return {"bytes": a + 16.0 * n * k, "flops": product * it * (1 + sweeps * 4 / 3)}


# -------------------------------------------------------------------- exact --
def _uniform_1d(case):
    """1-D mass m, gradient g and penalty t of the uniform grid: the 2-D operator is
    A = (t + g' m g) (x) m + m (x) (t + g' m g)."""
    n, P = case["n"], case["P"]
    _, mass, D = _reference_element(P)
    h, tau, N = 1.0 / n, case["tau"] * n, n * P
    lift = np.linalg.inv(mass) / h
    m, g, t = np.zeros((N, N)), np.zeros((N, N)), np.zeros((N, N))
    for e in range(n):
        f, l = e * P, e * P + P - 1          # first and last node
        sl = slice(f, f + P)
        m[sl, sl] = h * mass
        g[sl, sl] = D / h
        g[sl, f] += lift[:, 0]               # the left neighbour's trace (zero outside the domain)
        if e > 0:
            g[sl, f - 1] -= lift[:, 0]
            t[f, f] += tau
            t[f - 1, f - 1] += tau
            t[f, f - 1] -= tau
            t[f - 1, f] -= tau
        else:
            t[f, f] += tau
        if e == n - 1:
            g[sl, l] -= lift[:, P - 1]
            t[l, l] += tau
    return [torch.from_numpy(a).to(DEV) for a in (m, g, t)]


def _fast_solver(m, g, t):
    """Solves A(kappa = 1) U = F by simultaneous diagonalisation of the 1-D pencils."""
    K = t + g.T @ m @ g
    R = torch.linalg.cholesky(m)
    S = torch.linalg.solve_triangular(R, K, upper=False)
    S = torch.linalg.solve_triangular(R, S.T.contiguous(), upper=False)
    lam, Q = torch.linalg.eigh((S + S.T) / 2)
    V = torch.linalg.solve_triangular(R.T.contiguous(), Q, upper=True)   # V' m V = 1, V' K V = lam
    den = lam[:, None] + lam[None, :]
    return lambda F: V @ ((V.T @ F @ V) / den) @ V.T


def _refined(F, apply, solve, tol=1e-15, most=400):
    """Conjugate gradients on apply(U) = F with `solve` as the preconditioner."""
    U, R = torch.zeros_like(F), F.clone()
    Z = solve(R)
    D, rz = Z.clone(), (R * Z).sum()
    first = rz.clone()
    for _ in range(most):
        if float(rz) <= tol * tol * float(first):
            break
        Q = apply(D)
        a = rz / (D * Q).sum()
        U += a * D
        R = F - apply(U)
        Z = solve(R)
        new = (R * Z).sum()
        D = Z + (new / rz) * D
        rz = new
    return U


def exact(case, seed):
    kind = case["kind"]
    if kind == "spmv":
        rp, ci = _spmv_pattern(case)
        v, x, y = _spmv_values(case, len(ci), seed)
        b, n = case["b"], case["rows"]
        row = np.repeat(np.arange(n), np.diff(rp))
        part = torch.einsum("krc,kc->kr", v.reshape(-1, b, b), x.reshape(n, b)[torch.from_numpy(ci.astype(np.int64))])
        r = torch.zeros(n, b, dtype=torch.float64).index_add_(0, torch.from_numpy(row), part).reshape(-1)
        return (case["alpha"] * r + (case["beta"] * y if case["beta"] != 0 else 0)).to(DEV)
    if kind not in ("pcg", "kappa"):
        return None     # assembled on meshes (or through a hierarchy) that only the library builds
    n, P = case["n"], case["P"]
    m, g, t = _uniform_1d(case)
    solve = _fast_solver(m, g, t)
    F = _to_grid(_uniform_rhs(n, P, seed), n, P)
    if kind == "pcg":
        K = t + g.T @ m @ g
        U = _refined(F, lambda W: K @ W @ m.T + m @ W @ K.T, solve, most=4)
    else:
        kap = torch.from_numpy(_uniform_kappa(n, seed)).to(DEV)
        kap = _to_grid(kap[:, None].expand(-1, P * P).reshape(-1).contiguous(), n, P)
        U = _refined(F, lambda W: t @ W @ m.T + m @ W @ t.T + g.T @ (m @ (kap * (g @ W)) @ m.T)
                     + (m @ (kap * (W @ g.T)) @ m.T) @ g, solve)
    return {"x": _from_grid(U, n, P), "iterations": None}
