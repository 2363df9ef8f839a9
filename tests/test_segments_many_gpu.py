"""Segmented CG with more segments than one CTA of its scalar kernels takes
(32): copies of two meshes in one block-diagonal system, one-level Jacobi
preconditioner, each with its own right-hand side.

A segment's solve is that of its mesh alone up to rounding: the stopping test may
be met one iteration apart, and residual norms agree to 1e-6 of the largest (CG
amplifies rounding by less than the condition number, below 1e4, per digit kept
here).  The test sqrt(r.z) <= 1e-9 sqrt(r0.z0) bounds the residual by 1e-9
sqrt(cond) <= 1e-7 of the right-hand side.  Graph blocks and the host-driven loop
(profiling on) run the same kernels: equal bit for bit."""
import numpy as np
import pytest

import mgldg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nseg", [31, 33, 700, 2100])
@pytest.mark.parametrize("prec", [mgldg.PREC_FP64, mgldg.PREC_MIXED])
def test_segments(ctx, nseg, prec):
    meshes = [mgldg.disk_mesh(0.6), mgldg.disk_mesh(0.45)]
    pts, tri, off = mgldg.mesh_union([meshes[s % 2] for s in range(nseg)])
    kw = dict(tau0=2.0, tauD=2.0)
    one = dict(npre=1, npost=1, relaxation=mgldg.RELAX_JACOBI, omega=0.6, mean_project=0, precision=prec,
               solver=mgldg.COARSE_RELAXATION)
    prob = mgldg.CartesianProblem(ctx, 2, mesh=(pts, tri), agg_levels=1, agg_seed=1, **kw)
    mg = mgldg.Multigrid(ctx, prob.ops, [], **one)
    off = np.asarray(off, np.int64) * prob.npl
    b = np.random.default_rng(nseg).standard_normal(prob.ndof)
    maxit = 120
    x, its, hist = mgldg.pcg_segmented(ctx, prob.ops.A, b, off, mg, tol=1e-9, maxit=maxit)
    ctx.prof_enable(True)
    try:
        x2, its2, _ = mgldg.pcg_segmented(ctx, prob.ops.A, b, off, mg, tol=1e-9, maxit=maxit)
    finally:
        ctx.prof_enable(False)
    assert np.array_equal(x, x2) and np.array_equal(its, its2)
    alone = []
    for m in meshes:
        p = mgldg.CartesianProblem(ctx, 2, mesh=m, agg_levels=1, agg_seed=1, **kw)
        alone.append((p, mgldg.Multigrid(ctx, p.ops, [], **one)))
    for s in sorted({0, 1, nseg // 2, 31 % nseg, 32 % nseg, nseg - 1}):
        p, g = alone[s % 2]
        r = b[off[s]:off[s + 1]]
        _, hs = mgldg.pcg(ctx, p.ops.A, r, precon=g, tol=1e-9, maxit=maxit)
        m = min(its[s], len(hs))
        assert abs(int(its[s]) - len(hs)) <= 1
        assert np.abs(hist[s][:m] - hs[:m]).max() <= 1e-6 * hs.max()
    assert its.max() < maxit
    res = b - prob.ops.A.mv(x)
    for s in range(nseg):
        assert np.linalg.norm(res[off[s]:off[s + 1]]) <= 1e-7 * np.linalg.norm(b[off[s]:off[s + 1]])
