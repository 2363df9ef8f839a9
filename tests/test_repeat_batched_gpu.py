"""Multi-vector products of operators with repeated blocks (spmm_rep.cu) and
the block CG's fused passes: one Jacobi sweep per column and whole solves
against the single-vector path, around the tile edges (1, 32, 33, 34, 64, 65,
66 columns; rows below and above the table's limit).

FP64 sweeps sum the same products in the same order up to skipped zeros, so a
column agrees with the single-vector sweep to rounding (1e-13 of its largest
entry; a row has at most 5 * 16 products).  Solves to 1e-12 agree to 1e-10
(condition number below 3)."""
import ctypes as C

import numpy as np
import pytest

import mgldg

pytestmark = pytest.mark.gpu


def operator(ctx, b, n, seed):
    rng = np.random.default_rng(seed)
    few = int(round(b ** 0.5))
    lo = rng.standard_normal((b, b)) * 0.1
    lo[few:] = 0
    far = rng.standard_normal((b, b)) * 0.1
    far[:, [c for c in range(b) if c % few]] = 0
    dia = rng.standard_normal((b, b)) * 0.1
    dia = dia + dia.T + 4 * np.eye(b)
    rp, ci, bl = [0], [], []
    table = np.stack([lo, lo.T, far, far.T, dia, dia + 0.5 * np.eye(b)])
    for i in range(n):
        row = sorted((j, t) for j, t in ((i - 37, 2), (i - 1, 0), (i, 4 + (i % 11 == 0)), (i + 1, 1), (i + 37, 3))
                     if 0 <= j < n)
        ci += [j for j, _ in row]
        bl += [t for _, t in row]
        rp.append(len(ci))
    return mgldg.SparseBlockMatrix.from_csr(ctx, n, n, b, b, np.array(rp, np.int32), np.array(ci, np.int32), table[bl])


@pytest.mark.parametrize("b,n", [(4, 2047), (4, 2051), (9, 2048), (9, 4133), (16, 2050)])
@pytest.mark.parametrize("prec", [mgldg.PREC_FP64, mgldg.PREC_MIXED])
def test_columns_match_single(ctx, b, n, prec):
    import torch
    A = operator(ctx, b, n, b)
    ops = mgldg.LDGOperators.create_A(ctx, A)
    mg = mgldg.Multigrid(ctx, ops, [], solver=mgldg.COARSE_RELAXATION, relaxation=mgldg.RELAX_JACOBI, omega=0.7,
                         npre=1, npost=1, mean_project=0, precision=prec)
    rng = np.random.default_rng(n)
    for k in (1, 32, 33, 34, 64, 65, 66):
        F = rng.standard_normal((n * b, k))
        X, its, _ = mgldg.pcg_batched(ctx, ops.A, F, precon=mg, tol=1e-12, maxit=60)
        if prec == mgldg.PREC_FP64:
            # V-cycle of the one-level hierarchy: two sweeps from a given start
            X0 = rng.standard_normal((n * b, k))
            dB, dX = torch.from_numpy(F).cuda(), torch.from_numpy(X0).cuda()
            torch.cuda.synchronize()
            ctx.check(mgldg.lib().mgldg_mg_vcycle_batched_dev(ctx.h, mg.h, k, C.c_void_p(dB.data_ptr()),
                                                              C.c_void_p(dX.data_ptr())), "vcycle")
            got = dX.cpu().numpy()
        for c in {0, k // 2, k - 1}:
            x1, h1 = mgldg.pcg(ctx, ops.A, F[:, c], precon=mg, tol=1e-12, maxit=60)
            assert its[c] == len(h1)
            assert np.abs(X[:, c] - x1).max() <= 1e-10 * np.abs(x1).max()
            if prec == mgldg.PREC_FP64:
                want = mg.vcycle(F[:, c], X0[:, c])
                assert np.abs(got[:, c] - want).max() <= 1e-13 * np.abs(want).max()


def test_dense_coarse_columns(ctx):
    """The coarsest solve of all columns, with and without the mean
    projection: one V-cycle against the single-vector path (FP64 to rounding;
    the mixed form's FP32 sweeps differ by summation order, 1e-4 of the
    largest entry covers the coarse solve's condition number of about 500
    times 2^-24)."""
    import torch
    prob = mgldg.CartesianProblem(ctx, 2, 16)
    rng = np.random.default_rng(3)
    for mean in (0, 1):
        for prec, tol in ((mgldg.PREC_FP64, 1e-11), (mgldg.PREC_MIXED, 1e-4)):
            mg = mgldg.Multigrid(ctx, prob.ops, prob.T, npre=2, npost=2, solver=mgldg.COARSE_DENSE, max_levels=2,
                                 mean_project=mean, relaxation=mgldg.RELAX_JACOBI, omega=0.7, precision=prec)
            for k in (3, 64, 70):
                F = rng.standard_normal((prob.ndof, k))
                dB, dX = torch.from_numpy(F).cuda(), torch.zeros(prob.ndof, k, dtype=torch.float64, device="cuda")
                torch.cuda.synchronize()
                ctx.check(mgldg.lib().mgldg_mg_vcycle_batched_dev(ctx.h, mg.h, k, C.c_void_p(dB.data_ptr()),
                                                                  C.c_void_p(dX.data_ptr())), "vcycle")
                for c in {0, k - 1}:
                    want = mg.vcycle(F[:, c])
                    assert np.abs(dX[:, c].cpu().numpy() - want).max() <= tol * np.abs(want).max()
