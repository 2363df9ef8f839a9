"""Operators with repeated blocks and many row classes (repeat.cu): more
classes than a chunk of rows is sorted for (32), and so many that padding them
to whole groups is refused -- the single-vector kernels then have no table, and
no memory is held for one, while the multi-vector products take groups of four.

A row sums at most 5 blocks * 9 products in the first test: FP64 sweeps stay
below 1e-13, FP32 ones below 1e-5 of the row sums of magnitudes.  The second
operator is block diagonal with condition numbers below 3: solves to 1e-12 agree
with numpy to 1e-10.
"""
import numpy as np
import pytest

import mgldg
import test_repeat_gpu as base

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [mgldg.PREC_FP64, mgldg.PREC_MIXED])
def test_many_classes(ctx, prec):
    n, b, types = 32771, 9, 18
    rp, ci, vals = base.repeated_operator(n, b, 11, 61)
    row = np.repeat(np.arange(n), np.diff(rp))
    kind = (np.arange(n) // 37) % types
    vals[row == ci] = vals[row == ci][1] + (kind * 0.05)[:, None, None] * np.eye(b)
    A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, b, b, rp, ci, vals)
    ops = mgldg.LDGOperators.create_A(ctx, A)
    mg = mgldg.Multigrid(ctx, ops, [], solver=mgldg.COARSE_RELAXATION, relaxation=mgldg.RELAX_JACOBI, omega=0.6,
                         mean_project=0, precision=prec)
    rng = np.random.default_rng(5)
    x, f = rng.standard_normal(n * b), rng.standard_normal(n * b)
    got = mg.relax(0, 1, False, f, x).reshape(n, b)
    D = np.linalg.inv(vals[row == ci])
    t = f.reshape(n, b) - base.apply(rp, ci, vals, x)
    want = x.reshape(n, b) + 0.6 * np.einsum("nij,nj->ni", D, t)
    size = np.abs(x).reshape(n, b) + np.einsum(
        "nij,nj->ni", np.abs(D), np.abs(f.reshape(n, b)) + base.apply(rp, ci, np.abs(vals), np.abs(x)))
    tol = 1e-13 if prec == mgldg.PREC_FP64 else 1e-5
    assert (np.abs(got - want) <= tol * size).all()


def hierarchy(ctx, ops, prec=mgldg.PREC_FP64):
    return mgldg.Multigrid(ctx, ops, [], solver=mgldg.COARSE_RELAXATION, relaxation=mgldg.RELAX_JACOBI, omega=0.7,
                           npre=1, npost=1, mean_project=0, precision=prec)


def test_padding_refused(ctx):
    import torch

    n, b, kinds = 8200, 16, 2000
    rng = np.random.default_rng(2)
    d = rng.uniform(-1, 1, (n, b, b)) * 0.1 / b
    d = d + d.transpose(0, 2, 1) + 2 * np.eye(b)
    idx = np.arange(n, dtype=np.int32)
    rp = np.arange(n + 1, dtype=np.int32)
    A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, b, b, rp, idx, d[idx % kinds])
    ops = mgldg.LDGOperators.create_A(ctx, A)
    hierarchy(ctx, mgldg.LDGOperators.create_A(ctx, A.clone()))   # whatever is set up once is there
    ctx.sync()
    free = torch.cuda.mem_get_info()[0]
    mg = hierarchy(ctx, ops)
    ctx.sync()
    # inverse diagonal blocks of 16.8 MB, four vectors of 1 MB; the refused
    # table's images alone are more than 20 MB
    assert free - torch.cuda.mem_get_info()[0] <= 30 << 20
    F = rng.standard_normal((n * b, 5))
    want = np.linalg.solve(d[idx % kinds], F.reshape(n, b, 5)).reshape(n * b, 5)
    X, _, _ = mgldg.pcg_batched(ctx, ops.A, F, precon=mg, tol=1e-12, maxit=60)
    assert np.linalg.norm(X - want) <= 1e-10 * np.linalg.norm(want)
    for prec in (mgldg.PREC_FP64, mgldg.PREC_MIXED, mgldg.PREC_MIXED_F16):
        m = hierarchy(ctx, ops, prec)
        x, _ = mgldg.pcg(ctx, ops.A, F[:, 0], precon=m, tol=1e-12, maxit=60)
        assert np.linalg.norm(x - want[:, 0]) <= 1e-10 * np.linalg.norm(want[:, 0])
