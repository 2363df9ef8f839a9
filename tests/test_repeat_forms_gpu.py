"""Which forms run from the table of an operator's distinct blocks
(repeat.cu): both sides of the row limits and of the limits on images per row,
per block size and precision.  Checks and tolerances as in test_repeat_gpu.py
(rows of at most 5 blocks * 16 products)."""
import numpy as np
import pytest

import mgldg
import test_repeat_gpu as base

pytestmark = pytest.mark.gpu


# the operator has 8 images: the row limits decide
@pytest.mark.parametrize("b,n,prec", [(4, 39999, mgldg.PREC_FP64), (4, 40001, mgldg.PREC_FP64),
                                      (4, 65535, mgldg.PREC_MIXED), (4, 65539, mgldg.PREC_MIXED),
                                      (9, 32767, mgldg.PREC_MIXED), (9, 32791, mgldg.PREC_MIXED_F16),
                                      (9, 65571, mgldg.PREC_MIXED), (16, 8191, mgldg.PREC_MIXED),
                                      (16, 8192, mgldg.PREC_MIXED_F16)])
def test_row_limits(ctx, b, n, prec):
    base.test_table_sweep(ctx, b, n, prec)


@pytest.mark.parametrize("b,n", [(4, 50021), (9, 32801)])
def test_outer_products(ctx, b, n):
    base.test_table_cg(ctx, b, n)


# 4 + 18 + 18 images: 500 rows of 9 x 9 each in FP64, 160 rows of 16 x 16 each
# in FP32, 400 with FP16 values
@pytest.mark.parametrize("b,n,prec", [(9, 19999, mgldg.PREC_FP64), (9, 20000, mgldg.PREC_FP64),
                                      (9, 32771, mgldg.PREC_MIXED), (16, 8192, mgldg.PREC_FP64),
                                      (16, 8192, mgldg.PREC_MIXED), (16, 15999, mgldg.PREC_MIXED_F16),
                                      (16, 16000, mgldg.PREC_MIXED_F16)])
def test_image_limits(ctx, b, n, prec):
    rp, ci, vals = base.repeated_operator(n, b, 11, 61)
    row = np.repeat(np.arange(n), np.diff(rp))
    d = row == ci
    vals[d] = vals[d][1] + (((np.arange(n) // 37) % 18) * 0.05)[:, None, None] * np.eye(b)
    A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, b, b, rp, ci, vals)
    ops = mgldg.LDGOperators.create_A(ctx, A)
    mg = mgldg.Multigrid(ctx, ops, [], solver=mgldg.COARSE_RELAXATION, relaxation=mgldg.RELAX_JACOBI, omega=0.6,
                         mean_project=0, precision=prec)
    rng = np.random.default_rng(5)
    x, f = rng.standard_normal(n * b), rng.standard_normal(n * b)
    got = mg.relax(0, 1, False, f, x).reshape(n, b)
    D = np.linalg.inv(vals[d])
    want = x.reshape(n, b) + 0.6 * np.einsum("nij,nj->ni", D, f.reshape(n, b) - base.apply(rp, ci, vals, x))
    size = np.abs(x).reshape(n, b) + np.einsum(
        "nij,nj->ni", np.abs(D), np.abs(f.reshape(n, b)) + base.apply(rp, ci, np.abs(vals), np.abs(x)))
    err = np.abs(got - want)
    if prec == mgldg.PREC_MIXED_F16:
        # every block value within 2^-11 of the block's largest one
        slack = np.zeros((n, b))
        np.add.at(slack, row, (np.abs(vals).max(axis=(1, 2)) * 2.0 ** -11 *
                               np.abs(x).reshape(n, b)[ci].sum(axis=1))[:, None])
        err = np.maximum(0, err - np.einsum("nij,nj->ni", np.abs(D), slack))
    assert (err <= (1e-13 if prec == mgldg.PREC_FP64 else 1e-5) * size).all()
