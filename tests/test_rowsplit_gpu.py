"""Block rows dealt to several lane groups (rowsplit.cu): products and Jacobi
sweeps of 9 x 9, 25 x 25 and 27 x 27 blocks around the form's row limits and
CTA remainders, against numpy in FP64.

A row sums at most 19 * 27 products and then 27 more, so an FP64 result is
within 540 * 2^-53 < 1e-13 of sum |a x|, an FP32 one within 540 * 2^-24 =
3.3e-5 of it.
"""
import numpy as np
import pytest

import mgldg

pytestmark = pytest.mark.gpu


def operator(n, b, lo, hi, seed):
    rng = np.random.default_rng(seed)
    rp, ci = [0], []
    for i in range(n):
        k = min(n, int(rng.integers(lo, hi + 1)))
        c = {i} | {int(j) % n for j in i + 1 + rng.permutation(40)[:k - 1]}
        ci += sorted(c)
        rp.append(len(ci))
    v = rng.standard_normal((len(ci), b, b)) / b
    row = np.repeat(np.arange(n), np.diff(rp))
    d = row == np.array(ci)
    v[d] = v[d] + v[d].transpose(0, 2, 1) + 4 * np.eye(b)
    return np.array(rp, np.int32), np.array(ci, np.int32), v, row


def apply(row, ci, v, x):
    b = v.shape[1]
    y = np.zeros((row[-1] + 1, b))
    np.add.at(y, row, np.einsum("kij,kj->ki", v, x.reshape(-1, b)[ci]))
    return y


@pytest.mark.parametrize("b,n,lo,hi", [(27, 1, 1, 1), (27, 72, 10, 15), (27, 2047, 8, 14), (27, 2049, 8, 14),
                                       (25, 3, 2, 3), (25, 1023, 3, 6), (25, 1024, 3, 6), (25, 2050, 3, 6),
                                       (9, 117, 9, 12), (9, 4095, 8, 19), (9, 4096, 8, 19), (9, 1000, 3, 6)])
def test_split_rows(ctx, b, n, lo, hi):
    rp, ci, v, row = operator(n, b, lo, hi, 31 * b + n)
    rng = np.random.default_rng(n)
    x, f = rng.standard_normal(n * b), rng.standard_normal(n * b)
    Ax, size = apply(row, ci, v, x), apply(row, ci, np.abs(v), np.abs(x))
    D = np.linalg.inv(v[row == ci])
    want = x.reshape(n, b) + 0.6 * np.einsum("nij,nj->ni", D, f.reshape(n, b) - Ax)
    jsize = np.abs(x).reshape(n, b) + np.einsum("nij,nj->ni", np.abs(D), np.abs(f.reshape(n, b)) + size)
    for prec, tol in ((mgldg.PREC_FP64, 1e-13), (mgldg.PREC_MIXED, 3.3e-5)):
        A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, b, b, rp, ci, v)
        if prec == mgldg.PREC_FP64:
            got = A.mv(x, alpha=-2.0, beta=1.0, y=f).reshape(n, b)
            assert (np.abs(got - (f.reshape(n, b) - 2 * Ax)) <= tol * (np.abs(f.reshape(n, b)) + 2 * size)).all()
            assert (np.abs(A.mv(x).reshape(n, b) - Ax) <= tol * size).all()
        ops = mgldg.LDGOperators.create_A(ctx, A)
        mg = mgldg.Multigrid(ctx, ops, [], solver=mgldg.COARSE_RELAXATION, relaxation=mgldg.RELAX_JACOBI, omega=0.6,
                             mean_project=0, precision=prec)
        got = mg.relax(0, 1, False, f, x).reshape(n, b)
        assert (np.abs(got - want) <= tol * jsize).all(), (np.abs(got - want) / jsize).max()
