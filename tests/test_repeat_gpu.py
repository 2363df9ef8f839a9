"""Table form of level operators with few distinct blocks (repeat.cu).

The operator is built so that its blocks repeat, at sizes around the slot
kernels' edges: chunk remainders, one, two and four rows per lane pair, rows
of uneven length.  Sweeps are compared with a plain numpy evaluation in FP64.

Tolerances: a row sums at most 9 blocks * b products; the FP64 sweep is
within 9 * b * 2^-53 * sum |a x| of numpy's, below 1e-13 of the largest entry;
the mixed sweep within 9 * b * 2^-24 < 1e-5 * sum |a x| (b <= 16), taken
against the row sums of |A| |x|.
"""
import numpy as np
import pytest

import mgldg

pytestmark = pytest.mark.gpu


def repeated_operator(n, b, seed, chain):
    """Block rows with neighbours at +-1 and, for every third row, +-chain;
    four distinct off-diagonal blocks (two with few rows, two with few
    columns) and two diagonal ones."""
    rng = np.random.default_rng(seed)
    few = max(1, int(round(b ** 0.5)))
    off = rng.standard_normal((4, b, b)) * 0.1
    off[0, few:, :] = 0
    off[1, :b - few, :] = 0
    off[2, :, few:] = 0
    off[3, :, [c for c in range(b) if c % few]] = 0
    dia = rng.standard_normal((2, b, b)) * 0.1
    dia = dia + dia.transpose(0, 2, 1) + 4 * np.eye(b)     # the smoother inverts symmetric blocks
    rp, ci, bl = [0], [], []
    table = np.concatenate([off, dia])
    for i in range(n):
        row = {i: 4 + (i % 7 == 0)}
        for j, t in ((i - 1, 0), (i + 1, 1)) + (((i - chain, 2), (i + chain, 3)) if i % 3 == 0 else ()):
            if 0 <= j < n:
                row[j] = t
        for j in sorted(row):
            ci.append(j)
            bl.append(row[j])
        rp.append(len(ci))
    return np.array(rp, np.int32), np.array(ci, np.int32), table[bl]


def apply(rp, ci, vals, x):
    b = vals.shape[1]
    row = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    y = np.zeros((len(rp) - 1, b))
    np.add.at(y, row, np.einsum("kij,kj->ki", vals, x.reshape(-1, b)[ci]))
    return y


@pytest.mark.parametrize("prec", [mgldg.PREC_FP64, mgldg.PREC_MIXED, mgldg.PREC_MIXED_F16])
@pytest.mark.parametrize("b,n", [(4, 32768), (4, 32801), (9, 16384), (9, 16423), (16, 8192), (16, 8209), (16, 32770),
                                 (16, 131075)])
def test_table_sweep(ctx, b, n, prec):
    rp, ci, vals = repeated_operator(n, b, 100 * b + n % 97, 61)
    A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, b, b, rp, ci, vals)
    ops = mgldg.LDGOperators.create_A(ctx, A)
    mg = mgldg.Multigrid(ctx, ops, [], solver=mgldg.COARSE_RELAXATION, relaxation=mgldg.RELAX_JACOBI, omega=0.6,
                         mean_project=0, precision=prec)
    rng = np.random.default_rng(5)
    x, f = rng.standard_normal(n * b), rng.standard_normal(n * b)
    got = mg.relax(0, 1, False, f, x).reshape(n, b)
    row = np.repeat(np.arange(n), np.diff(rp))
    dia = vals[row == ci]
    u, inv = np.unique(dia.reshape(n, -1), axis=0, return_inverse=True)
    D = np.linalg.inv(u.reshape(-1, b, b))[inv.ravel()]
    t = f.reshape(n, b) - apply(rp, ci, vals, x)
    want = x.reshape(n, b) + 0.6 * np.einsum("nij,nj->ni", D, t)
    size = np.abs(x).reshape(n, b) + np.einsum(
        "nij,nj->ni", np.abs(D), np.abs(f.reshape(n, b)) + apply(rp, ci, np.abs(vals), np.abs(x)))
    # F16: every block value within 2^-11 of the block's largest one
    tol = {mgldg.PREC_FP64: 1e-13, mgldg.PREC_MIXED: 1e-5, mgldg.PREC_MIXED_F16: 1e-5}[prec]
    err = np.abs(got - want)
    if prec == mgldg.PREC_MIXED_F16 and b == 16:
        top = np.abs(vals).max(axis=(1, 2))
        slack = np.zeros((n, b))
        np.add.at(slack, row, (top * 2.0 ** -11 * np.abs(x).reshape(n, b)[ci].sum(axis=1))[:, None])
        err = np.maximum(0, err - np.einsum("nij,nj->ni", np.abs(D), slack))
    assert (err <= tol * size).all(), (err / size).max()


@pytest.mark.parametrize("b,n", [(4, 32801), (9, 16423), (16, 8209), (16, 131075)])
def test_table_cg(ctx, b, n):
    """The outer products: a CG solve (FP64 and double-float q = A d) with a
    one-level smoother as preconditioner reaches the solution (the system is
    well conditioned: 4 I plus small blocks, made symmetric)."""
    rp, ci, vals = repeated_operator(n, b, 3 * b + n % 89, 61)
    # symmetric pattern; A := A + A^T block by block keeps the blocks repeated
    pos = {}
    for i in range(n):
        for k in range(rp[i], rp[i + 1]):
            pos[(i, int(ci[k]))] = k
    keep = np.array([(int(j), i) in pos for i in range(n) for j in ci[rp[i]:rp[i + 1]]])
    row = np.repeat(np.arange(n), np.diff(rp))
    tr = np.array([pos[(int(j), int(i))] for i, j in zip(row[keep], ci[keep])])
    sym = vals[keep] + vals[tr].transpose(0, 2, 1)
    cnt = np.bincount(row[keep], minlength=n)
    rp2 = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32)
    ci2 = ci[keep]
    rng = np.random.default_rng(9)
    xt = rng.standard_normal(n * b)
    f = apply(rp2, ci2, sym, xt).ravel()
    for prec in (mgldg.PREC_FP64, mgldg.PREC_MIXED):
        A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, b, b, rp2, ci2, sym)
        ops = mgldg.LDGOperators.create_A(ctx, A)
        mg = mgldg.Multigrid(ctx, ops, [], solver=mgldg.COARSE_RELAXATION, relaxation=mgldg.RELAX_JACOBI, omega=0.6,
                             npre=1, npost=1, mean_project=0, precision=prec)
        x, hist = mgldg.pcg(ctx, ops.A, f, precon=mg, tol=1e-12, maxit=100)
        assert len(hist) < 100
        # residual below tol * ||f|| in the preconditioner's norm; condition number below 10
        assert np.linalg.norm(x - xt) <= 1e-10 * np.linalg.norm(xt)


def test_distinct_blocks_stay_general(ctx):
    """An operator without repeated blocks keeps the general kernels."""
    rng = np.random.default_rng(1)
    n, b = 8300, 16
    rp, ci, vals = repeated_operator(n, b, 7, 61)
    noise = 1e-3 * rng.standard_normal(vals.shape)
    vals = vals + noise + noise.transpose(0, 2, 1)
    x, f = rng.standard_normal(n * b), rng.standard_normal(n * b)
    row = np.repeat(np.arange(n), np.diff(rp))
    A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, b, b, rp, ci, vals)
    ops = mgldg.LDGOperators.create_A(ctx, A)
    mg = mgldg.Multigrid(ctx, ops, [], solver=mgldg.COARSE_RELAXATION, relaxation=mgldg.RELAX_JACOBI, omega=0.6,
                         mean_project=0)
    got = mg.relax(0, 1, False, f, x).reshape(n, b)
    D = np.linalg.inv(vals[row == ci])
    want = x.reshape(n, b) + 0.6 * np.einsum("nij,nj->ni", D, f.reshape(n, b) - apply(rp, ci, vals, x))
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
