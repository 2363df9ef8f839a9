"""Small and rectangular blocks: transfers of agglomerated meshes by entry
(k_spmv_entry), sweeps and double-float products of 6, 9 and 10 wide blocks
(k_jacobi_rows, k_spmv_rows, k_spmv_rows_df64), the dense coarsest solve of
odd sizes (coarse_row), against numpy in FP64.

Tolerances.  Transfers: at most 5 * 27 products, then alpha and beta, are
within 140 * 2^-53 < 1.6e-14 of sum |a x|.  Sweeps: at most 8 * 10 products
and 10 more are within 100 * 2^-53 < 1.2e-14 resp. 100 * 2^-24 < 6e-6 of the
sums of magnitudes.  Systems here have condition numbers below 3: a dense
solve of n < 1100 unknowns is within 3 * 3 n 2^-53 < 1.1e-12 and its FP32
form within 3 * 2^-23 < 4e-7 more; a V-cycle in FP32 is six steps of at most
200 products, 6 * 3 * 200 * 2^-24 < 2.2e-4.
"""
import numpy as np
import pytest

import mgldg


def operator(n, b, lo, hi, seed, scale=0.2):
    # diagonally dominant, symmetric diagonal blocks, all blocks distinct
    rng = np.random.default_rng(seed)
    rp, ci = [0], []
    for i in range(n):
        k = min(n, int(rng.integers(lo, hi + 1)))
        ci += sorted({i} | {int(j) % n for j in i + 1 + rng.permutation(40)[:k - 1]})
        rp.append(len(ci))
    ci = np.array(ci, np.int32)
    row = np.repeat(np.arange(n), np.diff(rp))
    v = rng.uniform(-1, 1, (len(ci), b, b)) * scale / (hi * b)
    d = row == ci
    v[d] = v[d] + v[d].transpose(0, 2, 1) + 2 * np.eye(b)
    return np.array(rp, np.int32), ci, v, row


def apply(row, n, ci, v, x):
    y = np.zeros((n, v.shape[1]))
    np.add.at(y, row, np.einsum("kij,kj->ki", v, x.reshape(-1, v.shape[2])[ci]))
    return y


@pytest.mark.gpu
@pytest.mark.parametrize("br,bc", [(3, 4), (4, 3), (6, 9), (9, 6), (10, 16), (16, 10), (4, 8), (8, 4), (10, 27),
                                   (27, 10)])
@pytest.mark.parametrize("n,nc", [(1, 1), (257, 63), (4099, 1021)])
def test_transfer_entries(ctx, br, bc, n, nc):
    rng = np.random.default_rng(100 * br + bc + n)
    cnt = rng.integers(0, min(nc, 5) + 1, n)
    rp = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.permutation(nc)[:k]) for k in cnt] + [[]]).astype(np.int32)
    row = np.repeat(np.arange(n), cnt)
    v = rng.standard_normal((len(ci), br, bc))
    x, f = rng.standard_normal(nc * bc), rng.standard_normal(n * br)
    A = mgldg.SparseBlockMatrix.from_csr(ctx, n, nc, br, bc, rp, ci, v)
    Ax, size = apply(row, n, ci, v, x), apply(row, n, ci, np.abs(v), np.abs(x))
    assert (np.abs(A.mv(x).reshape(n, br) - Ax) <= 1.6e-14 * size).all()
    got = A.mv(x, alpha=-2.0, beta=0.5, y=f).reshape(n, br)
    want = 0.5 * f.reshape(n, br) - 2 * Ax
    assert (np.abs(got - want) <= 1.6e-14 * (np.abs(f.reshape(n, br)) + 2 * size)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("b", [6, 9, 10])
@pytest.mark.parametrize("n", [1, 25, 41, 1217])
def test_sweeps_and_mixed_solves(ctx, b, n):
    rp, ci, v, row = operator(n, b, 1, 7, 7 * b + n)
    rng = np.random.default_rng(n)
    x, f = rng.standard_normal(n * b), rng.standard_normal((n, b))
    Ax, size = apply(row, n, ci, v, x), apply(row, n, ci, np.abs(v), np.abs(x))
    D = np.linalg.inv(v[row == ci])
    want = x.reshape(n, b) + 0.6 * np.einsum("nij,nj->ni", D, f - Ax)
    jsize = np.abs(x).reshape(n, b) + np.einsum("nij,nj->ni", np.abs(D), np.abs(f) + size)
    A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, b, b, rp, ci, v)
    ops = mgldg.LDGOperators.create_A(ctx, A)
    for prec, tol in ((mgldg.PREC_FP64, 1.2e-14), (mgldg.PREC_MIXED, 6e-6)):
        mg = mgldg.Multigrid(ctx, ops, [], solver=mgldg.COARSE_RELAXATION, relaxation=mgldg.RELAX_JACOBI, omega=0.6,
                             npre=2, npost=2, mean_project=0, precision=prec)
        got = mg.relax(0, 1, False, f.ravel(), x).reshape(n, b)
        assert (np.abs(got - want) <= tol * jsize).all(), (np.abs(got - want) / jsize).max()
        # the outer product (double-float in the mixed form) in a solve of a symmetric system
        sym = row == ci
        S = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, b, b, np.arange(n + 1, dtype=np.int32),
                                             np.arange(n, dtype=np.int32), v[sym])
        sops = mgldg.LDGOperators.create_A(ctx, S)
        smg = mgldg.Multigrid(ctx, sops, [], solver=mgldg.COARSE_RELAXATION, relaxation=mgldg.RELAX_JACOBI, omega=0.6,
                              npre=1, npost=1, mean_project=0, precision=prec)
        rhs = np.einsum("nij,nj->ni", v[sym], x.reshape(n, b))
        u, _ = mgldg.pcg(ctx, sops.A, rhs.ravel(), precon=smg, tol=1e-13, maxit=100)
        assert np.abs(u - x).max() <= 1e-12 * max(1.0, np.abs(x).max())


@pytest.mark.gpu
@pytest.mark.parametrize("b,n", [(1, 1), (3, 1), (3, 43), (3, 85), (3, 343), (4, 32), (9, 113)])
def test_dense_coarse_rows(ctx, b, n):
    rp, ci, v, row = operator(n, b, 1, 5, 3 * b + n)
    M = np.zeros((n * b, n * b))
    for k in range(len(ci)):
        M[row[k] * b:(row[k] + 1) * b, ci[k] * b:(ci[k] + 1) * b] += v[k]
    f = np.random.default_rng(n).standard_normal(n * b)
    want = np.linalg.solve(M, f)
    A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, b, b, rp, ci, v)
    ops = mgldg.LDGOperators.create_A(ctx, A)
    for prec, tol in ((mgldg.PREC_FP64, 1.1e-12), (mgldg.PREC_MIXED, 4e-7 + 1.1e-12)):
        mg = mgldg.Multigrid(ctx, ops, [], solver=mgldg.COARSE_DENSE, mean_project=0, precision=prec)
        assert np.linalg.norm(mg.vcycle(f) - want) <= tol * np.linalg.norm(want)


@pytest.mark.gpu
@pytest.mark.parametrize("bf,bc", [(3, 4), (6, 9), (10, 16), (4, 8), (10, 27)])
def test_vcycle_fp32_transfers(ctx, bf, bc):
    # four fine rows per coarse one, orthonormal columns; FP32 against FP64
    n = 4 * 257
    rp, ci, v, row = operator(n, bf, 1, 5, bf)
    rng = np.random.default_rng(bc)
    Q = np.linalg.qr(rng.standard_normal((n // 4, 4 * bf, bc)))[0].reshape(n, bf, bc)
    T = mgldg.SparseBlockMatrix.from_csr(ctx, n, n // 4, bf, bc, np.arange(n + 1, dtype=np.int32),
                                         (np.arange(n) // 4).astype(np.int32), Q)
    A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, bf, bf, rp, ci, v)
    ops = mgldg.LDGOperators.create_A(ctx, A)
    f = rng.standard_normal(n * bf)
    got = [mgldg.Multigrid(ctx, ops, [T], solver=mgldg.COARSE_RELAXATION, relaxation=mgldg.RELAX_JACOBI, omega=0.7,
                           npre=1, npost=1, mean_project=0, restriction=mgldg.RESTRICT_RAT, precision=p).vcycle(f)
           for p in (mgldg.PREC_FP64, mgldg.PREC_MIXED)]
    assert np.linalg.norm(got[1] - got[0]) <= 2.2e-4 * np.linalg.norm(got[0])


def test_pair_sum_is_as_accurate_as_fp64():
    # a host restatement of PairSum in FP32 (numpy rounds every operation):
    # three two-sums per pair against adding the pairs in FP64
    rng = np.random.default_rng(5)
    f = np.float32

    def two_sum(a, b):
        s = a + b
        bb = s - a
        return s, (a - (s - bb)) + (b - bb)

    n = 10000
    for B in (2, 3, 6, 10):
        hi = rng.standard_normal((B, n)).astype(f)
        hi[0, ::2] = -hi[1:, ::2].sum(0)                          # half of the sums cancel
        lo = (hi * rng.uniform(-1, 1, (B, n)) * 2.0**-22).astype(f)
        h, l, w = np.zeros(n, f), np.zeros(n, f), np.zeros(n, f)
        for k in range(B):
            h, e = two_sum(h, hi[k])
            t, e2 = two_sum(e, lo[k])
            l, e3 = two_sum(l, t)
            w = w + (e2 + e3)
        got = h.astype(np.float64) + (l.astype(np.float64) + w.astype(np.float64))
        fp64 = np.zeros(n)
        for k in range(B):
            fp64 = fp64 + (hi[k].astype(np.float64) + lo[k].astype(np.float64))
        exact = np.add.reduce(np.concatenate([hi, lo]).astype(np.longdouble), axis=0)
        size = np.abs(hi).sum(0)
        # FP64 rounds each of the 2 B sums (2^-53); the restatement only its last two
        assert (np.abs(got - exact) <= 2.0**-52 * size).all()
        assert np.sqrt(np.mean(((got - exact) / size) ** 2)) <= np.sqrt(np.mean(((fp64 - exact) / size) ** 2)) + 2.0**-54
