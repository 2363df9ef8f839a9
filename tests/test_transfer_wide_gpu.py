"""Table transfers (k_transfer) on operators so large that the restriction too
gives a thread several entries (from 2^19 of its rows' entries, four blocks per
row): a two-level V-cycle in both precisions against numpy in FP64.

Blocks as in test_transfer_tables_gpu.py: orthonormal columns, a fine operator of
condition number below 3, rows of at most 4 * 25 products; six steps stay within
6 * 3 * 200 u of the solution's norm, single entries within three times that of
the largest one.
"""
import numpy as np
import pytest

import mgldg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,n", [(4, 524291), (9, 233021), (16, 131075), (25, 83891)])
def test_wide_restriction(ctx, b, n):
    rng = np.random.default_rng(b + n)
    Q = np.linalg.qr(rng.standard_normal((4 * b, b)))[0].reshape(4, b, b)
    nc, idx = (n + 3) // 4, np.arange(n, dtype=np.int32)
    rp = np.arange(n + 1, dtype=np.int32)
    T = mgldg.SparseBlockMatrix.from_csr(ctx, n, nc, b, b, rp, idx // 4, Q[idx % 4])
    d = rng.uniform(-1, 1, (3, b, b)) * 0.1 / b
    d = d + d.transpose(0, 2, 1) + 2 * np.eye(b)
    ops = mgldg.LDGOperators.create_A(ctx, mgldg.SparseBlockMatrix.from_csr(ctx, n, n, b, b, rp, idx, d[idx % 3]))
    f = rng.standard_normal((n, b))

    def each(blocks, kind, x):          # blocks[kind[i]] x[i]
        y = np.empty_like(x)
        for k in range(len(blocks)):
            y[kind == k] = x[kind == k] @ blocks[k].T
        return y

    A = lambda x: each(d, idx % 3, x)
    Di = lambda x: each(np.linalg.inv(d), idx % 3, x)
    up = lambda xc: each(Q, idx % 4, xc[idx // 4])

    def down(r):
        y = np.zeros((nc, b))
        np.add.at(y, idx // 4, each(Q.transpose(0, 2, 1), idx % 4, r))
        return y

    # the coarse operator is block diagonal: one block per set of fine blocks
    nf = np.minimum(4, n - 4 * np.arange(nc))
    ckind = (np.arange(nc) * 4 % 3) * 4 + nf - 1
    C = np.zeros((12, b, b))
    for k in range(12):
        for j in range(k % 4 + 1):
            C[k] += Q[j].T @ d[(k // 4 + j) % 3] @ Q[j]
    w = 0.7
    x = w * Di(f)
    rc = down(f - A(x))
    Ci = np.linalg.pinv(C)
    xc = w * each(Ci, ckind, rc)
    xc = xc + w * each(Ci, ckind, rc - each(C, ckind, xc))
    x = x + up(xc)
    x = (x + w * Di(f - A(x))).ravel()
    for prec, u in ((mgldg.PREC_FP64, 2.0**-53), (mgldg.PREC_MIXED, 2.0**-24)):
        got = mgldg.Multigrid(ctx, ops, [T], solver=mgldg.COARSE_RELAXATION, relaxation=mgldg.RELAX_JACOBI, omega=w,
                              npre=1, npost=1, mean_project=0, restriction=mgldg.RESTRICT_RAT,
                              precision=prec).vcycle(f.ravel())
        tol = 6 * 3 * 200 * u
        assert np.linalg.norm(got - x) <= tol * np.linalg.norm(x)
        assert np.abs(got - x).max() <= 3 * tol * np.abs(x).max()
