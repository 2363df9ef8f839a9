"""Transfers with a table of blocks (k_transfer): both splits of their rows
over threads (from 2^19 entries on several entries each), remainders, in a
two-level V-cycle, FP32 against FP64; FP64 against numpy.

Four fine rows per coarse one and the last coarse row with fewer; the blocks of
four rows have orthonormal columns, the fine operator's condition number is
below 3 and rows have at most 4 * 25 products, so the FP32 V-cycle's six steps
stay within 6 * 3 * 200 * 2^-24 < 2.2e-4, an FP64 product within 110 * 2^-53
< 1.3e-14 of the sum of magnitudes.
"""
import numpy as np
import pytest

import mgldg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,n", [(4, 37), (4, 131071), (4, 131075), (9, 58255), (9, 58253), (16, 32767), (16, 32770),
                                 (16, 1000), (25, 20971), (25, 20975)])
def test_table_transfers(ctx, b, n):
    rng = np.random.default_rng(b + n)
    Q = np.linalg.qr(rng.standard_normal((4 * b, b)))[0].reshape(4, b, b)
    nc = (n + 3) // 4
    col = (np.arange(n) // 4).astype(np.int32)
    T = mgldg.SparseBlockMatrix.from_csr(ctx, n, nc, b, b, np.arange(n + 1, dtype=np.int32), col, Q[np.arange(n) % 4])
    x = rng.standard_normal((nc, b))
    for k in range(4):
        want, size = x[col[k::4]] @ Q[k].T, np.abs(x[col[k::4]]) @ np.abs(Q[k]).T
        assert (np.abs(T.mv(x.ravel()).reshape(n, b)[k::4] - want) <= 1.3e-14 * size).all()
    d = rng.uniform(-1, 1, (3, b, b)) * 0.1 / b
    d = d + d.transpose(0, 2, 1) + 2 * np.eye(b)
    A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, b, b, np.arange(n + 1, dtype=np.int32),
                                         np.arange(n, dtype=np.int32), d[np.arange(n) % 3])
    ops = mgldg.LDGOperators.create_A(ctx, A)
    f = rng.standard_normal(n * b)
    got = [mgldg.Multigrid(ctx, ops, [T], solver=mgldg.COARSE_RELAXATION, relaxation=mgldg.RELAX_JACOBI, omega=0.7,
                           npre=1, npost=1, mean_project=0, restriction=mgldg.RESTRICT_RAT, precision=p).vcycle(f)
           for p in (mgldg.PREC_FP64, mgldg.PREC_MIXED)]
    assert np.linalg.norm(got[1] - got[0]) <= 2.2e-4 * np.linalg.norm(got[0])
    # a fault in single rows, too: the largest entry's error
    assert np.abs(got[1] - got[0]).max() <= 2.2e-4 * np.abs(got[0]).max() * 3
