"""Which operators of a hierarchy get a table in the first multi-vector solve
(spmm_rep.cu): all large ones in FP64, the finest alone in the mixed form, told
from the number of setup launches; and products at the limits of both forms,
against the single-vector path (test_repeat_batched_gpu.py's check)."""
import numpy as np
import pytest

import mgldg
import test_repeat_batched_gpu as base

pytestmark = pytest.mark.gpu


def test_tables_built(ctx):
    b, n = 9, 6000
    rng = np.random.default_rng(4)
    launches = {}
    Q = np.linalg.qr(rng.standard_normal((2 * b, b)))[0].reshape(2, b, b)
    T = mgldg.SparseBlockMatrix.from_csr(ctx, n, n // 2, b, b, np.arange(n + 1, dtype=np.int32),
                                         (np.arange(n) // 2).astype(np.int32), Q[np.arange(n) % 2])
    F = rng.standard_normal((n * b, 3))
    for prec in (mgldg.PREC_FP64, mgldg.PREC_MIXED):
        ops = mgldg.LDGOperators.create_A(ctx, base.operator(ctx, b, n, b))
        mg = mgldg.Multigrid(ctx, ops, [T], solver=mgldg.COARSE_RELAXATION, relaxation=mgldg.RELAX_JACOBI, omega=0.6,
                             npre=1, npost=1, mean_project=0, restriction=mgldg.RESTRICT_RAT, precision=prec)
        before = ctx.prof()["setup"][0]
        mgldg.pcg_batched(ctx, ops.A, F, precon=mg, tol=1e-8, maxit=30)
        launches[prec] = ctx.prof()["setup"][0] - before
    assert launches[mgldg.PREC_MIXED] > 0
    assert launches[mgldg.PREC_FP64] == 2 * launches[mgldg.PREC_MIXED]


@pytest.mark.parametrize("b,n,prec", [(4, 19999, mgldg.PREC_MIXED), (4, 20000, mgldg.PREC_MIXED),
                                      (16, 3071, mgldg.PREC_FP64), (16, 3072, mgldg.PREC_FP64)])
def test_limits(ctx, b, n, prec):
    base.test_columns_match_single(ctx, b, n, prec)
