"""The coarsest level's dense inverse: elimination in one cluster's shared
memory (up to 448 unknowns) and by launches over all SMs, at the edges of the
cluster's column deal (8), of its rows per pass and of its range.

Orthogonal matrices, which need a row exchange in nearly every step: the
elimination's forward error is at most 2 n u ||L|| ||U|| <= 2 n u (n rho), with
multipliers of at most one and a growth rho taken as at most 4.
"""
import numpy as np
import pytest

import mgldg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 63, 64, 144, 257, 447, 448, 449])
def test_dense_inverse(ctx, n):
    rng = np.random.default_rng(n)
    Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, 1, 1, np.arange(0, n * n + 1, n, dtype=np.int32),
                                         np.tile(np.arange(n, dtype=np.int32), n), Q.ravel())
    mg = mgldg.Multigrid(ctx, mgldg.LDGOperators.create_A(ctx, A), [], solver=mgldg.COARSE_DENSE, mean_project=0,
                         relaxation=mgldg.RELAX_JACOBI, precision=mgldg.PREC_FP64)
    b = rng.standard_normal(n)
    x = mg.vcycle(b)
    assert np.linalg.norm(x - Q.T @ b) <= 8 * n * n * 2.0**-53 * np.linalg.norm(b)


def test_singular_is_refused(ctx):
    n = 16
    v = np.ones((n, n))
    A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, 1, 1, np.arange(0, n * n + 1, n, dtype=np.int32),
                                         np.tile(np.arange(n, dtype=np.int32), n), v.ravel())
    with pytest.raises(mgldg.MgldgError):
        mgldg.Multigrid(ctx, mgldg.LDGOperators.create_A(ctx, A), [], solver=mgldg.COARSE_DENSE, mean_project=0,
                        relaxation=mgldg.RELAX_JACOBI, precision=mgldg.PREC_FP64)
