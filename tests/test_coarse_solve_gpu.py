"""The coarsest level's dense solve at the lines between its two row loops
(wide loads from 257 to 2,048 unknowns), with odd sizes, whose rows start on an
odd entry every second time.

Householder reflections Q = I - 2 v v^T are their own inverses, so the solve of
Q x = b gives Q b; the elimination's forward error is at most 8 n^2 u ||b||
(2 n u ||L|| ||U|| with multipliers of at most one and a growth of at most 4).
A left out or doubled entry of a row changes x by about 2 ||b|| / n.
"""
import numpy as np
import pytest

import mgldg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [mgldg.PREC_FP64, mgldg.PREC_MIXED])
@pytest.mark.parametrize("n", [255, 256, 257, 258, 511, 2047, 2048, 2049])
def test_dense_solve(ctx, n, precision):
    rng = np.random.default_rng(n)
    v = rng.standard_normal(n)
    v /= np.linalg.norm(v)
    Q = np.eye(n) - 2.0 * np.outer(v, v)
    A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, 1, 1, np.arange(0, n * n + 1, n, dtype=np.int32),
                                         np.tile(np.arange(n, dtype=np.int32), n), Q.ravel())
    mg = mgldg.Multigrid(ctx, mgldg.LDGOperators.create_A(ctx, A), [], solver=mgldg.COARSE_DENSE, mean_project=0,
                         relaxation=mgldg.RELAX_JACOBI, precision=precision)
    b = rng.standard_normal(n)
    x = mg.vcycle(b)
    # FP32 right-hand side and result: half a unit in the last place each
    tol = 8 * n * n * 2.0**-53 + (2 * 2.0**-24 if precision == mgldg.PREC_MIXED else 0.0)
    assert np.linalg.norm(x - Q @ b) <= tol * np.linalg.norm(b)
