"""Gauss-Seidel passes whose CTAs have several times more rows than the
shared-memory ring has slots (k_gs_tiles): 30 meshes side by side in one
operator -- chains of rows, 5-point grids and rows without neighbours, so that
the CTAs run far apart -- against sequential sweeps in numpy.  Blocks of 10 in
FP64 have a warp count that is no power of two.

Off-diagonal blocks are scaled so that |Dinv| sum_j |A_ij| <= 1/2 in the
infinity norm; with omega = 0.8 the result is within 2.5 times one row update's
rounding, (m + 4) u (|Dinv| (|b| + |A| |x|) + |x|) for rows of m products.
"""
import numpy as np
import pytest

import mgldg

pytestmark = pytest.mark.gpu

N, COPIES = 400, 30


def pattern(kind):
    """neighbours of every row of one mesh"""
    if kind == "chain":
        return [[j for j in (i - 1, i + 1) if 0 <= j < N] for i in range(N)]
    if kind == "free":
        return [[] for _ in range(N)]
    pos = sorted((y // 4, x // 4, y % 4, x % 4, y, x) for y in range(20) for x in range(20))
    num = {(p[4], p[5]): k for k, p in enumerate(pos)}
    out = [None] * N
    for (y, x), k in num.items():
        out[k] = [num[q] for q in ((y, x + 1), (y + 1, x), (y, x - 1), (y - 1, x)) if q in num]
    return out


@pytest.mark.parametrize("b", [9, 10])
@pytest.mark.parametrize("reverse", [False, True])
def test_ring_wraps(ctx, b, reverse):
    rng = np.random.default_rng(b)
    rp, ci, vals, meshes = [0], [], [], []
    for c in range(COPIES):
        nb = pattern(("chain", "grid", "free")[c % 3])
        rows = []
        for i in range(N):
            cols = sorted(nb[i] + [i])
            v = rng.uniform(-1, 1, (len(cols), b, b))
            d = cols.index(i)
            v[d] = 0.1 * (v[d] + v[d].T) / b + 2 * np.eye(b)
            Dinv = np.linalg.inv(v[d])
            off = sum(np.abs(v[k]).sum(1).max() for k in range(len(cols)) if k != d)
            if off > 0:
                s = min(1.0, 0.5 / (off * np.abs(Dinv).sum(1).max()))
                for k in range(len(cols)):
                    if k != d:
                        v[k] *= s
            rows.append((cols, v, d, Dinv))
            rp.append(rp[-1] + len(cols))
            ci += [c * N + j for j in cols]
            vals.append(v)
        meshes.append(rows)
    n = N * COPIES
    f, x = rng.standard_normal((n, b)), rng.standard_normal((n, b))
    nsw = 2
    want = x.copy()
    dmax = 0.0
    for c, rows in enumerate(meshes):
        o = c * N
        for _ in range(nsw):
            for i in range(N - 1, -1, -1) if reverse else range(N):
                cols, v, d, Dinv = rows[i]
                t = f[o + i].copy()
                for k, j in enumerate(cols):
                    if k != d:
                        t -= v[k] @ want[o + j]
                want[o + i] += 0.8 * (Dinv @ t - want[o + i])
                dmax = max(dmax, np.abs(Dinv).sum(1).max())
    xm = max(np.abs(x).max(), np.abs(want).max())
    size = 2 * (np.abs(f).max() * dmax + xm)
    A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, b, b, np.array(rp, np.int32), np.array(ci, np.int32),
                                         np.concatenate(vals))
    ops = mgldg.LDGOperators.create_A(ctx, A)
    for prec, u in ((mgldg.PREC_FP64, 2.0**-53), (mgldg.PREC_MIXED, 2.0**-24)):
        mg = mgldg.Multigrid(ctx, ops, [], solver=mgldg.COARSE_RELAXATION, relaxation=mgldg.RELAX_GAUSS_SEIDEL,
                             omega=0.8, mean_project=0, precision=prec)
        first = None
        for _ in range(20):
            got = mg.relax(0, nsw, reverse, f.ravel(), x.ravel()).reshape(n, b)
            if first is None:
                first = got
                assert np.abs(got - want).max() <= 2.5 * (6 * b + 4) * u * size
            assert np.array_equal(got, first)
