"""Gauss-Seidel passes over tiles of rows (k_gs_tiles) against sequential
sweeps in numpy: every block size, tile remainders, both directions, one to
five sweeps (a pass takes four), unsymmetric patterns (rows that are waited for
but not read), rows with more blocks than the kernel's buffers (8) and columns
than a warp's lanes (32), CTAs with more rows than the shared-memory ring (64).

Off-diagonal blocks are scaled so that |Dinv| sum_j |A_ij| <= 1/2 in the
infinity norm: with omega = 0.8 a sweep damps earlier errors to 0.2 + 0.4 of
them, so the result is within 1 / (1 - 0.6) = 2.5 times one row update's
rounding, (m + 4) u (|Dinv| (|b| + |A| |x|) + |x|) for rows of m products.
"""
import numpy as np
import pytest

import mgldg

pytestmark = pytest.mark.gpu


def system(n, b, kind, seed):
    rng = np.random.default_rng(seed)
    nbr = [set() for _ in range(n)]
    if kind == "grid":                     # 5-point grid of 4 x 4 patches' order
        m = int(round(n**0.5))
        assert m * m == n
        w = 4 if m % 4 == 0 else 1
        pos = sorted(((y // w, x // w, y % w, x % w, y, x) for y in range(m) for x in range(m)))
        num = {(p[4], p[5]): k for k, p in enumerate(pos)}
        for (y, x), k in num.items():
            for dy, dx in ((0, 1), (1, 0), (0, -1), (-1, 0)):
                if (y + dy, x + dx) in num:
                    nbr[k].add(num[y + dy, x + dx])
    else:
        deg = {"band": 4, "wide": 11, "long": 45}[kind]
        for i in range(n):
            for j in rng.integers(max(0, i - 40), min(n, i + 41), rng.integers(0, deg + 1)):
                if j != i:
                    nbr[i].add(int(j))     # not symmetrised
    ci = [np.array(sorted(s | {i}), np.int32) for i, s in enumerate(nbr)]
    rp = np.concatenate([[0], np.cumsum([len(c) for c in ci])]).astype(np.int32)
    ci = np.concatenate(ci)
    row = np.repeat(np.arange(n), np.diff(rp))
    v = rng.uniform(-1, 1, (len(ci), b, b))
    d = row == ci
    v[d] = 0.1 * (v[d] + v[d].transpose(0, 2, 1)) / b + 2 * np.eye(b)
    Dinv = np.linalg.inv(v[d])
    off = np.abs(v).sum(2).max(1)
    off[d] = 0
    tot = np.zeros(n)
    np.add.at(tot, row, off)
    scale = 0.5 / (np.maximum(tot, 1e-30) * np.abs(Dinv).sum(2).max(1))
    v[~d] *= np.minimum(scale[row[~d]], 1.0)[:, None, None]
    return rp, ci, v, Dinv


def sweeps(rp, ci, v, Dinv, f, x, nsw, reverse, omega):
    x = x.copy()
    n = len(rp) - 1
    for _ in range(nsw):
        for i in range(n - 1, -1, -1) if reverse else range(n):
            k = np.arange(rp[i], rp[i + 1])
            k = k[ci[k] != i]
            t = f[i] - np.einsum("kij,kj->i", v[k], x[ci[k]])
            x[i] += omega * (Dinv[i] @ t - x[i])
    return x


@pytest.mark.parametrize("b,n,kind,nsw", [(1, 1, "band", 1), (3, 15, "band", 2), (4, 16, "grid", 2), (6, 17, "band", 5),
                                          (8, 64, "grid", 3), (9, 144, "grid", 2), (10, 257, "wide", 2),
                                          (16, 256, "grid", 4), (16, 100, "band", 1), (9, 1000, "long", 2),
                                          (16, 333, "long", 1), (6, 2000, "wide", 2), (1, 45001, "band", 2),
                                          (3, 20011, "wide", 1), (25, 60, "band", 2), (27, 33, "wide", 1)])
@pytest.mark.parametrize("reverse", [False, True])
def test_passes(ctx, b, n, kind, nsw, reverse):
    rp, ci, v, Dinv = system(n, b, kind, 7 * n + b)
    rng = np.random.default_rng(n)
    f, x = rng.standard_normal((n, b)), rng.standard_normal((n, b))
    want = sweeps(rp, ci, v, Dinv, f, x, nsw, reverse, 0.8)
    xm = max(np.abs(x).max(), np.abs(want).max())
    size = 2 * (np.abs(f).max() * np.abs(Dinv).sum(2).max() + xm)
    m = np.diff(rp).max() * b + b
    A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, b, b, rp, ci, v)
    ops = mgldg.LDGOperators.create_A(ctx, A)
    for prec, u in ((mgldg.PREC_FP64, 2.0**-53), (mgldg.PREC_MIXED, 2.0**-24)):
        mg = mgldg.Multigrid(ctx, ops, [], solver=mgldg.COARSE_RELAXATION, relaxation=mgldg.RELAX_GAUSS_SEIDEL,
                             omega=0.8, mean_project=0, precision=prec)
        got = [mg.relax(0, nsw, reverse, f.ravel(), x.ravel()).reshape(n, b) for _ in range(2)]
        assert np.array_equal(got[0], got[1])
        assert np.abs(got[0] - want).max() <= 2.5 * (m + 4) * u * size
