"""Caller's device vectors that start on an odd double (8-byte, not 16-byte
aligned): products, solves and V-cycles give what they give on aligned copies.

A row of the product has at most 5 b products: within (5 b + 5) 2^-52 of the sum
of magnitudes.  The solves run the same iterations up to rounding: to 1e-10, so
they agree to 1e-8 of the largest entry."""
import ctypes as C

import numpy as np
import pytest

import mgldg

pytestmark = pytest.mark.gpu


def pair(torch, v):
    """the vector at an aligned address and one entry further on"""
    buf = torch.zeros(len(v) + 1, dtype=torch.float64, device="cuda")
    u = buf[1:]
    u.copy_(torch.from_numpy(v))
    a = torch.from_numpy(v).cuda()
    assert a.data_ptr() % 16 == 0 and u.data_ptr() % 16 == 8
    return a, u


def ptr(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("b", [1, 3, 4, 6, 8, 9, 10, 16, 25, 27])
def test_product(ctx, b):
    import torch

    rng = np.random.default_rng(b)
    n = 301
    cols = [np.unique(np.r_[i, rng.integers(0, n, 4)]) for i in range(n)]
    rp = np.r_[0, np.cumsum([len(c) for c in cols])].astype(np.int32)
    v = rng.standard_normal((rp[-1], b, b))
    ci = np.concatenate(cols).astype(np.int32)
    A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, b, b, rp, ci, v)
    x, y = rng.standard_normal(n * b), rng.standard_normal(n * b)
    row = np.repeat(np.arange(n), np.diff(rp))
    want, size = y.reshape(n, b).copy(), np.abs(y).reshape(n, b).copy()
    np.add.at(want, row, 2 * np.einsum("kij,kj->ki", v, x.reshape(n, b)[ci]))
    np.add.at(size, row, 2 * np.einsum("kij,kj->ki", np.abs(v), np.abs(x).reshape(n, b)[ci]))
    for xs in pair(torch, x):
        for ys in pair(torch, y):
            torch.cuda.synchronize()
            ctx.check(mgldg.lib().mgldg_bsr_mv_dev(ctx.h, 2.0, A.h, ptr(xs), 1.0, ptr(ys)), "mv")
            ctx.sync()
            # rows of 5 b products and y
            assert (np.abs(ys.cpu().numpy().reshape(n, b) - want) <= (5 * b + 5) * 2.0**-52 * size).all()


# 16 x 16 blocks below and from the table kernels' limit on, and 9 x 9
@pytest.mark.parametrize("P,n", [(4, 16), (4, 128), (3, 32)])
@pytest.mark.parametrize("prec", [mgldg.PREC_FP64, mgldg.PREC_MIXED])
def test_solves(ctx, P, n, prec):
    import torch

    prob = mgldg.CartesianProblem(ctx, P, n, tau0=1.0 * n, tauD=1.0 * n)
    mg = mgldg.Multigrid(ctx, prob.ops, prob.T, npre=2, npost=2, relaxation=mgldg.RELAX_JACOBI, omega=0.6,
                         mean_project=0, precision=prec, solver=mgldg.COARSE_DENSE, max_levels=n.bit_length() - 2)
    b = np.random.default_rng(n).standard_normal(prob.ndof)
    L, got = mgldg.lib(), {}
    off = np.array([0, prob.ndof], np.int64)
    for k, bs in enumerate(pair(torch, b)):
        for form in ("pcg", "seg", "vcycle", "batch"):
            x = pair(torch, np.zeros(prob.ndof))[k]
            hist, it, its = np.zeros(60), C.c_int(), np.zeros(1, np.int32)
            torch.cuda.synchronize()
            A = prob.ops.A.h
            if form == "pcg":
                rc = L.mgldg_pcg_dev(ctx.h, mg.h, A, ptr(bs), ptr(x), 1e-10, 60, C.byref(it), hist)
            elif form == "seg":
                rc = L.mgldg_pcg_segmented_dev(ctx.h, mg.h, A, 1, off.ctypes.data_as(C.POINTER(C.c_int64)), ptr(bs),
                                               ptr(x), 1e-10, 60, its, hist)
            elif form == "vcycle":
                rc = L.mgldg_mg_vcycle_dev(ctx.h, mg.h, ptr(bs), ptr(x))
            else:
                rc = L.mgldg_pcg_batched_dev(ctx.h, mg.h, A, 1, ptr(bs), ptr(x), 1e-10, 60, its, hist)
            ctx.check(rc, form)
            ctx.sync()
            got[form, k] = x.cpu().numpy()
    for form in ("pcg", "seg", "vcycle", "batch"):
        scale = np.abs(got[form, 0]).max()
        assert np.abs(got[form, 1] - got[form, 0]).max() <= 1e-8 * scale


@pytest.mark.parametrize("k", [1, 2, 5, 64])
def test_columns(ctx, k):
    import torch

    prob = mgldg.CartesianProblem(ctx, 4, 64, tau0=64.0, tauD=64.0)
    mg = mgldg.Multigrid(ctx, prob.ops, prob.T, npre=1, npost=1, relaxation=mgldg.RELAX_JACOBI, omega=0.6,
                         mean_project=0, solver=mgldg.COARSE_DENSE, max_levels=5)
    B = np.random.default_rng(k).standard_normal(prob.ndof * k)
    got = []
    for q, bs in enumerate(pair(torch, B)):
        x = pair(torch, np.zeros(prob.ndof * k))[q]
        its, hist = np.zeros(k, np.int32), np.zeros(60 * k)
        torch.cuda.synchronize()
        ctx.check(mgldg.lib().mgldg_pcg_batched_dev(ctx.h, mg.h, prob.ops.A.h, k, ptr(bs), ptr(x), 1e-10, 60, its, hist),
                  "batched")
        ctx.sync()
        got.append(x.cpu().numpy())
    assert np.abs(got[1] - got[0]).max() <= 1e-8 * np.abs(got[0]).max()
