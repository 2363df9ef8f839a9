"""The CG's fused vector passes: odd lengths and a caller's x and b that are
8-byte aligned only give the solution, bit for bit the same as aligned ones
(the passes do the same operations per entry), in every precision and with and
without a preconditioner.  The systems are diagonally dominant (condition
number below 3), so a relative residual of 1e-13 leaves the solution within
1e-12."""
import ctypes as C

import numpy as np
import pytest

import mgldg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,n", [(1, 1), (3, 37), (3, 4099), (9, 16385), (16, 33)])
@pytest.mark.parametrize("prec", [None, mgldg.PREC_FP64, mgldg.PREC_MIXED])
def test_odd_and_unaligned(ctx, b, n, prec):
    import torch
    rng = np.random.default_rng(n)
    rp = np.concatenate([[0], np.cumsum([1 + (i > 0) + (i < n - 1) for i in range(n)])]).astype(np.int32)
    ci = np.concatenate([[j for j in (i - 1, i, i + 1) if 0 <= j < n] for i in range(n)]).astype(np.int32)
    row = np.repeat(np.arange(n), np.diff(rp))
    off = rng.standard_normal((b, b)) * 0.2 / b
    v = np.where((ci > row)[:, None, None], off, off.T)
    v[ci == row] = 2 * np.eye(b)
    xt = rng.standard_normal((n, b))
    f = np.zeros((n, b))
    np.add.at(f, row, np.einsum("kij,kj->ki", v, xt[ci]))
    A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, b, b, rp, ci, v)
    ops = mgldg.LDGOperators.create_A(ctx, A)
    mg = None
    if prec is not None:
        mg = mgldg.Multigrid(ctx, ops, [], solver=mgldg.COARSE_RELAXATION, relaxation=mgldg.RELAX_JACOBI, omega=0.8,
                             npre=1, npost=1, mean_project=0, precision=prec)
    got = []
    for off8 in (0, 1):
        fb = torch.zeros(n * b + 1, dtype=torch.float64, device="cuda")
        xb = torch.zeros_like(fb)
        fv, xv = fb[off8:off8 + n * b], xb[off8:off8 + n * b]
        # 16 x 16 products read x in 16-byte words, so there only b moves
        if b == 16:
            xv = xb[:n * b]
        fv.copy_(torch.from_numpy(f.ravel()))
        torch.cuda.synchronize()
        it = C.c_int()
        ctx.check(mgldg.lib().mgldg_pcg_dev(ctx.h, mg.h if mg else None, ops.A.h, C.c_void_p(fv.data_ptr()),
                                            C.c_void_p(xv.data_ptr()), 1e-13, 200, C.byref(it), np.zeros(200)), "pcg")
        ctx.sync()
        got.append(xv.cpu().numpy())
        assert np.abs(got[-1] - xt.ravel()).max() <= 1e-12 * max(1.0, np.abs(xt).max())
    assert np.array_equal(got[0], got[1])
