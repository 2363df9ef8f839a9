"""Hierarchies with dense coarsest levels of different sizes, created by several
host threads at once, each in its own context: one thread's launch limits must
not end in the other's launches.  Bound as in test_coarse_inverse_gpu.py."""
import threading

import numpy as np
import pytest

import mgldg

pytestmark = pytest.mark.gpu


def test_sizes_at_once():
    failed, done = [], threading.Event()
    start = threading.Barrier(4)

    def work(n, reps):
        try:
            ctx = mgldg.Context(0)
            rng = np.random.default_rng(n)
            Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
            A = mgldg.SparseBlockMatrix.from_csr(ctx, n, n, 1, 1, np.arange(0, n * n + 1, n, dtype=np.int32),
                                                 np.tile(np.arange(n, dtype=np.int32), n), Q.ravel())
            ops = mgldg.LDGOperators.create_A(ctx, A)
            b = rng.standard_normal(n)
            start.wait(60)
            k = 0
            while k < reps or (reps == 0 and not done.is_set()):
                mg = mgldg.Multigrid(ctx, ops, [], solver=mgldg.COARSE_DENSE, mean_project=0,
                                     relaxation=mgldg.RELAX_JACOBI, precision=mgldg.PREC_FP64)
                if k % 64 == 0:
                    x = mg.vcycle(b)
                    assert np.linalg.norm(x - Q.T @ b) <= 8 * n * n * 2.0**-53 * np.linalg.norm(b)
                k += 1
        except Exception as e:  # reported below, from the test's own thread
            failed.append(f"{n} unknowns: {e}")
        finally:
            if reps:
                done.set()

    threads = [threading.Thread(target=work, args=a) for a in ((448, 1000), (16, 0), (24, 0), (32, 0))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
