"""Conjugate gradients driven from the host (MGLDG_PCG_HOST_LOOP: one iteration
at a time, the V-cycle replayed from its own graph) against blocks of
iterations in one graph: the same kernels in the same order, so the same
solutions and histories bit for bit.  Odd and even numbers of sweeps (a sweep
swaps two arrays), V-cycles and relaxations called between the solves, one and
several levels, both smoothers, the segmented form."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import hashlib, json, sys
import numpy as np
import mgldg
ctx = mgldg.Context(0)
prob = mgldg.CartesianProblem(ctx, 3, 16, tau0=16.0, tauD=16.0)
n = prob.ndof
b = np.random.default_rng(1).standard_normal((3, n))
out = {}
for relax, omega in ((mgldg.RELAX_JACOBI, 0.6), (mgldg.RELAX_GAUSS_SEIDEL, 0.8)):
    for prec in (mgldg.PREC_FP64, mgldg.PREC_MIXED):
        for pre, post, levels in ((1, 1, 3), (1, 2, 3), (2, 2, 2), (1, 1, 1), (2, 1, 1)):
            T = prob.T if levels > 1 else []
            solver = mgldg.COARSE_DENSE if levels > 1 else mgldg.COARSE_RELAXATION
            mg = mgldg.Multigrid(ctx, prob.ops, T, npre=pre, npost=post, relaxation=relax, omega=omega, precision=prec,
                                 solver=solver, max_levels=levels, mean_project=0)
            h = hashlib.sha256()
            for k in range(3):
                try:        # unequal sweeps are no symmetric preconditioner
                    x, hist = mgldg.pcg(ctx, prob.ops.A, b[k], precon=mg, tol=1e-9, maxit=70)
                    h.update(x.tobytes() + hist.tobytes())
                except mgldg.MgldgError as e:
                    h.update(str(e).encode())
                if k == 0:
                    h.update(mg.vcycle(b[1]).tobytes())
                try:
                    x, its, hists = mgldg.pcg_segmented(ctx, prob.ops.A, b[k], [0, n], mg, tol=1e-9, maxit=60)
                    h.update(x.tobytes() + its.tobytes() + b"".join(v.tobytes() for v in hists))
                except mgldg.MgldgError as e:
                    h.update(str(e).encode())
                if k == 1:
                    h.update(mg.relax(0, 1, False, b[0], b[1]).tobytes())
            out[f"{relax} {prec} {pre} {post} {levels}"] = h.hexdigest()
print(json.dumps(out))
"""


def run(host_loop):
    env = dict(os.environ, PYTHONPATH=os.path.join(ROOT, "multigrid-ldg_gb300"))
    env.pop("MGLDG_PCG_HOST_LOOP", None)
    if host_loop:
        env["MGLDG_PCG_HOST_LOOP"] = "1"
    r = subprocess.run([sys.executable, "-c", SCRIPT], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_same_results():
    assert run(True) == run(False)
