"""Programmatic dependent launch changes timing only, for the even / odd kernels: the
FP32 stage (variant 6; 2 at order 7), the FP64 stage, gradient and divergence give
bit-identical results with the launch attribute on (default) and off
(DGC_STAGE_OVERLAP=0), the FP64 CG solve agrees to its tolerance.  The switch is read
once per process: one child process per setting, on meshes with one tile per SM,
where these kernels launch overlapped."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))

CHILD = r"""
import os, sys
import numpy as np
sys.path.insert(0, os.path.join(sys.argv[1], "dg-on-cuda_gb300"))
import torch
import dgc_gb300 as dg
from dgc_gb300 import meshes
res = {}
for phys in ("advection", "maxwell_te"):
    for tag, prec, N, n in (("f32", dg.F32, 4, 16), ("f32", dg.F32, 7, 9), ("f64", dg.F64, 3, 8), ("f64", dg.F64, 6, 16)):
        D = dg.Discretization(meshes.jittered_square(n, 7), phys, N, prec, ax=0.8, ay=0.6, bc=dg.BC_GAUSS)
        if prec == dg.F32:
            D.set_variant(6 if N <= 6 else 2)
        q0 = np.random.default_rng(N).standard_normal(D.Nf * D.K * D.Np)
        dt = 0.1 * D.info.min_edge / (N + 1) ** 2
        a, b, r = D.upload(q0), D.empty_state(), D.empty_state()
        for i in range(12):
            D.lserk4_step(a, b, r, i * dt, dt)
            a, b = b, a
        key = "%s_%s_%d_" % (phys, tag, N)
        res[key + "eager"] = a.cpu().numpy()
        fin = D.lserk4_run(D.upload(q0), D.empty_state(), D.empty_state(), 0.0, dt, 20, graph=True)
        res[key + "graph"] = fin.cpu().numpy()
        D.check()
D = dg.Discretization(meshes.jittered_square(16, 11), "laplace", 4, dg.F64, tau=dg.TAU_SCALED, dirichlet=True)
u = D.upload(np.random.default_rng(1).standard_normal(D.K * D.Np))
gx, gy = u, u
for i in range(6):  # each launch reads the one before
    gx, gy = D.grad(gx if i else u, sign=-1.0)
    gx = D.div(gx, gy, sign=1.0)
    gx = gx / gx.norm()
    gx = D.spd(D.laplace(gx))
    gx = gx / gx.norm()
res["chain"] = gx.cpu().numpy()
x, y = D.node_xy()
b = D.mass(D.upload((2 * np.pi ** 2 * np.sin(np.pi * x) * np.sin(np.pi * y)).reshape(-1)))
xs, st = D.pcg(b, mode=dg.SOLVE_FP64_PCG, rtol=1e-10, maxit=40000)
res["poisson"] = xs.cpu().numpy()
D.check()
np.savez(sys.argv[2], **res)
"""


@pytest.fixture(scope="module", autouse=True)
def built():
    from dgc_gb300 import build
    build.build()


def run_child(tmp_path, overlap):
    out = os.path.join(str(tmp_path), "overlap%d.npz" % overlap)
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT, out], env=dict(os.environ, DGC_STAGE_OVERLAP=str(overlap)),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    return np.load(out)


def test_results_with_and_without_launch_overlap(tmp_path):
    on, off = run_child(tmp_path, 1), run_child(tmp_path, 0)
    assert sorted(on.files) == sorted(off.files)
    for k in on.files:
        assert np.all(np.isfinite(on[k])), k
        if k == "poisson":
            # the dot products end in FP64 atomics, whose order varies from run to run
            assert np.linalg.norm(on[k] - off[k]) < 1e-9 * np.linalg.norm(off[k])
        else:
            assert np.array_equal(on[k].view(np.uint8), off[k].view(np.uint8)), k
