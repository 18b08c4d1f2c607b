"""Stage kernels on meshes with more full tiles than resident CTAs: several tiles per
persistent CTA (both buffers, their barrier phases, the per-tile reset of the inflow
list) and a ragged last one, against the oracle.  Smaller meshes are cut into one
tile per SM and reach none of these."""
import math

import numpy as np
import pytest

from conftest import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import dgc_gb300 as dg  # noqa: E402
from dgc_gb300 import meshes  # noqa: E402

KINDS = {"f64": (dg.F64, None), "blocked": (dg.F32, (5, 1)), "mapped": (dg.F32, (7, 3)), "even_odd": (dg.F32, (6, 2)),
         "compensated": (dg.F32C, None)}


def relerr(a, b):
    a, b = np.ravel(a), np.ravel(b)
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def make(n, phys, N, kind):
    prec, v = KINDS[kind]
    D = dg.Discretization(meshes.jittered_square(n, 90 + N), phys, N, prec, ax=0.8, ay=-0.6, bc=dg.BC_GAUSS)
    if v:
        D.set_variant(v[N > 6])
    return D


@pytest.mark.parametrize("N", range(1, 9))
@pytest.mark.parametrize("phys,okind", [("advection", oracle.ADVECTION), ("maxwell_te", oracle.MAXWELL_TE)])
@pytest.mark.parametrize("kind", KINDS)
def test_stage(kind, phys, okind, N):
    i = make(2, phys, N, kind).info
    per_wave = i.rhs_tile * i.rhs_blocks_per_sm * i.sm_count
    n = math.isqrt(per_wave // 2) + 2
    D = make(n, phys, N, kind)
    assert D.K > per_wave and D.K // i.rhs_tile >= i.sm_count  # as many full tiles, and more than are resident
    o = oracle.Oracle(*(lambda m: (m.xy, m.cells))(meshes.jittered_square(n, 90 + N)), N)
    p = oracle.problem(okind, 0.8, -0.6, dg.BC_GAUSS)
    q0 = np.random.default_rng(N).standard_normal(D.Nf * D.K * D.Np).astype(np.float32).astype(np.float64)
    ref = o.rhs(p, 0.3, q0)
    # rounding (6e-8, FP64 1.1e-16) through sums of up to 2 Np + 3 Nfp <= 117 terms of one magnitude
    tol = 1e-12 if kind == "f64" else 2e-5
    q = D.upload(q0)
    assert relerr(D.download(D.rhs(q, 0.3)), ref) < tol
    dt = 0.1 * D.info.min_edge / (N + 1) ** 2
    qb, res = D.empty_state(), D.empty_state()
    D.lserk4_step(q.clone(), qb, res, 0.3, dt)
    qo, _ = o.lserk4_step(p, 0.3, dt, q0, np.zeros_like(q0))
    assert relerr(D.download(qb), qo) < tol
    D.check()
