"""Inflow boundary values of the blocked FP32 stage kernels (advection): tiles
whose inflow nodes outnumber the list a CTA keeps of them, boundary faces along
the wind (a.n rounds to either sign), and tiles with and without a boundary,
against the oracle."""
import numpy as np
import pytest

from conftest import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import dgc_gb300 as dg  # noqa: E402
from dgc_gb300 import meshes  # noqa: E402

TOL32 = 2e-5  # the FP32 tolerance of the other stage tests
LIST = 256    # inflow nodes a CTA lists
WIND = (0.8, 0.6)


def relerr(a, b):
    a, b = np.ravel(a), np.ravel(b)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def loose_triangles(K, seed):
    """K triangles without common vertices: every face is a boundary face.  Of three,
    one has its first face along the wind and one inflow face, two have two inflow
    faces (a vertex pointing against the wind)."""
    rng = np.random.default_rng(seed)
    w = np.array(WIND)
    along = np.arange(K)[:, None] % 3 == 0
    p = rng.uniform(-0.6, 0.6, (K, 2))
    e = rng.uniform(0.2, 0.4, (K, 1)) * np.where(along, w * rng.choice([-1.0, 1.0], (K, 1)), [-w[1], w[0]])
    # third vertex on the left of the first edge: counter-clockwise
    t = rng.uniform(0.3, 0.7, (K, 1)) * e + rng.uniform(0.7, 1.0, (K, 1)) * np.stack([-e[:, 1], e[:, 0]], 1)
    xy = np.stack([p, p + e, p + t], 1).reshape(-1, 2)
    return meshes.Mesh(xy=xy, cells=np.arange(3 * K, dtype=np.int32).reshape(K, 3))


def check(D, m, variants):
    o = oracle.Oracle(m.xy, m.cells, D.N)
    p = oracle.problem(oracle.ADVECTION, *WIND, dg.BC_GAUSS)
    q0 = o.exact(p, 0.07)
    dt = 0.3 * D.info.min_edge / (D.N + 1) ** 2
    qo, _ = o.lserk4_step(p, 0.07, dt, q0, np.zeros_like(q0))
    ref = o.rhs(p, 0.07, q0)
    q = D.upload(q0)
    for v in variants:
        D.set_variant(v)
        assert relerr(D.download(D.rhs(q, 0.07)), ref) < TOL32, v
        qb, res = D.empty_state(), D.empty_state()
        D.lserk4_step(q.clone(), qb, res, 0.07, dt)
        assert relerr(D.download(qb), qo) < TOL32, v
    D.check()


@pytest.mark.parametrize("N", [1, 4, 8])
def test_more_inflow_nodes_than_listed(N):
    kw = dict(ax=WIND[0], ay=WIND[1], bc=dg.BC_GAUSS)
    variants = (5, 7) if N <= 6 else (1, 3)
    D = dg.Discretization(loose_triangles(7, N), "advection", N, dg.F32, **kw)
    D.set_variant(variants[0])
    te = D.info.rhs_tile
    K = te * D.info.sm_count + 3  # full tiles
    assert (te // 3 * 5) * (N + 1) > LIST
    m = loose_triangles(K, N)
    D = dg.Discretization(m, "advection", N, dg.F32, **kw)
    check(D, m, variants)


@pytest.mark.parametrize("n", [3, 40])
def test_tiles_with_and_without_boundary(n):
    m = meshes.jittered_square(n, 5)
    D = dg.Discretization(m, "advection", 4, dg.F32, ax=WIND[0], ay=WIND[1], bc=dg.BC_GAUSS)
    check(D, m, (5, 7))


@pytest.mark.parametrize("N", [2, 6, 7, 8])
@pytest.mark.parametrize("n", [24, 81])
def test_listed_and_unlisted_values_agree(N, n):
    """The batched launch evaluates inflow values where they are used, the stage
    kernel lists them (at orders 7, 8 only where a CTA has one tile, n = 24): the
    values, and so the states, are the same bits."""
    m = meshes.jittered_square(n, 6)
    D = dg.Discretization(m, "advection", N, dg.F32, ax=WIND[0], ay=WIND[1], bc=dg.BC_GAUSS)
    D.set_variant(5 if N <= 6 else 1)
    if n == 81 and N >= 7:
        assert -(-D.K // D.info.rhs_tile) > D.info.rhs_blocks_per_sm * D.info.sm_count
    o = oracle.Oracle(m.xy, m.cells, N)
    q = D.upload(o.exact(oracle.problem(oracle.ADVECTION, *WIND, dg.BC_GAUSS), 0.07))
    dt = 0.3 * D.info.min_edge / (N + 1) ** 2
    qb, res = D.empty_state(), D.empty_state()
    D.lserk4_step(q.clone(), qb, res, 0.07, dt)
    out = D.empty_state()
    dg.Batch([D]).lserk4_step([q.clone()], [out], [D.empty_state()], [0.07], [dt])
    assert torch.equal(out, qb)
    D.check()
