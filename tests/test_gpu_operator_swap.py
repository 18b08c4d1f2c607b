"""A caller's own CUDA graph, captured with operators that have the reflection
symmetry and replayed after dgc_set_operators took it away (and after it gave it
back): the replay gives the operators that are set, like a call outside the graph."""
import numpy as np
import pytest

from conftest import oracle  # noqa: F401

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import dgc_gb300 as dg  # noqa: E402
from dgc_gb300 import meshes  # noqa: E402


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def check(D, form, call, tol, changes=("any",)):
    """call() enqueues the operation and returns its output tensors (always the same ones)."""
    w = (dg.OP_DR_WEAK, dg.OP_DS_WEAK) if form == 0 else (dg.OP_DR_STRONG, dg.OP_DS_STRONG)
    Dr, Ds, L = D.operator(w[0]).copy(), D.operator(w[1]).copy(), D.operator(dg.OP_LIFT).copy()
    out = call()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call()
    g.replay()
    torch.cuda.synchronize()
    base = [o.clone() for o in out]
    rng = np.random.default_rng(3)
    for c in changes:
        if c == "any":
            new = [A + 0.1 * rng.standard_normal(A.shape) for A in (Dr, Ds, L)]
        else:  # still symmetric, but volume and flux terms no longer match
            new = [1.01 * Dr, 1.01 * Ds, L]
        D.set_operators(form, *new)
        call()
        torch.cuda.synchronize()
        want = [o.clone() for o in out]
        for o in out:
            o.zero_()
        g.replay()
        torch.cuda.synchronize()
        for o, x, b in zip(out, want, base):
            assert rel(x, b) > 1e-4  # the change shows
            assert rel(o, x) < tol
        D.set_operators(form, Dr, Ds, L)
        g.replay()
        torch.cuda.synchronize()
        for o, b in zip(out, base):
            assert torch.equal(o, b)
    D.check()


@pytest.mark.parametrize("N", range(1, 9))
@pytest.mark.parametrize("phys", ["advection", "maxwell_tm", "maxwell_te"])
@pytest.mark.parametrize("prec", [dg.F64, dg.F32])
def test_stage(prec, phys, N):
    D = dg.Discretization(meshes.jittered_square(7, N), phys, N, prec, ax=-0.7, ay=0.4)
    if prec == dg.F32:
        D.set_variant(6 if N <= 6 else 2)
    q = D.upload(np.random.default_rng(N).standard_normal(D.Nf * D.K * D.Np))
    out, qb, res = D.empty_state(), D.empty_state(), D.empty_state()

    def call():
        D.rhs(q, 0.3, out=out)
        res.zero_()
        D.lserk4_stage(0, q, qb, res, 0.3, 1e-3)
        return out, res

    # sums of up to 3 Np + 3 Nfp terms in another order: 1e-15 and 6e-8 per operation
    check(D, 0, call, 1e-12 if prec == dg.F64 else 2e-5, ("any",) if prec == dg.F64 else ("any", "scaled"))


@pytest.mark.parametrize("N", range(1, 9))
def test_laplace(N):
    D = dg.Discretization(meshes.jittered_square(7, N), "laplace", N, dg.F64)
    D.set_shift(2.5)
    u = D.upload(np.random.default_rng(N).standard_normal(D.K * D.Np))
    a, b = D.empty_state(), D.empty_state()

    def call():
        D.laplace(u, out=a)
        D.spd(u, out=b)
        return a, b

    check(D, 1, call, 1e-12)


@pytest.mark.parametrize("N", range(1, 9))
@pytest.mark.parametrize("phys", ["advection", "laplace"])
def test_grad_div(phys, N):
    D = dg.Discretization(meshes.jittered_square(7, N), phys, N, dg.F64)
    rng = np.random.default_rng(N)
    u, v = (D.upload(x) for x in rng.standard_normal((2, D.K * D.Np)))
    gx, gy, d = D.empty_state(), D.empty_state(), D.empty_state()

    def call():
        D.grad(u, sign=-1.0, out=(gx, gy))
        D.div(u, v, sign=1.0, out=d)
        return gx, gy, d

    check(D, 0, call, 1e-12)
