"""FP64 kernels in the even / odd basis of the reflection r <-> s against the
oracle (every order, meshes smaller than a tile, with a ragged last tile and with
many tiles), and the node-by-node kernels that operators without the symmetry
still run."""
import numpy as np
import pytest
import torch

import dgc_gb300 as dg
import oracle

pytestmark = pytest.mark.gpu

# rounding: the oracle and the kernels sum the same O(N^2) terms in another order
TOL = 1e-12
PHYS = [("advection", oracle.ADVECTION), ("maxwell_tm", oracle.MAXWELL_TM), ("maxwell_te", oracle.MAXWELL_TE)]


def rel(a, b):
    return np.linalg.norm(np.ravel(a) - np.ravel(b)) / np.linalg.norm(np.ravel(b))


@pytest.mark.parametrize("n", [1, 5, 23])
@pytest.mark.parametrize("N", range(1, 9))
def test_stage(N, n):
    m = dg.meshes.jittered_square(n, seed=N)
    o = oracle.Oracle(m.xy, m.cells, N)
    rng = np.random.default_rng(N)
    for name, kind in PHYS:
        D = dg.Discretization(m, name, N, dg.F64, ax=-0.7, ay=0.4)
        p = oracle.problem(kind, ax=-0.7, ay=0.4)
        q0 = rng.standard_normal(D.Nf * D.K * D.Np)
        q = D.upload(q0)
        ref = o.rhs(p, 0.3, q0)
        assert rel(D.download(D.rhs(q, 0.3)), ref) < TOL
        for dt in (1e-3, -1e-3):  # the time step is folded into the face factors, whose sign picks the upwind side
            qb, res = D.empty_state(), D.empty_state()
            D.lserk4_stage(0, q, qb, res, 0.3, dt)
            assert rel(D.download(res), dt * ref) < TOL
        D.check()


@pytest.mark.parametrize("n", [1, 4, 19])
@pytest.mark.parametrize("N", range(1, 9))
def test_laplace(N, n):
    m = dg.meshes.jittered_square(n, seed=10 + N)
    o = oracle.Oracle(m.xy, m.cells, N)
    D = dg.Discretization(m, "laplace", N, dg.F64, tau=dg.TAU_SCALED, dirichlet=True)
    u0 = np.random.default_rng(N).standard_normal(D.K * D.Np)
    u = D.upload(u0)
    assert rel(D.download(D.laplace(u)), o.laplace(u0, True, 1)) < TOL
    s = o.spd(u0, 1)
    assert rel(D.download(D.spd(u)), s) < TOL
    # shifted form S + shift J M
    D.set_shift(3.5)
    assert rel(D.download(D.spd(u)), s + 3.5 * D.download(D.mass(u))) < TOL
    D.check()


@pytest.mark.parametrize("n", [1, 4, 19])
@pytest.mark.parametrize("N", range(1, 9))
def test_grad_div(N, n):
    m = dg.meshes.jittered_square(n, seed=20 + N)
    o = oracle.Oracle(m.xy, m.cells, N)
    D = dg.Discretization(m, "laplace", N, dg.F64)
    rng = np.random.default_rng(N)
    u0, v0 = rng.standard_normal((2, D.K * D.Np))
    g, h = rng.standard_normal((2, D.info.num_boundary_faces * D.Nfp))
    u, v = D.upload(u0), D.upload(v0)
    gx, gy = D.grad(u, g=g, sign=-1.0)
    ref = o.grad(u0, g, -1.0)
    d = D.div(u, v, gx=g, gy=h, sign=0.5)
    assert rel(D.download(gx), ref[0]) < TOL and rel(D.download(gy), ref[1]) < TOL
    assert rel(D.download(d), o.div(u0, v0, g, h, 0.5)) < TOL
    # inputs off a 16-byte boundary take the node-by-node kernel
    shift = lambda t: torch.cat([t.new_zeros(1), t])[1:]  # noqa: E731
    us, vs = shift(u), shift(v)
    assert us.data_ptr() % 16 == 8
    gxs, gys = D.grad(us, g=g, sign=-1.0)
    assert rel(D.download(gxs), ref[0]) < TOL and rel(D.download(gys), ref[1]) < TOL
    assert rel(D.download(D.div(us, vs, gx=g, gy=h, sign=0.5)), D.download(d)) < TOL
    D.check()


@pytest.mark.parametrize("N,n", [(1, 9), (2, 1), (4, 23), (5, 40), (8, 7)])
def test_grad_div_without_kept_constants(N, n):
    """Advection handles keep no per-element constants: the same ones formed in the
    kernel, so the same bits as on a laplace handle."""
    m = dg.meshes.jittered_square(n, seed=3 + n)
    A, B = dg.Discretization(m, "laplace", N, dg.F64), dg.Discretization(m, "advection", N, dg.F64, ax=1.0, ay=0.5)
    u = torch.randn(A.K * A.NpP, dtype=torch.float64, device="cuda")
    gx, gy = A.grad(u)
    hx, hy = B.grad(u)
    valid = torch.arange(A.K * A.NpP, device="cuda") % A.NpP < A.Np
    for a, b in ((gx, hx), (gy, hy), (A.div(gx, gy), B.div(hx, hy))):
        assert torch.equal(a.reshape(-1)[valid], b.reshape(-1)[valid])


@pytest.mark.parametrize("n", [1, 4, 9])
@pytest.mark.parametrize("N", range(1, 9))
def test_fp32_stage(N, n):
    """dg_rhs_sym_kernel (variant 6, 2 at orders 7 and 8): less than a tile, whole
    tiles and a ragged last one; RHS, LSERK4 stage and classical RK4."""
    m = dg.meshes.jittered_square(n, seed=30 + N)
    o = oracle.Oracle(m.xy, m.cells, N)
    rng = np.random.default_rng(N)
    for name, kind in PHYS:
        D = dg.Discretization(m, name, N, dg.F32, ax=-0.7, ay=0.4)
        D.set_variant(6 if N <= 6 else 2)
        p = oracle.problem(kind, ax=-0.7, ay=0.4)
        q0 = rng.standard_normal(D.Nf * D.K * D.Np).astype(np.float32).astype(np.float64)
        q = D.upload(q0)
        ref = o.rhs(p, 0.3, q0)
        # FP32 rounding (6e-8) through sums of up to 100 terms of one magnitude
        assert rel(D.download(D.rhs(q, 0.3)), ref) < 2e-5
        dt = 0.1 * D.info.min_edge / (N + 1) ** 2
        qb, res = D.empty_state(), D.empty_state()
        D.lserk4_stage(0, q, qb, res, 0.3, dt)
        assert rel(D.download(res), dt * ref) < 2e-5
        work = [D.empty_state() for _ in range(3)]
        D.rk4_step(q, 0.3, dt, work)
        assert rel(D.download(q), o.rk4_step(p, 0.3, dt, q0)) < 2e-5
        D.check()


def test_fp32_operators_without_the_symmetry():
    """The blocked kernel takes over."""
    N = 6
    m = dg.meshes.jittered_square(6, seed=2)
    D = dg.Discretization(m, "maxwell_te", N, dg.F32)
    q = D.upload(np.random.default_rng(0).standard_normal(D.Nf * D.K * D.Np))
    Dr, Ds, L = (D.operator(w).copy() for w in (dg.OP_DR_WEAK, dg.OP_DS_WEAK, dg.OP_LIFT))
    Dr[3, 7] += 0.5
    D.set_operators(0, Dr, Ds, L)
    D.set_variant(5)
    want = D.rhs(q, 0.0).clone()
    D.set_variant(6)
    assert torch.equal(D.rhs(q, 0.0), want)


def test_operators_without_the_symmetry():
    """The node-by-node kernels take over, and give the caller's operators."""
    N = 4
    m = dg.meshes.jittered_square(6, seed=2)
    D = dg.Discretization(m, "advection", N, dg.F64, ax=0.8, ay=0.6, bc=dg.BC_ZERO)
    q = D.upload(np.random.default_rng(0).standard_normal(D.K * D.Np))
    base = D.download(D.rhs(q, 0.0))
    Dr, Ds, L = (D.operator(w).copy() for w in (dg.OP_DR_WEAK, dg.OP_DS_WEAK, dg.OP_LIFT))
    E = np.zeros_like(Dr)
    E[3, 7] = 0.5
    qa, qb, res = q.clone(), D.empty_state(), D.empty_state()
    D.lserk4_run(qa, qb, res, 0.0, 1e-3, 4)  # a cached graph holds the symmetric kernel
    D.set_operators(0, Dr + E, Ds, L)
    got = D.download(D.rhs(q, 0.0))
    # the change of the volume term: (ax rx + ay ry) E q
    g, _, _ = dg.host_mesh(m, N)
    qn = D.download(q).reshape(D.K, D.Np)
    want = base.reshape(D.K, D.Np) + (0.8 * g[:, :1] + 0.6 * g[:, 1:2]) * (qn @ E.T)
    assert rel(got, want) < TOL
    a = D.lserk4_run(q.clone(), qb, res, 0.0, 1e-3, 4, graph=False).clone()
    qa.copy_(q)
    assert torch.equal(D.lserk4_run(qa, qb, res, 0.0, 1e-3, 4), a)
    D.set_operators(0, Dr, Ds, L)
    assert rel(D.download(D.rhs(q, 0.0)), base) < 1e-14
