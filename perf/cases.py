"""The work a user of the library has it do, as cases that can be timed.

A case is a dict of plain values; `prepare` builds what a user's program holds
before the call (mesh handle, device state, right-hand side), `run` makes one
pass through the public entry points of dgc_gb300, and `exact` evaluates the
same discrete operators in FP64 with plain torch, from the mesh up, without the
library.  All meshes are the jittered square the package itself generates
(K = 2 n^2 triangles, orders 1..8); sizes follow the benchmark's workloads and
the tests.

Kinds
  step      one LSERK4 step (advection, Maxwell TM / TE) in FP64, FP32 or
            compensated FP32: the call of every time loop
  run       lserk4_run over a CUDA graph: a whole stretch of a small problem
  batch     one LSERK4 step of many independent FP32 instances
  graddiv   weak gradient and divergence (projection steps, post-processing)
  spd       one application of the IPDG operator: what user-side solvers call
  poisson   a whole Dirichlet Poisson solve, by solver mode
  stokes    one dual-splitting step of the Stokes example
  train     one gradient evaluation of the learned preconditioner's network
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "dg-on-cuda_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import dgc_gb300 as dg  # noqa: E402
from dgc_gb300 import meshes  # noqa: E402
from dgc_gb300 import stokes as st  # noqa: E402

_PREC = {"f64": dg.F64, "f32": dg.F32, "f32c": dg.F32C}
_MODE = {"pcg_f64": dg.SOLVE_FP64_PCG, "mixed_ir": dg.SOLVE_MIXED_IR, "two_level": dg.SOLVE_TWO_LEVEL,
         "two_level_mixed": dg.SOLVE_TWO_LEVEL_MIXED}


def listed():
    return [
        # the smallest call: one step on a coarse mesh, five launches of very little work each
        {"name": "adv_step_small", "kind": "step", "physics": "advection", "prec": "f64", "n": 8, "N": 3, "blocked": False},
        # plain method on the 32x32 advection mesh (K = 2048), twenty graphed steps towards T = 0.5
        {"name": "adv_run_k2048", "kind": "run", "physics": "advection", "prec": "f64", "n": 32, "N": 4, "steps": 20,
         "blocked": False},
        # the headline workload: Maxwell TE cavity at K = 32768, N = 6, mixed path
        {"name": "te_step_f32", "kind": "step", "physics": "maxwell_te", "prec": "f32", "n": 128, "N": 6, "blocked": True},
        # the same step on the plain FP64 path
        {"name": "te_step_f64", "kind": "step", "physics": "maxwell_te", "prec": "f64", "n": 128, "N": 6, "blocked": False},
        # long-time integration with the compensated FP32 state, a ragged size and an odd order
        {"name": "te_step_f32c", "kind": "step", "physics": "maxwell_te", "prec": "f32c", "n": 101, "N": 5, "blocked": False},
        # parameter study: mixed orders, sizes and physics in one persistent launch per stage
        {"name": "batch_24", "kind": "batch", "count": 24, "nmax": 160, "mix": 777},
        # gradient and divergence of a scalar / vector field on the Poisson mesh (K = 131072)
        {"name": "graddiv_f64", "kind": "graddiv", "prec": "f64", "n": 256, "N": 4},
        # matrix-free IPDG operator for a user's own Krylov solver, odd order
        {"name": "spd_f64", "kind": "spd", "prec": "f64", "n": 181, "N": 5},
        # plain FP64 block-Jacobi PCG to 1e-10, moderate mesh
        {"name": "poisson_pcg_f64", "kind": "poisson", "mode": "pcg_f64", "n": 48, "N": 4},
        # the fastest solver on the Poisson mesh (K = 131072), two-level preconditioner, FP32 inside
        {"name": "poisson_two_level", "kind": "poisson", "mode": "two_level_mixed", "n": 256, "N": 4},
        # one Stokes time step: grad / div, pressure solve, viscous solves
        {"name": "stokes_step", "kind": "stokes", "mode": "two_level_mixed", "n": 40, "N": 3},
        # training of the learned preconditioner: forward and backward over a batch of fields
        {"name": "mpnn_train", "kind": "train", "n": 128, "N": 4, "samples": 8, "layers": 4},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "run", "batch", "graddiv", "spd", "poisson", "stokes", "train"])
    if kind in ("step", "run"):
        N = rng.randint(1, 8)
        phys = rng.choice(["advection", "maxwell_tm", "maxwell_te"])
        prec = rng.choice(["f64", "f32", "f32", "f32c"])
        n = _logint(rng, 6, 150 if kind == "step" else 40)
        c = {"kind": kind, "physics": phys, "prec": prec, "n": n, "N": N, "blocked": prec == "f32" and rng.random() < 0.7}
        if kind == "run":
            c["steps"] = rng.choice([7, 20, 33, 40])
        return c
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 40), "nmax": rng.choice([24, 48, 96]), "mix": rng.randint(1, 10 ** 6)}
    if kind == "graddiv":
        return {"kind": kind, "prec": rng.choice(["f64", "f64", "f32"]), "n": _logint(rng, 10, 240), "N": rng.randint(1, 6)}
    if kind == "spd":
        return {"kind": kind, "prec": rng.choice(["f64", "f64", "f32"]), "n": _logint(rng, 10, 200), "N": rng.randint(1, 6)}
    if kind == "poisson":
        mode = rng.choice(["pcg_f64", "mixed_ir", "two_level", "two_level_mixed"])
        return {"kind": kind, "mode": mode, "n": _logint(rng, 12, 40 if mode == "pcg_f64" else 80), "N": rng.randint(2, 5)}
    if kind == "stokes":
        return {"kind": kind, "mode": rng.choice(["mixed_ir", "two_level_mixed"]), "n": _logint(rng, 10, 32),
                "N": rng.randint(2, 4)}
    return {"kind": "train", "n": _logint(rng, 16, 120), "N": rng.randint(2, 5), "samples": rng.randint(1, 8),
            "layers": rng.randint(2, 4)}


# ------------------------------------------------------------------ inputs

def _mesh(case, seed):
    return meshes.jittered_square(case["n"], 1000 + seed % 100003)


def _time_problem(case, seed):
    """Mesh, physics keywords and initial state [field][cell][node] from the node coordinates."""
    rng = np.random.default_rng([seed, 17])
    kw = {}
    if case["physics"] == "advection":
        th = rng.uniform(0.0, 2.0 * np.pi)
        kw = dict(ax=float(np.cos(th)), ay=float(np.sin(th)), bc=dg.BC_GAUSS, gx0=float(rng.uniform(-0.5, 0.5)),
                  gy0=float(rng.uniform(-0.5, 0.5)), gw=0.02)

        def q0(x, y):
            return np.exp(-((x - kw["gx0"]) ** 2 + (y - kw["gy0"]) ** 2) / kw["gw"])[None]
    else:
        # a few cavity modes with random amplitudes
        a = rng.normal(size=(3, 4))
        k = rng.integers(1, 4, size=(2, 4))

        def q0(x, y):
            q = np.zeros((3,) + x.shape)
            for i in range(4):
                cx, sx = np.cos(np.pi * k[0, i] * x), np.sin(np.pi * k[0, i] * x)
                cy, sy = np.cos(np.pi * k[1, i] * y), np.sin(np.pi * k[1, i] * y)
                if case["physics"] == "maxwell_te":
                    q[0] += a[0, i] * cx * sy
                    q[1] += a[1, i] * sx * cy
                    q[2] += a[2, i] * cx * cy
                else:
                    q[0] += a[0, i] * sx * cy
                    q[1] += a[1, i] * cx * sy
                    q[2] += a[2, i] * sx * sy
            return q
    return _mesh(case, seed), kw, q0


def _scalar_field(seed, modes=6):
    """A smooth random field u(x, y): a sum of Fourier modes."""
    rng = np.random.default_rng([seed, 29])
    k = rng.integers(1, 7, size=(2, modes))
    a = rng.normal(size=(2, modes)) / np.hypot(k[0], k[1])

    def u(x, y):
        r = np.zeros_like(x)
        for i in range(modes):
            r = r + a[0, i] * np.sin(np.pi * k[0, i] * x) * np.sin(np.pi * k[1, i] * y)
            r = r + a[1, i] * np.cos(np.pi * k[0, i] * x) * np.sin(np.pi * k[1, i] * y)
        return r
    return u


def _blocked_variant(N):
    return 5 if N <= 6 else 1


def _dt(D, N):
    return 0.5 * D.info.min_edge / (N + 1) ** 2


def _batch_specs(case):
    """Orders, sizes and physics of the instances: those of the batched workload (n
    log-uniform from 8, N in 2..8)."""
    rng = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["count"]):
        n = int(round(np.exp(rng.uniform(np.log(8), np.log(case["nmax"])))))
        N = int(rng.integers(2, 9))
        out.append({"n": n, "N": N, "prec": "f32",
                    "physics": ["advection", "maxwell_te", "maxwell_tm"][int(rng.integers(0, 3))]})
    return out


def _laplace(case, seed, prec=dg.F64):
    return dg.Discretization(_mesh(case, seed), "laplace", case["N"], prec, tau=dg.TAU_SCALED, dirichlet=True)


def prepare(case, seed):
    kind, N = case["kind"], case.get("N", 0)
    s = {"case": case}
    if kind in ("step", "run"):
        m, kw, q0 = _time_problem(case, seed)
        D = dg.Discretization(m, case["physics"], N, _PREC[case["prec"]], **kw)
        if case["blocked"]:
            D.set_variant(_blocked_variant(N))
        x, y = D.node_xy()
        s.update(D=D, q=D.upload(q0(x, y)), qa=D.empty_state(), qb=D.empty_state(), res=D.empty_state(), dt=_dt(D, N))
    elif kind == "batch":
        items = []
        for i, sp in enumerate(_batch_specs(case)):
            m, kw, q0 = _time_problem(sp, seed + 7919 * i)
            D = dg.Discretization(m, sp["physics"], sp["N"], dg.F32, **kw)
            D.set_variant(_blocked_variant(sp["N"]))
            x, y = D.node_xy()
            items.append((D, D.upload(q0(x, y)), _dt(D, sp["N"])))
        s.update(B=dg.Batch([d for d, _, _ in items]), q=[q for _, q, _ in items],
                 qb=[d.empty_state() for d, _, _ in items], res=[d.empty_state() for d, _, _ in items],
                 dt=[dt for _, _, dt in items], t=[0.0] * len(items))
    elif kind in ("graddiv", "spd"):
        D = _laplace(case, seed, _PREC[case["prec"]])
        x, y = D.node_xy()
        s.update(D=D, u=D.upload(_scalar_field(seed)(x, y)), out=D.empty_state())
        if kind == "graddiv":
            b = D.boundary_nodes()
            g = _scalar_field(seed + 1)(b[:, 0], b[:, 1])
            s.update(g=torch.from_numpy(np.ascontiguousarray(g)).cuda(), v=D.upload(_scalar_field(seed + 2)(x, y)),
                     gx=D.empty_state(), gy=D.empty_state())
    elif kind == "poisson":
        D = _laplace(case, seed)
        x, y = D.node_xy()
        D.block_jacobi()
        if case["mode"].startswith("two_level"):
            D.coarse_build(32)
        s.update(D=D, b=D.mass(D.upload(_scalar_field(seed, 12)(x, y))), x=D.empty_state())
    elif kind == "stokes":
        S = st.Stokes(_mesh(case, seed), N, consistent=True, rtol=1e-10, mode=_MODE[case["mode"]])
        vs = S.velocity_space
        x, y = (c.reshape(-1) for c in vs.node_xy())
        t, dt = 0.01 + 0.02 * (seed % 977) / 977.0, 1e-3
        prev, cur = st.exact_velocity(x, y, t - dt), st.exact_velocity(x, y, t)
        s.update(S=S, prev=[vs.upload(c) for c in prev], cur=[vs.upload(c) for c in cur], dt=dt,
                 bc=S.boundary_data(t, t - dt, dt), out=(S.empty(), S.empty()), p=S.empty())
    else:  # train
        D = _laplace(case, seed)
        net = dg.MPNN(D, layers=case["layers"], seed=1 + seed % 1000)
        net.set_weights(_train_weights(net.num_params, seed))
        X, T = _train_fields(case, seed, D.Np, D.NpP)
        s.update(net=net, D=D, X=torch.from_numpy(X).cuda().reshape(-1), T=torch.from_numpy(T).cuda().reshape(-1))
    return s


def _train_weights(num, seed):
    return (0.06 * np.random.default_rng([seed, 41]).standard_normal(num)).astype(np.float32)


def _train_fields(case, seed, Np, NpP):
    """Normalised residual / error fields [sample][cell][NpP] (padding 0)."""
    rng = np.random.default_rng([seed, 43])
    K = 2 * case["n"] ** 2
    cell = np.arange(K)[None, :, None] / K
    node = np.arange(Np)[None, None, :] / Np
    X = np.zeros((case["samples"], K, NpP), np.float32)
    T = np.zeros_like(X)
    ph = rng.uniform(0, 2 * np.pi, (case["samples"], 1, 1))
    X[:, :, :Np] = rng.standard_normal((case["samples"], K, Np)) * 0.7 + np.sin(40 * cell + 3 * node + ph)
    T[:, :, :Np] = np.cos(17 * cell + node + ph) + 0.1 * rng.standard_normal((case["samples"], K, Np))
    return X, T


# ------------------------------------------------------------------ one pass

def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "step":
        D = state["D"]
        # the step may use q as scratch (its stages alternate between the two
        # buffers), so a caller who keeps the old state hands over a copy
        state["qa"].copy_(state["q"])
        D.lserk4_step(state["qa"], state["qb"], state["res"], 0.0, state["dt"])
        return state["qb"]
    if kind == "run":
        state["qa"].copy_(state["q"])
        return state["D"].lserk4_run(state["qa"], state["qb"], state["res"], 0.0, state["dt"], c["steps"], graph=True)
    if kind == "batch":
        if "qa" not in state:
            state["qa"] = [torch.empty_like(q) for q in state["q"]]
        for a, q in zip(state["qa"], state["q"]):
            a.copy_(q)
        return state["B"].lserk4_step(state["qa"], state["qb"], state["res"], state["t"], state["dt"])
    if kind == "graddiv":
        D = state["D"]
        gx, gy = D.grad(state["u"], g=state["g"], sign=-1.0, out=(state["gx"], state["gy"]))
        d = D.div(state["u"], state["v"], out=state["out"])
        return {"gx": gx, "gy": gy, "div": d}
    if kind == "spd":
        return state["D"].spd(state["u"], out=state["out"])
    if kind == "poisson":
        state["x"].zero_()
        x, _ = state["D"].pcg(state["b"], state["x"], mode=_MODE[c["mode"]], rtol=1e-10, maxit=20000)
        return x
    if kind == "stokes":
        ux, uy, _ = state["S"].step(*state["prev"], *state["cur"], state["dt"], state["bc"], out=state["out"],
                                    p_out=state["p"])
        return {"ux": ux, "uy": uy, "p": state["p"]}
    loss, grad = state["net"].train_step(state["X"], state["T"], lr=0.0, want_grad=True)
    return {"loss": loss, "grad": grad}


# ------------------------------------------------------------------ what a pass cannot do without

def _dims(N):
    Np = (N + 1) * (N + 2) // 2
    return Np, (Np + 3) // 4 * 4, N + 1


def work(case):
    kind = case["kind"]
    if kind == "batch":
        ws = [work(dict(sp, kind="step")) for sp in _batch_specs(case)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    K = 2 * case["n"] ** 2
    Np, NpP, Nfp = _dims(case["N"])
    if kind in ("step", "run"):
        size = 4 if case["prec"] == "f32" else 8
        nf = 1 if case["physics"] == "advection" else 3
        rhs = K * 2 * (Np * Np * (2 if nf == 1 else 4) + nf * Np * 3 * Nfp)
        # state in, state out, geometry and neighbours once
        return {"bytes": K * (2 * nf * Np * size + 14 * (8 if case["prec"] == "f64" else 4) + 12),
                "flops": 5 * case.get("steps", 1) * rhs}
    size = 4 if case.get("prec") == "f32" else 8
    geo = K * (14 * size + 12)
    if kind == "graddiv":
        return {"bytes": K * Np * size * 6 + 2 * geo, "flops": K * 2 * (6 * Np * Np + 2 * Np * 3 * Nfp)}
    apply = K * 2 * (7 * Np * Np + 3 * Np * 3 * Nfp)
    if kind == "spd":
        return {"bytes": K * Np * size * 2 + geo, "flops": apply}
    if kind == "poisson":  # one apply at the least; the iterations are the solver's choice
        return {"bytes": K * Np * 16 + geo + K * Np * Np * 8, "flops": apply}
    if kind == "stokes":
        return {"bytes": K * Np * 8 * 7 + geo, "flops": 6 * apply}
    W, L, S = 64, case["layers"], case["samples"]
    return {"bytes": S * K * NpP * 8, "flops": 3 * S * K * 2 * (2 * W * NpP + L * 2 * W * W)}


# ------------------------------------------------------------------ the same values in 64 bits, by plain torch

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _jacobi(a, b, n, x):
    """Orthonormal Jacobi polynomials (Hesthaven & Warburton 2008, App. A)."""
    g0 = 2.0 ** (a + b + 1) / (a + b + 1) * math.gamma(a + 1) * math.gamma(b + 1) / math.gamma(a + b + 1)
    p0 = np.full_like(x, 1.0 / math.sqrt(g0))
    if n == 0:
        return p0
    g1 = (a + 1) * (b + 1) / (a + b + 3) * g0
    p1 = ((a + b + 2) * x / 2 + (a - b) / 2) / math.sqrt(g1)
    ao = 2 / (2 + a + b) * math.sqrt((a + 1) * (b + 1) / (a + b + 3))
    for i in range(1, n):
        h = 2 * i + a + b
        an = 2 / (h + 2) * math.sqrt((i + 1) * (i + 1 + a + b) * (i + 1 + a) * (i + 1 + b) / (h + 1) / (h + 3))
        bn = -(a * a - b * b) / h / (h + 2)
        p0, p1 = p1, ((x - bn) * p1 - ao * p0) / an
        ao = an
    return p1


def _djacobi(a, b, n, x):
    return np.zeros_like(x) if n == 0 else math.sqrt(n * (n + a + b + 1)) * _jacobi(a + 1, b + 1, n - 1, x)


def _lobatto(N):
    """Legendre-Gauss-Lobatto points: the ends and the roots of P_N'."""
    return np.concatenate([[-1.0], np.sort(np.polynomial.legendre.Legendre.basis(N).deriv().roots().real), [1.0]])


class _Element:
    """Reference triangle of order N on the alpha-optimised warp & blend nodes."""

    def __init__(self, N):
        alpha = [0.0, 0.0, 1.4152, 0.1001, 0.2751, 0.9808, 1.0999, 1.2832][N - 1]
        eq = np.linspace(-1.0, 1.0, N + 1)
        shift = _lobatto(N) - eq
        V1 = np.stack([_jacobi(0, 0, i, eq) for i in range(N + 1)], 1)

        def warp(r):
            P = np.stack([_jacobi(0, 0, i, r) for i in range(N + 1)], 1)
            w = P @ np.linalg.solve(V1, shift)
            inside = np.abs(r) < 1.0 - 1e-10
            return np.where(inside, w / np.where(inside, 1.0 - r * r, 1.0), 0.0)

        ij = [(i, j) for i in range(N + 1) for j in range(N + 1 - i)]
        L1 = np.array([i / N for i, _ in ij])
        L3 = np.array([j / N for _, j in ij])
        L2 = 1.0 - L1 - L3
        w1 = 4 * L2 * L3 * (1 + (alpha * L1) ** 2) * warp(L3 - L2)
        w2 = 4 * L1 * L3 * (1 + (alpha * L2) ** 2) * warp(L1 - L3)
        w3 = 4 * L1 * L2 * (1 + (alpha * L3) ** 2) * warp(L2 - L1)
        X = L3 - L2 + w1 - 0.5 * w2 - 0.5 * w3
        Y = (2 * L1 - L2 - L3) / math.sqrt(3.0) + 0.5 * math.sqrt(3.0) * (w2 - w3)
        b1 = (1 + math.sqrt(3.0) * Y) / 3
        b2 = (2 - 3 * X - math.sqrt(3.0) * Y) / 6
        b3 = (2 + 3 * X - math.sqrt(3.0) * Y) / 6
        self.N, self.Np, self.Nfp, self.NpP = N, len(ij), N + 1, (len(ij) + 3) // 4 * 4
        self.r, self.s = b3 - b2 - b1, b1 - b2 - b3
        r, s = self.r, self.s
        a = np.where(s < 1.0 - 1e-12, 2 * (1 + r) / np.where(s < 1.0 - 1e-12, 1 - s, 1.0) - 1, -1.0)
        V, Vr, Vs = [], [], []
        for i in range(N + 1):
            for j in range(N + 1 - i):
                fa, dfa = _jacobi(0, 0, i, a), _djacobi(0, 0, i, a)
                gb, dgb = _jacobi(2 * i + 1, 0, j, s), _djacobi(2 * i + 1, 0, j, s)
                h = 0.5 * (1 - s)
                hi, hm = h ** i, h ** max(i - 1, 0)
                V.append(math.sqrt(2.0) * fa * gb * (1 - s) ** i)
                dr = dfa * gb * (hm if i else 1.0)
                ds = dfa * gb * 0.5 * (1 + a) * (hm if i else 1.0) + fa * (dgb * hi - (0.5 * i * gb * hm if i else 0.0))
                Vr.append(2 ** (i + 0.5) * dr)
                Vs.append(2 ** (i + 0.5) * ds)
        V, Vr, Vs = (np.stack(v, 1) for v in (V, Vr, Vs))
        Minv = V @ V.T
        M = np.linalg.inv(Minv)
        self.fmask = np.array([[k for k, (i, j) in enumerate(ij) if i == 0],
                               [k for k, (i, j) in enumerate(ij) if i + j == N],
                               [k for k, (i, j) in enumerate(ij) if j == 0][::-1]])
        E = np.zeros((self.Np, 3 * self.Nfp))
        for f in range(3):
            x = r[self.fmask[f]] if f == 0 else s[self.fmask[f]]
            F = np.stack([_jacobi(0, 0, i, x) for i in range(N + 1)], 1)
            E[np.ix_(self.fmask[f], range(f * self.Nfp, (f + 1) * self.Nfp))] = np.linalg.inv(F @ F.T)
        t = lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(_dev())  # noqa: E731
        self.M, self.lift = t(M), t(Minv @ E)
        self.Dr, self.Ds = t(np.linalg.solve(V.T, Vr.T).T), t(np.linalg.solve(V.T, Vs.T).T)       # strong
        self.Wr, self.Ws = t(V @ Vr.T @ M), t(V @ Vs.T @ M)                                       # weak
        self.face_mass = t(E)


class _Plain:
    """The discrete operators on a mesh, FP64, one tensor expression each."""

    def __init__(self, m, N):
        e = self.e = _Element(N)
        d = _dev()
        c = m.cells.astype(np.int64)
        K = self.K = c.shape[0]
        P = m.xy[c]
        (x0, y0), (x1, y1), (x2, y2) = (P[:, i].T for i in range(3))
        xr, xs, yr, ys = 0.5 * (x1 - x0), 0.5 * (x2 - x0), 0.5 * (y1 - y0), 0.5 * (y2 - y0)
        J = xr * ys - xs * yr
        D = P[:, [1, 2, 0]] - P
        ln = np.sqrt((D ** 2).sum(-1))
        key = np.minimum(c, np.roll(c, -1, 1)) * (c.max() + 1) + np.maximum(c, np.roll(c, -1, 1))
        order = np.argsort(key.reshape(-1), kind="stable")
        srt = key.reshape(-1)[order]
        twin = np.full(3 * K, -1)
        eq = np.nonzero(srt[1:] == srt[:-1])[0]
        twin[order[eq]], twin[order[eq + 1]] = order[eq + 1], order[eq]
        bnd = np.nonzero(twin < 0)[0]
        bid = np.zeros(3 * K, np.int64)
        bid[bnd] = np.arange(bnd.size)
        l = np.stack([-0.5 * (e.r + e.s), 0.5 * (1 + e.r), 0.5 * (1 + e.s)])
        self.x, self.y = np.einsum("kv,vn->kn", P[..., 0], l), np.einsum("kv,vn->kn", P[..., 1], l)
        t = lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(d)  # noqa: E731
        self.J, self.fJ = t(J), t(0.5 * ln)
        self.rx, self.ry, self.sx, self.sy = t(ys / J), t(-xs / J), t(-yr / J), t(xr / J)
        self.nx, self.ny = t(D[..., 1] / ln), t(-D[..., 0] / ln)
        twin = twin.reshape(K, 3)
        self.inner = t(twin >= 0)[..., None]
        own = t(np.arange(K)[:, None, None] * e.Np + e.fmask[None])
        other = np.where(twin >= 0, twin, 0)
        other = other // 3 * e.Np
        nbn = e.fmask[np.where(twin >= 0, twin, 0) % 3][:, :, ::-1]
        self.vm = own
        self.vp = torch.where(self.inner, t(other[..., None] + nbn), own)
        self.bnode = t(bid.reshape(K, 3)[..., None] * e.Nfp + np.arange(e.Nfp))
        self.fx, self.fy = t(self.x.reshape(-1))[own], t(self.y.reshape(-1))[own]
        self.bx = self.fx.reshape(3 * K, e.Nfp)[t(bnd)].reshape(-1).cpu().numpy()
        self.by = self.fy.reshape(3 * K, e.Nfp)[t(bnd)].reshape(-1).cpu().numpy()
        h = 2 * self.J[:, None] / self.fJ
        hp = h.reshape(-1)[t(np.where(twin >= 0, twin, np.arange(3 * K).reshape(K, 3)))]
        self.tau = (N + 1.0) ** 2 / torch.minimum(h, hp)
        self.cellnbr = t(np.where(twin >= 0, twin // 3, -1))
        self.min_edge = float(ln.min())

    def faces(self, u):
        u = u.reshape(-1)
        return u[self.vm], u[self.vp]

    def lifted(self, flux):
        """LIFT(flux faceJ) / J of face-node values [K][3][Nfp]."""
        return (flux * self.fJ[..., None]).reshape(self.K, -1) @ self.e.lift.T / self.J[:, None]

    def d(self, u, weak):
        r = u @ (self.e.Wr if weak else self.e.Dr).T
        s = u @ (self.e.Ws if weak else self.e.Ds).T
        return (self.rx[:, None] * r + self.sx[:, None] * s, self.ry[:, None] * r + self.sy[:, None] * s)

    def rhs(self, physics, kw, q, t):
        nx, ny = self.nx[..., None], self.ny[..., None]
        if physics == "advection":
            a, b = self.faces(q[0])
            gx, gy = self.fx - kw["ax"] * t - kw["gx0"], self.fy - kw["ay"] * t - kw["gy0"]
            b = torch.where(self.inner, b, torch.exp(-(gx * gx + gy * gy) / kw["gw"]))
            an = kw["ax"] * nx + kw["ay"] * ny
            dx, dy = self.d(q[0], True)
            return [kw["ax"] * dx + kw["ay"] * dy - self.lifted(torch.where(an >= 0, a, b) * an)]
        te = physics == "maxwell_te"
        a, b = zip(*(self.faces(v) for v in q))
        wall = (-1.0, -1.0, 1.0) if te else (1.0, 1.0, -1.0)
        b = [torch.where(self.inner, v, w * u) for u, v, w in zip(a, b, wall)]
        sg = -1.0 if te else 1.0
        w = a[2] + b[2] + sg * (ny * (a[0] - b[0]) - nx * (a[1] - b[1]))
        f0, f1 = sg * 0.5 * ny * w, -sg * 0.5 * nx * w
        f2 = 0.5 * (sg * (ny * (a[0] + b[0]) - nx * (a[1] + b[1])) + a[2] - b[2])
        d2x, d2y = self.d(q[2], True)
        d1x, d0y = self.d(q[1], True)[0], self.d(q[0], True)[1]
        return [sg * d2y - self.lifted(f0), -sg * d2x - self.lifted(f1), sg * (d0y - d1x) - self.lifted(f2)]

    # Carpenter & Kennedy (1994), five-stage fourth-order 2N-storage scheme
    A = (0.0, -567301805773 / 1357537059087, -2404267990393 / 2016746695238, -3550918686646 / 2091501179385,
         -1275806237668 / 842570457699)
    B = (1432997174477 / 9575080441755, 5161836677717 / 13612068292357, 1720146321549 / 2090206949498,
         3134564353537 / 4481467310338, 2277821191437 / 14882151754819)
    C = (0.0, 1432997174477 / 9575080441755, 2526269341429 / 6820363962896, 2006345519317 / 3224310063776,
         2802321613138 / 2924317926251)

    def step(self, physics, kw, q, t, dt):
        res = [torch.zeros_like(v) for v in q]
        for a, b, c in zip(self.A, self.B, self.C):
            r = self.rhs(physics, kw, q, t + c * dt)
            res = [a * x + dt * y for x, y in zip(res, r)]
            q = [x + b * y for x, y in zip(q, res)]
        return q

    def native(self, fields):
        out = torch.zeros(self.K, len(fields), self.e.NpP, dtype=torch.float64, device=fields[0].device)
        out[:, :, :self.e.Np] = torch.stack(fields, 1)
        return out.reshape(-1)

    def laplace(self, u):
        nx, ny = self.nx[..., None], self.ny[..., None]
        um, up = self.faces(u)
        du = torch.where(self.inner, um - up, 2 * um)
        ux, uy = self.d(u, False)
        qx, qy = ux - self.lifted(0.5 * nx * du), uy - self.lifted(0.5 * ny * du)
        (xm, xp), (ym, yp) = self.faces(qx), self.faces(qy)
        dq = torch.where(self.inner, (xm - xp) * nx + (ym - yp) * ny, torch.zeros_like(du))
        return self.d(qx, False)[0] + self.d(qy, False)[1] - self.lifted(0.5 * (dq + 2 * self.tau[..., None] * du))

    def spd(self, u):
        return -self.J[:, None] * (self.laplace(u) @ self.e.M)

    def solve(self, b):
        """Conjugate gradients to 1e-13 with the elements' own stiffness blocks."""
        e = self.e
        Dx = self.rx[:, None, None] * e.Dr + self.sx[:, None, None] * e.Ds
        Dy = self.ry[:, None, None] * e.Dr + self.sy[:, None, None] * e.Ds
        B = self.J[:, None, None] * (Dx.transpose(1, 2) @ e.M @ Dx + Dy.transpose(1, 2) @ e.M @ Dy)
        for f in range(3):
            F = torch.zeros(e.Np, e.Np, dtype=torch.float64, device=b.device)
            ix = torch.from_numpy(e.fmask[f]).to(b.device)
            F[ix[:, None], ix[None]] = e.face_mass[ix, f * e.Nfp:(f + 1) * e.Nfp]
            B += (self.tau[:, f] * self.fJ[:, f])[:, None, None] * F
        Bi = torch.linalg.inv(B)
        x, r = torch.zeros_like(b), b.clone()
        z = torch.einsum("kij,kj->ki", Bi, r)
        p, rz, stop = z, (r * z).sum(), 1e-26 * (b * b).sum()
        for i in range(20000):
            S = self.spd(p)
            al = rz / (p * S).sum()
            x, r = x + al * p, r - al * S
            if i % 25 == 0 and (r * r).sum() <= stop:
                break
            z = torch.einsum("kij,kj->ki", Bi, r)
            rz, old = (r * z).sum(), rz
            p = z + rz / old * p
        return x


def _f32(v):
    return v.to(torch.float32).to(torch.float64)


def _state(p, q0, prec):
    q = [torch.from_numpy(np.ascontiguousarray(v)).to(_dev()) for v in q0(p.x, p.y)]
    return [_f32(v) for v in q] if prec == "f32" else q


def _split(v):
    hi = v.to(torch.float32).to(torch.float64)
    return torch.cat([hi, v - hi])


def _exact_steps(case, seed, steps):
    m, kw, q0 = _time_problem(case, seed)
    p = _Plain(m, case["N"])
    q = _state(p, q0, case["prec"])
    dt = 0.5 * p.min_edge / (case["N"] + 1) ** 2
    for i in range(steps):
        q = p.step(case["physics"], kw, q, i * dt, dt)
    return p.native(q)


def _field(p, u, prec):
    v = torch.from_numpy(np.ascontiguousarray(u(p.x, p.y))).to(_dev())
    return _f32(v) if prec == "f32" else v


def exact(case, seed):
    kind, prec = case["kind"], case.get("prec")
    if kind == "step":
        q = _exact_steps(case, seed, 1)
        return _split(q) if prec == "f32c" else q  # a compensated state is hi and lo
    if kind == "run":
        q = _exact_steps(case, seed, case["steps"])
        return _split(q) if prec == "f32c" else q
    if kind == "batch":
        return [_exact_steps(sp, seed + 7919 * i, 1) for i, sp in enumerate(_batch_specs(case))]
    if kind == "stokes":
        return None
    p = _Plain(_mesh(case, seed), case["N"])
    if kind == "spd":
        return p.native([p.spd(_field(p, _scalar_field(seed), prec))])
    if kind == "graddiv":
        u, v = _field(p, _scalar_field(seed), prec), _field(p, _scalar_field(seed + 2), prec)
        g = torch.from_numpy(_scalar_field(seed + 1)(p.bx, p.by)).to(_dev())
        nx, ny = p.nx[..., None], p.ny[..., None]

        def mean(w, data=None, sign=1.0):
            a, b = p.faces(w)
            ext = sign * a + (0.0 if data is None else data[p.bnode])
            return 0.5 * (a + torch.where(p.inner, b, ext))
        um = mean(u, g, -1.0)
        dx, dy = p.d(u, True)
        flux = nx * mean(u) + ny * mean(v)
        return {"gx": p.native([p.lifted(nx * um) - dx]), "gy": p.native([p.lifted(ny * um) - dy]),
                "div": p.native([p.lifted(flux) - dx - p.d(v, True)[1]])}
    if kind == "poisson":
        if case["n"] > 64:
            return None
        f = _field(p, _scalar_field(seed, 12), None)
        return p.native([p.solve(p.J[:, None] * (f @ p.e.M))])
    return _exact_train(case, seed, p)


def _exact_train(case, seed, p):
    e, W, L = p.e, 64, case["layers"]
    num = 2 * W * e.NpP + W + e.NpP + L * (2 * W * W + W)
    w = torch.from_numpy(_train_weights(num, seed)).to(_dev())
    w = w.to(torch.bfloat16).to(torch.float64).requires_grad_(True)
    at = 0

    def take(*shape):
        nonlocal at
        n = math.prod(shape)
        at += n
        return w[at - n:at].reshape(shape)
    win, bi = take(W, e.NpP), take(W)
    layers = [(take(W, W), take(W, W), take(W)) for _ in range(L)]
    wout, bo = take(e.NpP, W), take(e.NpP)
    X, T = (torch.from_numpy(v).to(_dev()).double() for v in _train_fields(case, seed, e.Np, e.NpP))
    has = (p.cellnbr >= 0)[..., None]
    ix = p.cellnbr.clamp(min=0)
    loss, grad = 0.0, torch.zeros_like(w)
    for x, t in zip(X, T):
        h = x @ win.T + bi
        for ws, wn, b in layers:
            m = (h[ix] * has).sum(1)
            h = h + torch.relu(h @ ws.T + m @ wn.T + b)
        d = (h @ wout.T + bo - t)[:, :e.Np]
        tv = t[:, :e.Np]
        part = (d * p.spd(d)).sum() / (tv * p.spd(tv)).sum() / case["samples"]
        grad += torch.autograd.grad(part, w, retain_graph=True)[0]
        loss += float(part.detach())
    return {"loss": loss, "grad": grad}
