"""The network's kernels at the sizes where their tiles end: fewer nodes than one
tile, one past a tile, several samples whose fields straddle tiles; caller arrays
off a 16-byte boundary."""
import numpy as np
import pytest
import torch

import dgc_gb300 as dg
from dgc_gb300 import meshes

import mpnn_ref

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(np.ravel(a) - np.ravel(b)) / np.linalg.norm(np.ravel(b))


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n,N,S", [(1, 1, 1), (3, 4, 2), (4, 2, 4), (8, 8, 1), (9, 3, 3), (20, 4, 5)])
def test_forward_and_gradients(n, N, S, offset):
    m = meshes.jittered_square(n, 5 + n)
    D = dg.Discretization(m, "laplace", N, dg.F64, tau=dg.TAU_SCALED, dirichlet=True)
    L = 2
    net = dg.MPNN(D, layers=L, seed=1)
    net.set_loss(dg.MPNN_LOSS_L2)
    K, Np, npi = D.K, D.Np, D.NpP
    rng = np.random.default_rng(n)
    w = (rng.standard_normal(net.num_params) * 0.15).astype(np.float32)
    net.set_weights(w)
    x = rng.standard_normal((S * K, npi)).astype(np.float32)
    t = rng.standard_normal((S * K, npi)).astype(np.float32)

    def dev(a):
        b = torch.zeros(a.size + offset, dtype=torch.float32, device="cuda")
        b[offset:] = torch.from_numpy(a.reshape(-1)).cuda()
        return b[offset:]

    nbr = dg.host_mesh(m, N)[1]
    loss, grad = net.train_step(dev(x), dev(t), lr=0.0, want_grad=True)
    lr, gr = mpnn_ref.loss_and_grad(w, x.astype(np.float64), t.astype(np.float64), nbr, K, npi, Np, L)
    # FP32 sums of up to S K = 4000 products of O(1) values against float64
    assert abs(loss - lr) < 1e-5 * lr
    assert rel(grad.cpu().numpy(), gr) < 2e-5
    y = net.forward(dev(x[:K]))
    assert rel(y.cpu().numpy(), mpnn_ref.forward(w, x[:K].astype(np.float64), nbr, K, npi, L)[0]) < 5e-6
    D.check()


@pytest.mark.parametrize("n,N,S", [(1, 1, 2), (3, 4, 3), (9, 8, 2), (20, 3, 5), (40, 4, 7)])
def test_energy_loss_over_many_fields(n, N, S):
    """The S applies of all samples go through one pair of launches, tiles field after
    field: fields smaller than a tile, partly filled tiles, more tiles than CTAs."""
    m = meshes.jittered_square(n, 40 + n)
    D = dg.Discretization(m, "laplace", N, dg.F64, tau=dg.TAU_SCALED, dirichlet=True)
    L = 2
    net = dg.MPNN(D, layers=L, seed=1)
    K, Np, npi = D.K, D.Np, D.NpP
    rng = np.random.default_rng(n)
    w = (rng.standard_normal(net.num_params) * 0.15).astype(np.float32)
    net.set_weights(w)
    x = rng.standard_normal((S * K, npi)).astype(np.float32)
    t = rng.standard_normal((S * K, npi)).astype(np.float32)
    loss, grad = net.train_step(torch.from_numpy(x).cuda().reshape(-1), torch.from_numpy(t).cuda().reshape(-1),
                                lr=0.0, want_grad=True)

    def spd(v):  # the FP64 form on one native-layout field
        return D.spd(torch.from_numpy(np.ascontiguousarray(v).reshape(-1)).cuda()).cpu().numpy().reshape(K, npi)

    lr, gr = mpnn_ref.loss_and_grad(w, x.astype(np.float64), t.astype(np.float64), dg.host_mesh(m, N)[1], K, npi, Np, L,
                                    spd=spd)
    # random fields load all modes, so S d carries FP32's own relative error: sums of
    # at most 3 Np + 9 (N + 1) = 216 products, 216 x 6e-8 at worst
    assert abs(loss - lr) < 1.3e-5 * lr
    assert rel(grad.cpu().numpy(), gr) < 3e-5
    D.check()
