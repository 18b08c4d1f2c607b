"""The two-level cycle's fused kernels (step + block-Jacobi, block-Jacobi +
correction, restriction of r - w S z) at every order, on meshes of a few elements,
with ragged last groups and with aggregates of more than 32 cells."""
import numpy as np
import pytest
import torch

import dgc_gb300 as dg
from dgc_gb300 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dirichlet", [True, False])
@pytest.mark.parametrize("n,cells", [(4, 8), (9, 50)])
@pytest.mark.parametrize("N", range(1, 9))
def test_two_level_modes_solve_every_order(N, n, cells, dirichlet):
    m = meshes.jittered_square(n, 60 + N)
    D = dg.Discretization(m, "laplace", N, dg.F64, tau=dg.TAU_SCALED, dirichlet=dirichlet)
    x, y = D.node_xy()
    f = np.sin(np.pi * x) * np.cos(2 * np.pi * y) + x * y
    b = D.mass(D.upload(f.reshape(-1)))
    D.coarse_build(cells)
    ref, _ = D.pcg(b, mode=dg.SOLVE_FP64_PCG, rtol=1e-12)
    for mode in (dg.SOLVE_TWO_LEVEL, dg.SOLVE_TWO_LEVEL_MIXED):
        u, st = D.pcg(b, mode=mode, rtol=1e-11)
        assert st["converged"]
        # both residuals are below 1e-11; the systems' condition is below 1e5 at these sizes
        assert (torch.linalg.norm(u - ref) / torch.linalg.norm(ref)).item() < 1e-6
        assert st["final_relres"] <= 1e-11
    D.check()


@pytest.mark.parametrize("n,cells", [(80, 2), (33, 1)])
def test_coarse_product_across_passes(n, cells):
    """More aggregates than one pass of the FP32 coarse product holds of its vector
    (4096), and fewer: against the FP64 product."""
    D = dg.Discretization(meshes.jittered_square(n, 3), "laplace", 1, dg.F64, tau=dg.TAU_SCALED, dirichlet=True)
    D.coarse_build(cells)
    na = D.coarse_info()[1]
    assert na > 4096 if n == 80 else 0 < na < 4096
    r = D.upload(np.random.default_rng(n).standard_normal(D.K * D.Np))
    a, b = D.coarse_apply(r, precision=dg.F32), D.coarse_apply(r)
    # FP32 rounding (6e-8) of a random r, whose modes the inverse scales like the
    # result's own, over sums of a few hundred roundings
    assert (torch.linalg.norm(a - b) / torch.linalg.norm(b)).item() < 1e-4
    D.check()
