"""Tile code of a batch by the handles' variant: the blocked tiles for the blocked
and for the even / odd variant (5 and 6; 1 and 2 at orders 7, 8), the node-by-node
ones for every other."""
import pytest

from conftest import oracle  # noqa: F401

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import dgc_gb300 as dg  # noqa: E402
from dgc_gb300 import meshes  # noqa: E402


@pytest.mark.parametrize("N", [1, 4, 6, 7, 8])
@pytest.mark.parametrize("phys", ["advection", "maxwell_te"])
def test_batch_code_by_variant(N, phys):
    blk = 5 if N <= 6 else 1
    D = dg.Discretization(meshes.jittered_square(9, N), phys, N, dg.F32)
    q = D.upload(torch.randn(D.Nf * D.K * D.Np, dtype=torch.float64, generator=torch.manual_seed(N)).numpy())
    dt = 0.3 * D.info.min_edge / (N + 1) ** 2

    def alone(v):
        D.set_variant(v)
        qb = D.empty_state()
        D.lserk4_step(q.clone(), qb, D.empty_state(), 0.1, dt)
        return qb

    def batched(v):
        D.set_variant(v)
        qb = D.empty_state()
        dg.Batch([D]).lserk4_step([q.clone()], [qb], [D.empty_state()], [0.1], [dt])
        return qb

    ref0, ref_blk = alone(0), alone(blk)
    assert not torch.equal(ref0, ref_blk)  # the comparison below tells the codes apart
    for v in range(D.num_variants()):
        assert torch.equal(batched(v), ref_blk if v in (blk, blk + 1) else ref0), v
    D.check()
