"""First use of a solver or network on a stream that does not wait for the default
stream, while the default stream is busy: the work buffers allocated then are cleared
before the call's kernels use them."""
import numpy as np
import pytest

from conftest import oracle  # noqa: F401

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import dgc_gb300 as dg  # noqa: E402
from dgc_gb300 import meshes  # noqa: E402

BUSY = 200_000_000  # clock cycles, about 0.1 s


def on_side_stream(call):
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    torch.cuda._sleep(BUSY)
    with torch.cuda.stream(side):
        out = call()
    side.synchronize()
    torch.cuda.synchronize()
    return out


def laplace():
    D = dg.Discretization(meshes.jittered_square(16, 11), "laplace", 4, dg.F64)
    x, y = D.node_xy()
    b = D.mass(D.upload((2 * np.pi ** 2 * np.sin(np.pi * x) * np.sin(np.pi * y)).reshape(-1)))
    D.block_jacobi()
    D.coarse_build(8)
    return D, b


@pytest.mark.parametrize("mode", [dg.SOLVE_TWO_LEVEL, dg.SOLVE_TWO_LEVEL_MIXED])
def test_first_two_level_solve(mode):
    D, b = laplace()
    x0 = D.empty_state()
    x, st = on_side_stream(lambda: D.pcg(b, x0, mode=mode, rtol=1e-10, maxit=2000))
    assert st["converged"]
    want, ref = D.pcg(b, mode=mode, rtol=1e-10, maxit=2000)
    # the iteration counts agree but for the order of the FP64 atomic sums
    assert abs(st["iterations"] - ref["iterations"]) <= 8
    assert float((x - want).norm()) < 1e-8 * float(want.norm())


def test_first_training_step():
    D, _ = laplace()
    rng = np.random.default_rng(0)
    X, T = (torch.from_numpy(rng.standard_normal((2, D.K, D.NpP)).astype(np.float32)).cuda().reshape(-1)
            for _ in range(2))

    def net():
        n = dg.MPNN(D, layers=2, seed=3)
        n.set_weights((0.06 * np.random.default_rng(1).standard_normal(n.num_params)).astype(np.float32))
        return n

    a, b = net(), net()
    loss, grad = on_side_stream(lambda: a.train_step(X, T, lr=0.0, want_grad=True))
    wl, wg = b.train_step(X, T, lr=0.0, want_grad=True)
    g, w = (np.asarray(v.cpu() if hasattr(v, "cpu") else v, dtype=np.float64) for v in (grad, wg))
    # FP32 atomic sums in another order
    assert abs(loss - wl) < 1e-5 * abs(wl) and np.linalg.norm(g - w) < 1e-4 * np.linalg.norm(w)
