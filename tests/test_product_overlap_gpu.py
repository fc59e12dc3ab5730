"""Single-right-hand-side products from a few V units to many, back to back: the kernels of
consecutive products overlap at their ends, and each must still see what the one before wrote."""
import pytest

import hmgpu
from tests import geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 700, 5003, 40000])
@pytest.mark.parametrize("precision", ["f64", "f32", "mixed"])
def test_chained_products_equal_separate_ones(gpu, n, precision):
    """x <- H x / |H x| twelve times without a wait, from a graph's replay too, equals the same
    with a wait after every product, bit for bit, and so does the other V schedule."""
    import torch
    P = geometry.sphere(n, seed=n)
    T = hmgpu.ClusterTree(P, max_points_per_leaf=16, gpu=True)
    H = hmgpu.HMatrix(hmgpu.Kernel("laplace", P), T, T, eta=1.0, eps=1e-5, precision=precision)
    dt = torch.float64 if precision == "f64" else torch.float32
    x0 = torch.randn(n, device=gpu, dtype=dt, generator=torch.Generator(gpu).manual_seed(1))

    def chain(step, wait):
        x = x0.clone()
        for _ in range(12):
            y = step(x)
            if wait:
                torch.cuda.synchronize()
            x = y / y.norm()
            if wait:
                torch.cuda.synchronize()
        return x

    want = chain(lambda x: H * x, True)
    assert torch.equal(chain(lambda x: H * x, False), want)
    xg, yg = torch.empty(n, device=gpu, dtype=dt), torch.empty(n, device=gpu, dtype=dt)
    G = hmgpu.Graph(H, xg, yg)

    def replay(x):
        xg.copy_(x)
        return G.launch()

    assert torch.equal(chain(replay, False), want)
    t = H.tuning()
    H.set_tuning(8, 32, t["multi_rhs_from"], not t["v_dynamic"])
    assert torch.equal(chain(lambda x: H * x, False), want)
    assert H.status() == 0
