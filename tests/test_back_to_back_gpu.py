"""Products directly behind one another on a stream, each reading what the one before wrote, with no
other kernel between: a product's first kernel starts while the last one of the product before ends."""
import pytest

import hmgpu
from tests import geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 700, 5003, 40000])
@pytest.mark.parametrize("precision", ["f64", "f32", "mixed"])
@pytest.mark.parametrize("nrhs", [1, 5, 32, 50])
def test_chain_equals_waited_chain(gpu, n, precision, nrhs):
    """a -> b -> a ... eight times, ten chains, against the same with a wait after every product."""
    import torch
    P = geometry.sphere(n, seed=n)
    T = hmgpu.ClusterTree(P, max_points_per_leaf=16, gpu=True)
    H = hmgpu.HMatrix(hmgpu.Kernel("laplace", P), T, T, eta=1.0, eps=1e-5, precision=precision)
    dt = torch.float64 if precision == "f64" else torch.float32
    # eight products grow by up to (n / 4 pi)^8 and stay within FP32
    x = 1e-6 * torch.randn(nrhs, n, device=gpu, dtype=dt, generator=torch.Generator(gpu).manual_seed(1))
    x = x[0] if nrhs == 1 else x.t()

    def chain(wait):
        a, b = x.clone(memory_format=torch.preserve_format), torch.zeros_like(x, memory_format=torch.preserve_format)
        torch.cuda.synchronize()
        for _ in range(4):
            hmgpu.mul_(b, H, a)
            if wait:
                torch.cuda.synchronize()
            hmgpu.mul_(a, H, b)
            if wait:
                torch.cuda.synchronize()
        return a

    want = chain(True)
    assert torch.isfinite(want).all()
    for _ in range(10):
        assert torch.equal(chain(False), want)
    assert H.status() == 0
