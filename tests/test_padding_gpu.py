"""Panel rows are padded to a multiple of four columns: the padding must hold zeros whatever the
device memory held before, for every product multiplies it by zero."""
import pytest

import hmgpu
from tests import geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "f32", "mixed"])
@pytest.mark.parametrize("nrhs", [1, 8, 32])
def test_products_are_finite_on_dirty_memory(gpu, precision, nrhs, tmp_path):
    import torch

    def dirty():  # memory that the next allocations are likely to get, full of NaN
        t = torch.full((1 << 27,), float("nan"), dtype=torch.float64, device=gpu)
        torch.cuda.synchronize()
        del t
        torch.cuda.empty_cache()

    dt = torch.float64 if precision == "f64" else torch.float32
    for n, kind, dims, leaf, eta in ((77, "dipolar", 3, 16, 1.0), (701, "laplace", 1, 17, 1.5), (83, "laplace", 1, 5, 1.0)):
        P = geometry.cube(n, seed=n)
        for k in range(3):
            dirty()
            T = hmgpu.ClusterTree(P, max_points_per_leaf=leaf, dims=dims, gpu=True)
            H = hmgpu.HMatrix(hmgpu.Kernel(kind, P), T, T, eta=eta, eps=1e-6, precision=precision)
            x = torch.ones(nrhs, n * dims, device=gpu, dtype=dt)
            x = x[0] if nrhs == 1 else x.t()
            y = H * x
            assert torch.isfinite(y).all(), (n, k)
            H.save(tmp_path / "h.bin")
            dirty()
            assert torch.equal(hmgpu.HMatrix.load(tmp_path / "h.bin") * x, y)
