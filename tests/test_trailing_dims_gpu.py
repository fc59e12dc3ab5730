"""mul_ with tensors of more than two dimensions, columns one after another in memory: every column of
the second dimension is multiplied."""
import pytest

import hmgpu
from tests import geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [1, 2, 5])
def test_three_dimensions(gpu, nrhs):
    import torch
    P = geometry.sphere(700, seed=1)
    T = hmgpu.ClusterTree(P, max_points_per_leaf=16, gpu=True)
    H = hmgpu.HMatrix(hmgpu.Kernel("laplace", P), T, T, eta=1.0, eps=1e-5, precision="f64")
    X = torch.randn(nrhs, 700, device=gpu, dtype=torch.float64, generator=torch.Generator(gpu).manual_seed(3)).t()
    want = H * X
    Y = torch.zeros(nrhs, 700, device=gpu, dtype=torch.float64).t()
    hmgpu.mul_(Y.unsqueeze(2), H, X.unsqueeze(2))
    assert torch.equal(Y, want)
