"""Multi-right-hand-side products captured by the caller: the first product of a handle, which makes its
scratch, in a capture that allows allocation."""
import numpy as np
import pytest

import hmgpu
from tests import geometry

pytestmark = pytest.mark.gpu


def _matrix(precision, gpu, n=3001):
    P = geometry.sphere(n, seed=n)
    T = hmgpu.ClusterTree(P, max_points_per_leaf=16, gpu=True)
    return hmgpu.HMatrix(hmgpu.Kernel("laplace", P), T, T, eta=1.0, eps=1e-5, precision=precision)


def _columns(H, nrhs, precision, gpu, seed):
    import torch
    dt = torch.float64 if precision == "f64" else torch.float32
    return torch.randn(nrhs, H.shape[1], device=gpu, dtype=dt, generator=torch.Generator(gpu).manual_seed(seed)).t()


@pytest.mark.parametrize("precision", ["f64", "f32", "mixed"])
@pytest.mark.parametrize("nrhs", [8, 20])
@pytest.mark.parametrize("eager_between", [False, True])
def test_first_product_in_a_capture(gpu, precision, nrhs, eager_between):
    import torch
    H = _matrix(precision, gpu)
    X = _columns(H, nrhs, precision, gpu, 1)
    want = [_matrix(precision, gpu) * X, None]
    X2 = _columns(H, nrhs, precision, gpu, 2)
    want[1] = _matrix(precision, gpu) * X2
    Xg = X.clone(memory_format=torch.preserve_format)
    Y = torch.zeros(nrhs, H.shape[0], device=gpu, dtype=X.dtype).t()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="relaxed"):
        hmgpu.mul_(Y, H, Xg)
    assert not Y.any()  # captured, not run
    if eager_between:
        assert torch.equal(H * X2, want[1])
    junk = [np.full(1 << k, -1, np.int64) for k in range(4, 16) for _ in range(4)]  # freed host memory is reused
    for x, w in ((X, want[0]), (X2, want[1]), (X, want[0])):
        Xg.copy_(x)
        g.replay()
        assert torch.equal(Y, w)
    assert torch.equal(H * X, want[0]) and H.status() == 0
    del junk


@pytest.mark.parametrize("precision", ["f64", "f32", "mixed"])
@pytest.mark.parametrize("warm,nrhs", [(32, 8), (32, 18), (64, 20), (20, 16), (8, 32), (8, 3), (5, 40)])
def test_capture_after_another_count(gpu, precision, warm, nrhs):
    """A capture that forbids allocation, after a product with another number of columns."""
    import torch
    H = _matrix(precision, gpu)
    X = _columns(H, nrhs, precision, gpu, 1)
    want = _matrix(precision, gpu) * X
    H * _columns(H, warm, precision, gpu, 2)
    Y = torch.zeros(nrhs, H.shape[0], device=gpu, dtype=X.dtype).t()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        hmgpu.mul_(Y, H, X)
    for _ in range(2):
        Y.zero_()
        g.replay()
        if precision == "f32":  # a column's sum depends on the width of its pass
            assert torch.linalg.norm((Y - want).double()) <= 1e-5 * torch.linalg.norm(want.double())
        else:
            assert torch.equal(Y, want)
    assert torch.equal(H * X, want) and H.status() == 0
