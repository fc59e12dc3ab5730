"""Products whose x and y share memory: x is read as a whole before y is written, at every size, so
y = H y in place and overlapping vectors give the bits of a product into memory of its own."""
import ctypes as C

import pytest

import hmgpu
from hmgpu import _lib
from tests import geometry

pytestmark = pytest.mark.gpu


def _matrix(n, precision, gpu, seed=1):
    import torch
    P = geometry.sphere(n, seed=n)
    T = hmgpu.ClusterTree(P, max_points_per_leaf=16, gpu=True)
    H = hmgpu.HMatrix(hmgpu.Kernel("laplace", P), T, T, eta=1.0, eps=1e-5, precision=precision)
    dt = torch.float64 if precision == "f64" else torch.float32
    return H, torch.randn(n, device=gpu, dtype=dt, generator=torch.Generator(gpu).manual_seed(seed))


@pytest.mark.parametrize("n", [40, 700, 5003, 40000])
@pytest.mark.parametrize("precision", ["f64", "f32", "mixed"])
def test_one_column(gpu, n, precision):
    import torch
    H, x = _matrix(n, precision, gpu)
    want = H * x
    for _ in range(20):
        z = x.clone()
        hmgpu.mul_(z, H, z)
        assert torch.equal(z, want)
    for shift in (-5, 3):  # y a few entries before or behind x
        buf = torch.zeros(n + 8, device=gpu, dtype=x.dtype)
        xs, ys = buf[5:5 + n], buf[5 + shift:5 + shift + n]
        xs.copy_(x)
        hmgpu.mul_(ys, H, xs)
        assert torch.equal(ys, want)
    z = x.clone()
    G = hmgpu.Graph(H, z, z)
    z.copy_(x)
    assert torch.equal(G.launch(), want)
    z.copy_(x)
    stream = torch.cuda.current_stream(gpu).cuda_stream
    assert _lib.lib().hmgpu_matvec_noalloc(H._h, C.c_void_p(z.data_ptr()), C.c_void_p(z.data_ptr()),
                                           C.c_void_p(stream)) == 0
    assert torch.equal(z, want)
    _, smap = H.index_maps()
    xp = x[torch.tensor(smap - 1, device=gpu)].contiguous()
    S = H.shard(0, 2)
    rows = S.rows[1] - S.rows[0]
    own = S.mul_permuted(torch.empty(rows, device=gpu, dtype=x.dtype), xp)
    z = xp.clone()
    assert torch.equal(S.mul_permuted(z[:rows], z), own)


@pytest.mark.parametrize("precision", ["f64", "f32", "mixed"])
@pytest.mark.parametrize("nrhs", [2, 3, 18])
def test_several_columns(gpu, precision, nrhs):
    """In place, and (from three columns on) with y two columns behind x in one array."""
    import torch
    H, _ = _matrix(700, precision, gpu)
    n = H.shape[1]
    dt = torch.float64 if precision == "f64" else torch.float32
    X = torch.randn(nrhs, n, device=gpu, dtype=dt, generator=torch.Generator(gpu).manual_seed(nrhs)).t()
    want = H * X
    Z = X.clone(memory_format=torch.preserve_format)
    hmgpu.mul_(Z, H, Z)
    assert torch.equal(Z, want)
    if nrhs >= 3:
        buf = torch.zeros(nrhs + 2, n, device=gpu, dtype=dt).t()
        buf[:, :nrhs].copy_(X)
        hmgpu.mul_(buf[:, 2:], H, buf[:, :nrhs])
        assert torch.equal(buf[:, 2:], want)
