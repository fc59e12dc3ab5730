"""Shards without rows: more ranks than row tiles. Their product does nothing and succeeds; the others
give the whole product's rows."""
import ctypes as C

import pytest

import hmgpu
from hmgpu import _lib
from tests import geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "f32", "mixed"])
def test_more_ranks_than_tiles(gpu, precision):
    import torch
    P = geometry.cube(200, seed=4)
    T = hmgpu.ClusterTree(P, max_points_per_leaf=32)
    H = hmgpu.HMatrix(hmgpu.Kernel("laplace", P), T, T, eta=2.0, eps=1e-6, precision=precision)
    world = H.info()["n_tiles"] + 5
    dt = torch.float64 if precision == "f64" else torch.float32
    x = torch.randn(200, dtype=dt, device=gpu, generator=torch.Generator(gpu).manual_seed(2))
    tmap, smap = H.index_maps()
    xp = x[torch.tensor(smap - 1, device=gpu)].contiguous()
    ref = (H * x)[torch.tensor(tmap - 1, device=gpu)]
    stream = torch.cuda.current_stream(gpu).cuda_stream
    empty = 0
    for r in range(world):
        S = H.shard(r, world)
        b, e = S.rows
        y = torch.full((e - b + 1,), 7.0, dtype=dt, device=gpu)  # the C entry wants an address for no rows, too
        assert _lib.lib().hmgpu_matvec_shard(S._h, C.c_void_p(xp.data_ptr()), C.c_void_p(y.data_ptr()),
                                             C.c_void_p(stream)) == 0, _lib.lib().hmgpu_last_error()
        assert torch.equal(y[:-1], ref[b:e]) and y[-1] == 7.0
        empty += b == e
    assert empty >= 5
