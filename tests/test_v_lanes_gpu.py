"""FP32 V rows have half the lanes, with two sums each, where a matrix's V rows are up to 2 GB: the bits of
a row's sum must not depend on it, so a shard below the line gives the rows of a matrix above."""
import pytest

import hmgpu
from tests import geometry

pytestmark = pytest.mark.gpu


def test_shards_of_a_matrix_above_the_line(gpu):
    import torch
    P = geometry.film(1024, 1024)
    n = P.shape[1]
    T = hmgpu.ClusterTree(P, max_points_per_leaf=64, gpu=True)
    H = hmgpu.HMatrix(hmgpu.Kernel("laplace", P), T, T, eta=2.0, eps=1e-4, precision="f32")
    x = torch.randn(n, device=gpu, generator=torch.Generator(gpu).manual_seed(2))
    tmap, smap = H.index_maps()
    ref = (H * x)[torch.tensor(tmap - 1, device=gpu)]
    xp = x[torch.tensor(smap - 1, device=gpu)].contiguous()
    for world in (1, 4, 64):
        for r in sorted({0, world // 2, world - 1}):
            S = H.shard(r, world)
            b, e = S.rows
            y = torch.full((e - b,), float("nan"), device=gpu)
            assert torch.equal(S.mul_permuted(y, xp), ref[b:e]), (world, r)


@pytest.mark.parametrize("leaf", [3, 16, 33, 64, 129])
def test_members_of_a_batch_and_schedules(gpu, leaf):
    """Rows of one to some hundred vectors, in both schedules, alone and in a batch."""
    import torch
    members, xs = [], []
    for n in (600, 5000, 20000):
        P = geometry.film(n // 40, 40, seed=leaf)
        T = hmgpu.ClusterTree(P, max_points_per_leaf=leaf, gpu=True)
        members.append(hmgpu.HMatrix(hmgpu.Kernel("laplace", P), T, T, eta=1.5, eps=1e-5, precision="f32"))
        xs.append(torch.randn(P.shape[1], device=gpu, generator=torch.Generator(gpu).manual_seed(n)))
    want = [H * x for H, x in zip(members, xs)]
    assert torch.equal(hmgpu.batch(members) * torch.cat(xs), torch.cat(want))
    for H, x, w in zip(members, xs, want):
        t = H.tuning()
        for dynamic in (0, 1):
            H.set_tuning(16, 32, t["multi_rhs_from"], dynamic)
            assert torch.equal(H * x, w)
