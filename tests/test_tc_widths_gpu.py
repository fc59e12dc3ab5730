"""Tensor-core passes 16, 32 and 64 right-hand sides wide (mixed precision): the columns at the edges
of each width, whole and lean handles, against the oracle's FP64 product (src/mult.jl:6-32) of the
same H-matrix, and bitwise equal whatever the width of the pass they are in."""
import numpy as np
import pytest

import hmgpu
from oracle import oracle as O
from tests import geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lean", [False, True])
@pytest.mark.parametrize("leaf", [9, 64])
def test_columns_do_not_depend_on_the_width(gpu, lean, leaf):
    import torch
    P = geometry.film(47, 41, seed=leaf)
    T = O.Tree(P.T, leaf)
    Ho = O.HMatrix(O.Kernel("laplace", P.T, P.T), T, T, eta=1.5, eps=1e-5, nthreads=8)
    H = hmgpu.HMatrix.from_flat(Ho.m, Ho.n, Ho.target_index_map, Ho.source_index_map, Ho.dense_block_indices,
                                Ho.dense_blocks, Ho.U_block_indices, Ho.U_matrices, Ho.V_block_indices,
                                Ho.V_matrices, precision="mixed", lean=lean)
    X = np.random.default_rng(leaf).standard_normal((81, Ho.n)).astype(np.float32)
    Xd = torch.tensor(X, device=gpu).t()
    Y = H * Xd  # 64 and 17 columns: a 64-wide and a 32-wide pass
    ref = np.stack([Ho.mul(x.astype(np.float64)) for x in X], 1)
    err = np.linalg.norm(Y.double().cpu().numpy() - ref, axis=0) / np.linalg.norm(ref, axis=0)
    assert err.max() <= 1e-5  # the FP32 bar; the mixed form's own is held elsewhere
    for nrhs in (3, 15, 16, 17, 32, 33, 64, 65, 80):
        assert torch.equal(H * Xd[:, :nrhs], Y[:, :nrhs]), nrhs
    assert H.status() == 0
