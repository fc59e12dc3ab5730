"""Multi-right-hand-side products over the row counts and widths of the micro-kernel: panels of up
to 16, 32, 48 and 64 rows (leaf sizes around each), V items of one warp and of a CTA (few and
many columns), against the oracle's product (src/mult.jl:6-32) of the same H-matrix."""
import numpy as np
import pytest

import hmgpu
from oracle import oracle as O
from tests import geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf", [5, 16, 17, 33, 48, 49, 64, 65, 130])
def test_rows_and_widths(gpu, leaf):
    """FP64 within 1e-12 and FP32 within 1e-5 of the FP64 oracle, as for every product; the
    columns do not depend on how many there are beside them within a width."""
    import torch
    P = geometry.film(61, 53, seed=leaf)
    T = O.Tree(P.T, leaf)
    Ho = O.HMatrix(O.Kernel("laplace", P.T, P.T), T, T, eta=1.5, eps=1e-5, nthreads=8)
    flat = (Ho.m, Ho.n, Ho.target_index_map, Ho.source_index_map, Ho.dense_block_indices, Ho.dense_blocks,
            Ho.U_block_indices, Ho.U_matrices, Ho.V_block_indices, Ho.V_matrices)
    X = np.random.default_rng(leaf).standard_normal((Ho.n, 32))
    X = X.astype(np.float32).astype(np.float64)
    ref = np.stack([Ho.mul(X[:, k]) for k in range(32)], 1)
    for precision, tol, dt in (("f64", 1e-12, torch.float64), ("f32", 1e-5, torch.float32)):
        H = hmgpu.HMatrix.from_flat(*flat, precision=precision)
        Xd = torch.tensor(X.T.copy(), dtype=dt, device=gpu).t()
        for nrhs, wide in ((3, 8), (9, 16), (17, 32)):
            Y = H * Xd[:, :nrhs]
            assert torch.equal(Y, (H * Xd[:, :wide])[:, :nrhs])
            err = np.linalg.norm(Y.double().cpu().numpy() - ref[:, :nrhs], axis=0) / np.linalg.norm(ref[:, :nrhs], axis=0)
            assert err.max() <= tol, (precision, nrhs)
        assert H.status() == 0
