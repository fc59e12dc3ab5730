"""The Jacobi SVD of the recompression (src/aca.jl:123-143) over core sizes: groups of lanes up
to 64 terms, a CTA above, with both matrices in shared memory, one, or none."""
import numpy as np
import pytest

import hmgpu
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 3, 8, 9, 16, 17, 20, 21, 24, 25, 28, 29, 32, 33, 40, 41, 48, 49, 63, 64, 65, 100, 131, 170])
@pytest.mark.parametrize("decay", [0.0, 8.0])
def test_svd_recompress_core_sizes(gpu, k, decay):
    """Every factor bitwise the oracle's, whose sweep visits the pairs one by one."""
    rng = np.random.default_rng(1000 + k)
    U = rng.standard_normal((k + 3, k)) * np.logspace(0, -decay, k)
    V = rng.standard_normal((k, k + 5))
    if k > 2:
        V[k // 2] = 0.0  # a zero singular value: products of exactly zero
    eps = 1e-5 if decay else 0.0
    Us, Vs = hmgpu.SVD_recompress(U, V, eps)
    Uo, Vo = O.svd_recompress(U, V, eps)
    np.testing.assert_array_equal(Us, Uo)
    np.testing.assert_array_equal(Vs, Vo)
