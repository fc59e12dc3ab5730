"""Products of matrices with more row units than resident CTAs, most of them so short that a CTA's
warps are done with a unit at once: the ticket of the next unit must reach every warp before it is
overwritten. Against the dense product of the same blocks (src/mult.jl:80-146)."""
import numpy as np
import pytest

import hmgpu

pytestmark = pytest.mark.gpu


def _thin(rows, per, width, seed):
    """Rows in tiles of `per`: every third tile a dense block of `width` columns, every third a rank-1
    block, the others covered by rank-0 blocks alone. Returns from_flat's arguments and y(X)."""
    rng = np.random.default_rng(seed)
    tiles = rows // per
    n = 4 * width
    dense, dd, ui, ud, vi, vd, parts = [], [], [], [], [], [], []
    for t in range(tiles):
        r0, c0 = t * per, int(rng.integers(0, n - width + 1))
        if t % 3 == 0:
            A = rng.standard_normal((per, width))
            dense.append([r0 + 1, r0 + per, c0 + 1, c0 + width, sum(a.size for a in dd)])
            dd.append(A.reshape(-1))
            parts.append((r0, c0, A))
        else:
            k = 1 if t % 3 == 1 else 0
            U, V = rng.standard_normal((per, k)), rng.standard_normal((k, width))
            ui.append([r0 + 1, r0 + per, len(vi) + 1, len(vi) + k, sum(a.size for a in ud)])
            for q in range(k):
                vi.append([c0 + 1, c0 + width, sum(a.size for a in vd)])
                vd.append(V[q])
            ud.append(U.reshape(-1))
            parts.append((r0, c0, U @ V))
    cat = lambda a: np.concatenate(a) if a else np.zeros(0)
    flat = (rows, n, np.arange(1, rows + 1), np.arange(1, n + 1), np.array(dense), cat(dd), np.array(ui), cat(ud),
            np.array(vi), cat(vd))

    def y(X):
        Y = np.zeros((rows, X.shape[1]))
        for r0, c0, A in parts:
            Y[r0:r0 + per] = A @ X[c0:c0 + A.shape[1]]
        return Y

    return flat, y


@pytest.mark.parametrize("precision,tol", [("f64", 1e-12), ("f32", 1e-5)])
@pytest.mark.parametrize("nrhs", [3, 8, 16, 32])
def test_short_tiles_several_columns(gpu, precision, tol, nrhs):
    import torch
    flat, ref = _thin(9 * 2400, 9, 4, seed=nrhs)
    H = hmgpu.HMatrix.from_flat(*flat, precision=precision)
    X = np.random.default_rng(nrhs + 1).standard_normal((H.shape[1], nrhs)).astype(np.float32).astype(np.float64)
    want = ref(X)
    dt = torch.float64 if precision == "f64" else torch.float32
    Xd = torch.tensor(X.T.copy(), dtype=dt, device=gpu).t()
    first = H * Xd
    assert np.linalg.norm(first.double().cpu().numpy() - want) <= tol * np.linalg.norm(want)
    for _ in range(50):
        assert torch.equal(H * Xd, first)


@pytest.mark.parametrize("precision,tol", [("f64", 1e-12), ("f32", 1e-5), ("mixed", 1e-5)])
def test_tiles_without_columns_one_column(gpu, precision, tol):
    """Tiles covered by rank-0 blocks alone come one after another, at the end of the list."""
    import torch
    flat, ref = _thin(9 * 6000, 9, 4, seed=7)
    H = hmgpu.HMatrix.from_flat(*flat, precision=precision)
    x = np.random.default_rng(8).standard_normal((H.shape[1], 1)).astype(np.float32).astype(np.float64)
    want = ref(x)[:, 0]
    xd = torch.tensor(x[:, 0], dtype=torch.float64 if precision == "f64" else torch.float32, device=gpu)
    first = H * xd
    assert np.linalg.norm(first.double().cpu().numpy() - want) <= tol * np.linalg.norm(want)
    assert (first.cpu().numpy()[want == 0.0] == 0.0).all()
    for _ in range(50):
        assert torch.equal(H * xd, first)
