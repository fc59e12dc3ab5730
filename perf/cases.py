"""The work that a program gives this framework, as cases that can be timed.

A case is one of three things a program does through the public entry points:

  product   y = H x (mul!) with an H-matrix that the program keeps, for one or several
            right-hand sides, in each storage precision;
  batch     one product of many small H-matrices as one block-diagonal operator, replayed
            from a CUDA graph;
  assemble  cluster tree, H-matrix and its first product, from points on the host: what a
            new geometry costs.

Point sets and parameters are those of the tests and of the benchmark: the unit circle with the
2-D log kernel, points in a cube and on a sphere, the jittered film, and the demagnetising
tensor, whose points own three rows and columns each.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(1, os.path.abspath("hmatrixgpu.jl_gb300"))
import hmgpu  # noqa: E402


def _case(name, op, geometry, n, kernel, leaf, eta, eps, precision, nrhs=1, members=1):
    return {"name": name, "op": op, "geometry": geometry, "n": n, "kernel": kernel, "leaf": leaf, "eta": eta,
            "eps": eps, "precision": precision, "nrhs": nrhs, "members": members}


def listed():
    return [
        # a boundary-element problem on a curve, FP64 as the reference has it: iterations of a
        # small solver, where a product's launches count more than its bytes
        _case("circle-1000 f64 x1", "product", "circle", 1000, "log2d", 64, 1.5, 1e-6, "f64"),
        # a screened potential on a surface mesh of ordinary size, FP32
        _case("sphere-20011 f32 x1", "product", "sphere", 20011, "yukawa", 32, 1.5, 1e-5, "f32"),
        # the benchmark's headline: one field evaluation on a film of a million cells
        _case("film-1048576 f32 x1", "product", "film", 1 << 20, "laplace", 64, 2.0, 1e-4, "f32"),
        # the default precision on a volume at a tight tolerance
        _case("cube-40960 f64 x1", "product", "cube", 40960, "laplace", 64, 2.0, 1e-6, "f64"),
        # the demagnetising field of cells with three components, a handful of states at once
        _case("dipolar-300 f64 x6", "product", "cube", 300, "dipolar", 16, 1.0, 1e-6, "f64", 6),
        # a block solver's columns in plain FP32
        _case("film-262144 f32 x32", "product", "film", 1 << 18, "laplace", 64, 2.0, 1e-4, "f32", 32),
        # the same in mixed precision, on a film that is not square
        _case("film-500500 mixed x32", "product", "film", 500500, "laplace", 64, 2.0, 1e-4, "mixed", 32),
        # many columns on a volume at a tight tolerance: 64 and a remainder
        _case("cube-32768 mixed x70", "product", "cube", 32768, "laplace", 64, 2.0, 1e-6, "mixed", 70),
        # many bodies of different sizes, one product each per step
        _case("batch-12 spheres f32 x1", "batch", "sphere", 24000, "yukawa", 32, 1.5, 1e-5, "f32", 1, 12),
        # a new film geometry: tree, assembly and first product
        _case("assemble film-262144 f32", "assemble", "film", 1 << 18, "laplace", 64, 2.0, 1e-4, "f32"),
        # the default precision at a tight tolerance: the assembly itself is most of the work
        _case("assemble cube-32768 f64", "assemble", "cube", 32768, "laplace", 64, 2.0, 1e-6, "f64"),
        # a small body with the demagnetising tensor, for many products with many columns
        _case("assemble dipolar-216 mixed", "assemble", "cube", 216, "dipolar", 16, 1.0, 1e-6, "mixed"),
    ]


# geometry, kernel, leaf sizes, eta, tolerances, points from, to
_KINDS = [
    ("circle", "log2d", (64,), 1.5, (1e-6,), 500, 20000),
    ("sphere", "yukawa", (16, 32), 1.5, (1e-5,), 700, 131072),
    ("cube", "laplace", (32, 64), 2.0, (1e-4, 1e-5, 1e-6), 300, 40960),
    ("film", "laplace", (64,), 2.0, (1e-4,), 2000, 1 << 20),
    ("cube", "dipolar", (16,), 1.0, (1e-6,), 60, 216),
]


def _log_uniform(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    geometry, kernel, leaves, eta, tols, lo, hi = rng.choice(_KINDS)
    leaf, eps = rng.choice(leaves), rng.choice(tols)
    u = rng.random()
    if u < 0.1:
        n = _log_uniform(rng, 2000, 24000)
        c = _case("", "batch", "sphere", n, "yukawa", 32, 1.5, 1e-5, rng.choice(("f32", "f64", "mixed")), 1,
                  rng.randint(2, 12))
    elif u < 0.3:
        n = _log_uniform(rng, lo, min(hi, {"cube": 32768, "film": 1 << 18, "sphere": 65536}.get(geometry, hi)))
        c = _case("", "assemble", geometry, n, kernel, leaf, eta, eps, rng.choice(("f64", "f32", "mixed")))
    else:
        precision = rng.choice(("f64", "f32", "f32", "mixed"))
        nrhs = 1 if rng.random() < 0.4 else _log_uniform(rng, 2, 70)
        if precision != "mixed" and nrhs > 1:  # columns times points as the largest listed ones have
            hi = min(hi, max(2 * lo, (1 << 23) // nrhs))
        if precision == "f64":
            hi = min(hi, 1 << 18)
        c = _case("", "product", geometry, _log_uniform(rng, lo, hi), kernel, leaf, eta, eps, precision, nrhs)
    del c["name"]
    return c


def _points(geometry, n, seed):
    """3 x n points, as the tests and the benchmark make them."""
    rng = np.random.default_rng(seed)
    if geometry == "circle":
        i = np.arange(1, n + 1, dtype=np.float64)
        return np.stack([np.sin(i * 2 * np.pi / n), np.cos(i * 2 * np.pi / n), np.zeros(n)])
    if geometry == "sphere":
        v = rng.standard_normal((3, n))
        return v / np.linalg.norm(v, axis=0)
    if geometry == "film":  # a grid of cells, about square, the last row ragged
        nx = int(math.isqrt(n - 1)) + 1
        k = np.arange(n)
        g = np.stack([k // nx, k % nx, np.zeros(n)]).astype(np.float64)
        return g + 0.05 * rng.standard_normal(g.shape)
    return rng.random((n, 3)).T.copy()


def _dims(case):
    return 3 if case["kernel"] == "dipolar" else 1


def _dtype(case):
    return torch.float64 if case["precision"] == "f64" else torch.float32


def _assemble(case, P):
    T = hmgpu.ClusterTree(P, max_points_per_leaf=case["leaf"], dims=_dims(case), gpu=True)
    return hmgpu.HMatrix(hmgpu.Kernel(case["kernel"], P), T, T, eta=case["eta"], eps=case["eps"],
                         precision=case["precision"])


def _member_points(case, seed):
    """Member sizes spread over a factor of twelve below n, and their points."""
    k = case["members"]
    return [_points(case["geometry"], max(200, int(case["n"] * 12.0 ** (-i / max(1, k - 1)))), 1000 * seed + i)
            for i in range(k)]


def _vectors(case, n, seed):
    """x as the entry points take it: a vector, or columns one after another."""
    g = torch.Generator("cuda").manual_seed(seed)
    x = torch.randn((case["nrhs"], n), generator=g, device="cuda", dtype=torch.float64).to(_dtype(case))
    return x[0].contiguous() if case["nrhs"] == 1 else x.t()


def _like(case, m):
    y = torch.empty((case["nrhs"], m), device="cuda", dtype=_dtype(case))
    return y[0] if case["nrhs"] == 1 else y.t()


def prepare(case, seed):
    if case["op"] == "batch":
        members = [_assemble(case, P) for P in _member_points(case, seed)]
        H = hmgpu.batch(members)
        x, y = _vectors(case, H.shape[1], seed), _like(case, H.shape[0])
        return {"op": "batch", "graph": hmgpu.Graph(H, x, y)}
    P = _points(case["geometry"], case["n"], seed)
    n = _dims(case) * case["n"]
    state = {"op": case["op"], "x": _vectors(case, n, seed)}
    if case["op"] == "product":
        return state | {"H": _assemble(case, P), "y": _like(case, n)}
    return state | {"case": case, "P": P}


def run(state):
    if state["op"] == "product":
        return hmgpu.mul_(state["y"], state["H"], state["x"])
    if state["op"] == "batch":
        return state["graph"].launch()
    H = _assemble(state["case"], state["P"])
    out = {"y": H * state["x"]}
    info = H.info()  # what the program logs of the matrix it got
    out |= {k: info[k] for k in ("admissible_leaves", "full_leaves", "max_rank", "total_rank", "dense_entries",
                                 "far_entries")}
    target, source = H.index_maps()
    return out | {"target": target, "source": source}


@functools.lru_cache(maxsize=None)
def _stored(items):
    """(stored entries, sum over blocks of r^2 (m + n), total rank, rows and columns) of a case's H-matrices."""
    case = dict(items)
    sets = _member_points(case, 1) if case["op"] == "batch" else [_points(case["geometry"], case["n"], 1)]
    entries = qr = rank = n = 0
    for P in sets:
        H = _assemble(case | {"precision": "f32"}, P)
        i, (_, a) = H.info(), H.blocks()
        a = a.astype(np.float64)
        entries += i["dense_entries"] + i["far_entries"]
        qr += float(((a[:, 1] - a[:, 0] + a[:, 3] - a[:, 2] + 2) * a[:, 4] ** 2).sum()) if len(a) else 0.0
        rank += i["total_rank"]
        n += P.shape[1] * _dims(case)
    return entries, qr, rank, n


def work(case):
    entries, qr, rank, n = _stored(tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "nrhs", "precision"))))
    es, nrhs = (8 if case["precision"] == "f64" else 4), case["nrhs"]
    product = {"bytes": es * (entries + nrhs * 2 * n), "flops": 2.0 * nrhs * entries}
    if case["op"] != "assemble":
        return product
    # every stored entry is generated and written, then read by the first product; an entry is
    # about 10 operations, the elimination of the terms before it, QR and the factors about 9 r^2 (m + n)
    return {"bytes": 24 * n + es * entries + product["bytes"], "flops": product["flops"] + 10.0 * entries + 9.0 * qr}


def _rows(kernel, X, Y):
    """Kernel values of target points X against source points Y (rows x columns) in FP64."""
    d = X[:, :, None] - Y[:, None, :]
    if kernel == "dipolar":
        r2 = (d * d).sum(0)
        r5 = (r2 * r2 * r2.sqrt()).masked_fill(r2 == 0, 1.0)
        K = torch.empty((X.shape[1], 3, Y.shape[1], 3), dtype=X.dtype, device=X.device)
        for a in range(3):
            for b in range(3):
                v = -3.0 * d[a] * d[b]
                if a == b:
                    v = v + r2
                K[:, a, :, b] = (v / r5 / (4 * math.pi)).masked_fill(r2 == 0, 0.0)
        return K.reshape(3 * X.shape[1], 3 * Y.shape[1])
    r = (d * d).sum(0).sqrt_()
    at0 = r == 0
    if kernel == "log2d":
        near = r < 1e-12
        return (-torch.log(r.masked_fill_(near, 1.0)) / (2 * math.pi)).masked_fill_(near, 1.0)
    r.masked_fill_(at0, 1.0)
    v = torch.exp(-r) / r if kernel == "yukawa" else 1.0 / (4 * math.pi * r)
    return v.masked_fill_(at0, 0.0)


def _dense_product(case, P, x):
    """K x summed over all points in FP64."""
    Pt = torch.tensor(P, device="cuda", dtype=torch.float64)
    step = max(1, (1 << 26) // (Pt.shape[1] * _dims(case) ** 2))
    return torch.cat([_rows(case["kernel"], Pt[:, i:i + step], Pt) @ x for i in range(0, Pt.shape[1], step)])


def exact(case, seed):
    sets = _member_points(case, seed) if case["op"] == "batch" else [_points(case["geometry"], case["n"], seed)]
    d = _dims(case)
    if sum((d * P.shape[1]) ** 2 for P in sets) * (16 + case["nrhs"]) > 1.5e11:
        return None
    x = _vectors(case, d * sum(P.shape[1] for P in sets), seed).double()
    y, at = [], 0
    for P in sets:
        n = d * P.shape[1]
        y.append(_dense_product(case, P, x[at:at + n]))
        at += n
    y = torch.cat(y)
    y = y if y.dim() == 1 else y.t().contiguous().t()
    return {"y": y} if case["op"] == "assemble" else y
