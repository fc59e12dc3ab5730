"""The assembly kernels' FP64 operations on the integer pipes against the FP64 instructions, bit for bit
(any NaN equals any NaN), over random and special operands: a user kernel whose entry (i, j) is 1 where
an operation on operands made from i and j differs."""
import numpy as np
import pytest

import hmgpu

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "hm_soft64.cuh"
__device__ unsigned long long mix(unsigned long long z) {  // splitmix64
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
__device__ bool same(double u, double v) {
  return (u != u && v != v) || __double_as_longlong(u) == __double_as_longlong(v);
}
__device__ double hmgpu_entry(const double *x, const double *y, const double *p, int a, int b) {
  const long long i = (long long)x[1], j = (long long)y[1];
  const unsigned long long h = mix(i * 100003 + j + (unsigned long long)p[0] * 7919);
  unsigned long long u = mix(h), v = mix(h + 1);
  const int kind = (int)(h % 6);
  if (kind < 4) {  // exponents near each other, so that quotients and sums round; significands near ends
    const unsigned long long e = 1023 - 30 + (h >> 32) % 60, f = e + (h >> 40) % 5 - 2;
    u = (u & 0x800fffffffffffffull) | (e << 52);
    v = (v & 0x800fffffffffffffull) | (f << 52);
    if (kind == 1) u |= 0x000ffffffffffff0ull;
    if (kind == 2) v = (v & 0xfff000000000000full);
    if (kind == 3) v = (v & 0xfff0000000000000ull) | ((u + ((h >> 50) & 3)) & 0x000fffffffffffffull);
  }  // kind 4: any bits; kind 5: one operand from the table of special values
  double s = __longlong_as_double((long long)u), t = __longlong_as_double((long long)v);
  if (kind == 5) {
    if (h & (1ull << 60)) s = p[1 + (h >> 8) % 40];
    if (h & (1ull << 61)) t = p[1 + (h >> 16) % 40];
  }
  bool ok = same(hm::dmul(s, t), __dmul_rn(s, t)) && same(hm::ddiv(s, t), __ddiv_rn(s, t));
  ok = ok && same(hm::dsqrt(s), __dsqrt_rn(s)) && same(hm::dsqrt(t), __dsqrt_rn(t));
  ok = ok && same(hm::dadd(s, t), __dadd_rn(s, t)) && same(hm::dsub(s, t), __dsub_rn(s, t));
  return ok ? 0.0 : 1.0;
}
"""

TINY = np.finfo(np.float64).tiny
SPECIAL = [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, TINY, -TINY, TINY - 5e-324, 2 * TINY, 3 * TINY, 1.0, -1.0,
           1.0 + 2.0 ** -52, 1.0 - 2.0 ** -53, 2.0, 4.0, 4.0 - 2.0 ** -51, 2.0 ** 52, 2.0 ** 53 - 1, 2.0 ** 511, 2.0 ** 512,
           2.0 ** 1022, 2.0 ** -511, 2.0 ** -512, 2.0 ** -537, 2.0 ** -538, np.finfo(np.float64).max, -np.finfo(np.float64).max,
           np.finfo(np.float64).max / 2, 1e-300, 1e300, 1e-160, 1e160, 3.0, 0.1, 1 / 3, 1e-15, 4 * np.pi]


@pytest.mark.parametrize("seed", range(6))
def test_bits_equal_the_instructions(gpu, seed):
    """9 million operand pairs per seed."""
    assert len(SPECIAL) == 40
    n = 3000
    P = np.stack([np.arange(n) * 1e-3, np.arange(n, dtype=np.float64), np.zeros(n)])
    T = hmgpu.ClusterTree(P, max_points_per_leaf=64)
    K = hmgpu.Kernel("user", P, user=SOURCE, params=[float(seed)] + SPECIAL)
    _, _, V = hmgpu.sparsify_hmatrix(K, T, T, eta=1e9, triplets=True)
    assert V.size == n * n
    assert V.sum() == 0.0
