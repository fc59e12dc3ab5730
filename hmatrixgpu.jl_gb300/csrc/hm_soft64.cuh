// IEEE FP64 division and square root (round to nearest even) on the integer pipes, and FP64
// additions and multiplications as FMAs, for the assembly kernels.
//
// The FP64 pipe of this GPU retires 1.67 additions or multiplications and 1.98 FMAs per clock
// and SM; a division or a square root, a dozen dependent FP64 instructions, takes it 4.4 clocks. The
// integer pipes have room for 64 to 128 operations in the same clock and are idle beside it.
// Measured, results per clock and SM (by the FP64 instructions in brackets): quotients 0.84 (0.23),
// roots 1.14 (0.22); sums as fma(a, 1, b) and products as fma(a, b, -0) 1.99 (1.67). On the
// integer pipes a product takes some 80 instructions, with its checks, and the QR and Jacobi
// kernels took twice as long with them.
//
// Every result is the correctly rounded one, bit for bit what the FP64 instruction gives
// (NaN payloads aside). Operands or results outside the normal range (zeros, subnormals,
// infinities, NaN, overflow) take the FP64 instructions.
//
// The header is also compiled by NVRTC with the entry kernels: it includes nothing.
#pragma once

namespace hm {

// not literals: FMAs with known ones and zeros would be turned back into additions and products
static __constant__ double kOne64 = 1.0, kMinusOne64 = -1.0, kMinusZero64 = -0.0;

__device__ __forceinline__ double dadd(double a, double b) { return __fma_rn(a, kOne64, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __fma_rn(b, kMinusOne64, a); }
__device__ __forceinline__ double dmul(double a, double b) { return __fma_rn(a, b, kMinusZero64); }

__device__ __forceinline__ unsigned s64_lo(unsigned long long v) { return static_cast<unsigned>(v); }
__device__ __forceinline__ unsigned s64_hi(unsigned long long v) { return static_cast<unsigned>(v >> 32); }
__device__ __forceinline__ unsigned long long s64_mul(unsigned a, unsigned b) {
  return static_cast<unsigned long long>(a) * b;
}
__device__ __forceinline__ unsigned long long s64_bits(double d) {
  return static_cast<unsigned long long>(__double_as_longlong(d));
}
__device__ __forceinline__ double s64_double(unsigned long long u) {
  return __longlong_as_double(static_cast<long long>(u));
}
// the 21 leading bits of a normal number's significand, hidden bit included
__device__ __forceinline__ unsigned s64_top(unsigned h) { return (h & 0xfffffu) | 0x100000u; }

__device__ __noinline__ double ddiv_any(double a, double b) { return __ddiv_rn(a, b); }
__device__ __noinline__ double dsqrt_any(double s) { return __dsqrt_rn(s); }

// 2^31 times an approximate value y in [1/2, 1], as an integer below 2^31
__device__ __forceinline__ unsigned s64_fixed(float y) {
  unsigned b = __float_as_uint(y);
  b = min(max(b, 0x3f000000u), 0x3f7fffffu);
  return ((b | 0x800000u) << 8) >> 1;
}

// a / b: the quotient of the significands in digits of 20, 20 and 13 bits, each estimated from
// the remainder's leading 32 bits and an approximate reciprocal (Knuth, The Art of Computer
// Programming, vol. 2, 4.3.1, the digit estimate of algorithm D). The reciprocal is made an
// underestimate (2^-23 from the operand's cut, one ulp of rcp.approx, less than the 8 ulps
// taken off), so that every remainder is >= 0 and below three divisors, and the last below
// two. The exact remainder then decides the rounding.
__device__ __forceinline__ double ddiv(double a, double b) {
  const unsigned long long ab = s64_bits(a), bb = s64_bits(b);
  const unsigned ah = s64_hi(ab), bh = s64_hi(bb);
  const unsigned ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu;
  // normal operands, and a quotient exponent of at least 1 after the shift below
  if (!(ea - 1u < 2046u && eb - 1u < 2046u && ea - eb + 1021u < 2044u)) return ddiv_any(a, b);
  const unsigned long long ma = (static_cast<unsigned long long>(s64_top(ah)) << 32) | s64_lo(ab);
  const unsigned long long mb = (static_cast<unsigned long long>(s64_top(bh)) << 32) | s64_lo(bb);
  const unsigned mbl = s64_lo(mb), mbh = s64_hi(mb);
  const unsigned less = ma < mb ? 1u : 0u;
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;"
      : "=f"(y)
      : "f"(__uint_as_float(0x3f800000u | ((bh & 0xfffffu) << 3) | (s64_lo(bb) >> 29))));
  const unsigned Y = s64_fixed(y) - 0x400u;
  auto times_b = [&](unsigned q) { return s64_mul(q, mbl) + (static_cast<unsigned long long>(q * mbh) << 32); };
  const unsigned long long A = ma << less;  // in [mb, 2 mb)
  const unsigned q1 = static_cast<unsigned>(s64_mul(static_cast<unsigned>(A >> 22), Y) >> 41);
  unsigned long long R = (A << 20) - times_b(q1);
  const unsigned q2 = static_cast<unsigned>(s64_mul(static_cast<unsigned>(R >> 24), Y) >> 39);
  R = (R << 20) - times_b(q2);
  const unsigned q3 = static_cast<unsigned>(s64_mul(static_cast<unsigned>(R >> 24), Y) >> 46);
  R = (R << 13) - times_b(q3);
  unsigned long long q = (static_cast<unsigned long long>(q1) << 33) + (static_cast<unsigned long long>(q2) << 13) + q3;
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const bool more = R >= mb;
    R -= more ? mb : 0ull;
    q += more;
  }
  unsigned long long m = q >> 1;  // q has 54 bits: its last is the first beyond the significand
  m += (s64_lo(q) & 1u) && (R != 0ull || (s64_lo(m) & 1u));
  const unsigned e = ea - eb + 1022u - less;  // m brings the hidden bit
  return s64_double((static_cast<unsigned long long>(e) << 52) + m +
                    (static_cast<unsigned long long>((ah ^ bh) & 0x80000000u) << 32));
}

// sqrt(s): with f in [1, 4) the significand under an even exponent, an approximate 1 / sqrt(f)
// gives sqrt(f) to 22 bits; a Newton step on the exact residual gives 43; the exact remainder of that
// one more, to within one unit of the last place; and its own remainder, exact again, decides the
// rounding (Newton with exact remainders, as in Zimmermann, "Karatsuba Square Root", 1999). A
// square root is never halfway between two numbers.
__device__ __forceinline__ double dsqrt(double s) {
  const unsigned long long b = s64_bits(s);
  const unsigned h = s64_hi(b), l = s64_lo(b);
  if (!(h - 0x00100000u < 0x7fe00000u)) return dsqrt_any(s);  // not positive, normal and finite
  const unsigned e = h >> 20, odd = (e & 1u) ^ 1u;
  const unsigned long long m = ((static_cast<unsigned long long>(s64_top(h)) << 32) | l) << odd;  // f 2^52
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;"
      : "=f"(y)
      : "f"(__uint_as_float(((127u + odd) << 23) | ((h & 0xfffffu) << 3) | (l >> 29))));
  const unsigned Y = s64_fixed(y);
  const unsigned X1 = s64_hi(s64_mul(s64_hi(m << 10), Y));  // sqrt(f) 2^29
  const long long r1 = static_cast<long long>((m << 6) - s64_mul(X1, X1));  // residual, times 2^58
  const int d1 = static_cast<int>((static_cast<long long>(static_cast<int>(r1 >> 8)) * static_cast<int>(Y)) >> 32);
  const unsigned long long X2 = (static_cast<unsigned long long>(X1) << 21) + static_cast<long long>(d1);  // 2^50
  const unsigned xl = s64_lo(X2), xh = s64_hi(X2);
  // f 2^100 - X2^2: its low 64 bits are all of it
  const long long r2 = static_cast<long long>(
      (m << 48) - (s64_mul(xl, xl) + (static_cast<unsigned long long>(2u * xl * xh) << 32)));
  const int c = static_cast<int>((static_cast<long long>(static_cast<int>(r2 >> 32)) * static_cast<int>(Y)) >> 32) >> 16;
  const unsigned long long r4 = X2 << 2;  // sqrt(f) 2^52, to be corrected by c
  const unsigned long long t = 2 * r4 + static_cast<long long>(c);
  const long long rem = static_cast<long long>((static_cast<unsigned long long>(r2) << 4) -
                                               t * static_cast<unsigned long long>(static_cast<long long>(c)));
  long long r = static_cast<long long>(r4) + c;
  r += rem > r ? 1 : rem <= -r ? -1 : 0;
  const unsigned er = static_cast<unsigned>(static_cast<int>(e - 1023u - odd) >> 1) + 1022u;  // r brings the hidden bit
  return s64_double((static_cast<unsigned long long>(er) << 52) + static_cast<unsigned long long>(r));
}

}  // namespace hm
