// Correctly rounded FP64 division and square root on the integer pipe.
//
// GB300 executes one FP64 warp instruction per ~64 cycles per SM
// sub-partition, while its integer and FP32 pipes accept a warp instruction
// every cycle or two.  An IEEE double division costs about nine FP64
// instructions (a reciprocal seed refined by Newton steps in FP64 plus the
// rounding correction), so the FP64-bound face kernels spend about half of
// their FP64 pipe time in divisions.  Here the quotient is computed exactly
// in 64-bit integer arithmetic instead:
//
//   * a, b normal: a / b = rho 2^k with rho = mA / mb in [1, 2), mb the 53-bit
//     mantissa of b and mA that of a, doubled where it is below mb.
//   * Q = floor(rho 2^53), 54 bits, is formed by schoolbook long division in
//     two digits with a 32-bit fixed-point reciprocal y of mb (the method of
//     division by invariant integers: T. Granlund, P. Montgomery, PLDI 1994;
//     N. Moller, T. Granlund, IEEE Trans. Computers 60(2), 2011): y is the
//     FP32 reciprocal of b's top 24 bits refined by one Newton step, kept
//     below the exact value, so each digit is low by a few units at most and
//     each remainder, formed modulo 2^64, is non-negative and fits.  One
//     comparison of the last remainder with mb makes Q exact.
//   * A quotient of two 53-bit integers is never halfway between two 53-bit
//     numbers (odd 54-bit Q times mb would need more than 53 bits), so
//     (Q + 1) >> 1 is the quotient rounded to nearest.
//
// Bounds (y below by at most 1.5 2^-30, first digit low by less than 6 units,
// second by less than 2) hold for any seed within the documented error of
// rcp.approx (1 ulp).  A division is about 55 instructions; the earlier form,
// with a 64-bit reciprocal and 128-bit remainders, was about 170 and left the
// ALU pipe nearly as busy as the FP64 pipe.
//
// Results are therefore the IEEE round-to-nearest quotients, bit for bit.
// Operands outside the fast path (zero, subnormal, infinite or NaN divisor,
// subnormal, infinite or NaN dividend, a quotient outside the normal range)
// take the ordinary division, which gives the IEEE result for them too.
//
// A divisor used with several dividends is prepared once (den_prep); each
// quotient then costs the two digits (quot).
//
// The same file holds the integer forms of the correctly rounded products by
// constants (small integers, powers of two, literals such as 1/6) and of the
// density guard r + 1e-30; they are described beside their code.
//
// The square root follows the same pattern: m in [1, 4) with an even exponent
// left over, y from the FP32 inverse square root and one Newton step, the
// first digit m y, the second from the remainder, Q = floor(sqrt(m) 2^53)
// made exact by one comparison of m 2^106 - Q^2 with 2 Q, and (Q + 1) >> 1
// (the root of a 53-bit number is never a rounding midpoint).
#pragma once

#include <stdint.h>

namespace pda {

// several quotients by one divisor (the divisor's reciprocal formed once)
struct Quot2 {
  double q0, q1;
};
struct Quot3 {
  double q0, q1, q2;
};
struct Quot4 {
  double q0, q1, q2, q3;
};

namespace ip {

#if defined(__CUDACC__)

__device__ __forceinline__ float rcp_seed_f32(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ uint64_t mant53(uint64_t u) {
  return (u & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
}

// low 64 bits of q m (m < 2^53): a 32x32 wide product and a 32-bit one
__device__ __forceinline__ uint64_t mul_lo(uint32_t q, uint64_t m) {
  return (uint64_t)q * (uint32_t)m + ((uint64_t)(q * (uint32_t)(m >> 32)) << 32);
}

// fixed-point seed: r in [1/2, 1] as an FP32 value to r 2^32 - 3 2^9, rounded
// to a multiple of 2^9 (r + 1 - 3 2^-23 lies in [1, 2), so its fraction bits
// are that number)
__device__ __forceinline__ uint32_t seed_bits(float r) {
  return __float_as_uint(r + __uint_as_float(0x3F7FFFFAu)) << 9;
}

// The fast paths take operands whose biased exponent lies in [768, 1280),
// 2^-255 <= |x| < 2^257: products and quotients of such operands are normal,
// so no other exponent is checked.  exp_window(high word) is below 2^30 for
// these and not below for any other (subnormal, infinite and NaN among them).
__device__ __forceinline__ uint32_t exp_window(uint32_t h) { return 2u * h - (768u << 21); }
__device__ __forceinline__ uint32_t hi_word(double x) { return (uint32_t)__double2hiint(x); }
__device__ __forceinline__ uint32_t lo_word(double x) { return (uint32_t)__double2loint(x); }
__device__ __forceinline__ double from_words(uint32_t h, uint32_t l) { return __hiloint2double((int)h, (int)l); }
// sign and exponent bits; mantissa bits with the leading one.  Sign and
// exponent fields add and subtract modulo 2^32: the sign bit as exclusive or.
__device__ __forceinline__ uint32_t sign_exp(uint32_t h) { return h & 0xFFF00000u; }
__device__ __forceinline__ uint32_t mant_hi(uint32_t h) { return (h & 0x000FFFFFu) | 0x00100000u; }

template <typename... T>
__device__ __forceinline__ bool in_window(T... x) {
  return (exp_window(hi_word(x)) | ...) < (1u << 30);
}

// a prepared divisor
struct Den {
  double b;
  uint64_t mb;  // 53-bit mantissa
  uint32_t y;   // 2^32 2^52 / mb, low by at most 1.5 2^-30 of itself
  uint32_t w;   // exp_window
};

__device__ __forceinline__ Den den_prep(double b) {
  Den D;
  const uint32_t h = hi_word(b), l = lo_word(b);
  D.b = b;
  D.w = exp_window(h);
  const uint32_t mh = mant_hi(h);
  D.mb = (uint64_t)mh << 32 | l;
  // mb 2^-52 with 31 fraction bits, truncated.  (The funnel shift intrinsic is volatile assembly: with it the compiler
  // kept equal quotients apart, 74 per first-order 1D row instead of 47, and V + J of 10^6 cells took 1000 us, not 847.)
  const uint32_t bh = mh << 11 | l >> 21;
  // the top 23 fraction bits as an FP32 number in [1, 2)
  const uint32_t y0 = seed_bits(rcp_seed_f32(__uint_as_float((bh >> 8) + 0x3F000000u)));
  // Newton: e = 1 - y0 b in units of 2^-31, made low by 2 units so that y stays low
  const uint32_t e = 0x7FFFFFFEu - __umulhi(y0, bh);
  D.y = y0 + __umulhi(y0, 2u * e);
  return D;
}

// results outside the fast path: zero dividends, and the ordinary division
static __device__ __noinline__ double quot_special(double a, double b) {
  const uint64_t ua = (uint64_t)__double_as_longlong(a), ub = (uint64_t)__double_as_longlong(b);
  const uint32_t eb = (uint32_t)(ub >> 52) & 0x7FFu;
  if ((ua << 1) == 0 && eb - 1u < 0x7FEu)  // +-0 / normal
    return __longlong_as_double((long long)((ua ^ ub) & 0x8000000000000000ull));
  return a / b;
}

// RN(a / b) for a prepared divisor
__device__ __forceinline__ double quot(double a, const Den &D) {
  const uint32_t h = hi_word(a), l = lo_word(a);
  if ((exp_window(h) | D.w) >= (1u << 30)) return quot_special(a, D.b);
  const uint64_t ma = (uint64_t)mant_hi(h) << 32 | l;
  const bool ge = ma >= D.mb;
  // sign and (biased exponent - 1): the mantissa's leading bit, and a carry, add one
  const uint32_t eb = sign_exp(h) - sign_exp(hi_word(D.b)) + (ge ? 1022u << 20 : 1021u << 20);
  // rho = mA / mb in [1, 2); Q = floor(rho 2^53) in two digits
  const uint64_t mA = ge ? ma : ma << 1;
  const uint32_t q1 = __umulhi((uint32_t)(mA >> 22), D.y);       // rho 2^30, low by less than 6
  const uint64_t r1 = (mA << 30) - mul_lo(q1, D.mb);             // in [0, 6 mb)
  const uint32_t q2 = __umulhi((uint32_t)(r1 >> 24), D.y) >> 5;  // r1 2^23 / mb, low by less than 2
  const uint64_t r2 = (r1 << 23) - mul_lo(q2, D.mb);             // in [0, 2 mb)
  const uint32_t t = (q2 + (r2 >= D.mb ? 2u : 1u)) >> 1;         // Q's rounding bit added, dropped
  const uint64_t m = ((uint64_t)(eb + (q1 >> 10)) << 32 | (q1 << 22)) + t;
  return __longlong_as_double((long long)m);
}

__device__ __forceinline__ double div(double a, double b) { return quot(a, den_prep(b)); }
__device__ __forceinline__ Quot2 div2(double a0, double a1, double b) {
  const Den D = den_prep(b);
  return {quot(a0, D), quot(a1, D)};
}
__device__ __forceinline__ Quot3 div3(double a0, double a1, double a2, double b) {
  const Den D = den_prep(b);
  return {quot(a0, D), quot(a1, D), quot(a2, D)};
}
__device__ __forceinline__ Quot4 div4(double a0, double a1, double a2, double a3, double b) {
  const Den D = den_prep(b);
  return {quot(a0, D), quot(a1, D), quot(a2, D), quot(a3, D)};
}

__device__ __forceinline__ float rsqrt_seed_f32(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

static __device__ __noinline__ double sqrt_special(double x) {
  const uint64_t ux = (uint64_t)__double_as_longlong(x);
  if ((ux << 1) == 0) return x;  // +-0
  return ::sqrt(x);
}

// RN(sqrt(x))
__device__ __forceinline__ double sqrt(double x) {
  const uint64_t ux = (uint64_t)__double_as_longlong(x);
  const uint32_t ex = (uint32_t)(ux >> 52);
  if (ex - 1u >= 0x7FEu) return sqrt_special(x);  // zero, subnormal, infinite, NaN, negative
  const uint32_t odd = (ex & 1u) ^ 1u;            // parity of ex - 1023
  const uint64_t m = mant53(ux) << odd;           // m 2^-52 in [1, 4)
  const uint32_t mh = (uint32_t)(m >> 22);        // with 30 fraction bits, truncated
  const uint32_t y0 = seed_bits(
      rsqrt_seed_f32(__uint_as_float(((127u + odd) << 23) | ((uint32_t)(ux >> 29) & 0x7FFFFFu))));
  // Newton: e = 1 - m y0^2 in units of 2^-30, made low by 3 units; y = 2^32 / sqrt(m), low by at most 2^-29.3 of itself
  const uint32_t e = 0x3FFFFFFDu - __umulhi(mh, __umulhi(y0, y0));
  const uint32_t y = y0 + __umulhi(y0, 2u * e);
  const uint32_t s1 = __umulhi(mh, y);                        // sqrt(m) 2^30, low by less than 7
  const uint64_t r1 = (m << 8) - (uint64_t)s1 * s1;           // m 2^60 - s1^2 < 2^35
  const uint32_t q2 = __umulhi((uint32_t)(r1 >> 3), y) >> 5;  // (sqrt(m) 2^30 - s1) 2^23, low by less than 2
  const uint64_t Q = ((uint64_t)s1 << 23) + q2;
  const uint64_t r2 = (r1 << 46) - (((uint64_t)s1 * q2) << 24) - (uint64_t)q2 * q2;  // m 2^106 - Q^2
  const uint32_t t = (q2 + (r2 > 2 * Q ? 2u : 1u)) >> 1;
  const uint64_t hi = (uint64_t)((ex + 1u - odd + 1021u) >> 1) << 52;
  return __longlong_as_double((long long)(hi + ((uint64_t)s1 << 22) + t));
}

// Out-of-line forms for kernels where code size and compile time matter more
// than the last cycles (row tables, Jacobians, reduced-order model): a call
// costs a few integer and move instructions, which do not touch the FP64 pipe.
static __device__ __noinline__ double div_call(double a, double b) { return div(a, b); }
static __device__ __noinline__ double sqrt_call(double x) { return sqrt(x); }
// Several quotients by one divisor, out of line: one division call per
// quotient.  A call that returns one double keeps its result in registers;
// sharing the reciprocal through a call that returns two or more quotients
// (or stores them) measured slower in the face kernels, and so did forming
// the reciprocal out of line with the quotients in place (more code).
__device__ __forceinline__ Quot2 div2_call(double a0, double a1, double b) { return {div_call(a0, b), div_call(a1, b)}; }
__device__ __forceinline__ Quot3 div3_call(double a0, double a1, double a2, double b) {
  return {div_call(a0, b), div_call(a1, b), div_call(a2, b)};
}
__device__ __forceinline__ Quot4 div4_call(double a0, double a1, double a2, double a3, double b) {
  return {div_call(a0, b), div_call(a1, b), div_call(a2, b), div_call(a3, b)};
}

// ---------------------------------------------------------------------------
// Exact-by-construction products and sums on the integer pipe.
//
// The WENO and Rusanov expressions multiply by small integers (3, 5, 7, 11),
// by 1/2 and 1/4, by constants (1/6, 13/12, 2e-6), and add 1e-30 to a
// density.  Each of these has an IEEE round-to-nearest result that integer
// arithmetic forms from the bit pattern at a fraction of an FP64
// instruction's cost on GB300, so they leave the FP64 pipe to the products
// and sums of two variables:
//   * RN(K x), K a small integer: the 53-bit mantissa times K fits 57 bits;
//     it is shifted back to 53 bits with round to nearest, ties to even, and
//     a carry into bit 53 moves into the exponent field by adding the
//     mantissa (implicit bit included) to the exponent minus one;
//   * RN(x y): the 106-bit product of the mantissas from four 32-bit products,
//     rounded in the same way;
//   * x * 2^-S is exact while the result stays normal: S is subtracted from
//     the exponent field;
//   * RN(r + 1e-30) = r whenever 1e-30 is below half a unit in the last place
//     of r: for |r| >= 2^-44 the nearest neighbour of r lies at least 2^-97
//     (about 6.3e-30) away on either side.
// Operands outside these fast paths (zero, tiny, huge, infinite or NaN) take
// the ordinary FP64 operation, so every result is the IEEE one bit for bit.
// Executed instructions, measured on loops of one operation: division 68
// (a call included), root 66, product 37, square 36, product by a constant
// 33, by a small integer 29, x / 2 11, guard 6; about 6 fewer each without
// the check of their operands.  (Earlier forms: division 170, product by a
// small integer 43, x / 2 15, guard 9.)  An FP64 instruction takes the time
// of 64 issue slots.
// (out of line: in place, the compiler executes them ahead of the branch, on the pipe that is to be spared)
static __device__ __noinline__ double mul_call(double a, double b) {
  // zero times finite, as in fields at rest
  const uint32_t ah = hi_word(a), bh = hi_word(b);
  if (((ah << 1 | lo_word(a)) == 0 || (bh << 1 | lo_word(b)) == 0) && (ah & 0x7FF00000u) != 0x7FF00000u &&
      (bh & 0x7FF00000u) != 0x7FF00000u)
    return from_words((ah ^ bh) & 0x80000000u, 0u);
  return a * b;
}
static __device__ __noinline__ double add_call(double a, double b) { return a + b; }

// The product of two 53-bit mantissas xh:xl, yh:yl, P in [2^104, 2^106), as
// 32-bit words (four 32 x 32-bit products; the middle sum fits 64 bits)
struct Prod {
  uint32_t w3, w2, w1, w0;
};
__device__ __forceinline__ Prod mant_product(uint32_t xh, uint32_t xl, uint32_t yh, uint32_t yl) {
  const uint64_t p = (uint64_t)xl * yl;
  const uint64_t t = (uint64_t)xl * yh + (uint64_t)xh * yl + (p >> 32);
  const uint64_t h = (uint64_t)xh * yh + (t >> 32);
  return {(uint32_t)(h >> 32), (uint32_t)h, (uint32_t)t, (uint32_t)p};
}

// A product's bits: the top 53 bits of P (shifted down by 52, or 53 where
// P >= 2^105), rounded by the bits below, ties to even where TIES (they can
// occur).  eb: sign and exponent field sum less the bias and one.
template <bool TIES>
__device__ __forceinline__ double round_product(const Prod &p, uint32_t eb) {
  const uint32_t top = p.w3 >> 9, s = 20u + top;
  const uint32_t m1 = __funnelshift_r(p.w2, p.w3, s), m0 = __funnelshift_r(p.w1, p.w2, s);
  const uint32_t w = __funnelshift_r(p.w0, p.w1, s);
  uint32_t up = w >> 31;
  if (TIES && w == 0x80000000u && p.w0 == 0) up = m0 & 1u;
  const uint64_t m = ((uint64_t)(m1 + eb + (top << 20)) << 32 | m0) + up;
  return __longlong_as_double((long long)m);
}

// RN(x c) for a positive constant c (a literal: its words fold at compile
// time).  Where c's mantissa MC is odd, MX MC is a rounding midpoint only for
// MX = 3 2^51 (the product needs at least 51 trailing zero bits, all of them
// MX's), with kept part (3 MC - 1) / 2: for MC = 1 mod 4 that is odd and
// rounding up gives the even neighbour, so no tie needs to be detected (1/6,
// 13/12 and 2e-6 are such constants).
__device__ __forceinline__ double mul_const_u(double x, const double c) {
  const uint32_t h = hi_word(x), ch = hi_word(c), cl = lo_word(c);
  const uint32_t eb = sign_exp(h) + sign_exp(ch) - (1024u << 20);
  const Prod p = mant_product(mant_hi(h), lo_word(x), mant_hi(ch), cl);
  return (cl & 3u) == 1u ? round_product<false>(p, eb) : round_product<true>(p, eb);
}

// RN(x y)
__device__ __forceinline__ double mul_u(double x, double y) {
  const uint32_t h = hi_word(x), g = hi_word(y);
  const uint32_t eb = sign_exp(h) + sign_exp(g) - (1024u << 20);
  return round_product<true>(mant_product(mant_hi(h), lo_word(x), mant_hi(g), lo_word(y)), eb);
}

// RN(x^2)
__device__ __forceinline__ double square_u(double x) {
  const uint32_t h = hi_word(x);
  const uint32_t eb = 2u * sign_exp(h) - (1024u << 20);
  const uint32_t mh = mant_hi(h), l = lo_word(x);
  return round_product<true>(mant_product(mh, l, mh, l), eb);
}

// The forms *_u do not check their operands: a caller with several products
// checks all their operands at once (in_window), so that the products lie in
// one basic block and overlap.  Normal operands suffice where the result is
// normal.

// RN(K x) for an integer constant 2 < K < 16 that is not a power of two: the
// 53-bit mantissa times K fits 57 bits and is shifted back by s bits
template <int K>
__device__ __forceinline__ double mul_small_u(double x) {
  static_assert(K > 2 && K < 16 && (K & (K - 1)) != 0, "K: a small integer that is not a power of two");
  constexpr int KB = K >= 8 ? 3 : (K >= 4 ? 2 : 1);  // floor(log2 K)
  const uint32_t h = hi_word(x);
  // P = m K in [2^(52+KB), 2^(54+KB)); s = KB or KB + 1 puts P >> s in [2^52, 2^53)
  const uint64_t pl = (uint64_t)lo_word(x) * K;
  const uint32_t p0 = (uint32_t)pl, p1 = mant_hi(h) * K + (uint32_t)(pl >> 32);
  const uint32_t s = (p1 >> (21 + KB)) + KB;
  const uint32_t m1 = p1 >> s, m0 = __funnelshift_r(p0, p1, s);
  // the s bits shifted out, at the top of a word, plus one where the kept part is odd
  const uint32_t w = __funnelshift_r(0u, p0, s) + (m0 & 1u);
  const uint64_t m = ((uint64_t)(m1 + sign_exp(h) + (s << 20) - (1u << 20)) << 32 | m0) + (w > 0x80000000u ? 1u : 0u);
  return __longlong_as_double((long long)m);
}

// The same with the check of their operands
__device__ __forceinline__ double mul(double x, double y) {
  return in_window(x, y) ? mul_u(x, y) : mul_call(x, y);
}
template <int K>
__device__ __forceinline__ double mul_small(double x) {
  return in_window(x) ? mul_small_u<K>(x) : mul_call(x, (double)K);
}
// the product out of line, where code size matters more than a call
static __device__ __noinline__ double mul_out(double x, double y) { return mul(x, y); }

// x / 2, unchecked
__device__ __forceinline__ double half_u(double x) { return from_words(hi_word(x) - (1u << 20), lo_word(x)); }
// x * 2^-S (S = 1, 2): exact for a normal result
template <int S>
__device__ __forceinline__ double mul_pow2_neg(double x) {
  static_assert(S >= 1 && S <= 8, "S");
  const uint32_t h = hi_word(x);
  if (exp_window(h) >= (1u << 30)) return mul_call(x, 1.0 / (double)(1 << S));
  return from_words(h - ((uint32_t)S << 20), lo_word(x));
}

// RN(r + 1e-30): r for 2^-44 <= |r| < infinity
__device__ __forceinline__ double add_1em30(double r) {
  if (2u * hi_word(r) - (979u << 21) >= (0x7FFu - 979u) << 21) return add_call(r, 1.e-30);
  return r;
}

#endif  // __CUDACC__

}  // namespace ip
}  // namespace pda
