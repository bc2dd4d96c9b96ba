// Correctly rounded FP64 quotients and square roots for the plain FP64
// kernels, in 64-bit integers.
//
// GB300 executes FP64 at 1.7 lanes per clock and SM: a warp's FP64
// instruction occupies its sub-partition's unit for 64 cycles, and four
// sub-partitions together take one every 19 cycles, in which the SM could
// issue 76 others. The FP64 kernels are bound by the number of FP64
// instructions. A quotient by a divisor that does not change (node mass,
// reference length) takes one high product of 64-bit integers with the
// divisor's reciprocal; a square root and the reciprocal of its result take
// Newton's iteration on integers from the FP32 approximation. The last bit is
// then decided from the part of the result below it, and in the rare case
// that the error of that part could matter, by the exact remainder, computed
// modulo 2^64 (it is small). No FP64 instruction, and the bits of the IEEE
// operations.
//  (Reciprocal multiplication with a remainder check: Granlund, Montgomery,
//  "Division by invariant integers using multiplication", PLDI 1994; Newton's
//  iteration for the inverse square root: Brent, Zimmermann, "Modern Computer
//  Arithmetic", 2010, 1.5 and 4.2.)
//
// The functions hold for normal numbers away from the ends of the range
// (in_range); callers take the general operations elsewhere. They compile for
// the host too, where tests compare them with the general operations on
// operands chosen to lie next to rounding boundaries.
#ifndef MFG_EXACT_CUH
#define MFG_EXACT_CUH

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define MFG_HD __host__ __device__ __forceinline__
#else
#define MFG_HD inline
#endif

namespace mfg {

MFG_HD int32_t hi_word(double x) {
#ifdef __CUDA_ARCH__
  return __double2hiint(x);
#else
  uint64_t u;
  std::memcpy(&u, &x, 8);
  return static_cast<int32_t>(u >> 32);
#endif
}

// 2^-800 <= |x| < 2^801: far enough from both ends for every product and
// residual below (divisors are held to 2^-100 .. 2^100 by exact_reciprocal).
MFG_HD bool in_range(double x) {
  const uint32_t e = (static_cast<uint32_t>(hi_word(x)) >> 20) & 0x7FFu;
  return e - (1023u - 800u) <= 1600u;
}

// x == 0 without an FP64 instruction (a comparison is one).
MFG_HD bool is_zero(double x) {
#ifdef __CUDA_ARCH__
  return ((__double2hiint(x) & 0x7FFFFFFF) | __double2loint(x)) == 0;
#else
  return x == 0.0;
#endif
}

MFG_HD uint64_t bits_of(double x) {
#ifdef __CUDA_ARCH__
  return static_cast<uint64_t>(__double_as_longlong(x));
#else
  uint64_t u;
  std::memcpy(&u, &x, 8);
  return u;
#endif
}

MFG_HD double from_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(static_cast<long long>(u));
#else
  double x;
  std::memcpy(&x, &u, 8);
  return x;
#endif
}

MFG_HD uint64_t mul_high(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return static_cast<uint64_t>((static_cast<unsigned __int128>(a) * b) >> 64);
#endif
}

// The 53-bit significand of a normal number, and the same with its leading bit
// at bit 63.
MFG_HD uint64_t significand(uint64_t u) {
  return (u & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
}
MFG_HD int32_t exponent_bits(uint64_t u) { return static_cast<int32_t>(u >> 52) & 0x7FF; }

// Reciprocal of a divisor for div_known(): floor(2^127 / D) for its
// significand D at bit 63 (2^64 - 1 for a power of two), or 0 when the divisor
// is outside 2^-100 .. 2^100 and its quotients need the general division.
// Set-up, on the device too.
//
// From the FP64 quotient, off by less than 2^12, and its exact remainder
// 2^127 - R D in two words (a 128-bit division takes ten times as long): the
// remainder over D corrects R to the last unit or the one beside it, and the
// loops below settle that.
MFG_HD uint64_t exact_reciprocal(double d) {
  if (!(d >= 0x1p-100 && d <= 0x1p100)) return 0;
  const uint64_t D = significand(bits_of(d)) << 11;
  if (D == 0x8000000000000000ull) return ~0ull;
  const double Df = static_cast<double>(D);  // exact: 53 bits
  uint64_t R = static_cast<uint64_t>(0x1p127 / Df);  // below 2^64 - 2^10: D is 2^63 + 2^11 or more
  uint64_t lo = 0 - R * D;
  int64_t hi = static_cast<int64_t>(0x8000000000000000ull - mul_high(R, D) - (R * D != 0));
  const double rest = static_cast<double>(hi) * 0x1p64 + static_cast<double>(lo);
  R += static_cast<uint64_t>(static_cast<int64_t>(floor(rest / Df)));
  lo = 0 - R * D;
  hi = static_cast<int64_t>(0x8000000000000000ull - mul_high(R, D) - (R * D != 0));
  for (; hi < 0; --R) {  // remainder below 0: D more
    lo += D;
    hi += lo < D;
  }
  for (; hi > 0 || lo >= D; ++R) {
    hi -= lo < D;
    lo -= D;
  }
  return R;
}

// x / d, correctly rounded, for in_range(x) and a positive normal d, from R:
// within (-kBelow, kAbove) of 2^127 / D, D the significand of d at bit 63.
//
// P = high(X R) is then X 2^63 / D less at most 1 + kBelow and more at most
// kAbove; doubled where X < D, so that its leading bit is bit 63, twice that.
// Bits 11 and up are the quotient's 53, and it is rounded by bit 10 unless
// the bits below are within that error of one half; there the sign of the
// exact remainder against the midpoint decides (a quotient is never halfway
// between two numbers).
template <int kBelow, int kAbove>
MFG_HD double div_recip(double x, double d, uint64_t R) {
  const uint64_t xb = bits_of(x), db = bits_of(d);
  uint64_t P = mul_high(significand(xb) << 11, R);
  const uint32_t n = static_cast<uint32_t>(P >> 63);
  P <<= 1u - n;
  const uint64_t c = P >> 11;
  uint32_t up = static_cast<uint32_t>(P >> 10) & 1u;
  constexpr uint32_t lo = 2 * (kBelow + 1), width = lo + 2 * kAbove;
  if ((static_cast<uint32_t>(P) & 0x7FFu) - (0x400u - lo) < width) {
    // 2^(s + 1) X - (2 c + 1) D > 0, X and D as 53-bit integers
    const uint64_t D = significand(db);
    const int64_t t = static_cast<int64_t>((significand(xb) << (54u - n)) - (2 * c + 1) * D);
    up = t > 0;
  }
  const int64_t e = exponent_bits(xb) - exponent_bits(db) + 1021 + static_cast<int32_t>(n);
  return from_bits((static_cast<uint64_t>(e) << 52) + c + up + (xb & 0x8000000000000000ull));
}

// x / d, correctly rounded, for R = exact_reciprocal(d) (not 0) and
// in_range(x).
MFG_HD double div_known(double x, double d, uint64_t R) { return div_recip<1, 0>(x, d, R); }

// Approximation of 1 / sqrt(u), 1 <= u < 4, with relative error below 2^-22.
MFG_HD float rsqrt_start(float u) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(u));
  return y;
#else
  return 1.0f / std::sqrt(u);
#endif
}

MFG_HD uint32_t float_bits(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  uint32_t u;
  std::memcpy(&u, &x, 4);
  return u;
#endif
}
MFG_HD float float_from_bits(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x;
  std::memcpy(&x, &u, 4);
  return x;
#endif
}

// l = sqrt(s), correctly rounded, for in_range(s) and s > 0, and R within
// (-3, 3) of 2^127 / L, L the significand of l at bit 63, for
// div_recip<3, 3>(). False when l is rounded up to a power of two: then R is
// not set (and callers take the general operations).
//
// s = u 2^(2k), 1 <= u < 4; g = sqrt(u), y = 1 / g. Y0 is y to 22 bits (scaled
// by 2^32), Y to 42 (2^64), Ga g to 41 (2^42, off by less than 3 units) and G,
// corrected by its exact remainder u - Ga^2 (below 2^46, scaled by 2^84), to 63
// (2^63, low by at most 1.1 units and high by less than 0.1). l is rounded as
// in div_recip().
//
// The start y0 approximates 1 / sqrt(root_operand(s)), u cut to 24 bits.
MFG_HD uint32_t root_odd(uint64_t sb) { return ~static_cast<uint32_t>(sb >> 52) & 1u; }
MFG_HD float root_operand(double s) {
  const uint64_t sb = bits_of(s);
  return float_from_bits(((127u + root_odd(sb)) << 23) |
                         (static_cast<uint32_t>(sb >> 29) & 0x7FFFFFu));
}
MFG_HD bool sqrt_recip(double s, float y0, double& l, uint64_t& R) {
  const uint64_t sb = bits_of(s);
  const uint32_t odd = root_odd(sb);                 // u >= 2
  const uint64_t U = significand(sb) << (10 + odd);  // u 2^62
  uint32_t yb = float_bits(y0);
  yb = yb < 0x3F7FFFFFu ? yb : 0x3F7FFFFFu;  // below 1, and no less than 1 / 2
  yb = yb > 0x3F000000u ? yb : 0x3F000000u;
  const uint32_t Y0 = (yb << 8) | 0x80000000u;
  // y (1 + e / 2), e = 1 - u y^2
  const int64_t e = static_cast<int64_t>(0x4000000000000000ull -
                                         mul_high(U, static_cast<uint64_t>(Y0) * Y0));
  const uint64_t Y =
      (static_cast<uint64_t>(Y0) << 32) +
      static_cast<uint64_t>((static_cast<int64_t>(Y0 >> 1) * static_cast<int32_t>(e >> 11)) >> 19);
  const uint64_t Ga = mul_high(U, Y) >> 20;
  const int64_t rest = static_cast<int64_t>((U << 22) - Ga * Ga);
  const uint64_t G =
      (Ga << 21) +
      static_cast<uint64_t>((static_cast<int64_t>(static_cast<int32_t>(rest >> 15)) *
                             static_cast<int32_t>(static_cast<uint32_t>(Y >> 32) >> 1)) >> 38);
  const uint64_t c = G >> 11;
  uint32_t up = static_cast<uint32_t>(G >> 10) & 1u;
  if ((static_cast<uint32_t>(G) & 0x7FFu) - 0x3FEu < 3u)  // u 2^104 > (c + 1/2)^2
    up = static_cast<int64_t>((U << 42) - c * c - c) > 0;
  const uint64_t m = c + up;
  const int64_t k = (exponent_bits(sb) + 1021 + static_cast<int32_t>(1u - odd)) >> 1;
  l = from_bits((static_cast<uint64_t>(k) << 52) + m);
  if (m >> 53) return false;
  // y (1 + e), e = 1 - l y
  const uint64_t L = m << 11;
  const int64_t el = static_cast<int64_t>(0x8000000000000000ull - mul_high(L, Y));
  R = Y + static_cast<uint64_t>((static_cast<int64_t>(Y >> 32) * el) >> 31);
  return true;
}

// f / l, correctly rounded, from R of sqrt_recip(); in_range(f).
MFG_HD double div_root(double f, double l, uint64_t R) { return div_recip<3, 3>(f, l, R); }

// a b, correctly rounded: the product of the significands, its last bit by
// the bits below and, in the one case in 2048 where those say exactly one
// half, by the part of the product below them. General operation where an
// operand or the product is not a normal number.
MFG_HD double mul_exact(double a, double b) {
  const uint64_t ab = bits_of(a), bb = bits_of(b);
  const uint32_t ea = static_cast<uint32_t>(ab >> 52) & 0x7FFu;
  const uint32_t eb = static_cast<uint32_t>(bb >> 52) & 0x7FFu;
  const uint64_t A = significand(ab) << 11, B = significand(bb) << 11;
  uint64_t P = mul_high(A, B);
  const uint32_t n = static_cast<uint32_t>(P >> 63);
  P <<= 1u - n;
  const uint64_t c = P >> 11;
  uint32_t up = static_cast<uint32_t>(P >> 10) & 1u;
  if ((static_cast<uint32_t>(P) & 0x7FFu) == 0x400u && A * B == 0)
    up = static_cast<uint32_t>(c) & 1u;  // halfway: to even
  const uint32_t e = ea + eb - 1024u + n;
  if (ea - 1u < 2046u && eb - 1u < 2046u && e < 2045u)
    return from_bits((static_cast<uint64_t>(e) << 52) + c + up +
                     ((ab ^ bb) & 0x8000000000000000ull));
#ifdef __CUDA_ARCH__
  // (not C++: the compiler would run the product ahead of the test)
  double r;
  asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
  return r;
#else
  return a * b;
#endif
}

}  // namespace mfg

#endif
