// Correctly rounded FP64 quotients and square roots for the plain FP64
// kernels, in fewer FP64 instructions than the general operations.
//
// GB300 executes FP64 at 2 lanes per clock and SM, so an FP64 instruction
// takes the pipe as long as 64 issue slots; the FP64 kernels are bound by
// the number of FP64 instructions. Two methods cut it without changing a bit:
//  - a quotient by a divisor that does not change (node mass, reference
//    length) with the divisor's correctly rounded reciprocal at hand: one
//    product, its exact residual by FMA and one correction (P. Markstein,
//    "Computation of elementary functions on the IBM RISC System/6000
//    processor", IBM J. Res. Dev. 34, 1990; Brisebarre, Muller, Raina,
//    "Accelerating correctly rounded floating-point division when the
//    divisor is known in advance", IEEE Trans. Comp. 53, 2004);
//  - a square root together with the reciprocal of the result, by coupled
//    Newton (Goldschmidt) iterations on g = sqrt(s) and h = 1 / (2 sqrt(s))
//    from an approximate reciprocal square root, the last two steps of g
//    with the exact residual s - g^2 (same paper, and Cornea, Harrison,
//    Tang, "Scientific Computing on Itanium-based Systems", 2002).
// Both assume that nothing over- or underflows on the way; in_range() tests
// that, and callers take the general operations outside it. The functions
// compile for the host too, where tests compare them with the general
// operations on operands chosen to lie next to rounding boundaries.
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

MFG_HD double fma64(double a, double b, double c) {
#ifdef __CUDA_ARCH__
  return __fma_rn(a, b, c);
#else
  return std::fma(a, b, c);
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

// The reciprocal that div_known() takes, or 0 when the divisor is outside
// 2^-100 .. 2^100 and its quotients need the general division. Host set-up.
inline double exact_reciprocal(double d) {
  return d >= std::ldexp(1.0, -100) && d <= std::ldexp(1.0, 100) ? 1.0 / d : 0.0;
}

// x / d, correctly rounded, for rd = RN(1 / d) (not 0) and in_range(x); a
// zero x gives a zero. 3 FP64 instructions.
MFG_HD double div_known(double x, double d, double rd) {
  const double q = x * rd;
  const double r = fma64(-q, d, x);
  return fma64(r, rd, q);
}

// x * 2^k for a normal x and a normal result, without an FP64 instruction.
template <int k>
MFG_HD double scale_exponent(double x) {
#ifdef __CUDA_ARCH__
  return __hiloint2double(__double2hiint(x) + k * (1 << 20), __double2loint(x));
#else
  return std::ldexp(x, k);
#endif
}

// l = sqrt(s) and y = 1 / l, both correctly rounded, from an approximation y0
// of 1 / sqrt(s) with relative error below 2^-19; in_range(s). The first
// three FMAs leave g = sqrt(s) and h = 1 / (2 sqrt(s)) with relative errors
// below 2^-37, the next two round g (its error far below an ulp), the next
// two bring y to about an ulp; then g is corrected by its exact residual, the
// correction off by no more than about 2^-53 of an ulp, and y by its own. The
// one exception is y for an l whose significand is all ones (see all_ones).
// 12 FP64 instructions.
MFG_HD void sqrt_recip(double s, double y0, double& l, double& y) {
  double g = s * y0;
  double h = scale_exponent<-1>(y0);
  const double r = fma64(-h, g, 0.5);
  g = fma64(g, r, g);
  h = fma64(h, r, h);
  g = fma64(fma64(-g, g, s), h, g);
  y = scale_exponent<1>(h);
  y = fma64(y, fma64(-y, g, 1.0), y);
  l = fma64(fma64(-g, g, s), scale_exponent<-1>(y), g);
  y = fma64(y, fma64(-y, l, 1.0), y);
}

// Possibly a number whose significand is all ones, for which the last step of
// a reciprocal is known to fail (Markstein): the low word says enough.
MFG_HD bool all_ones(double x) {
#ifdef __CUDA_ARCH__
  return __double2loint(x) == -1;
#else
  uint64_t u;
  std::memcpy(&u, &x, 8);
  return static_cast<uint32_t>(u) == 0xFFFFFFFFu;
#endif
}

#ifdef __CUDACC__
// Approximate reciprocal square root, the start of sqrt_recip().
__device__ __forceinline__ double rsqrt_start(double s) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
  return y;
}
#endif

}  // namespace mfg

#endif
