// hmn_div.cuh -- correctly rounded FP64 division and square root without
// branches, for quotients that share a denominator.
//
// Division: P. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", IBM J. Res. Develop. 34(1), 1990; J.-M. Muller
// et al., "Handbook of Floating-Point Arithmetic" (2nd ed., 2018), section
// 4.7; N. Brisebarre, J.-M. Muller, S. K. Raina, "Accelerating correctly
// rounded floating-point division when the divisor is known in advance",
// IEEE Trans. Comput. 53(8), 2004.
//
//  * reciprocal: from an approximation y0 of 1/b with e = 1 - b y0, the
//    third-order step y1 = y0 + y0 (e + e^2) leaves a relative error of |e|^3
//    and one rounding, so y1 is within one ulp of 1/b; one Newton-Raphson
//    step more gives RN(1/b) exactly, unless the significand of b is 1.11...1
//    (Markstein's theorem for the reciprocal);
//  * quotient: with y = RN(1/b), q0 = RN(a y), r = RN(a - b q0), the quotient
//    is q = RN(q0 + r y): one multiplication and two FMAs.  Why one
//    correction is enough: scale a, b to [1, 2).  (i) a >= b: q0 is within
//    one ulp u of a/b, r is exact, and the only rounding boundaries in reach
//    are q0 +- u/2.  Write r = b u/2 + k w with w the last place of r and k a
//    whole number, never 0 (a/b is no midpoint).  With b y = 1 + eps, |eps| <=
//    b 2^-54, r y - u/2 = (u/2) eps + k w y; the second term is the larger
//    one because b^2 < 4.  (ii) a < b: q0 is within (1 + a)/2 ulp, below 1.5;
//    for boundaries at q0 +- u/2 as before; to pass q0 +- 3u/2 wrongly, a
//    would have to lie within a few last places of 2, and then so does b, a/b
//    lies next to a floating-point number and no boundary is near.
//
// Square root: third-order iteration from y0 ~ 1/sqrt(x) with t = RN(x y0),
// e = 1 - t y0, c = e/2 + 3 e^2/8: g = t + t c is within 0.75 ulp of s =
// sqrt(x), h = y0/2 + c y0/2 has a relative error below 1.25 2^-53, and RN(g
// + h (x - g^2)) is RN(s) (Handbook, section 4.8).  Why: scale x to [1, 4).
// g + h (x - g^2) = s - (s - g)^2 / (2 s) + (s - g) eps, and a midpoint m
// next to s satisfies x - m^2 = k 2^-106 with k = 7 (mod 8), since the square
// of an odd number is 1 (mod 8): where k is not -1 the distance to m exceeds
// the error; k = -1 holds only for x = 1 + 2^-52 and x = 4 - 2^-51, which the
// test of these operations runs over all exponents.
//
// The theorems assume that no intermediate overflows or underflows.  The
// operations check the operands' exponents instead of branching: a
// denominator outside [2^-500, 2^500], a nonzero numerator outside that range
// in magnitude, a radicand outside it (zero included) and a denominator with
// an all-ones significand set `bad`, and the caller then recomputes with IEEE
// operations.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace hmn {

// |x| in [2^-500, 2^501): biased exponent in [523, 1523].  The high word
// shifted left by one drops the sign and puts the exponent in bits 21..31,
// so the test is one shift-add and one unsigned compare.
__device__ __forceinline__ bool fin_range(double x) {
  const unsigned t = (unsigned)__double2hiint(x) << 1;
  return t - (523u << 21) < (1001u << 21);
}

// x in [2^LO, 2^HI) and positive (a sign bit makes the difference large)
template <int LO = -500, int HI = 501>
__device__ __forceinline__ bool pos_range(double x) {
  return (unsigned)__double2hiint(x) - ((unsigned)(1023 + LO) << 20) < ((unsigned)(HI - LO) << 20);
}

// |x| below 2^HI (infinities and NaN are not)
template <int HI>
__device__ __forceinline__ bool below(double x) {
  return ((unsigned)__double2hiint(x) & 0x7fffffffu) < ((unsigned)(1023 + HI) << 20);
}

__device__ __forceinline__ bool is_zero(double x) {
  return (((unsigned)__double2hiint(x) & 0x7fffffffu) | (unsigned)__double2loint(x)) == 0u;
}

// all-ones significand: the low word and the 20 significand bits of the high
// word are all ones
__device__ __forceinline__ bool ones_significand(double b) {
  return (((unsigned)__double2hiint(b) | 0xfff00000u) & (unsigned)__double2loint(b)) == 0xffffffffu;
}

// approximate reciprocal and reciprocal square root: the largest relative
// error over all high words is 2^-19.9 (measured), so the cube of twice that
// leaves the third-order steps below 0.03 ulp off before their rounding
__device__ __forceinline__ double rcp_approx(double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  return y;
}
__device__ __forceinline__ double rsqrt_approx(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}

// 1/b within about one ulp, without branches (two Newton-Raphson steps from
// the approximation); for the mixed-precision form, which is not bound to
// IEEE quotients.  A zero b gives NaN where IEEE gives infinity.
__device__ __forceinline__ double rcp_nr(double b) {
  double y = rcp_approx(b);
  double e = __fma_rn(-b, y, 1.0);
  y = __fma_rn(y, e, y);
  e = __fma_rn(-b, y, 1.0);
  return __fma_rn(y, e, y);
}

// RN(1/b) of a b that the caller has checked
__device__ __forceinline__ double recip_core(double b) {
  double y = rcp_approx(b);
  double e = __fma_rn(-b, y, 1.0);
  y = __fma_rn(y, __fma_rn(e, e, e), y);  // within one ulp of 1/b
  e = __fma_rn(-b, y, 1.0);
  return __fma_rn(y, e, y);
}

// RN(1/b) of either sign; sets bad where b is out of range or has an all-ones
// significand.  (The kernels pair div_rn below with reciprocals formed on the
// host; tests/div_check.cu checks it with these.)
__device__ __forceinline__ double recip_rn(double b, bool& bad) {
  bad = bad || !fin_range(b) || ones_significand(b);
  return recip_core(b);
}

// RN(a/b) from y = RN(1/b); sets bad where a is out of range (zero excepted,
// which is exact and keeps its sign)
__device__ __forceinline__ double div_rn(double a, double b, double y, bool& bad) {
  const bool zero = is_zero(a);
  bad = bad || !(fin_range(a) || zero);
  const double q0 = a * y;
  const double r = __fma_rn(-b, q0, a);
  const double q = __fma_rn(r, y, q0);
  return zero ? q0 : q;
}

// The same for a denominator that has to be positive: sets bad where b is not.
__device__ __forceinline__ double recip_pos(double b, bool& bad) {
  bad = bad | !pos_range(b) | ones_significand(b);
  return recip_core(b);
}

// RN(a/b), b positive, y = RN(1/b).  The remainder is formed with the other
// sign, b q0 - a: it is +0 where the quotient is exact, its product with -y
// is then -0, and adding -0 keeps q0 and the sign of a zero quotient, so no
// select is needed.
__device__ __forceinline__ double div_pos(double a, double b, double y, bool& bad) {
  bad = bad | !(fin_range(a) | is_zero(a));
  const double q0 = a * y;
  const double r = __fma_rn(b, q0, -a);
  return __fma_rn(-r, y, q0);
}

// RN(sqrt(x)); sets bad where x is not in the positive range
__device__ __forceinline__ double sqrt_pos(double x, bool& bad) {
  bad = bad | !pos_range(x);
  const double y = rsqrt_approx(x), h0 = 0.5 * y;
  const double t = x * y;
  const double e = __fma_rn(-t, y, 1.0);
  const double c = e * __fma_rn(0.375, e, 0.5);
  const double g = __fma_rn(t, c, t), h = __fma_rn(h0, c, h0);
  return __fma_rn(h, __fma_rn(-g, g, x), g);
}

// Division policy of hmn_math.cuh with the operations above, for positive
// denominators: `bad` records whether any result since construction may
// differ from the IEEE operation, in which case the caller recomputes the
// whole expression with PlainDiv.
//
// Measured against quotients with two corrections and selects for the sign of
// a zero, reciprocals with one more FMA and CUDA's sqrt, whose slow path is a
// branch (the stage is bound by dependent FP64 instructions): march stage at
// 256^3 8.13 -> 7.10 ms, 97x75x62 box 17.3 -> 15.3 ms for 16 steps, 48 KH
// boxes 76.5 -> 67.6 ms for 16 steps, a tube's step chain 6 % shorter.
struct FastDiv {
  static constexpr bool flags = true;  // results may be refused
  bool bad = false;
  // what the hydrodynamic flux asks of its operands beyond the above
  template <int LO, int HI>
  __device__ __forceinline__ void need_pos(double x) { bad = bad | !pos_range<LO, HI>(x); }
  template <int HI>
  __device__ __forceinline__ void need_below(double x) { bad = bad | !below<HI>(x); }
  __device__ __forceinline__ double rec(double b) { return recip_pos(b, bad); }
  __device__ __forceinline__ double div(double a, double b, double y) { return div_pos(a, b, y, bad); }
  __device__ __forceinline__ double root(double x) { return sqrt_pos(x, bad); }
};

}  // namespace hmn
