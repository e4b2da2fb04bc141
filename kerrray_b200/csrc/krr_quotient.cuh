// Correctly rounded FP64 quotients without branches, several to one denominator: the reference
// order's divisions.
//
// A compiled FP64 division tests its operands and branches to a slow path, so the 17 divisions
// of a metric evaluation (by 7 different denominators) and the 6 of an error norm ran one after
// the other, about 100 cycles each: the reference-order kernels waited on them for most of
// their time (at 64^2, 4.9 cycles per instruction with one warp per scheduler, 3.0 of them the
// fixed latency of a dependent instruction).  Here a denominator's reciprocal is shared, nothing
// branches, and the quotients of one evaluation overlap.  The values are those of IEEE division
// bit for bit (for b as below and no overflow or underflow on the way; the callers check):
//
//   y   1/b by two Newton steps from the hardware reciprocal.  That is within a relative 2^-19 of
//       1/b (2^-19.9 over all 2^20 upper words of a fraction), so y before its last rounding is
//       within 2^-76 and |y - 1/b| <= (1/2 + 2^-23) ulp(y);
//   q0  within (1/2 + 2^-51) ulp of a/b: a (y + lo) with lo = (1 - b y) y, or RN(a y) corrected
//       once by its residual;
//   r   a - b q0, exact (a multiple of ulp(b) ulp(q0), at most 2^53 of them);
//   q   RN(q0 + r y): before its rounding it differs from a/b by |a/b - q0| |1 - b y|.
//
// Scale a and b to [1, 2) and let u be the quotient's ulp.  Every rounding boundary m of the
// quotient is a multiple of u/2, so a - b m, which is not zero, is at least ulp(b) u / 2 and a/b
// lies u / (2^53 b) or more from m.  The difference above is at most (1/2 + 2^-51) u times
// b (1/2 + 2^-23) 2^-53 (ulp(y) = 2^-53 for 1/b in (1/2, 1]).  It is the smaller of the two, and q
// therefore RN(a/b), if b^2 < 4 (1 - 2^-22 - 2^-49): for every b whose fraction does not begin with
// 20 ones, b < 2 - 2^-20 and b^2 < 4 (1 - 2^-20 + 2^-42).  A zero numerator gives +0 whatever its
// sign.  The last step, correcting a nearly correct quotient by its exact residual, is Markstein's
// (IBM J. Res. Dev. 34 (1990) 111).
#pragma once

#include <cuda_runtime.h>

namespace krr {

struct Recip {
  double b, y, lo, e;  // the denominator, 1/b, (1 - b y) y, 1 - b y
};

__device__ __forceinline__ double recip_nearest(double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  y = fma(fma(-b, y, 1.0), y, y);
  return fma(fma(-b, y, 1.0), y, y);
}

__device__ __forceinline__ Recip recip(double b) {
  Recip d;
  d.b = b;
  d.y = recip_nearest(b);
  d.e = fma(-b, d.y, 1.0);
  d.lo = d.e * d.y;
  return d;
}

// a / b with the shared reciprocal: four operations.
__device__ __forceinline__ double quotient(double a, const Recip& d) {
  const double q0 = fma(a, d.y, a * d.lo);
  return fma(fma(-d.b, q0, a), d.y, q0);
}

// 1 / b: q0 = y.
__device__ __forceinline__ double quotient_one(const Recip& d) { return fma(d.e, d.y, d.y); }

// a / b for a denominator of its own: y, then two residual corrections.
__device__ __forceinline__ double quotient(double a, double b) {
  const double y = recip_nearest(b);
  const double q0 = a * y;
  const double q1 = fma(fma(-b, q0, a), y, q0);
  return fma(fma(-b, q1, a), y, q1);
}

// The test on a denominator's fraction, for several denominators by minima: 0 where the first 20
// of its 52 bits are all ones.
__device__ __forceinline__ unsigned fraction_gap(double b) {
  return (~(unsigned)__double2hiint(b)) & 0x000fffffu;
}

// Whether |x| lies in [2^LO, 2^HI) (false for NaN and infinities).
template <int LO, int HI>
__device__ __forceinline__ bool within(double x) {
  return ((unsigned)__double2hiint(x) & 0x7fffffffu) - ((unsigned)(1023 + LO) << 20) < ((unsigned)(HI - LO) << 20);
}

// a / b for any operands: branch-free in the range where that holds (|b| in [2^-400, 2^400], a 0 or
// |a| in [2^-900, 2^900), which leaves |a / b| normal or its residual exact), else by IEEE division
// out of line.
static __device__ __noinline__ double quotient_ieee(double a, double b) { return a / b; }

__device__ __forceinline__ double quotient_any(double a, double b) {
  const unsigned ha = (unsigned)__double2hiint(a) & 0x7fffffffu, hb = (unsigned)__double2hiint(b) & 0x7fffffffu;
  const double q = quotient(a, b);
  const bool ok = hb - 0x26f00000u < 0x32000000u && fraction_gap(b) != 0u &&
                  (a == 0.0 || ha - 0x20b00000u < 0x3e800000u);
  return ok ? q : quotient_ieee(a, b);
}

}  // namespace krr
