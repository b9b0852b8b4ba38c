// gb_fx64.cuh -- fixed-point arithmetic of the FP64 hopping term (host and device).
//
// GB300 issues FP64 at 2 lanes per clock and SM, and 32 x 32 -> 64 bit integer multiply-adds
// at 61 (both measured): one real product of the SU(3) multiplication as three integer
// multiply-adds costs about a tenth of the double-precision fused multiply-add.  A number is
// a signed 64-bit integer in units that its site (spinors) or its operator (links) fixes,
// kept as two signed 32-bit limbs, v = hi 2^32 + lo.
//
//   spinor  |v| < 2^60: units of 2^-60 of the site's own power of two, the smallest above its
//           largest |re|, |im| (a double keeps 53 bits below itself, a site at least 59 below
//           its largest component); the two-spinors and their sums over legs follow exactly
//   link    round(u 2^(61 - k)), k the operator's exponent, chosen so that the absolute values
//           of a row (6 reals) sum to at most 1.5 2^k: -U/2 with U in SU(3) has k = 0 and
//           a resolution of 2^-61
//   dot     hh = sum hi hi and mid = sum (hi lo + lo hi), the lo lo products (below 2^-60 of the
//           largest value) dropped; the result hh + mid / 2^32 is rounded once, to 2^-58 of
//           the largest term
//
// No sum overflows: with sum |u| <= 1.5 2^k, sum |hi_u| 2^31 <= 1.5 2^60 (+ 3 2^31) and
// sum |lo_u hi_h| <= 6 2^31 2^29 = 6 2^60, so |mid| < 7.6 2^60 < 2^63; |hh| <= 1.5 2^58 and
// eight legs stay below 2^62.
//
// The error is a fixed part of the unit, where FP64's is one of each sum's own terms.  With terms of the unit's
// size it is below the FP64 kernel's (tests/cpp/test_fx64.cpp measures both against long double): sums are
// exact, where FP64 rounds each of them at 2^-53.  A sum of terms far below the unit would keep fewer bits than a
// double: kernels find those (fx_site_exponent, deriv_fx_kernel in gb_dhop_fx.cu) and take them in FP64.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define GB_HD __host__ __device__ __forceinline__
#else
#define GB_HD inline
#endif

namespace gb {
namespace fx {

// Biased binary exponents of the largest component of the sites that the fixed-point path
// takes.  A site of zeros has exponent 0; any other outside (also infinities and NaN) is
// marked kBad, and the outputs next to it go to the FP64 arithmetic.
constexpr int kEmin = 100, kEmax = 1900, kBad = 4095;

// (hi, lo) limbs of a value
GB_HD void split(long long v, int& hi, int& lo) {
  lo = int(uint32_t(uint64_t(v)));
  hi = int(uint32_t(uint64_t(v) >> 32) + (uint32_t(lo) >> 31));
}

// limbs of a link value, with lo > -2^31 so that both limbs can be negated
GB_HD void split_link(long long v, int& hi, int& lo) {
  if (uint32_t(uint64_t(v)) == 0x80000000u) v += 1;
  split(v, hi, lo);
}

// The double with the words (whi, wlo) as an integer in units of 2^(E - 1023 - 59): a value
// of exponent E lands in [2^59, 2^60).  E is at least the value's exponent and at least kEmin;
// zeros (and subnormals, far below the unit) give 0.
GB_HD long long from_words(uint32_t whi, uint32_t wlo, int E) {
  const uint32_t a = whi & 0x7fffffffu;
  const uint32_t sh = uint32_t(E + 4 - int(a >> 20));
  const uint64_t w = (uint64_t((a << 11) | (wlo >> 21) | 0x80000000u) << 32) | uint64_t(wlo << 11);
  uint64_t m;
#ifdef __CUDA_ARCH__
  asm("shr.u64 %0, %1, %2;" : "=l"(m) : "l"(w), "r"(sh));  // shifts of 64 and more give 0
#else
  m = sh < 64 ? w >> sh : 0;
#endif
  const long long s = (long long)(int(whi) >> 31);
  return (long long)(m ^ uint64_t(s)) - s;
}

// a b + c on signed 32-bit factors: one integer multiply-add, for factors that the compiler
// takes as 32-bit numbers (see opaque).  The sum wraps as unsigned: mid starts at 2^63.
GB_HD long long mad(int a, int b, long long c) {
  return (long long)(uint64_t(c) + uint64_t((long long)a * (long long)b));
}

// Hides where a limb comes from.  The compiler otherwise sees the shifts of the 64-bit value it
// was cut from, widens the products to 64 x 64 bits and emits three times the instructions.
GB_HD void opaque(int& limb) {
#ifdef __CUDA_ARCH__
  asm("" : "+r"(limb));
#else
  (void)limb;
#endif
}

// A dot starts from (kStartHh, kStartMid): mid carries 2^63 so that its upper word is read as
// unsigned, and 2^31 to round hh + mid / 2^32 to nearest; hh gives the 2^31 back.
constexpr long long kStartHh = -0x80000000ll;
constexpr long long kStartMid = (long long)0x8000000080000000ull;
GB_HD long long join(long long hh, long long mid) { return hh + (long long)(uint64_t(mid) >> 32); }

// the exponent (of 2) of a result's unit, for spinor exponent E and link exponent k
GB_HD int result_exponent(int E, int k) { return E - 1023 - 56 + k; }

}  // namespace fx
}  // namespace gb
