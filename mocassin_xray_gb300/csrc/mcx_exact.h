/* mcx_exact.h - FP64 operations done on the bits or by a known reciprocal, for the
 * device (GB300 does two FP64 operations a cycle and SM) and, for their tests, the host.
 */
#ifndef MCX_EXACT_H
#define MCX_EXACT_H

#include "mcx_fmath.h"

#if !defined(__CUDA_ARCH__)
#include <math.h>
#endif

/* the upper and lower half of a double */
MCX_FM_FN int mcx_hi(double x) {
#if defined(__CUDA_ARCH__)
  return __double2hiint(x);
#else
  return (int)(uint32_t)(mcx_fm_bits(x) >> 32);
#endif
}
MCX_FM_FN int mcx_lo(double x) {
#if defined(__CUDA_ARCH__)
  return __double2loint(x);
#else
  return (int)(uint32_t)mcx_fm_bits(x);
#endif
}
MCX_FM_FN double mcx_fma(double a, double b, double c) {
#if defined(__CUDA_ARCH__)
  return __fma_rn(a, b, c);
#else
  return fma(a, b, c);
#endif
}

/* Whether old + v is exact, seen from the bits of old >= 0 and of an FP32 value
 * v > 0: both are multiples of the last place of a sum one binade above the larger.
 * Integer work instead of FP64 additions and compares (which kept the transport's
 * FP64 pipe 47 % busy).  False where it cannot be seen. */
MCX_FM_FN bool exactSum(double old, double v) {
  const unsigned long long bo = (unsigned long long)mcx_fm_bits(old);
  const int eo = (int)(bo >> 52), ev = (int)((unsigned)mcx_hi(v) >> 20);
  if ((unsigned)(ev - 1) >= 0x7feu) return false;            // v infinite, NaN, 0 or subnormal
  if ((unsigned)(eo - 1) >= 0x7feu) return bo == 0ull;       // old the same, or negative: 0 + v is v
  if (eo > ev) return eo - ev <= 28 && (bo & 1ull) == 0ull;             // v's last place is at least 2^(ev - 23)
  const int sh = ev + 1 - eo;
  return sh <= 52 && (bo << (64 - sh)) == 0ull;
}

/* Markstein's division (P. W. Markstein, IBM J. Res. Dev. 34 (1990) 111): a / d
 * correctly rounded from r, the correctly rounded 1 / d, in five operations.
 * The first correction makes the quotient faithful, so that the second's
 * remainder is exact and its sum rounds to a / d.  Exponents within 2^450 keep
 * every intermediate normal; others, and zeros of d, infinities and NaN, take
 * the division itself. */
MCX_FM_FN double eqDivide(double a, double d, double r) {
  const int ha = mcx_hi(a), hd = mcx_hi(d);
  const unsigned ea = ((unsigned)ha >> 20) & 0x7ffu, ed = ((unsigned)hd >> 20) & 0x7ffu;
  if (ed - 573u < 900u) {
    if (ea - 573u < 900u) {
      double q = a * r;
      q = mcx_fma(mcx_fma(-q, d, a), r, q);
      return mcx_fma(mcx_fma(-q, d, a), r, q);
    }
    if (((ha & 0x7fffffff) | mcx_lo(a)) == 0) return a * r;   // a signed zero
  }
  return a / d;
}

#endif
