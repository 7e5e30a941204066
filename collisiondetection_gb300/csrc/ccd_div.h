// Correctly rounded binary64 division on the FP32 and integer pipes.
//
// GB300 issues one FP64 warp instruction per SM about every 19 cycles, and a
// division is some ten of them: half of the root solver's FP64 work, and 564
// cycles of every dependent chain through it.  The FP32 and integer pipes are
// otherwise idle there and issue 40 to 80 times as fast.
//
// The quotient of the significands is estimated in FP32: the leading 24 bits
// of a and b with an approximate reciprocal, then one correction from the FP32
// remainder with the trailing 29 bits, which leaves an error below 2^10 units
// in the last of 53 places.  The exact remainder of that estimate fits 64
// bits, so the integer pipe computes it modulo 2^64; its FP32 quotient by b
// gives the missing units, and a last comparison of the new remainder with
// b / 2 rounds to nearest (a quotient of two 53-bit significands is never
// half-way between two others).  Operands that are zero, subnormal, infinite
// or NaN, and quotients that might be, take the operator.
#pragma once

#include <string.h>

#include "ccd_common.h"

namespace ccd {

CCD_HD uint64_t bits_of(double x) {
  uint64_t u;
  memcpy(&u, &x, sizeof u);
  return u;
}
CCD_HD double double_of(uint64_t u) {
  double x;
  memcpy(&x, &u, sizeof x);
  return x;
}
CCD_HD float float_of(uint32_t u) {
  float x;
  memcpy(&x, &u, sizeof x);
  return x;
}

// a / b for normal a and b with a normal quotient; y: 1 / (b's leading 24 bits
// as a number in [1, 2)) to 2^-23.
CCD_HD double div_significands(uint64_t ua, uint64_t ub, float bh, float y) {
  const uint64_t kMant = (1ull << 52) - 1, kOne = 1ull << 52;
  const uint64_t A = (ua & kMant) | kOne, B = (ub & kMant) | kOne;
  const float ah = float_of(0x3f800000u | (uint32_t)((ua & kMant) >> 29));
  const float al = (float)(uint32_t)(ua & 0x1fffffffu) * 0x1p-52f;
  const float bl = (float)(uint32_t)(ub & 0x1fffffffu) * 0x1p-52f;
  float qh = ah * y;
  float rr = fmaf(-bh, qh, ah);
  rr = rr + al;
  rr = fmaf(-bl, qh, rr);
  float ql = rr * y;
  const bool less = A < B;  // quotient in (1/2, 1): one more place
  const float s = less ? 2.0f : 1.0f;
  qh *= s;
  ql *= s;
  uint64_t Q = ((uint64_t)(uint32_t)(qh * 0x1p30f) << 22) + (uint64_t)((int64_t)(int32_t)(ql * 0x1p48f) * 16);
  int64_t r = (int64_t)((A << (less ? 53 : 52)) - B * Q);
  const float e = (float)(int32_t)(r >> 32) * y * 0x1p-20f;
#if defined(__CUDA_ARCH__)
  const int32_t d = __float2int_rn(e);
#else
  const int32_t d = (int32_t)lrintf(e);
#endif
  Q += (uint64_t)(int64_t)d;
  r -= (int64_t)d * (int64_t)B;
  if (r + r > (int64_t)B)
    Q++;
  else if (-(r + r) > (int64_t)B)
    Q--;
  const int64_t e2 = (int64_t)((ua >> 52) & 0x7ff) - (int64_t)((ub >> 52) & 0x7ff) + 1022 - (less ? 1 : 0);
  return double_of(((ua ^ ub) & 0x8000000000000000ull) | (((uint64_t)e2 << 52) + Q));
}

// a / b, correctly rounded.
CCD_HD double exact_div(double a, double b) {
#if defined(__CUDA_ARCH__)
  const uint64_t ua = bits_of(a), ub = bits_of(b);
  const int ea = (int)((ua >> 52) & 0x7ff), eb = (int)((ub >> 52) & 0x7ff);
  // Exponents within 2^+-500 of 1 keep the quotient normal.
  if ((unsigned)(ea - 523) > 1000u || (unsigned)(eb - 523) > 1000u) return a / b;
  const float bh = float_of(0x3f800000u | (uint32_t)((ub >> 29) & 0x7fffffu));
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(bh));
  return div_significands(ua, ub, bh, y);
#else
  return a / b;
#endif
}

}  // namespace ccd
