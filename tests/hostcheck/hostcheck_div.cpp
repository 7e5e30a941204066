// Host build of the division on the FP32 and integer pipes (csrc/ccd_div.h).
#include <cmath>
#include <cstdint>

#include "../../collisiondetection_gb300/csrc/ccd_div.h"

// Quotients with the reciprocal estimate `ulps` units in the last place off
// the FP32 quotient.
extern "C" void hc_div(const double *a, const double *b, int64_t n, int ulps, double *q) {
  for (int64_t i = 0; i < n; i++) {
    const uint64_t ua = ccd::bits_of(a[i]), ub = ccd::bits_of(b[i]);
    const float bh = ccd::float_of(0x3f800000u | (uint32_t)((ub >> 29) & 0x7fffffu));
    float y = 1.0f / bh;
    for (int k = 0; k < (ulps < 0 ? -ulps : ulps); k++) y = std::nextafterf(y, ulps > 0 ? 2.0f : 0.0f);
    q[i] = ccd::div_significands(ua, ub, bh, y);
  }
}
