// Host build of the sextics that wait (csrc/ccd_classify.h): rows whose
// distance sextic waits are decided from their side lists and, in full, from
// all their lists.
#include <cmath>
#include <cstdint>

#include "../../collisiondetection_gb300/csrc/ccd_classify.h"

namespace {

// out: 0 the sextic does not wait, 1 settled without it, 2 not.  hit: the
// decision from all lists.
template <class P>
void check(const double *x, double eta, uint8_t &out, uint8_t &hit) {
  constexpr int K = P::kSlots, kDist = ccd::cls::Row<P>::kDist;
  double dist[7];
  P::coeffs(x, eta, kDist, dist);
  const unsigned wait = ccd::cls::waits(dist);
  out = hit = 0;
  if (!(wait & ccd::cls::kWaits)) return;
  ccd::SpanList l[K];
  double t = 0.0;
  for (int k = 0; k < K; k++) {
    double op[7];
    uint8_t st = 0;
    P::coeffs(x, eta, k, op);
    l[k].clear();
    ccd::sign_spans(op, P::degree(k), l[k], P::want_pos(k), st);
  }
  out = ccd::cls::settled_without_sextic<K>(x, l, (wait & ccd::cls::kZeroAtStart) != 0) ? 1 : 2;
  if constexpr (K == 4) {
    hit = ccd::vf_combine(l[0], l[1], l[2], l[3], t);
  } else {
    ccd::SpanList cop, par;
    ccd::ee_split_parallel(x, l[0], cop, par);
    hit = ccd::ee_combine(cop, par, l[1], l[2], l[3], l[4], t);
  }
}

}  // namespace

extern "C" void hc_wait(int kind, int64_t n, const double *x, const double *eta, uint8_t *out, uint8_t *hit) {
  for (int64_t i = 0; i < n; i++) {
    if (kind == 0)
      check<ccd::VFPolys>(x + 24 * i, eta[i], out[i], hit[i]);
    else
      check<ccd::EEPolys>(x + 24 * i, eta[i], out[i], hit[i]);
  }
}

extern "C" void hc_waits(int64_t n, const double *op, uint8_t *out) {
  for (int64_t i = 0; i < n; i++) out[i] = (uint8_t)ccd::cls::waits(op + 7 * i);
}
