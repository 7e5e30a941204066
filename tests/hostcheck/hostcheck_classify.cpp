// Host build of csrc/ccd_classify.h: every row that the FP32 stage passes on is
// decided twice, from all its interval lists and from the lists that the
// classification leaves to the root finder.
#include <cmath>
#include <cstdint>
#include <cstring>

#include "../../collisiondetection_gb300/csrc/ccd_classify.h"
#include "../../collisiondetection_gb300/csrc/ccd_cull32.h"

namespace {

template <class P>
bool combine(const double *x, const ccd::SpanList *l, double &t, bool &parallel) {
  parallel = false;
  if constexpr (P::kSlots == 4) {
    return ccd::vf_combine(l[0], l[1], l[2], l[3], t);
  } else {
    ccd::SpanList cop, par;
    ccd::ee_split_parallel(x, l[0], cop, par);
    parallel = par.n > 0;
    return ccd::ee_combine(cop, par, l[1], l[2], l[3], l[4], t);
  }
}

// out: 0 rejected by the FP32 stage, 1 decided by the classification, 2 some
// lists stand in, 3 the same but left to a second round (parallel edges), 4
// every list solved.  differs: the two decisions.
template <class P>
void check(const double *x, double eta, uint8_t &out, uint8_t &differs, int &jobs, int &solved) {
  constexpr int K = P::kSlots;
  out = differs = 0;
  jobs = solved = 0;
  if (K == 4 ? ccd::vf_rejects(x, eta) : ccd::ee_rejects(x, eta)) return;
  float w[64];
  bool bounded = true;
  ccd::SpanList full[K], part[K];
  bool queued[K];
  for (int k = 0; k < K; k++) {
    double op[7];
    uint8_t st = 0;
    P::coeffs(x, eta, k, op);
    bounded = ccd::cls::Row<P>::put(w, k, op) && bounded;
    double copy[7];
    std::memcpy(copy, op, sizeof copy);
    queued[k] = ccd::reduce_poly(copy, P::degree(k)) > 2;
    full[k].clear();
    ccd::sign_spans(op, P::degree(k), full[k], P::want_pos(k), st);
  }
  ccd::cls::Need need{false, (1u << K) - 1u, 0u};
  if (bounded) need = ccd::cls::decide<P>(w);
  double t0 = -1.0, t1 = -1.0;
  bool par;
  const bool h0 = combine<P>(x, full, t0, par);
  for (int k = 0; k < K; k++) {
    jobs += queued[k];
    solved += queued[k] && !need.miss && ((need.solve >> k) & 1u);
  }
  if (need.miss) {
    out = 1;
    differs = h0;
    return;
  }
  out = need.solve == (1u << K) - 1u ? 4 : 2;
  for (int k = 0; k < K; k++) {
    part[k] = full[k];
    if (!((need.solve >> k) & 1u)) ccd::cls::stand_in(need.near, part[k]);
  }
  const bool h1 = combine<P>(x, part, t1, par);
  if (out == 2 && par) {
    out = 3;
    return;
  }
  differs = h0 != h1 || (h0 && std::memcmp(&t0, &t1, sizeof t0) != 0);
}

}  // namespace

extern "C" void hc_classify(int kind, int64_t n, const double *x, const double *eta, uint8_t *out, uint8_t *differs,
                            int *jobs, int *solved) {
  for (int64_t i = 0; i < n; i++) {
    if (kind == 0)
      check<ccd::VFPolys>(x + 24 * i, eta[i], out[i], differs[i], jobs[i], solved[i]);
    else
      check<ccd::EEPolys>(x + 24 * i, eta[i], out[i], differs[i], jobs[i], solved[i]);
  }
}
