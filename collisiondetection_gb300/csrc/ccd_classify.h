// Which polynomials of a vertex-face or edge-edge row have to be solved.
//
// The reference's decision (src/CTCD.cpp:310-410, 477-507) depends on its
// interval lists only through the times they share: spans of one list that
// touch act as one span, spans that overlap pairwise have a common point, and
// the time reported is the least point of the common set.  So a list is needed
// only near times at which every other list may be present.
//
// [0, 1] is cut into 256 cells and each polynomial's sign on a cell is bounded
// in FP32, from the FP64 coefficients that the reference itself forms (scaled
// to sum|c| = 1): its values at the cell's ends, less h^2/8 times a bound of
// |p''| (the Bernstein coefficients of p'') and the evaluation's rounding.
//
//   * a cell is empty when some polynomial has the wrong sign all over it by
//     more than kMargin: the spans of a list end at the polynomial's roots and
//     hold the wanted sign at their midpoints, so the list has no part there;
//   * a row whose cells are all empty misses, and nothing of it is solved;
//   * a "side" polynomial (all but the distance sextic) that has the wanted
//     sign by kMargin on every cell that is not empty and on its neighbours
//     covers all of them: those cells stand for its list.
//
// The loops over a lane's cells stay rolled: a small batch's build kernel is
// bound by fetching its instructions once.
//
// What is left for the root finder is mostly the distance sextic of the rows
// that collide.  The times reported stay the root finder's own, bit for bit:
// an end of a list that stands in lies four cells from any time at which the
// lists can meet.
//
// The margin against the root finder's accuracy: its roots are those of a
// polynomial within some hundred ulps of the given one, so a sign held by 1e-5
// of the coefficients' sum does not change.  What it does badly are sextics
// (nearly squares of the coplanarity cubic, whose simple roots they double)
// with a double root r beside a double root near -r: those came out up to 5e-3
// off where the moduli agreed to 1%, and at most 1.5e-3 elsewhere, |p| < 1e-7.
// A row is left to the solver when its sextic is below kMirror on the mirror
// image of a cell on which it is below kMargin (from the fifth cell on: a
// contact earlier than that has its mirror image among the start's cells).  On
// the host (tests/test_classify_host.py and test_classify_edges_host.py draw
// the same families), 137 M rows of twelve families -- random, integer
// lattices, coplanar, parallel, tangential, flat sheets, scales from 1e-6 to
// 1e4, mirrored roots from t = 5e-5 on -- gave no row that the full solve
// decides otherwise, and no contact time that differs in a bit.
#pragma once

#include <string.h>

#include "ccd_ctcd64.h"

namespace ccd {
namespace cls {

constexpr int kLanes = 32;           // a warp's lanes take the cells of one row,
constexpr int kPer = 8;              // eight consecutive ones each
constexpr float kCell = 1.0f / (kLanes * kPer);
constexpr float kMargin = 1e-5f;
constexpr float kMirror = 1e-4f;
constexpr float kRound = 1.5e-6f;    // coefficients and Horner steps in FP32, sum|c| = 1
// Coefficients further apart than this are left to the solver: with roots 30
// orders of magnitude apart it can lose one and report a span without the
// wanted sign (1 in 10^6 rows with coordinates between 1e-20 and 1e20; none in
// 7 million with this bound).
constexpr float kLeast = 1e-30f;
constexpr int kRuns = 3;             // runs of non-empty cells kept; more are left to the solver

// FP32 coefficients (ascending powers, sum|c| = 1) of the degree-N polynomial
// op (reference order, highest power first), then the error bound of a cell on
// [0, 1] and that of one on [-1, 0].  False when op is not finite or vanishes.
template <int N>
CCD_NOINLINE bool take(const double *op, float *p) {
  double m = 0.0;
CCD_UNROLL
  for (int i = 0; i <= N; i++) m = smax(m, fabs(op[i]));
  if (!(m > 1e-200) || !(m < 1e200)) return false;
  // the power of two that brings m into [1, 2)
  uint64_t bits;
  memcpy(&bits, &m, sizeof bits);
  bits = (2046ull - (bits >> 52)) << 52;
  double scale;
  memcpy(&scale, &bits, sizeof scale);
  float a[N + 1], s = 0.0f;
  bool even = true;
CCD_UNROLL
  for (int i = 0; i <= N; i++) {
    a[i] = (float)(op[N - i] * scale);
    even = even && (op[N - i] == 0.0 || fabsf(a[i]) > kLeast);
    s += fabsf(a[i]);
  }
  const float r = 1.0f / s;
  float d[N - 1], sum = 0.0f, most = 0.0f;
CCD_UNROLL
  for (int i = 0; i <= N; i++) {
    a[i] *= r;
    p[i] = a[i];
    if (i >= 2) {
      d[i - 2] = (float)(i * (i - 1)) * a[i];
      sum += fabsf(d[i - 2]);
    }
  }
CCD_UNROLL
  for (int j = 0; j <= N - 2; j++) {
    float v = 0.0f, c = 1.0f;  // C(j, i) / C(N - 2, i)
CCD_UNROLL
    for (int i = 0; i <= j; i++) {
      v += c * d[i];
      if (i < j) c = c * ((float)(j - i) / (float)(N - 2 - i));
    }
    most = fmaxf(most, fabsf(v));
  }
  const float bend = kCell * kCell * 0.13f;  // > h^2 / 8
  p[N + 1] = bend * most + kRound;
  p[N + 2] = bend * sum + kRound;
  return even && s == s;
}

template <int N>
CCD_HD float at(const float *p, float t) {
  float v = p[N];
CCD_UNROLL
  for (int i = N - 1; i >= 0; i--) v = fmaf(v, t, p[i]);
  return v;
}

// A row's polynomials: the distance sextic, then the sides.
template <class Polys>
struct Row {
  static constexpr int K = Polys::kSlots;
  static constexpr int kDist = K == 4 ? 3 : 0;
  static constexpr int NS = K == 4 ? 3 : 4;  // degree of the sides
  static constexpr int kSides = K - 1;
  static constexpr int kWords = 9 + kSides * (NS + 3);
  static constexpr unsigned kAll = (1u << K) - 1u;
  static CCD_HD int slot_of(int side) { return K == 4 ? side : side + 1; }

  // Takes slot k's polynomial into the row's words w; false when it cannot be
  // bounded (the row is left to the solver).
  static CCD_HD bool put(float *w, int k, const double *op) {
    if (op[0] == 0.0) return false;
    if (k == kDist) return take<6>(op, w);
    return take<NS>(op, w + 9 + (K == 4 ? k : k - 1) * (NS + 3));
  }

  // Cells of one lane (bit i: cell 8 * lane + i) on which the sextic may be
  // <= kMargin; mirrored: on the mirror image of one of them, four cells or
  // more from the start, it may be <= kMirror.
  static CCD_HD unsigned near_contact(const float *w, int lane, bool &mirrored) {
    const float t0 = (float)(lane * kPer) * kCell;
    unsigned open = 0;
    float prev = at<6>(w, t0);
CCD_ROLLED
    for (int i = 0; i < kPer; i++) {
      const float next = at<6>(w, t0 + (float)(i + 1) * kCell);
      if (!(fminf(prev, next) - w[7] > kMargin)) open |= 1u << i;
      prev = next;
    }
    mirrored = false;
    const unsigned test = lane == 0 ? open & 0xf0u : open;
    if (test) {
      prev = at<6>(w, -t0);
CCD_ROLLED
      for (int i = 0; i < kPer; i++) {
        const float next = at<6>(w, -(t0 + (float)(i + 1) * kCell));
        if (((test >> i) & 1u) && !(fminf(prev, next) - w[8] > kMirror)) mirrored = true;
        prev = next;
      }
    }
    return open;
  }

  // Cells of the lane on which side s is < -kMargin all over; good: it is
  // > kMargin on all of them.
  static CCD_HD unsigned outside(const float *w, int s, int lane, bool &good) {
    const float *p = w + 9 + s * (NS + 3);
    const float t0 = (float)(lane * kPer) * kCell;
    unsigned out = 0;
    float prev = at<NS>(p, t0), least = prev;
CCD_ROLLED
    for (int i = 0; i < kPer; i++) {
      const float next = at<NS>(p, t0 + (float)(i + 1) * kCell);
      if (fmaxf(prev, next) + p[NS + 1] < -kMargin) out |= 1u << i;
      least = fminf(least, next);
      prev = next;
    }
    good = least - p[NS + 1] > kMargin;
    return out;
  }
};

// Outcome for a row: nothing to solve (miss), or the slots to solve and the
// lanes (bits of `near`) whose cells stand for the other lists.
struct Need {
  bool miss;
  unsigned solve, near;
};

// Runs of set bits.
CCD_HD int runs(unsigned m) {
  unsigned s = m & ~(m << 1);
  int n = 0;
  for (; s; s &= s - 1) n++;
  return n;
}

// The lists that stand in for a slot's: the runs of near's lanes.
CCD_HD void stand_in(unsigned near, SpanList &out) {
  out.clear();
  int lane = 0;
  while (lane < kLanes) {
    if (!((near >> lane) & 1u)) {
      lane++;
      continue;
    }
    const int first = lane;
    while (lane < kLanes && ((near >> lane) & 1u)) lane++;
    out.push((double)first / kLanes, (double)lane / kLanes);
  }
}

// ------------------------------------------------------------------ sextics that wait
// A distance sextic whose last two coefficients are this small beside the
// largest has roots at (or within rounding of) t = 0: features that start in
// contact with their common plane, as the edges of a flat sheet do.  Such a
// solve can run through all 20 shifts (some 13,000 steps, against about 20
// for others), and the row's other lists usually share no time beyond 0, so
// it waits for them.  On a flat sheet in rigid motion with jitter, 86% of the
// solver steps of these sextics are saved.
// (24 meshes, sheets among them: 465 -> 202 ms with it and the classification.)
constexpr double kWaitTail = 1e-9;
constexpr unsigned kWaits = 1;        // the sextic waits for the row's other lists
constexpr unsigned kZeroAtStart = 2;  // and vanishes exactly at t = 0 beside other terms

// What distance sextic op (reference order) is, in these bits.
CCD_HD unsigned waits(const double *op) {
  double m = 0.0, sum = 0.0;
CCD_UNROLL
  for (int c = 0; c <= 6; c++) {
    m = smax(m, fabs(op[c]));
    sum += fabs(op[c]);
  }
  // not one that is infinite or NaN: the solver reports it in the row's status
  if (!(sum < 1e300) || !(fabs(op[5]) + fabs(op[6]) <= kWaitTail * m)) return 0;
  bool other = false;
CCD_UNROLL
  for (int c = 1; c < 6; c++) other = other || op[c] != 0.0;
  return kWaits | (op[6] == 0.0 && op[0] != 0.0 && other ? kZeroAtStart : 0);
}

// Whether the N side lists of a row share a time; beyond: one after t = 0.
template <int N>
CCD_HD bool sides_meet(const SpanList *l, bool &beyond) {
  bool meets = false;
  beyond = false;
  for (int i = 0; i < l[0].n; i++)
    for (int j = 0; j < l[1].n; j++) {
      const double lo1 = smax(l[0].s[i].l, l[1].s[j].l), hi1 = smin(l[0].s[i].u, l[1].s[j].u);
      if (lo1 > hi1) continue;
      for (int k = 0; k < l[2].n; k++) {
        const double lo2 = smax(lo1, l[2].s[k].l), hi2 = smin(hi1, l[2].s[k].u);
        if (lo2 > hi2) continue;
        for (int m = 0; m < (N == 4 ? l[N - 1].n : 1); m++) {
          const double lo = N == 4 ? smax(lo2, l[N - 1].s[m].l) : lo2, hi = N == 4 ? smin(hi2, l[N - 1].s[m].u) : hi2;
          if (lo > hi) continue;
          meets = true;
          if (hi > 0.0) beyond = true;
        }
      }
    }
  return meets;
}

// Whether a row of K lists misses whatever its waiting sextic's list is: its
// side lists share no time; or, of an edge-edge row x, they share t = 0 alone,
// the sextic vanishes there exactly and the edges are parallel there: the
// sextic's list holds the span [0, 0], which counts as parallel and rules out
// every combination that touches it.
template <int K>
CCD_HD bool settled_without_sextic(const double *x, const SpanList *l, bool zero_at_start) {
  bool beyond;
  if (K == 4) return !sides_meet<3>(l, beyond);
  if (!sides_meet<4>(l + 1, beyond)) return true;
  if (beyond || !zero_at_start) return false;
  SpanList start, cop, par;
  start.n = 1;
  start.s[0] = Span{0.0, 0.0};
  ee_split_parallel(x, start, cop, par);
  return par.n > 0;
}

#if !defined(__CUDA_ARCH__)
// The same decision as the warp's (stages.cuh), one lane after another.
template <class Polys>
inline Need decide(const float *w) {
  typedef Row<Polys> R;
  Need r{false, R::kAll, 0u};
  unsigned live[kLanes];
  bool good[R::kSides][kLanes], any = false;
  for (int l = 0; l < kLanes; l++) {
    bool mirrored;
    const unsigned open = R::near_contact(w, l, mirrored);
    if (mirrored) return r;
    unsigned out = 0;
    for (int s = 0; s < R::kSides; s++) out |= R::outside(w, s, l, good[s][l]);
    live[l] = open & ~out;
    any = any || live[l];
  }
  if (!any) {
    r.miss = true;
    return r;
  }
  unsigned near = 0, solve = 1u << R::kDist;
  for (int l = 0; l < kLanes; l++)
    if (live[l] || (l > 0 && (live[l - 1] & 0xf0u)) || (l + 1 < kLanes && (live[l + 1] & 0x0fu))) near |= 1u << l;
  if (runs(near) > kRuns) return r;
  for (int s = 0; s < R::kSides; s++)
    for (int l = 0; l < kLanes; l++)
      if (((near >> l) & 1u) && !good[s][l]) solve |= 1u << R::slot_of(s);
  r.near = near;
  r.solve = solve;
  return r;
}
#endif

}  // namespace cls
}  // namespace ccd
