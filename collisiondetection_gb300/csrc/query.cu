// One vertex-face or edge-edge row in FP64: a single query.
//
// A lone lane takes a row's lists one after another, each a root solve of some
// 100 us of dependent FP64 operations and cold code.  Here a cluster of blocks
// takes them at once, one warp on an SM of its own per list (five warps on one
// SM would share its FP64 pipe), and the first empty list stops the others
// through their shared memory: a query ends with the list that settles it, and
// takes the longest of its lists instead of their sum.  A solve whose shifts
// fail goes on with a stage's remaining shifts at once, one per lane
// (ccd_jt_shifts.h).  Polynomials, solver and decision are those of the
// one-lane kernel, operation for operation.
//
// Medians of whole queries on benchmark rows, one lane and this kernel (us):
// vertex-face rows that hit 383 and 223, that miss 117 and 49; edge-edge 607
// and 258, 216 and 49.  A row that its first list settles without a solve: 46
// and 50.  A larger FP64 batch has rows enough for its lanes.
#include <cooperative_groups.h>

#include "ccd_ctcd64.h"
#include "ccd_jt_shifts.h"
#include "narrow.cuh"

namespace ccd {
namespace {

// Shifts of a stage that one lane tries before the rest run at once: more than
// in the pool, whose other solves wait.  With 2, a query that a few failed
// shifts settle took 1.33 ms where one lane takes 1.05; with 4 it takes 0.84,
// and the longest ones (all shifts fail) 5.1 instead of 4.3 (one lane: 100).
constexpr int kShiftsAlone = 4;

// What the cluster's first block gathers of each list.
struct Lists {
  SpanList l[8];
  uint8_t status[8], empty[8];
};

// Runs the solve that lane 0 has started in `shared` to its end, by the warp;
// false once *stop is set.
__device__ bool solve(jt::LocalStorage &shared, const volatile int *stop) {
  const unsigned kFull = 0xffffffffu;
  const jt::LocalState s{&shared};
  for (;;) {
    const int mode = s.I(jt::MODE);
    if (mode == jt::kDone) return true;
    if (__any_sync(kFull, *stop != 0)) return false;
    if (mode != jt::kInit && s.I(jt::CNT) >= kShiftsAlone) {
      jt::LocalStorage own = shared;
      if (!jt::shifts::run(own, kShiftsAlone, stop)) return false;
      if (threadIdx.x == 0) shared = own;
    } else if (threadIdx.x == 0) {
      jt::step(s);
    }
    __syncwarp();
  }
}

// Spans of op (reduced to degree deg) from a finished solve.
__device__ void solved_spans(const double *op, int deg, jt::LocalStorage &shared, SpanList &out, bool want_pos,
                             uint8_t &status) {
  const jt::LocalState s{&shared};
  double tr[6];
  for (int i = 0; i < deg; i++) tr[i] = s.Z(i);
  status |= (uint8_t)s.I(jt::STATUS);
  root_spans(op, deg, tr, s.I(jt::ROOTS), out, want_pos);
}

template <class Polys>
__global__ void __launch_bounds__(32) query_kernel(PrimBatch b) {
  namespace cg = cooperative_groups;
  constexpr int K = Polys::kSlots;
  const cg::cluster_group cluster = cg::this_cluster();
  const int slot = (int)cluster.block_rank(), lane = threadIdx.x;
  __shared__ Lists lists;
  __shared__ jt::LocalStorage state;
  __shared__ int stop;
  if (lane == 0) stop = 0;
  cluster.sync();
  double x[24];
  bool ordinary = true;
#pragma unroll
  for (int j = 0; j < 24; j++) {
    x[j] = __ldg(b.rows + j);
    ordinary = ordinary && fabs(x[j]) < 1e30;
  }
  const double eta = __ldg(b.eta);
  ordinary = ordinary && fabs(eta) < 1e30;
  double op[7];
  SpanList sl;
  sl.clear();
  uint8_t status = 0;
  int deg = 0;
  bool working = false, empty = true;  // a list that is given up counts as empty
  // One empty list settles the row.  Not where numbers may overflow: the
  // solver reports those in the row's status, list by list.
  const auto listed = [&]() {
    empty = sl.n == 0;
    if (K == 5 && slot == 0) {  // only spans at which the edges are not parallel count
      SpanList cop, par;
      ee_split_parallel(x, sl, cop, par);
      empty = cop.n == 0;
    }
    if (lane == 0 && empty && ordinary)
      for (int r = 0; r < K; r++) *(volatile int *)cluster.map_shared_rank(&stop, r) = 1;
  };
  // First the lists that take no iteration, in every block: many rows end
  // there, and a block that has begun to iterate stops only between steps.
  if (slot < K) {
    const bool pos = Polys::want_pos(slot);
    Polys::coeffs(x, eta, slot, op);
    deg = reduce_poly(op, Polys::degree(slot));
    if (deg <= 2) {
      low_degree_spans(op, deg, sl, pos);
    } else if (sign_possible(op, deg, pos)) {
      if (lane == 0) jt::start(jt::LocalState{&state}, op, deg);
      __syncwarp();
      working = jt::LocalState{&state}.I(jt::MODE) != jt::kDone;
      if (!working) solved_spans(op, deg, state, sl, pos, status);
    }
    if (!working) listed();
  }
  cluster.sync();
  if (slot < K) {
    if (working && solve(state, &stop)) {
      solved_spans(op, deg, state, sl, Polys::want_pos(slot), status);
      listed();
    }
    if (lane == 0) {
      Lists *to = cluster.map_shared_rank(&lists, 0);
      to->l[slot] = sl;
      to->status[slot] = status;
      to->empty[slot] = empty;
    }
  }
  cluster.sync();
  if (slot != 0 || lane != 0) return;
  // The lists in the order of the one-lane test, which ends at an empty one.
  status = 0;
  bool h = true;
  for (int k = 0; k < K && h; k++) {
    status |= lists.status[k];
    h = !lists.empty[k];
  }
  double t = 0.0;
  if (h) {
    if constexpr (K == 4) {
      h = vf_combine(lists.l[0], lists.l[1], lists.l[2], lists.l[3], t);
    } else {
      SpanList cop, par;
      ee_split_parallel(x, lists.l[0], cop, par);
      h = ee_combine(cop, par, lists.l[1], lists.l[2], lists.l[3], lists.l[4], t);
    }
  }
  b.hit[0] = h;
  if (h) b.t[0] = t;
  if (b.status) b.status[0] = status;
  b.counters->survivors += 1;
  b.counters->hits += h;
  b.counters->status_flags += status != 0;
}

template <class Polys>
cudaError_t launch(const PrimBatch &b, int blocks, cudaStream_t s) {
  cudaLaunchAttribute cluster;
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim.x = (unsigned)blocks;
  cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(32);
  cfg.stream = s;
  cfg.attrs = &cluster;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, query_kernel<Polys>, b);
}

}  // namespace

cudaError_t launch_query(const PrimBatch &b, cudaStream_t s) {
  return b.kind == kVF ? launch<VFPolys>(b, 4, s) : launch<EEPolys>(b, 8, s);
}

}  // namespace ccd
