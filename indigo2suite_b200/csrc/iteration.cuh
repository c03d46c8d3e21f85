// End of an iteration, shared by every relax kernel (one launch per iteration
// or resident): the last block of the iteration records it, rotates the
// frontier slots and picks the style of the next iteration. Included by each
// translation unit that instantiates relax kernels.
#pragma once
#include "common.cuh"
#include "mlp.cuh"

namespace i2 {

// ---------------------------------------------------------------------------
// Selection of the next variant.

// Fixed frontier-size rule: union-find for CC on symmetric graphs where
// union_find_pays (common.cuh, with both sides measured), bottom-up pull for BFS
// levels whose frontier carries more than 1/16 of the edges
// (direction-optimising BFS), otherwise the edge-balanced push, which measured
// fastest of the push styles on every family tried.
// Union-find replaces the whole traversal, so it is a choice made once, before
// the first iteration, by both selectors; the per-iteration picks are among the
// propagation styles.
static __device__ bool union_find_first(const GStats& gs, int algo, int allowed, int next_iter) {
  return algo == kCC && next_iter == 0 && ((allowed >> kUnionFind) & 1) && union_find_pays(gs.nodes, gs.avgdeg);
}

// The learned selector overrides the rule only where it predicts the rule's
// style at least 2^kLearnedMargin (about 11%) slower than its own pick: the
// rule is its fallback, and small mispredictions between close styles do not
// cost time.
constexpr float kLearnedMargin = 0.15f;

static __device__ int heuristic_pick(const GStats& gs, int algo, int allowed, int size, unsigned long long edges) {
  (void)size;
  const float fe = (float)edges;
  const float E = (float)gs.edges;
  auto ok = [&](int v) { return (allowed >> v) & 1; };
  if (algo == kBFS && ok(kPullFrontier) && fe > E * (1.f / 16.f)) return kPullFrontier;
  return ok(kVPCta) ? kVPCta : kVPThread;
}

// Executed by every thread of one block, on the head S in shared memory: picks
// the variant for the next launch from the frontier in slot `nxt`, whose
// features the caller has put into S.feat, and sets go (and, when the
// traversal ends, the loop condition of the graph). `cond` tells whether
// another launch will happen; `force` >= 0 overrides the pick (the compress
// launch of union-find CC).
// The learned selector is re-evaluated when the frontier's entries or edges
// moved by more than a factor 1.5 since its last evaluation, or 16 iterations
// passed; otherwise the previous choice stands (long tails of small, similar
// frontiers do not pay for an inference each). On graphs with more vertices
// than any it was trained on it defers to the frequency rule (no inference):
// measured on RMAT-24 and RMAT-26 BFS, its picks there cost 1.08-1.38x the
// rule's time even with the size features clamped to the training range.
template <class H>
static __device__ void select_next(const Ctx& c, H& S, int next_iter, int nxt, bool cond, int force) {
  const unsigned long long p = S.slot[nxt].packed;
  const int n = slot_size(p);
  const unsigned e = slot_edges(p);
  int v = S.fixed_variant;
  if constexpr (H::kSelect) {
    const int mode = S.mode;
    [[maybe_unused]] const float* y = nullptr;
    bool learned = false, infer = false;
    if constexpr (H::kNetwork) {
      __shared__ float h1[kHidden], h2[kHidden], out[kOut];
      learned = c.mlp && c.gs.nodes <= kMaxTrainedNodes;
      const long long sn = S.sel_n, se = S.sel_e;
      const bool moved = next_iter == 0 || 2LL * n > 3LL * sn || 3LL * n < 2LL * sn || 2LL * e > 3LL * se ||
                         3LL * e < 2LL * se || next_iter - S.sel_iter >= 16;
      infer = mode == 2 && learned && cond && moved && force < 0;
      if (infer) mlp_forward_block(c.mlp, S.feat, h1, h2, out);
      y = out;
    }
    if (threadIdx.x == 0) {
      if (mode == 3) {
        v = next_iter >= S.then_at ? S.then_variant : S.fixed_variant;
      } else if ((mode == 1 || mode == 2) && union_find_first(c.gs, S.algo, S.allowed, next_iter)) {
        v = kUnionFind;
      } else if (mode == 1 || (mode == 2 && !learned)) {
        v = heuristic_pick(c.gs, S.algo, S.allowed, n, e);
      } else if (mode == 2) {
        v = S.variant;
        if (infer) {
          const int h = heuristic_pick(c.gs, S.algo, S.allowed, n, e);
          float best = 3.0e38f;
          int bv = -1;
          for (int k = 0; k < kOut; ++k)  // per-iteration styles only (see union_find_first)
            if (k != kUnionFind && ((S.allowed >> k) & 1) && y[k] < best) {
              best = y[k];
              bv = k;
            }
          v = (bv >= 0 && best + kLearnedMargin < y[h]) ? bv : h;
          S.sel_n = n;
          S.sel_e = e;
          S.sel_iter = next_iter;
        }
      }
    }
  }
  if (threadIdx.x == 0) {
    if (force >= 0) v = force;
    S.variant = v;
    if (cond) atomicAdd(&c.ctl->hist[v], 1);
    S.go = cond ? 1 : 0;
    // the graph's loop condition starts at 1 and keeps its value between launches
    if (c.use_loop && !cond) cudaGraphSetConditional((cudaGraphConditionalHandle)c.loop_h, 0u);
  }
}

// Edges that the next near set should carry: the budget, or more where the
// far pile is large. A move reads the whole pile, about 20 ps an entry, which
// is the time of 2 relaxed edges; near sets of fewer edges than that spend
// most of the traversal in moves. RMAT-25 ordered (12 M entries on the pile),
// ms: no growth 16.7 (25 moves, 5.6 ms), 1 edge per entry 14.7, 2 14.1,
// 3 15.8; RMAT-22 (2 M entries), where the budget is the larger: 2.07 with all.
constexpr long long kMoveEdgesPerEntry = 2;
static __device__ __forceinline__ long long near_budget(const CtlHead& S) {
  const int np = S.split == 1 ? 1 - S.pcur : S.pcur;  // the pile the next move reads
  return max(-(long long)S.delta, kMoveEdgesPerEntry * (long long)S.psize[np]);
}

// Edge budget of the SSSP near/far ordering (whole block; kBlock bins): the
// first bin at which each histogram's running edge count reaches the budget
// (kHistBins if it never does): [0] the next frontier's, [1] the pile's. The
// next frontier's histogram is then cleared for the next launch's pushes.
static_assert(kHistBins == kBlock, "one histogram bin per thread");
static __device__ void budget_quantiles(const Ctx& c, const CtlHead& S, int* q) {
  __shared__ unsigned long long part[kBlock / kWarp];
  __shared__ int sq[2];
  const unsigned long long B = (unsigned long long)near_budget(S);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int which = 0; which < 2; ++which) {
    unsigned long long* h = c.hist + which * kHistBins;
    const unsigned long long x = *(volatile unsigned long long*)&h[threadIdx.x];
    unsigned long long incl = x;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) part[wid] = incl;
    if (threadIdx.x == 0) sq[which] = kHistBins;
    __syncthreads();
    for (int w = 0; w < wid; ++w) incl += part[w];
    if (incl >= B && incl - x < B) sq[which] = threadIdx.x;
    __syncthreads();
  }
  q[0] = sq[0];
  q[1] = sq[1];
  c.hist[threadIdx.x] = 0ull;
}

// Thread 0 of the last block, edge budget: the next launch of the ordering.
// `q` are the histogram quantiles, `n`/`e` the next frontier's entries and
// edges. Returns whether another launch follows; *clear_pile is set when the
// pile histogram must be cleared (a move rebuilds it from the entries it keeps).
static __device__ int budget_next(CtlHead& S, const int* q, long long n, unsigned e, int nxt, int* clear_pile) {
  const long long B = -(long long)S.delta, near = near_budget(S);
  const int shift = S.hshift;
  const int was = S.split;
  const int p = S.pcur;
  int cond = n > 0;
  *clear_pile = 0;
  if (was == 1) {  // the move emptied pile p onto the other one
    S.psize[p] = 0;
    S.pmin[p] = kInf;
    S.pcur = 1 - p;
  }
  S.split = 0;
  const int np = S.pcur;
  // move next when the frontier is empty, or so small that its last
  // iterations would cost more launches than edges (it is carried along)
  if (S.psize[np] > 0 && (n == 0 || (was == 0 && (long long)e * 16 < B))) {
    // at the budget's quantile of the pile (and above the pile's lower bound,
    // so that a live entry moves, or the move learns the bound)
    const int pm = S.pmin[np];
    long long T = q[1] < kHistBins ? (long long)S.pbase + ((long long)(q[1] + 1) << shift) : (long long)kInf;
    if (pm != kInf) T = max(T, (long long)pm + 1);
    T = min(T, (long long)kInf);
    S.prev_threshold = S.threshold;
    S.threshold = (int)T;
    int lo = pm != kInf ? pm : S.pbase;  // the smallest value the move can carry
    if (n > 0) lo = min(lo, S.slot[nxt].mindist);
    S.hbase = lo;
    S.pbase = (int)T;                       // kept values are at or above T
    S.split = 1;
    *clear_pile = 1;
    return 1;
  }
  if (n > 0 && was != 3 && (long long)e > 2 * near && q[0] < kHistBins) {
    const long long T = (long long)S.hbase + ((long long)(q[0] + 1) << shift);
    if (T < (long long)S.threshold) {  // trim the next frontier to about that many edges
      S.threshold = (int)T;
      S.split = 3;
    }
  }
  S.hbase = S.slot[nxt].mindist;
  return cond;
}

// Last block of a relax launch: record the launch, advance the iteration and
// decide whether the loop continues. The head is read once (with the counts
// that every block has added), advanced in shared memory by thread 0 while the
// second warp writes the record and computes the next frontier's features, and
// written back with one store per thread.
template <class H>
static __device__ __forceinline__ void finish_iteration(const Ctx& c, H& S, int i, int cur, int nxt, int old) {
  __shared__ int s_cond, s_force, s_clear;
  __shared__ int s_q[2];
  const unsigned long long t1 = globaltimer();
  load_head(c, S);
  if (threadIdx.x == 0) s_clear = 0;
  __syncthreads();
  if (S.variant == kUnionFind && S.uf_phase == 0) uf_sample_giant(c, S);  // whole block
  if (S.delta < 0) {
    int q[2];
    budget_quantiles(c, S, q);
    if (threadIdx.x == 0) {
      s_q[0] = q[0];
      s_q[1] = q[1];
    }
    __syncthreads();
  }
  const unsigned long long dt = t1 - S.tstart;
  if (threadIdx.x / kWarp == 1) {
    const int lane = threadIdx.x % kWarp;
    if (c.recs && i < c.rec_cap) {
      IterRec& r = c.recs[i];
      if (lane == 0) {
        const Slot& f = S.slot[cur];
        r.iter = i;
        r.variant = S.variant;
        r.size = slot_size(f.packed);
        r.hsize = slot_size(f.hpacked);
        r.edges = slot_edges(f.packed);
        r.maxdeg = f.maxdeg;
        r.mindist = f.mindist;
        r.visited = S.visited;
        r.t_ns = dt;
        r.kind = S.split;
        r.threshold = S.threshold;
        r.pile = S.delta != 0 ? S.psize[S.split == 1 ? 1 - S.pcur : S.pcur] : 0u;
      }
      if (lane < kFeatures) r.feat[lane] = S.feat[lane];
    }
    if (lane < kFeatures) {
      const Slot& f = S.slot[nxt];
      S.feat[lane] = frontier_feature(lane, c.gs, S.algo, i + 1, slot_size(f.packed), slot_size(f.hpacked),
                                      slot_edges(f.packed), f.maxdeg, S.visited);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    S.relax_ns += dt;
    Slot& so = S.slot[old];
    so.packed = 0;
    so.hpacked = 0;
    so.maxdeg = 0;
    so.mindist = kInf;
    S.done = 0;
    S.chunk = 0;
    S.tstart = ~0ull;
    S.iter = i + 1;
    const Slot& sn = S.slot[nxt];
    const long long n = slot_size(sn.packed);
    int cond = n > 0;
    if (S.delta < 0) {
      cond = budget_next(S, s_q, n, slot_edges(sn.packed), nxt, &s_clear);
    } else if (S.delta > 0) {
      if (S.split) {  // this launch emptied pile pcur onto the other one
        const int p = S.pcur;
        S.psize[p] = 0;
        S.pmin[p] = kInf;
        S.pcur = 1 - p;
        S.split = 0;
      }
      const int p = S.pcur;
      if (n == 0 && S.psize[p] > 0) {
        // next launch splits the pile at a raised threshold
        const long long lo = max((long long)S.threshold, (long long)S.pmin[p]);
        S.prev_threshold = S.threshold;
        S.threshold = (int)min(lo + (long long)S.delta, (long long)kInf);
        S.split = 1;
        cond = 1;
      }
    }
    int force = -1;
    if (S.variant == kUnionFind) {
      if (S.uf_phase < 2) {  // the next union-find launch follows
        S.uf_phase += 1;
        force = kUnionFind;
        cond = 1;
      } else {
        S.uf_phase = 0;  // labels final; nothing was pushed
      }
    }
    if (cond && i + 1 >= S.iter_cap) {
      atomicOr(&c.ctl->status, kStatusIterCap);
      cond = 0;
    }
    s_cond = cond;
    s_force = force;
  }
  __syncthreads();
  if (s_clear) c.hist[kHistBins + threadIdx.x] = 0ull;  // read above; the move rebuilds it
  select_next(c, S, i + 1, nxt, s_cond != 0, s_force);
  __syncthreads();
  store_head(c, S);
}

}  // namespace i2
