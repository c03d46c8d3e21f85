// B200 relaxation engine: device graphs, traversal runs and the C ABI of
// include/i2b200.h for BFS, SSSP and CC.
//
// A traversal is: reset the control block, fill dist/labels and seed F_0, then
// one relaxation per iteration until the frontier is empty (the do-while of the
// reference's host drivers, e.g.
// BFS_CUDA_V_Data_Push_..._Warp_..._NonDup.cu:112-122). In the default loop
// mode (I2_LOOP_GRAPH) that is two launches: k_start, and one cooperative
// launch that runs every iteration itself, its blocks meeting at a bounded
// barrier between iterations (relax_resident, relax.cuh). I2_LOOP_RELAUNCH is a
// CUDA graph whose WHILE conditional node launches one kernel per iteration:
// the fixed style's, or the dispatch kernel whose blocks branch on the style
// picked for this iteration. Either way the last block of an iteration picks
// the next style on the device, so there is no host round trip per iteration.
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <numeric>
#include <vector>
#include "../../include/i2b200.h"
#include "common.cuh"
#include "engine.h"
#include "host_graph.h"
#include "mlp.cuh"
#include "relax.cuh"
#include "iteration.cuh"

namespace i2 {

static_assert(sizeof(IterRec) == sizeof(i2_iter_record), "record layout");
static_assert((int)kNumVariants == (int)I2_NUM_VARIANTS, "variant count");

// ---------------------------------------------------------------------------
// Init kernels.

// Counts of a frontier that is not listed: every vertex with edges (records and
// features show what a listed one would).
static __device__ __forceinline__ void whole_slot(const Ctx& c, Slot& s) {
  s.packed = ((unsigned long long)c.gs.linked << 32) | (unsigned)c.g.edges;
  s.hpacked = (unsigned long long)c.gs.nheavy << 32;
  s.maxdeg = c.gs.maxdeg;
  s.mindist = c.gs.first;
}

// dist[v] = INF (BFS/SSSP) or v (CC). For CC every vertex enters F_0, unless
// union-find runs from the first iteration (CtlHead::whole): it reads no
// frontier, so none is built.
template <int ALG>
__global__ void __launch_bounds__(kBlock) k_fill(Ctx c) {
  __shared__ Stage s;
  stage_init(s);
  Acc a;
  acc_init(a);
  __syncthreads();
  const int V = c.g.nodes;
  if (ALG == kCC && c.ctl->whole) {
    const unsigned stride = gridDim.x * kBlock;
    for (unsigned v = blockIdx.x * kBlock + threadIdx.x; v < (unsigned)V; v += stride) c.dist[v] = (int)v;
    if (blockIdx.x == 0 && threadIdx.x == 0) whole_slot(c, c.ctl->slot[0]);
    return;
  }
  for (long long base = (long long)blockIdx.x * kBlock; base < V; base += (long long)gridDim.x * kBlock) {
    const int v = (int)base + threadIdx.x;
    const bool in = (unsigned)v < (unsigned)V;  // v may pass INT_MAX
    constexpr bool kAll = ALG == kCC || ALG == kMIS;  // every vertex starts in F_0
    const int deg = (kAll && in) ? c.g.nindex[v + 1] - c.g.nindex[v] : 0;
    // MIS: a vertex without neighbours is in the set at once
    if (in) c.dist[v] = ALG == kCC ? v : ALG == kMIS ? (deg == 0 ? kMisIn : kMisUndecided) : kInf;
    if (kAll) {
      const bool put = in && deg > 0;  // vertices without edges are already final
      const unsigned word = __ballot_sync(0xffffffffu, put);
      if ((threadIdx.x & 31) == 0 && word) c.bm[0][v >> 5] = word;
      if (put) {
        a.mindist = min(a.mindist, v);
        stage_entry(c, s, a, 0, v, deg);
      }
      stage_flush(c, s, 0);
    }
  }
  if (ALG == kCC || ALG == kMIS) {
    stage_flush(c, s, 0);
    acc_reduce(a, s);
    if (threadIdx.x == 0) {
      const Acc& r = s.red[0];
      Slot& sl = c.ctl->slot[0];
      if (r.maxdeg) atomicMax(&sl.maxdeg, r.maxdeg);
      if (r.mindist != kInf) atomicMin(&sl.mindist, r.mindist);
    }
  }
}

// Whole block: the features of the seeded frontier F_0, and the first style.
static __device__ void select_first(const Ctx& c, SelectHead& S) {
  if (threadIdx.x < kFeatures) {
    const Slot& f = S.slot[0];
    S.feat[threadIdx.x] = frontier_feature(threadIdx.x, c.gs, S.algo, 0, slot_size(f.packed), slot_size(f.hpacked),
                                           slot_edges(f.packed), f.maxdeg, S.visited);
  }
  __syncthreads();
  select_next(c, S, 0, 0, true, -1);
  __syncthreads();
}

// One block: seed the sources (BFS/SSSP) and select the first variant.
template <int ALG>
__global__ void __launch_bounds__(kBlock) k_seed(Ctx c) {
  Ctl* ctl = c.ctl;
  if (ALG != kCC && ALG != kMIS) {
    const int ns = c.srcs ? ctl->nsrc : 1;
    for (int j = threadIdx.x; j < ns; j += blockDim.x) {
      const int v = c.srcs ? c.srcs[j] : ctl->src;
      const int deg = c.g.nindex[v + 1] - c.g.nindex[v];
      const unsigned bit = 1u << (v & 31);
      if (atomicOr(&c.bm[0][v >> 5], bit) & bit) continue;
      c.dist[v] = 0;
      atomicAdd((unsigned long long*)&ctl->visited, 1ull);
      Slot& sl = ctl->slot[0];
      atomicMin(&sl.mindist, 0);
      if (deg == 0) {
        atomicAnd(&c.bm[0][v >> 5], ~bit);  // nothing to propagate
        continue;
      }
      atomicMax(&sl.maxdeg, deg);
      const unsigned long long b = atomicAdd(&sl.packed, (1ull << 32) | (unsigned)deg);
      c.wl[0][slot_size(b)] = v;
      c.woff[0][slot_size(b)] = slot_edges(b);
      if (deg >= c.heavy) {
        const int t = heavy_tiles(deg);
        const unsigned long long hb = atomicAdd(&sl.hpacked, (1ull << 32) | (unsigned)t);
        c.hwl[0][slot_size(hb)] = v;
        c.htoff[0][slot_size(hb)] = slot_edges(hb);
      }
    }
  } else if (threadIdx.x == 0) {
    ctl->visited = c.g.nodes;
  }
  __threadfence();
  __syncthreads();
  // the head with the seeded frontier: its features, and the first style
  __shared__ SelectHead S;
  load_head(c, S);
  __syncthreads();
  select_first(c, S);
  store_head(c, S);
}

// Per-run parameters, passed by value to k_reset so that queued runs never
// share a host buffer.
struct RunParams {
  int algo, mode, fixed_variant, allowed, src, nsrc, iter_cap, delta, hold, stall_ms, then_at, then_variant, hshift, whole;
  unsigned uf_step;
  bool operator!=(const RunParams& o) const { return std::memcmp(this, &o, sizeof(RunParams)) != 0; }
};

// The head of a run with these parameters (all its other words are zero).
static __device__ __forceinline__ void reset_head(CtlHead& S, const RunParams& p) {
  for (int k = 0; k < 3; ++k) S.slot[k].mindist = kInf;
  S.tstart = ~0ull;
  S.iter_cap = p.iter_cap;
  S.mode = p.mode;
  S.fixed_variant = p.fixed_variant;
  S.variant = p.fixed_variant;
  S.allowed = p.allowed;
  S.src = p.src;
  S.nsrc = p.nsrc;
  S.algo = p.algo;
  S.delta = p.delta;
  S.hshift = p.hshift;
  S.then_at = p.then_at;
  S.then_variant = p.then_variant;
  S.hold = p.hold;
  S.whole = p.whole;
  S.uf_step = p.uf_step;
  S.stall_ns = (unsigned long long)p.stall_ms * 1000000ull;
  S.threshold = p.delta > 0 ? p.delta : kInf;  // sources start at 0
  S.pmin[0] = kInf;
  S.pmin[1] = kInf;
}

__global__ void k_reset(Ctl* ctl, RunParams p) {
  unsigned* w = reinterpret_cast<unsigned*>(ctl);
  for (unsigned k = threadIdx.x; k < sizeof(Ctl) / sizeof(unsigned); k += blockDim.x) w[k] = 0u;
  __syncthreads();
  if (threadIdx.x == 0) reset_head(*ctl, p);
}

// Start of a resident traversal: control block, bitmaps and values in one
// kernel. Where no frontier of many vertices is to be built (one source,
// union-find from the first iteration, MIS, whose first iteration takes every
// vertex) it seeds the frontier and selects the first variant too, so that the
// traversal is two launches; CC by propagation has k_fill and k_seed after it,
// runs from many sources k_seed. Five nodes of a CUDA graph
// (memset, reset, fill, seed, conditional loop) took 16-20 us more: SSSP on RMAT
// with 3,001 vertices 151 -> 130 us, BFS RMAT-20 138 -> 118; and instantiating
// the graph cost a new graph's first traversal 0.25 ms.
template <int ALG>
__global__ void __launch_bounds__(kBlock) k_start(const __grid_constant__ Ctx c, RunParams p, unsigned words) {
  const bool single = (ALG == kBFS || ALG == kSSSP) && !c.srcs;
  const bool whole = single || ALG == kMIS || (ALG == kCC && p.whole);
  const int V = c.g.nodes;
  const int src = single ? p.src : -1;
  const int deg = single ? c.g.nindex[src + 1] - c.g.nindex[src] : 0;
  const unsigned stride = gridDim.x * kBlock;
  const unsigned tid = blockIdx.x * kBlock + threadIdx.x;
  // bitmaps, far-pile bitmap and histograms; a vertex without edges is never in a frontier
  const unsigned sword = deg > 0 ? (unsigned)src >> 5 : ~0u;
  for (unsigned w = tid; w < words; w += stride) c.bm[0][w] = w == sword ? 1u << (src & 31) : 0u;
  if (whole || ALG == kBFS || ALG == kSSSP) {
    // values, 16 bytes a store (the array starts on a 256-byte boundary)
    const unsigned quads = (unsigned)V >> 2;
    int4* d4 = reinterpret_cast<int4*>(c.dist);
    for (unsigned q = tid; q < quads; q += stride) {
      const int v = (int)(q << 2);
      d4[q] = ALG == kMIS  ? make_int4(kMisUndecided, kMisUndecided, kMisUndecided, kMisUndecided)
              : ALG == kCC ? make_int4(v, v + 1, v + 2, v + 3)
                         : make_int4(v == src ? 0 : kInf, v + 1 == src ? 0 : kInf, v + 2 == src ? 0 : kInf,
                                     v + 3 == src ? 0 : kInf);
    }
    for (unsigned v = (quads << 2) + tid; v < (unsigned)V; v += stride)
      c.dist[v] = ALG == kMIS ? (int)kMisUndecided : ALG == kCC ? (int)v : (int)v == src ? 0 : kInf;
  }
  if (blockIdx.x != 0) return;
  __shared__ SelectHead S;
  for (unsigned k = threadIdx.x; k < sizeof(Ctl) / sizeof(unsigned); k += kBlock)
    reinterpret_cast<unsigned*>(c.ctl)[k] = 0u;
  if (threadIdx.x < kHeadWords) reinterpret_cast<unsigned*>(&S)[threadIdx.x] = 0u;
  __syncthreads();
  if (threadIdx.x == 0) {
    reset_head(S, p);
    Slot& sl = S.slot[0];
    if (single) {
      S.visited = 1;
      sl.mindist = 0;
      if (deg > 0) {
        sl.maxdeg = deg;
        sl.packed = (1ull << 32) | (unsigned)deg;
        c.wl[0][0] = src;
        c.woff[0][0] = 0;
        if (deg >= c.heavy) {
          sl.hpacked = (1ull << 32) | (unsigned)heavy_tiles(deg);
          c.hwl[0][0] = src;
          c.htoff[0][0] = 0;
        }
      }
    } else if (whole) {
      S.whole = 1;
      S.visited = V;
      whole_slot(c, sl);
    }
  }
  __syncthreads();
  if (whole) select_first(c, S);
  store_head(c, S);
}

// ---------------------------------------------------------------------------
// Graph maintenance kernels.

// Sets bit 8 of *bad when a weight is negative (SSSP needs weights >= 0).
__global__ void k_negative_weights(const int* w, long long n, int* bad) {
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  int neg = 0;
  for (long long e = tid; e < n; e += stride) neg |= w[e] < 0;
  if (__any_sync(0xffffffffu, neg) && (threadIdx.x & 31) == 0) atomicOr(bad, 8);
}

__global__ void k_validate(DGraph g, int* bad) {
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long v = tid; v < g.nodes; v += stride)
    if (g.nindex[v + 1] < g.nindex[v]) atomicOr(bad, 1);
  for (long long e = tid; e < g.edges; e += stride)
    if ((unsigned)g.nlist[e] >= (unsigned)g.nodes) atomicOr(bad, 2);
  if (tid == 0 && (g.nindex[0] != 0 || g.nindex[g.nodes] != g.edges)) atomicOr(bad, 4);
}

struct DevStats {
  unsigned long long hub;  // largest degree << 32 | ~vertex: the lowest ID on ties
  unsigned long long counts;  // heavy vertices << 32 | vertices with edges
  unsigned firstinv;       // INT_MAX - the smallest of them (0: none)
  unsigned winv;           // INT_MAX - smallest weight (0: no weights)
  int unsorted;
  int asym;
  int pad;
  double sumsq;
  double wsum;
};

__global__ void k_degree_stats(DGraph g, int heavy, DevStats* st) {
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  unsigned long long hub = 0;
  int nh = 0, nl = 0;
  unsigned firstinv = 0;
  double s2 = 0.0;
  for (long long v = tid; v < g.nodes; v += stride) {
    const int b = g.nindex[v], e = g.nindex[v + 1];
    const int d = e - b;
    hub = max(hub, ((unsigned long long)d << 32) | (unsigned)~v);
    nh += d >= heavy;
    if (d > 0) {
      ++nl;
      firstinv = max(firstinv, (unsigned)INT_MAX - (unsigned)v);
    }
    s2 += (double)d * d;
  }
  unsigned winv = 0;
  double ws = 0.0;
  if (g.eweight)
    for (long long e = tid; e < g.edges; e += stride) {
      const int w = g.eweight[e];
      winv = max(winv, (unsigned)INT_MAX - (unsigned)w);
      ws += (double)w;
    }
  // one set of atomics per block: from every thread they were 0.4 ms on one line
  nh = __reduce_add_sync(0xffffffffu, nh);
  nl = __reduce_add_sync(0xffffffffu, nl);
  firstinv = __reduce_max_sync(0xffffffffu, firstinv);
  winv = __reduce_max_sync(0xffffffffu, winv);
  for (int o = 16; o > 0; o >>= 1) {
    hub = max(hub, __shfl_down_sync(0xffffffffu, hub, o));
    s2 += __shfl_down_sync(0xffffffffu, s2, o);
    ws += __shfl_down_sync(0xffffffffu, ws, o);
  }
  __shared__ int snh[kWarp], snl[kWarp];
  __shared__ unsigned swi[kWarp], sfi[kWarp];
  __shared__ unsigned long long shub[kWarp];
  __shared__ double ss2[kWarp], sws[kWarp];
  const int wid = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    shub[wid] = hub;
    snh[wid] = nh;
    snl[wid] = nl;
    sfi[wid] = firstinv;
    swi[wid] = winv;
    ss2[wid] = s2;
    sws[wid] = ws;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int k = 1; k < nwarp; ++k) {
    hub = max(hub, shub[k]);
    nh += snh[k];
    nl += snl[k];
    firstinv = max(firstinv, sfi[k]);
    winv = max(winv, swi[k]);
    s2 += ss2[k];
    ws += sws[k];
  }
  atomicMax(&st->hub, hub);
  atomicAdd(&st->counts, ((unsigned long long)(unsigned)nh << 32) | (unsigned)nl);
  // most blocks find these two no further on than others have
  if (firstinv > *(volatile unsigned*)&st->firstinv) atomicMax(&st->firstinv, firstinv);
  if (winv > *(volatile unsigned*)&st->winv) atomicMax(&st->winv, winv);
  atomicAdd(&st->sumsq, s2);
  if (g.eweight) atomicAdd(&st->wsum, ws);
}

// Adjacency lists strictly increasing (sorted, no duplicates)? One thread per
// CSR entry, using the starting-point array for the entry's row.
__global__ void k_sorted(DGraph g, const int* __restrict__ sp, DevStats* st) {
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  int uns = 0;
  for (long long e = 1 + tid; e < g.edges; e += stride)
    uns |= (sp[e] == sp[e - 1]) && (g.nlist[e] <= g.nlist[e - 1]);
  if (uns) atomicOr(&st->unsorted, 1);
}

// For every entry (u, v, w): is (v, u, w) present? One thread per entry,
// binary search in v's sorted adjacency.
__global__ void k_symmetry(DGraph g, const int* __restrict__ sp, DevStats* st) {
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  int asym = 0;
  for (long long k = tid; k < g.edges && !asym; k += stride) {
    const int u = sp[k];
    const int v = g.nlist[k];
    int lo = g.nindex[v], hi = g.nindex[v + 1] - 1, pos = -1;
    while (lo <= hi) {
      const int mid = lo + ((hi - lo) >> 1);  // lo + hi may exceed INT_MAX
      if ((unsigned)mid >= (unsigned)g.edges) {
        asym = 1;  // cannot happen on a validated CSR; refuse rather than read out of bounds
        break;
      }
      const int x = g.nlist[mid];
      if (x == u) { pos = mid; break; }
      if (x < u) lo = mid + 1; else hi = mid - 1;
    }
    if (pos < 0 || (g.eweight && g.eweight[pos] != g.eweight[k])) asym = 1;
  }
  if (asym) atomicOr(&st->asym, 1);
}

// sp[k] = row of CSR entry k; one warp per vertex, coalesced stores.
__global__ void k_build_sp(DGraph g, int* sp) {
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  for (long long v = warp; v < g.nodes; v += nwarps)
    for (long long k = g.nindex[v] + lane; k < g.nindex[v + 1]; k += 32) sp[k] = (int)v;
}

// Reference synthetic weights (include/sssp_vertex_cuda.h:127-137) on the device.
__global__ void k_synth_weights(DGraph g, int* w) {
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = tid; i < g.nodes; i += stride)
    for (int j = g.nindex[i]; j < g.nindex[i + 1]; ++j) {
      const int prod = (int)((unsigned)i * (unsigned)g.nlist[j]);
      int x = 1 + (prod % g.nodes);
      w[j] = x < 0 ? -x : x;
    }
}

// Reached vertices and the sum of their degrees (E_r).
__global__ void k_reached(DGraph g, const int* dist, unsigned long long* out) {
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  unsigned long long nv = 0, ne = 0;
  for (long long v = tid; v < g.nodes; v += stride)
    if (dist[v] != kInf) {
      nv++;
      ne += (unsigned long long)(g.nindex[v + 1] - g.nindex[v]);
    }
  for (int o = 16; o > 0; o >>= 1) {
    nv += __shfl_down_sync(0xffffffffu, nv, o);
    ne += __shfl_down_sync(0xffffffffu, ne, o);
  }
  __shared__ unsigned long long sv[kWarp], se[kWarp];
  if ((threadIdx.x & 31) == 0) {
    sv[threadIdx.x >> 5] = nv;
    se[threadIdx.x >> 5] = ne;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
    nv += sv[k];
    ne += se[k];
  }
  atomicAdd(&out[0], nv);
  atomicAdd(&out[1], ne);
}

// Values of a traversal on the degree-ordered copy, back in original IDs:
// out[v] = copy[inv[v]] (coalesced inv read and write, gathered copy read).
__global__ void k_unpermute(const int* __restrict__ copy, const int* __restrict__ inv, int n,
                            int* __restrict__ out) {
  const int stride = gridDim.x * blockDim.x;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) out[v] = copy[inv[v]];
}

// CC on the degree-ordered copy labels each vertex with its component's
// smallest copy ID; the caller's labels are the smallest original IDs. First
// mn[r] = min { v : label of copy vertex inv[v] is r } (one atomicMin per
// distinct label in a warp, by its lowest lane, which holds the smallest v
// since a warp covers consecutive v; skipped when mn[r] is already smaller,
// as it soon is for the giant component), then out[v] = mn[label(inv[v])].
__global__ void k_cc_min_init(int* __restrict__ mn, int n) {
  const int stride = gridDim.x * blockDim.x;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) mn[v] = INT_MAX;
}

__global__ void k_cc_min_original(const int* __restrict__ copy_label, const int* __restrict__ inv, int n,
                                  int* mn) {
  const int stride = gridDim.x * blockDim.x;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
    const int r = copy_label[inv[v]];
    const unsigned peers = __match_any_sync(__activemask(), r);
    if ((int)(threadIdx.x & 31) == __ffs(peers) - 1 && v < *(volatile int*)&mn[r]) atomicMin(&mn[r], v);
  }
}

__global__ void k_cc_labels(const int* __restrict__ copy_label, const int* __restrict__ inv,
                            const int* __restrict__ mn, int n, int* __restrict__ out) {
  const int stride = gridDim.x * blockDim.x;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) out[v] = mn[copy_label[inv[v]]];
}

// ---------------------------------------------------------------------------
// Kernel tables.

// The selectors' per-iteration kernel; `wide`: the form compiled for the fixed
// styles' resident blocks per SM (graphs of kWideSelectorNodes vertices or more).
static KernelFn dispatch_kernel(int algo, bool wide) {
  if (algo == kBFS) return dispatch_fn<kBFS>(wide);
  if (algo == kSSSP) return dispatch_fn<kSSSP>(wide);
  return dispatch_fn<kCC>(wide);  // MIS never dispatches
}

// One launch per iteration in style v: in a run of that style alone (mode 0), or
// in one whose style may change.
static KernelFn relax_kernel(int algo, int mode, int v, bool near_far, bool wide) {
  if (near_far && algo == kSSSP && v == kVPCta) return near_far_kernel(false);
  if (algo == kBFS) return relax_fn<kBFS>(v, mode != 0, wide);
  if (algo == kSSSP) return relax_fn<kSSSP>(v, mode != 0, wide);
  if (algo == kCC) return relax_fn<kCC>(v, mode != 0, wide);
  return mis_kernel(false);  // one style
}

// Kernel of a resident traversal: fixed style v (mode 0) or the per-iteration
// pick (v < 0; `wide`: the form compiled for more resident blocks).
static KernelFn resident_kernel(int algo, int v, bool near_far, bool wide) {
  if (algo == kMIS) return mis_kernel(true);  // one style
  if (near_far && algo == kSSSP && v == kVPCta) return near_far_kernel(true);
  if (algo == kBFS) return resident_fn<kBFS>(v, wide);
  if (algo == kSSSP) return resident_fn<kSSSP>(v, wide);
  return resident_fn<kCC>(v, wide);
}

static KernelFn fill_kernel(int algo) {
  if (algo == kBFS) return k_fill<kBFS>;
  if (algo == kSSSP) return k_fill<kSSSP>;
  if (algo == kCC) return k_fill<kCC>;
  return k_fill<kMIS>;
}
static KernelFn seed_kernel(int algo) {
  if (algo == kBFS) return k_seed<kBFS>;
  if (algo == kSSSP) return k_seed<kSSSP>;
  if (algo == kCC) return k_seed<kCC>;
  return k_seed<kMIS>;
}

// ---------------------------------------------------------------------------
// Device state helpers.

int cuda_status(cudaError_t e) {
  if (e == cudaSuccess) return I2_OK;
  if (e == cudaErrorMemoryAllocation) return I2_ERR_NOMEM;
  if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) return I2_ERR_NO_DEVICE;
  return I2_ERR_CUDA;
}

#define I2_CK(call)                         \
  do {                                      \
    cudaError_t e_ = (call);                \
    if (e_ != cudaSuccess) {                \
      cudaGetLastError();                   \
      return cuda_status(e_);               \
    }                                       \
  } while (0)

static int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 1;
  }
  return n;
}

// Preferred shared-memory carveout (percent of the unified L1/shared storage)
// for the relax kernels; -1 leaves the choice to the driver. A large carveout
// costs L1 capacity, which the adjacency reads use. It is an attribute of the
// kernels, which all graphs share, and decides how many blocks of one fit an SM:
// a change invalidates the grids that every graph has kept (g_carveout_set).
static std::atomic<int> g_carveout{-1};
static std::atomic<unsigned> g_carveout_set{0};  // changes so far

int grid_for(KernelFn fn, int max_per_sm) {
  cudaFuncSetAttribute((const void*)fn, cudaFuncAttributePreferredSharedMemoryCarveout, g_carveout.load());
  int per = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void*)fn, kBlock, 0);
  per = std::max(1, std::min(per, max_per_sm));
  return per * sm_count();
}

// Per-device selector parameters.
static std::mutex g_mlp_mu;
static float* g_mlp_dev[64] = {nullptr};

const float* mlp_device_params() {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(g_mlp_mu);
  return (dev >= 0 && dev < 64) ? g_mlp_dev[dev] : nullptr;
}

int mlp_install(const float* params, int count) {
  if (!params || count != kParams) return I2_ERR_ARG;
  int dev = 0;
  I2_CK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return I2_ERR_ARG;
  std::lock_guard<std::mutex> lk(g_mlp_mu);
  if (!g_mlp_dev[dev]) I2_CK(cudaMalloc(&g_mlp_dev[dev], sizeof(float) * kParams));
  I2_CK(cudaMemcpy(g_mlp_dev[dev], params, sizeof(float) * kParams, cudaMemcpyHostToDevice));
  return I2_OK;
}

}  // namespace i2

using namespace i2;

// ---------------------------------------------------------------------------
// Graph handle.

struct ExecKey {
  int algo, mode, variant, multi, near_far;
  bool operator<(const ExecKey& o) const {
    if (algo != o.algo) return algo < o.algo;
    if (mode != o.mode) return mode < o.mode;
    if (variant != o.variant) return variant < o.variant;
    if (multi != o.multi) return multi < o.multi;
    return near_far < o.near_far;
  }
};

struct ExecEntry {
  cudaGraphExec_t ex = nullptr;
  cudaGraphNode_t reset = nullptr;
  RunParams last{};
  Ctx ctx{};
};

struct i2_graph {
  DGraph g{};
  GStats gs{};
  int hub = 0;  // highest-degree vertex, the lowest ID on ties
  int device = 0;
  bool owns = false;
  int* d_nindex = nullptr;
  int* d_nlist = nullptr;
  int* d_eweight = nullptr;
  bool owns_weights = false;
  int* d_sp = nullptr;
  int heavy = 4096;
  int blocks_per_sm = 8;  // cap; the occupancy of each kernel decides below it
  // workspace
  bool ws_ready = false;
  char* ws_base = nullptr;     // one block: values, frontier lists, bitmaps, control block, records
  char* heavy_base = nullptr;  // one block: the heavy lists (sized by the heavy threshold)
  int* dist = nullptr;
  int* wl[3] = {nullptr, nullptr, nullptr};
  unsigned* woff[3] = {nullptr, nullptr, nullptr};
  int* hwl[3] = {nullptr, nullptr, nullptr};
  unsigned* htoff[3] = {nullptr, nullptr, nullptr};
  unsigned* bm[3] = {nullptr, nullptr, nullptr};
  unsigned* fbm = nullptr;  // far-pile bitmap, allocated after bm[2]
  unsigned long long* hist = nullptr;  // near/far distance histograms, after fbm
  int* pile[2] = {nullptr, nullptr};
  int bm_words = 0;
  bool resident_ok = true;  // cleared if the device refuses the cooperative launch
  Ctl* ctl = nullptr;
  IterRec* recs = nullptr;
  int rec_cap = 0;
  int* srcs = nullptr;
  int srcs_cap = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev2 = nullptr, ev3 = nullptr;
  Ctl* h_ctl = nullptr;  // pinned
  int* h_stage = nullptr;  // pinned, kStageInts ints (results of small graphs on their way to the caller)
  bool staged = false;     // the last run's result has reached the caller's array
  std::map<ExecKey, ExecEntry> execs;
  std::map<const void*, int> grids;  // launch grids of the resident traversals' kernels
  unsigned grids_of = 0;             // g_carveout_set they belong to
  std::vector<cudaGraph_t> graphs;
  int last_iters = 0;
  // sweep scratch
  int* snap_dist = nullptr;
  unsigned* snap_bm = nullptr;
  int* snap_wl = nullptr;
  int* snap_hwl = nullptr;
  // degree-ordered copy (i2_graph_reorder): BFS and SSSP run on it, their
  // sources mapped by inv and their results gathered back to original IDs
  i2_graph* twin = nullptr;
  int* d_inv = nullptr;         // original ID -> copy's ID (device)
  std::vector<int> h_inv;       // the same on the host, to map sources
  bool last_on_twin = false;    // the last traversal ran on the copy (records)
};

namespace i2 {

// ---------------------------------------------------------------------------
// Device memory pool and pinned control blocks.

namespace {
struct DevPool {
  cudaMemPool_t pool = nullptr;
  cudaStream_t s = nullptr;  // allocations and frees are ordered on it
  cudaStream_t copy[2] = {nullptr, nullptr};  // uploads (several at once share them: each waits for both)
};
std::mutex g_pool_mu;
DevPool g_pools[64];
std::mutex g_ctl_mu;
std::vector<Ctl*> g_ctl_free;  // pinned host control blocks of freed graphs
}  // namespace

static DevPool* dev_pool() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    cudaGetLastError();
    return nullptr;
  }
  std::lock_guard<std::mutex> lk(g_pool_mu);
  DevPool& p = g_pools[dev];
  if (!p.pool) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    cudaStream_t s = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    unsigned long long keep = ~0ull;  // never hand reserved memory back on its own
    if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess ||
        cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) {
      cudaGetLastError();
      cudaMemPoolDestroy(pool);
      return nullptr;
    }
    for (cudaStream_t& cs : p.copy)
      if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        if (p.copy[0]) cudaStreamDestroy(p.copy[0]);
        p.copy[0] = p.copy[1] = nullptr;
        cudaStreamDestroy(s);
        cudaMemPoolDestroy(pool);
        return nullptr;
      }
    p.pool = pool;
    p.s = s;
  }
  return &p;
}

cudaError_t dev_alloc_bytes(void** ptr, size_t bytes) {
  *ptr = nullptr;
  DevPool* p = dev_pool();
  if (!p) return cudaErrorInitializationError;
  cudaError_t e = cudaMallocFromPoolAsync(ptr, bytes, p->pool, p->s);
  if (e == cudaErrorMemoryAllocation) {
    // Reserved but unused blocks may be too fragmented to serve the request:
    // hand them back and try once more.
    cudaGetLastError();
    cudaStreamSynchronize(p->s);
    cudaMemPoolTrimTo(p->pool, 0);
    e = cudaMallocFromPoolAsync(ptr, bytes, p->pool, p->s);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(p->s);  // usable by every stream from here
  if (e != cudaSuccess) *ptr = nullptr;
  return e;
}

static void dev_free_all(void* const* ptrs, int n) {
  DevPool* p = dev_pool();
  if (!p) return;
  bool waited = false;
  for (int k = 0; k < n; ++k) {
    if (!ptrs[k]) continue;
    if (!waited) cudaDeviceSynchronize();
    waited = true;
    cudaFreeAsync(ptrs[k], p->s);
  }
}

void dev_free(void* ptr) { dev_free_all(&ptr, 1); }

int dev_trim() {
  DevPool* p = dev_pool();
  if (!p) return I2_ERR_NO_DEVICE;
  I2_CK(cudaStreamSynchronize(p->s));
  I2_CK(cudaMemPoolTrimTo(p->pool, 0));
  return I2_OK;
}

static cudaError_t ctl_host_get(Ctl** out) {
  {
    std::lock_guard<std::mutex> lk(g_ctl_mu);
    if (!g_ctl_free.empty()) {
      *out = g_ctl_free.back();
      g_ctl_free.pop_back();
      return cudaSuccess;
    }
  }
  return cudaMallocHost(out, sizeof(Ctl));
}

static void ctl_host_put(Ctl* c) {
  if (!c) return;
  std::lock_guard<std::mutex> lk(g_ctl_mu);
  g_ctl_free.push_back(c);
}

// Results of up to kStageInts values go to the caller through a pinned block,
// copied with the report before its one wait for the device; a copy into
// pageable memory waits by itself after that. Blocks of freed graphs are kept
// for the next ones, at most kStageKept of them. Host BFS call, us, pinned /
// pageable: ER 1,000 106 / 115, 16,000 143 / 154, 65,000 175 / 186, 131,072 208 /
// 225, 262,144 275 / 288, 524,288 412 / 380, 10^6 631 / 545 (the host's copy out
// of the block is then the longer one). The limit keeps a graph's block at 256
// KB; up to 2^18 values would gain the same 10-16 us for four times that.
constexpr int kStageInts = 1 << 16;
constexpr size_t kStageKept = 16;
static std::mutex g_stage_mu;
static std::vector<int*> g_stage_free;

static bool stage_get(i2_graph* g) {
  if (g->g.nodes > kStageInts) return false;
  if (g->h_stage) return true;
  {
    std::lock_guard<std::mutex> lk(g_stage_mu);
    if (!g_stage_free.empty()) {
      g->h_stage = g_stage_free.back();
      g_stage_free.pop_back();
      return true;
    }
  }
  if (cudaMallocHost(&g->h_stage, sizeof(int) * kStageInts) == cudaSuccess) return true;
  cudaGetLastError();
  g->h_stage = nullptr;
  return false;
}

static void stage_put(i2_graph* g) {
  if (!g->h_stage) return;
  {
    std::lock_guard<std::mutex> lk(g_stage_mu);
    if (g_stage_free.size() < kStageKept) {
      g_stage_free.push_back(g->h_stage);
      g->h_stage = nullptr;
    }
  }
  if (g->h_stage) cudaFreeHost(g->h_stage);
  g->h_stage = nullptr;
}

static void drop_execs(i2_graph* g) {
  for (auto& kv : g->execs) cudaGraphExecDestroy(kv.second.ex);
  g->execs.clear();
  g->grids.clear();
}

static void free_graph_state(i2_graph* g) {
  drop_execs(g);
  for (auto gr : g->graphs) cudaGraphDestroy(gr);
  g->graphs.clear();
  // one wait for the device, then every block back to the pool
  void* blocks[] = {g->ws_base, g->heavy_base, g->pile[0],  g->pile[1], g->srcs,  g->snap_dist,
                    g->snap_bm, g->snap_wl,    g->snap_hwl, g->d_sp,    g->d_inv, nullptr,
                    nullptr,    nullptr};
  int nb = 11;
  if (g->owns) {
    blocks[nb++] = g->d_nindex;
    blocks[nb++] = g->d_nlist;
  }
  if (g->owns || g->owns_weights) blocks[nb++] = g->d_eweight;
  dev_free_all(blocks, nb);
  g->d_inv = nullptr;
  if (g->h_ctl) ctl_host_put(g->h_ctl);
  stage_put(g);
  if (g->ev0) cudaEventDestroy(g->ev0);
  if (g->ev1) cudaEventDestroy(g->ev1);
  if (g->ev2) cudaEventDestroy(g->ev2);
  if (g->ev3) cudaEventDestroy(g->ev3);
  if (g->stream) cudaStreamDestroy(g->stream);
  if (g->twin) i2_graph_free(g->twin);
  g->twin = nullptr;
}

static int compute_stats(i2_graph* g) {
  DevStats* st = nullptr;
  I2_CK(dev_alloc(&st, sizeof(DevStats)));
  static_assert(sizeof(DevStats) <= sizeof(Ctl), "read back through the pinned control block");
  DevStats& h = *reinterpret_cast<DevStats*>(g->h_ctl);
  cudaError_t e = cudaMemsetAsync(st, 0, sizeof(DevStats), g->stream);
  if (e == cudaSuccess) {
    k_degree_stats<<<4 * sm_count(), 256, 0, g->stream>>>(g->g, g->heavy, st);
    e = cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, g->stream);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
  dev_free(st);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return cuda_status(e);
  }
  GStats& s = g->gs;
  s.nodes = g->g.nodes;
  s.edges = g->g.edges;
  s.maxdeg = (int)(h.hub >> 32);
  g->hub = (int)~(unsigned)h.hub;
  s.nheavy = (int)(h.counts >> 32);
  s.linked = (int)(unsigned)h.counts;
  s.first = s.linked ? INT_MAX - (int)h.firstinv : kInf;
  s.wmin = g->g.eweight && h.winv ? (int)((unsigned)INT_MAX - h.winv) : 1;
  s.symmetric = -1;  // decided on first need (ensure_symmetry)
  const double mean = (double)g->g.edges / (double)g->g.nodes;
  const double var = std::max(0.0, h.sumsq / (double)g->g.nodes - mean * mean);
  s.avgdeg = (float)mean;
  s.degcv = mean > 0 ? (float)(std::sqrt(var) / mean) : 0.f;
  s.wmean = (g->g.eweight && g->g.edges > 0) ? (float)(h.wsum / (double)g->g.edges) : 1.f;
  return I2_OK;
}

static int finish_setup(i2_graph* g) {
  I2_CK(cudaGetDevice(&g->device));
  I2_CK(cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking));
  I2_CK(cudaEventCreate(&g->ev0));
  I2_CK(cudaEventCreate(&g->ev1));
  I2_CK(cudaEventCreate(&g->ev2));
  I2_CK(cudaEventCreate(&g->ev3));
  I2_CK(ctl_host_get(&g->h_ctl));
  g->g.vec_ok = ((((uintptr_t)g->g.nlist) & 15) == 0 && (((uintptr_t)g->g.eweight) & 15) == 0) ? 1 : 0;
  return compute_stats(g);
}

// Words of the bitmap block: 4 bitmaps, then (8-byte aligned) the two
// distance histograms of the budgeted near/far ordering.
static size_t hist_offset_words(const i2_graph* g) { return (4ull * g->bm_words + 1) & ~1ull; }
static size_t bm_block_words(const i2_graph* g) { return hist_offset_words(g) + 2ull * 2 * kHistBins; }

// The three frontiers' heavy lists, one block for the six arrays.
static int alloc_heavy(i2_graph* g) {
  if (g->heavy_base) return I2_OK;
  const size_t n = ((size_t)std::max(1, g->gs.nheavy) + 63) & ~(size_t)63;  // 256-byte boundaries
  I2_CK(dev_alloc(&g->heavy_base, sizeof(int) * 6 * n));
  for (int k = 0; k < 3; ++k) {
    g->hwl[k] = reinterpret_cast<int*>(g->heavy_base) + (size_t)(2 * k) * n;
    g->htoff[k] = reinterpret_cast<unsigned*>(g->heavy_base) + (size_t)(2 * k + 1) * n;
  }
  return I2_OK;
}

static int ensure_workspace(i2_graph* g) {
  if (g->ws_ready) return I2_OK;
  const long long V = g->g.nodes;
  g->bm_words = (int)((V + 31) / 32);
  g->rec_cap = (int)std::min<long long>(V + 2, 1 << 16);
  int st = alloc_heavy(g);
  if (st) return st;
  // one block, every array on a 256-byte boundary
  size_t at = 0;
  const auto take = [&](size_t bytes) {
    const size_t o = at;
    at += (bytes + 255) & ~(size_t)255;
    return o;
  };
  const size_t o_dist = take(sizeof(int) * V);
  size_t o_wl[3], o_off[3];
  for (int k = 0; k < 3; ++k) {
    o_wl[k] = take(sizeof(int) * V);
    o_off[k] = take(sizeof(unsigned) * V);
  }
  // the three frontier bitmaps, the far-pile bitmap and the near/far distance
  // histograms (cleared together before every run)
  const size_t o_bm = take(sizeof(unsigned) * bm_block_words(g));
  const size_t o_ctl = take(sizeof(Ctl));
  const size_t o_recs = take(sizeof(IterRec) * g->rec_cap);
  I2_CK(dev_alloc(&g->ws_base, at));
  const auto ptr = [&](size_t o) { return static_cast<void*>(g->ws_base + o); };
  g->dist = static_cast<int*>(ptr(o_dist));
  for (int k = 0; k < 3; ++k) {
    g->wl[k] = static_cast<int*>(ptr(o_wl[k]));
    g->woff[k] = static_cast<unsigned*>(ptr(o_off[k]));
  }
  unsigned* bm = static_cast<unsigned*>(ptr(o_bm));
  for (int k = 0; k < 3; ++k) g->bm[k] = bm + (size_t)k * g->bm_words;
  g->fbm = bm + 3ull * g->bm_words;
  g->hist = reinterpret_cast<unsigned long long*>(bm + hist_offset_words(g));
  g->ctl = static_cast<Ctl*>(ptr(o_ctl));
  g->recs = static_cast<IterRec*>(ptr(o_recs));
  g->ws_ready = true;
  return I2_OK;
}

static size_t pile_capacity(const i2_graph* g) { return (size_t)g->g.nodes + 1; }

static int ensure_piles(i2_graph* g) {
  if (g->pile[0]) return I2_OK;
  // each pile: nodes + 1 vertices, then their degrees (a full pile sends
  // vertices to the next frontier instead)
  for (int k = 0; k < 2; ++k) I2_CK(dev_alloc(&g->pile[k], sizeof(int) * 2 * pile_capacity(g)));
  drop_execs(g);  // graphs bake the context
  return I2_OK;
}

static int ensure_sp(i2_graph* g) {
  if (g->d_sp) return I2_OK;
  I2_CK(dev_alloc(&g->d_sp, sizeof(int) * ((size_t)g->g.edges + 4)));
  k_build_sp<<<8 * sm_count(), 256, 0, g->stream>>>(g->g, g->d_sp);
  I2_CK(cudaStreamSynchronize(g->stream));
  g->g.sp = g->d_sp;
  return I2_OK;
}

// Pull variants read a vertex's out-list as its in-list, so they need every
// (u, v, w) to have a (v, u, w) partner. Checked once, on first need.
static int ensure_symmetry(i2_graph* g) {
  if (g->gs.symmetric >= 0) return I2_OK;
  int st = ensure_sp(g);
  if (st) return st;
  DevStats* d = nullptr;
  I2_CK(dev_alloc(&d, sizeof(DevStats)));
  DevStats h{};
  cudaMemcpy(d, &h, sizeof(h), cudaMemcpyHostToDevice);
  const int grid = 8 * sm_count();
  k_sorted<<<grid, 256, 0, g->stream>>>(g->g, g->d_sp, d);
  cudaStreamSynchronize(g->stream);
  cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
  if (!h.unsorted) {
    k_symmetry<<<grid, 256, 0, g->stream>>>(g->g, g->d_sp, d);
    cudaStreamSynchronize(g->stream);
    cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
  }
  cudaError_t e = cudaGetLastError();
  dev_free(d);
  if (e != cudaSuccess) return cuda_status(e);
  g->gs.symmetric = (!h.unsorted && !h.asym) ? 1 : 0;
  drop_execs(g);  // graphs bake the statistics into their arguments
  return I2_OK;
}

// Styles applicable to this graph and algorithm: pull and union-find read a
// vertex's out-list as its in-list (symmetric graphs only), the edge sweeps
// need sp[], and union-find computes CC labels only.
// Smallest graph (vertices) on which the selectors' union-find CC runs as
// union-find's own kernel (run_traversal). The line was drawn before that kernel
// chose its blocks by the graph's size; below it, us, own kernel / the selectors':
// RMAT-20 145 / 168, ER 600,000 159 / 176, ER 2 x 10^6 199 / 200, grid 300^2 116 /
// 122, 1000^2 146 / 142, 2000^2 224 / 266. It has not been moved.
constexpr long long kUnionFindKernelNodes = 1LL << 22;

// Whether the learned selector picks styles here. Where it defers to the rule for
// the whole traversal (no parameters, or a graph larger than any it was trained
// on) the traversal is the rule's, by the rule's kernels (SSSP on a grid of
// 6000^2, ms: 52.4 as the rule's, 59.7 in the selectors' kernel).
// SSSP on graphs of skewed degrees is the rule's too: the network mostly picks
// the rule's style there, whose own kernel has more blocks and the long tiles, and
// where it picks another it loses. us, by the network / the rule: RMAT-20 786 / 658,
// RMAT-18 307 / 282, RMAT-12 184 / 144, RMAT-20 with edge factor 4 2,942 / 385, 32
// 1,282 / 944, power-law pairs on 10^6 vertices 1,462 / 987; of 33 graphs of 2^10 to
// 2^21 vertices none was faster by the network.
static bool learned_here(const i2_graph* g, int algo) {
  return mlp_device_params() && (long long)g->g.nodes <= kMaxTrainedNodes &&
         !(algo == I2_SSSP && g->gs.degcv > 1.f);
}

// Whether the selectors run in the form compiled for more resident blocks.
static bool wide_selector(const i2_graph* g) { return (long long)g->g.nodes >= kWideSelectorNodes; }

// Whether a resident traversal takes its kernel's form for more resident blocks
// per SM. The selectors': graphs of kWideSelectorNodes vertices or more. The
// edge-balanced style: graphs of skewed degrees, where the tiles of the hubs
// keep more warps busy than 5 blocks have, at the price of spills that cost the
// short iterations of other graphs. us, 6 / 5 blocks: SSSP RMAT 10^6 678 / 711,
// 4 x 10^6 2,102 / 2,204, 25 x 10^6 degree-ordered 10,122 / 10,978; CC RMAT
// 4 x 10^6 1,854 / 2,104, 25 x 10^6 ordered 11,630 / 12,792; but ER 2 x 10^6
// SSSP 1,388 / 1,367, CC 1,104 / 966, grid 10^6 SSSP 2,358 / 2,078.
static bool wide_form(const i2_graph* g, int variant) {
  return variant == kVPCta ? g->gs.degcv > 1.f : wide_selector(g);
}

// Most resident blocks per SM of a style's kernel on this graph. The
// edge-balanced push of BFS and SSSP takes 4 of the 5 it is compiled for on
// sparse graphs of even degrees (average below 6: grids, road networks) of 2^24
// vertices and more, where the blocks push one another's lines out of L2. 5 / 4
// blocks: SSSP grid 7000^2 70.5 / 65.8 ms, 6000^2 52.2 / 48.6, 5000^2 28.7 / 26.8,
// ER 4 x 10^7 with 4 entries a vertex 21.9 / 21.2, BFS grid 6000^2 5.76 / 5.56. ER
// with 8 entries a vertex gains nothing (2^24 BFS 2.35 / 2.40) and CC, whose first
// iteration holds every vertex, loses (ER 4 x 10^7 with 4 entries 39.8 / 41.9).
// Smaller sparse graphs would gain too (grid 2000^2 SSSP 4.47 / 4.31, BFS 1.71 /
// 1.60); there the line is with the learned selector, which would then lose to the
// rule on grids (its picks are from times at 5 blocks).
// Union-find on graphs of average degree 6 or more takes about one block per SM
// for every 2^11 vertices an SM has, 8 chunks a warp: more warps link trees that the
// others have not joined yet, and meet at the same roots. Sparser graphs have few
// links at a time and keep every block (a caterpillar of 4 x 10^5 vertices 92, 125-168
// by size). us, 1 / 2 / 3 / 4 / 6 blocks: RMAT-17 110 / 122 / 153 /
// 193 / 204, RMAT-18 117 / 172 / 198 / 215 / 305, RMAT-20 171 / 140 / 144 / 168 /
// 187, RMAT-22 473 / 295 / 235 / 213 / 186, ER 3 x 10^5 139 / 138 / 200 / 255 /
// 371, 6 x 10^5 175 / 170 / 163 / 192 / 301, 2 x 10^6 304 / 219 / 200 / 192 / 195;
// grid 300^2 121 / 108 / 112 / 134 / 116, 2000^2 705 / 408 / 312 / 262 / 224.
static int style_blocks(const i2_graph* g, int algo, int variant) {
  if (variant == kUnionFind) {
    const long long per_block = 8LL * kWarp * kWarpsPerBlock, sms = sm_count();
    const long long blocks = (g->g.nodes + per_block * sms / 2) / (per_block * sms);
    const long long most = std::min(g->blocks_per_sm, I2_UF_MIN_BLOCKS);
    return (int)(g->gs.avgdeg < 6.f ? most : std::min(std::max(1LL, blocks), most));
  }
  const bool sparse = variant == kVPCta && (algo == I2_BFS || algo == I2_SSSP) && g->g.nodes >= (1 << 24) &&
                      g->gs.degcv <= 1.f && g->gs.avgdeg < 6.f;
  return sparse ? std::min(g->blocks_per_sm, 4) : g->blocks_per_sm;
}

static int allowed_mask(const i2_graph* g, int algo) {
  int m = 0;
  for (int v = 0; v < kNumVariants; ++v) m |= 1 << v;
  if (g->gs.symmetric != 1) m &= ~((1 << kPullFrontier) | (1 << kPullTopo) | (1 << kUnionFind));
  if (!g->d_sp) m &= ~(1 << kEdgeTopo);
  if (algo != I2_CC) m &= ~(1 << kUnionFind);
  return m;
}

static Ctx make_ctx(const i2_graph* g) {
  Ctx c{};
  c.g = g->g;
  c.gs = g->gs;
  c.dist = g->dist;
  for (int k = 0; k < 3; ++k) {
    c.wl[k] = g->wl[k];
    c.woff[k] = g->woff[k];
    c.hwl[k] = g->hwl[k];
    c.htoff[k] = g->htoff[k];
    c.bm[k] = g->bm[k];
  }
  c.ctl = g->ctl;
  c.recs = g->recs;
  c.rec_cap = g->rec_cap;
  c.heavy = g->heavy;
  c.bm_words = g->bm_words;
  c.pile_cap = (unsigned)std::min<size_t>(pile_capacity(g), 0xffffffffu);
  for (int k = 0; k < 2; ++k) {
    c.pile[k] = g->pile[k];
    c.pdeg[k] = g->pile[k] ? g->pile[k] + pile_capacity(g) : nullptr;
  }
  c.fbm = g->fbm;
  c.hist = g->hist;
  c.mlp = mlp_device_params();
  c.srcs = nullptr;
  return c;
}

// Default edge budget of the near/far ordering per SM (I2_SSSP_BUDGET_AUTO):
// about 7 warp tiles for each resident warp of the edge-balanced kernel.
// RMAT-22 SSSP (ms, device-timed): plain 2.57; budget 1M 2.95, 2M 2.57,
// 4M 2.38, 8M 2.60, 16M 2.97 edges.
constexpr int kBudgetEdgesPerSM = 28672;

// Near/far ordering applies to SSSP with the fixed edge-balanced push only
// (the style that implements the split launches). Returns the ordering's
// Ctl::delta: > 0 a fixed threshold step, < 0 minus an edge budget, 0 off.
// A fixed step relaxes up to 2.2x fewer edges on RMAT graphs, but the step
// that wins moves with the graph. The edge budget instead keeps each near
// frontier at about B edges: enough to fill the GPU, few enough that
// distances settle before their vertices relax.
// Smallest graph (CSR entries) on which the selectors' SSSP takes the budgeted
// ordering (skewed degrees only; see run_traversal).
constexpr long long kBudgetRuleEdges = 1LL << 26;

static int pick_order(const i2_graph* g, int algo, int mode, int variant, int step, int budget) {
  if (algo != I2_SSSP || mode != 0 || variant != kVPCta) return 0;
  if (step > 0) return step;
  if (budget == I2_SSSP_BUDGET_AUTO) {
    // Twice the budget on graphs of 2^30 CSR entries or more. RMAT-26 on its
    // degree-ordered copy, per traversal: 35.9 ms at the base budget (4.2 M
    // edges), 34.6 at 6 M, 34.1 at 8.4 M, 34.2 at 10 M, 35.7 at 12 M; on
    // RMAT-22 (2^27 entries) the base budget is the fastest.
    int b = std::max(1 << 16, sm_count() * kBudgetEdgesPerSM);
    if ((long long)g->g.edges >= (1LL << 30)) b *= 2;
    return -b;
  }
  if (budget > 0) return -budget;
  return 0;
}

// Histogram bin width of the edge budget: the largest power of two not above
// the smallest weight, the step by which distances grow per hop. (On RMAT-22
// with weights in [1, 255] most distances from the hub are below 32: the
// minimum over many paths takes the light edges, so bins sized by the mean
// weight put the whole budget quantile into the first bin.)
static int budget_shift(const i2_graph* g) {
  const int wm = g->gs.wmin > 1 ? g->gs.wmin : 1;
  int s = 0;
  while ((2LL << s) <= wm) ++s;  // floor(log2(wmin))
  return s;
}

// Whether union-find links in ascending order (body_union): on graphs of low
// average degree, and on graphs numbered with the hubs in front (the
// degree-ordered copies among them), where the first vertices' links already
// tie most of the graph to the smallest IDs. First launch, us, ascending /
// spread, on degree-ordered copies: RMAT 10^6 33 / 294, 9 x 10^6 123 / 362,
// 25 x 10^6 253 / 511. Whole run: degree-ordered RMAT-18 84 / 174, RMAT-20 140 /
// 336; pairs whose ends' IDs fall like a power p of a uniform number, 2 x 10^6
// vertices: p = 4 154 / 290, p = 2 187 / 258, p = 1.7 194 / 355, p = 1.3 289-382 /
// 187-289. A hub in the first 64th by chance (RMAT-16 to 20, within the noise;
// RMAT-20 up to 1.4x for spread) is why the line lies as low as 1/256.
static bool union_in_order(const i2_graph* g) {
  return g->gs.avgdeg < 6.f || g->hub < g->g.nodes / 256;
}

// A step near the golden section of n that is coprime to n: multiples of it
// mod n visit every index once, neighbours in time far apart (union-find).
static unsigned spread_step(unsigned n) {
  unsigned s = (unsigned)(n * 0.6180339887498949) | 1u;
  while (s < 3 || std::gcd(s, n) != 1) s += 2;  // 1 means ascending order
  return s;
}

static RunParams make_params(const i2_graph* g, int algo, int mode, int variant, int src, int nsrc, int cap,
                             int delta = 0) {
  RunParams p{};
  p.algo = algo;
  p.mode = mode;
  p.fixed_variant = variant < 0 ? 0 : variant;
  p.allowed = allowed_mask(g, algo);
  p.src = src;
  p.nsrc = nsrc;
  p.delta = delta;
  p.hshift = budget_shift(g);
  p.uf_step = algo != I2_CC ? 0 : union_in_order(g) ? 1u : spread_step((unsigned)((g->g.nodes + 31LL) / 32));
  // Test hook: withhold the first barrier release of a resident traversal,
  // so that every block's bounded wait runs out (I2_STALL_MS bounds it).
  const char* hold = std::getenv("I2_TEST_HOLD_BARRIER");
  p.hold = (hold && hold[0] == '1') ? 1 : 0;
  const char* stall = std::getenv("I2_STALL_MS");
  p.stall_ms = stall ? std::max(1, std::atoi(stall)) : 10000;
  // a split launch moves at least one pile entry into a frontier, or learns
  // the pile's exact minimum for the next one
  p.iter_cap = cap > 0 ? cap : (int)std::min<long long>((long long)g->g.nodes * (delta != 0 ? 3 : 1) + 2, INT_MAX);
  return p;
}

static int add_kernel_node(cudaGraph_t gr, cudaGraphNode_t* node, const cudaGraphNode_t* deps, int ndeps,
                           KernelFn fn, int grid, Ctx* ctx) {
  cudaKernelNodeParams p{};
  p.func = (void*)fn;
  p.gridDim = dim3(grid);
  p.blockDim = dim3(kBlock);
  p.sharedMemBytes = 0;
  void* args[1] = {ctx};
  p.kernelParams = args;
  p.extra = nullptr;
  I2_CK(cudaGraphAddKernelNode(node, gr, deps, ndeps, &p));
  return I2_OK;
}

static int build_exec(i2_graph* g, int algo, int mode, int variant, bool multi, const RunParams& rp,
                      ExecEntry** out) {
  ExecKey key{algo, mode, mode == 0 ? variant : -1, multi ? 1 : 0, rp.delta != 0 ? 1 : 0};
  auto it = g->execs.find(key);
  if (it != g->execs.end()) {
    *out = &it->second;
    return I2_OK;
  }
  cudaGraph_t gr;
  I2_CK(cudaGraphCreate(&gr, 0));
  g->graphs.push_back(gr);
  cudaGraphConditionalHandle loop_h;
  I2_CK(cudaGraphConditionalHandleCreate(&loop_h, gr, 1, cudaGraphCondAssignDefault));
  Ctx c = make_ctx(g);
  c.srcs = multi ? g->srcs : nullptr;
  c.loop_h = (unsigned long long)loop_h;
  c.use_loop = 1;
  // bitmaps <- 0
  cudaGraphNode_t n_ms, n_reset, n_fill, n_seed, n_loop;
  cudaMemsetParams ms{};
  ms.dst = g->bm[0];
  ms.value = 0;
  ms.elementSize = 4;
  ms.width = bm_block_words(g);  // frontier and far-pile bitmaps, histograms
  ms.height = 1;
  ms.pitch = 0;
  I2_CK(cudaGraphAddMemsetNode(&n_ms, gr, nullptr, 0, &ms));
  // control block <- run parameters
  {
    cudaKernelNodeParams kp{};
    Ctl* ctl = g->ctl;
    RunParams p = rp;
    void* args[2] = {&ctl, &p};
    kp.func = (void*)k_reset;
    kp.gridDim = dim3(1);
    kp.blockDim = dim3(32);
    kp.kernelParams = args;
    I2_CK(cudaGraphAddKernelNode(&n_reset, gr, &n_ms, 1, &kp));
  }
  int st = add_kernel_node(gr, &n_fill, &n_reset, 1, fill_kernel(algo), grid_for(fill_kernel(algo), 8), &c);
  if (st) return st;
  st = add_kernel_node(gr, &n_seed, &n_fill, 1, seed_kernel(algo), 1, &c);
  if (st) return st;
  cudaGraphNodeParams cp{};
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = loop_h;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  I2_CK(cudaGraphAddNode(&n_loop, gr, &n_seed, 1, &cp));
  cudaGraph_t body = cp.conditional.phGraph_out[0];
  // The loop body is one kernel, launched once per iteration: the fixed style's,
  // or the dispatch kernel whose blocks branch on the style the previous
  // iteration selected.
  {
    cudaGraphNode_t n;
    KernelFn fn = mode == 0 ? relax_kernel(algo, 0, variant, rp.delta != 0, wide_form(g, variant))
                            : dispatch_kernel(algo, wide_selector(g));
    st = add_kernel_node(body, &n, nullptr, 0, fn, grid_for(fn, style_blocks(g, algo, mode == 0 ? variant : -1)), &c);
    if (st) return st;
  }
  ExecEntry e;
  I2_CK(cudaGraphInstantiate(&e.ex, gr, 0));
  e.reset = n_reset;
  e.last = rp;
  e.ctx = c;
  auto ins = g->execs.emplace(key, e);
  *out = &ins.first->second;
  return I2_OK;
}

// Launch the traversal graph with this run's parameters. Changing the reset
// node's arguments affects only launches made after the change.
static int launch_exec(i2_graph* g, ExecEntry* e, const RunParams& rp, cudaStream_t s) {
  if (e->last != rp) {
    cudaKernelNodeParams kp{};
    Ctl* ctl = g->ctl;
    RunParams p = rp;
    void* args[2] = {&ctl, &p};
    kp.func = (void*)k_reset;
    kp.gridDim = dim3(1);
    kp.blockDim = dim3(32);
    kp.kernelParams = args;
    I2_CK(cudaGraphExecKernelNodeSetParams(e->ex, e->reset, &kp));
    e->last = rp;
  }
  I2_CK(cudaGraphLaunch(e->ex, s));
  return I2_OK;
}

typedef void (*StartFn)(Ctx, RunParams, unsigned);
static StartFn start_kernel(int algo) {
  if (algo == kBFS) return k_start<kBFS>;
  if (algo == kSSSP) return k_start<kSSSP>;
  if (algo == kCC) return k_start<kCC>;
  return k_start<kMIS>;
}

// The kernels of a resident traversal and their grids.
struct ResidentPlan {
  KernelFn loop = nullptr;   // every iteration, one cooperative launch
  KernelFn fill = nullptr;   // a first frontier of many vertices (else null)
  KernelFn seed = nullptr;   // its seeding, or that of many sources (else null)
  StartFn start = nullptr;
  int loop_grid = 0, loop_blocks = 0, fill_grid = 0, start_grid = 0;
};

// Looks the kernels up before the traversal's first event: a kernel's first use
// in a process loads it (0.5-15 ms), which the report's device time must not hold.
static ResidentPlan plan_resident(i2_graph* g, int algo, int mode, int variant, bool multi, const RunParams& rp) {
  const unsigned set = g_carveout_set.load();
  if (g->grids_of != set) g->grids.clear();
  g->grids_of = set;
  const auto grid = [g](const void* fn, int max_per_sm) {
    auto it = g->grids.find(fn);
    if (it == g->grids.end()) it = g->grids.emplace(fn, grid_for((KernelFn)fn, max_per_sm)).first;
    return it->second;
  };
  const auto load = [g](const void* fn) {
    if (g->grids.count(fn)) return;
    g->grids.emplace(fn, 0);
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, fn) != cudaSuccess) cudaGetLastError();  // its launch reports it
  };
  ResidentPlan p;
  const int v = mode == 0 ? variant : -1;
  p.loop = resident_kernel(algo, v, rp.delta != 0, wide_form(g, v));
  p.loop_blocks = style_blocks(g, algo, v);
  p.loop_grid = grid((const void*)p.loop, p.loop_blocks);
  p.start = start_kernel(algo);
  load((const void*)p.start);
  const long long units = (long long)g->g.nodes / 4 + (long long)bm_block_words(g);
  p.start_grid = (int)std::max(1LL, std::min(8LL * sm_count(), units / (4 * kBlock)));
  const bool frontier = algo == I2_CC && !rp.whole;
  if (frontier) {
    p.fill = fill_kernel(algo);
    p.fill_grid = grid((const void*)p.fill, 8);
  }
  if (frontier || multi) {
    p.seed = seed_kernel(algo);
    load((const void*)p.seed);
  }
  return p;
}

// A resident traversal: its start (one kernel; with the frontier's own kernels
// where many vertices are in it), and one cooperative launch that runs every
// iteration.
static cudaError_t launch_resident(i2_graph* g, const ResidentPlan& p, bool multi, const RunParams& rp,
                                   cudaStream_t s) {
  Ctx c = make_ctx(g);
  c.srcs = multi ? g->srcs : nullptr;
  p.start<<<p.start_grid, kBlock, 0, s>>>(c, rp, (unsigned)bm_block_words(g));
  if (p.fill) p.fill<<<p.fill_grid, kBlock, 0, s>>>(c);
  if (p.seed) p.seed<<<1, kBlock, 0, s>>>(c);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  void* args[1] = {&c};
  e = cudaLaunchCooperativeKernel((const void*)p.loop, dim3(p.loop_grid), dim3(kBlock), args, 0, s);
  if (e == cudaErrorCooperativeLaunchTooLarge) {  // another thread changed the carveout meanwhile
    cudaGetLastError();
    const int grid = g->grids[(const void*)p.loop] = grid_for(p.loop, p.loop_blocks);
    e = cudaLaunchCooperativeKernel((const void*)p.loop, dim3(grid), dim3(kBlock), args, 0, s);
  }
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

// Reset the bitmaps and the control block on the stream (host-driven paths).
static int prepare_run(i2_graph* g, cudaStream_t s, const RunParams& rp) {
  I2_CK(cudaMemsetAsync(g->bm[0], 0, sizeof(unsigned) * bm_block_words(g), s));
  k_reset<<<1, 32, 0, s>>>(g->ctl, rp);
  I2_CK(cudaGetLastError());
  return I2_OK;
}

// Host-driven loop (one control-block read per iteration, like the reference's
// do-while). Each relax launch is bracketed by CUDA events on the launching
// stream; their sum is returned in *relax_ms.
static int run_host_loop(i2_graph* g, cudaStream_t s, int algo, bool multi, double* relax_ms) {
  Ctx c = make_ctx(g);
  c.srcs = multi ? g->srcs : nullptr;
  KernelFn ff = fill_kernel(algo);
  ff<<<grid_for(ff, 8), kBlock, 0, s>>>(c);
  seed_kernel(algo)<<<1, kBlock, 0, s>>>(c);
  Ctl* h = g->h_ctl;
  double total = 0.0;
  for (;;) {
    I2_CK(cudaMemcpyAsync(h, g->ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s));
    I2_CK(cudaStreamSynchronize(s));
    // the last launch's decision: another frontier, a near/far split, the
    // compress launch of union-find, or the end (including the iteration cap)
    if (!h->go || (h->status & kStatusIterCap)) break;
    KernelFn fn = relax_kernel(algo, h->mode, h->variant, h->delta != 0, wide_form(g, h->variant));
    I2_CK(cudaEventRecord(g->ev2, s));
    fn<<<grid_for(fn, style_blocks(g, algo, h->variant)), kBlock, 0, s>>>(c);
    I2_CK(cudaGetLastError());
    I2_CK(cudaEventRecord(g->ev3, s));
    I2_CK(cudaEventSynchronize(g->ev3));
    float ms = 0.f;
    I2_CK(cudaEventElapsedTime(&ms, g->ev2, g->ev3));
    total += ms;
  }
  *relax_ms = total;
  return I2_OK;
}

static int fill_report(i2_graph* g, cudaStream_t s, int algo, i2_report* rep, double host_relax_ms, int* host_out) {
  // the counts join the control block (zeroed when the run began): one copy back
  k_reached<<<std::min(4 * sm_count(), g->g.nodes / 1024 + 1), 256, 0, s>>>(g->g, g->dist, g->ctl->reached);
  I2_CK(cudaGetLastError());
  I2_CK(cudaMemcpyAsync(g->h_ctl, g->ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s));
  if (host_out && stage_get(g))
    I2_CK(cudaMemcpyAsync(g->h_stage, g->dist, sizeof(int) * (size_t)g->g.nodes, cudaMemcpyDeviceToHost, s));
  I2_CK(cudaStreamSynchronize(s));
  if (host_out && g->h_stage && !(g->h_ctl->status & kStatusStall)) {
    std::memcpy(host_out, g->h_stage, sizeof(int) * (size_t)g->g.nodes);
    g->staged = true;
  }
  const Ctl* h = g->h_ctl;
  g->last_iters = h->iter;
  if (rep) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, g->ev0, g->ev1);
    rep->seconds = ms * 1e-3;
    rep->relax_seconds = host_relax_ms >= 0.0 ? host_relax_ms * 1e-3 : h->relax_ns * 1e-9;
    rep->iterations = h->iter;
    for (int k = 0; k < 16; ++k) rep->variant_hist[k] = h->hist[k];
    rep->reached_vertices = (long long)h->reached[0];
    rep->reached_edges = (long long)h->reached[1];
  }
  if (h->status & kStatusStall) return I2_ERR_STALL;
  if (h->status & kStatusIterCap) return I2_ERR_ITER_CAP;
  (void)algo;
  return I2_OK;
}

// BFS, SSSP or (symmetric graphs) CC of a graph that has a degree-ordered
// copy: the traversal runs on the copy (same options, on the caller's stream
// or the graph's), from the mapped sources, and a gather puts its values into
// this graph's result buffer in original IDs. Levels and distances do not
// depend on the numbering, so the result is the one the original CSR gives;
// CC labels are mapped to each component's smallest original ID. The
// report's seconds are the copy's (init and iterations) plus the mapping's.
static int run_on_twin(i2_graph* g, int algo, int src, const int* srcs_host, int nsrc, const i2_opts* opts,
                       i2_report* rep) {
  std::vector<int> mapped;
  if (srcs_host) {
    if (nsrc < 1) return I2_ERR_ARG;
    mapped.resize(nsrc);
    for (int j = 0; j < nsrc; ++j) {
      if (srcs_host[j] < 0 || srcs_host[j] >= g->g.nodes) return I2_ERR_ARG;
      mapped[j] = g->h_inv[srcs_host[j]];
    }
  } else if (src < 0 || src >= g->g.nodes) {
    return I2_ERR_ARG;
  }
  int st = ensure_workspace(g);
  if (st) return st;
  i2_opts o{};
  if (opts) o = *opts;
  cudaStream_t s = o.stream ? (cudaStream_t)o.stream : g->stream;
  o.stream = (void*)s;
  st = run_traversal(g->twin, algo, srcs_host ? 0 : g->h_inv[src], srcs_host ? mapped.data() : nullptr, nsrc, &o,
                     rep);
  if (st && st != I2_ERR_ITER_CAP) return st;
  g->last_on_twin = true;
  g->last_iters = g->twin->last_iters;
  const int n = g->g.nodes;
  if (rep) I2_CK(cudaEventRecord(g->ev2, s));
  const int grid = (int)std::min<long long>(4LL * sm_count(), (n + 255) / 256);
  if (algo == I2_CC) {
    int* mn = g->wl[0];  // free while the original CSR is not traversed
    k_cc_min_init<<<grid, 256, 0, s>>>(mn, n);
    k_cc_min_original<<<grid, 256, 0, s>>>(g->twin->dist, g->d_inv, n, mn);
    k_cc_labels<<<grid, 256, 0, s>>>(g->twin->dist, g->d_inv, mn, n, g->dist);
  } else {
    k_unpermute<<<grid, 256, 0, s>>>(g->twin->dist, g->d_inv, n, g->dist);
  }
  I2_CK(cudaGetLastError());
  if (rep) {  // the copy's traversal time (its report) plus the mapping
    I2_CK(cudaEventRecord(g->ev3, s));
    I2_CK(cudaEventSynchronize(g->ev3));
    float ms = 0.f;
    I2_CK(cudaEventElapsedTime(&ms, g->ev2, g->ev3));
    rep->seconds += ms * 1e-3;
  }
  return st;
}

int run_traversal(i2_graph* g, int algo, int src, const int* srcs_host, int nsrc, const i2_opts* opts,
                  i2_report* rep, int* host_out) {
  if (!g) return I2_ERR_ARG;
  if (algo < I2_BFS || algo > I2_MIS) return I2_ERR_ARG;
  g->staged = false;
  I2_CK(cudaSetDevice(g->device));
  if (g->twin && (algo == I2_BFS || algo == I2_SSSP)) return run_on_twin(g, algo, src, srcs_host, nsrc, opts, rep);
  if (g->twin && algo == I2_CC) {
    // A component's smallest original ID follows from the copy's labels only
    // where components are the same vertex sets in both (symmetric edges);
    // the copy's adjacency is sorted, so its check decides set symmetry.
    int st = ensure_symmetry(g->twin);
    if (st) return st;
    if (g->twin->gs.symmetric == 1) return run_on_twin(g, algo, 0, nullptr, 0, opts, rep);
  }
  g->last_on_twin = false;
  i2_opts o{};
  if (opts) o = *opts;
  if (o.loop_mode < I2_LOOP_GRAPH || o.loop_mode > I2_LOOP_RELAUNCH) return I2_ERR_ARG;
  const bool sourced = algo == I2_BFS || algo == I2_SSSP;
  if (sourced && !srcs_host && (src < 0 || src >= g->g.nodes)) return I2_ERR_ARG;
  if (algo == I2_SSSP) {
    if (!g->g.eweight) return I2_ERR_ARG;
    if (g->gs.wmin < 0) return I2_ERR_UNSUPPORTED;
  }
  int st = ensure_workspace(g);
  if (st) return st;
  if (algo == I2_MIS) {  // one style; the set is defined on undirected graphs
    st = ensure_symmetry(g);
    if (st) return st;
    if (g->gs.symmetric != 1) return I2_ERR_UNSUPPORTED;
    o.variant = kVPWarp;
    o.then_at = 0;
    o.sssp_delta = 0;
    o.sssp_budget = 0;
  }
  int mode = 0, variant = o.variant;
  if (variant == I2_AUTO_HEURISTIC) mode = 1;
  else if (variant == I2_AUTO_LEARNED) mode = learned_here(g, algo) ? 2 : 1;
  else if (variant < 0 || variant >= kNumVariants) return I2_ERR_ARG;
  if (o.then_at < 0) return I2_ERR_ARG;
  if (o.then_at > 0) {  // a fixed switch of style: per-iteration dispatch
    if (mode != 0 || o.then_variant < 0 || o.then_variant >= kNumVariants) return I2_ERR_ARG;
    mode = 3;
  }
  // SSSP on a graph of skewed degrees (coefficient of variation above 1) with
  // 2^26 CSR entries or more, from one source: both selectors run the
  // edge-balanced push in the budgeted near/far ordering for the whole
  // traversal (the per-iteration styles cannot take part in its moves and
  // trims). us, plain / budgeted: RMAT-22 2,120 / 1,901, RMAT-23 4,367 / 3,403,
  // RMAT-26 in degree order 45,829 / 29,035, RMAT-21 1,144 / 1,131; but RMAT-20 654 /
  // 772, RMAT-18 283 / 328, ER 2^22 2,405 / 2,787, grid 2048^2 4,242 / 4,895, which
  // keep the per-iteration rule. (At a budget of 10^6 edges ER 2^22 takes 2,027 and
  // 2^23 3,741 for 4,860: the rule has no budget for such graphs.)
  // CC on a symmetric graph of 2^22 vertices or more where union-find pays:
  // both selectors take it before the first iteration, so it runs as
  // union-find's own kernel; on smaller graphs in the selectors' kernel
  // (kUnionFindKernelNodes).
  if (algo == I2_CC && (mode == 1 || mode == 2) && (long long)g->g.nodes >= kUnionFindKernelNodes) {
    st = ensure_symmetry(g);
    if (st) return st;
    if (((allowed_mask(g, algo) >> kUnionFind) & 1) && union_find_pays(g->g.nodes, g->gs.avgdeg)) {
      mode = 0;
      variant = kUnionFind;
    }
  }
  if (algo == I2_SSSP && (mode == 1 || mode == 2) && !srcs_host && o.sssp_delta <= 0 &&
      (long long)g->g.edges >= kBudgetRuleEdges && g->gs.degcv > 1.f) {
    mode = 0;
    variant = kVPCta;
    if (o.sssp_budget <= 0) o.sssp_budget = I2_SSSP_BUDGET_AUTO;
  }
  // sp[] is for the edge sweeps, which the frequency rule never picks
  if (mode >= 2 || variant == kEdgeTopo) {
    st = ensure_sp(g);
    if (st) return st;
  }
  if (mode != 0 || variant == kPullFrontier || variant == kPullTopo || variant == kUnionFind) {
    st = ensure_symmetry(g);
    if (st) return st;
  }
  // The frequency rule picks the edge-balanced push for every iteration of SSSP,
  // and of CC where union-find does not pay: that style's own kernel runs them.
  // SSSP, us, own kernel / the selectors': RMAT 10^6 655 / 785, degree-ordered
  // 2.5 x 10^6 1,086 / 1,205, 5.5 x 10^5 374 / 399.
  if (mode == 1 && (algo == I2_SSSP ||
                    (algo == I2_CC && !(((allowed_mask(g, algo) >> kUnionFind) & 1) &&
                                        union_find_pays(g->g.nodes, g->gs.avgdeg))))) {
    mode = 0;
    variant = kVPCta;
    o.sssp_delta = 0;  // options of the fixed style: not the rule's
    o.sssp_budget = 0;
  }
  if ((mode == 0 || mode == 3) && !((allowed_mask(g, algo) >> variant) & 1)) return I2_ERR_UNSUPPORTED;
  if (mode == 3 && !((allowed_mask(g, algo) >> o.then_variant) & 1)) return I2_ERR_UNSUPPORTED;
  cudaStream_t s = o.stream ? (cudaStream_t)o.stream : g->stream;
  const bool multi = srcs_host != nullptr;
  if (multi) {
    if (nsrc < 1) return I2_ERR_ARG;
    for (int j = 0; j < nsrc; ++j)
      if (srcs_host[j] < 0 || srcs_host[j] >= g->g.nodes) return I2_ERR_ARG;
    if (g->srcs_cap < nsrc) {
      dev_free(g->srcs);
      g->srcs = nullptr;
      I2_CK(dev_alloc(&g->srcs, sizeof(int) * nsrc));
      g->srcs_cap = nsrc;
      // graphs bake the source pointer: rebuild them
      drop_execs(g);
    }
    I2_CK(cudaMemcpyAsync(g->srcs, srcs_host, sizeof(int) * nsrc, cudaMemcpyHostToDevice, s));
  }
  const int delta = pick_order(g, algo, mode, variant, o.sssp_delta, o.sssp_budget);
  if (delta != 0) {
    st = ensure_piles(g);
    if (st) return st;
  }
  RunParams rp = make_params(g, algo, mode, variant, src, nsrc, o.iter_cap, delta);
  if (mode == 3) {
    rp.then_at = o.then_at;
    rp.then_variant = o.then_variant;
  }
  // union-find from the first iteration: fixed, or by the selectors' rule
  rp.whole = algo == I2_CC && ((mode == 0 && variant == kUnionFind) ||
                                  ((mode == 1 || mode == 2) && ((rp.allowed >> kUnionFind) & 1) &&
                                   union_find_pays(g->g.nodes, g->gs.avgdeg)));
  ExecEntry* ex = nullptr;
  const bool graph_loop = o.loop_mode == I2_LOOP_GRAPH || o.loop_mode == I2_LOOP_RELAUNCH;
  // Resident traversal where the device takes the cooperative launch; a graph
  // with one launch per iteration otherwise.
  bool resident = o.loop_mode == I2_LOOP_GRAPH && g->resident_ok;
  // a stream under capture gets the graph, whose launch it refuses
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (resident && (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone)) {
    cudaGetLastError();
    resident = false;
  }
  if (graph_loop && !resident) {
    st = build_exec(g, algo, mode, variant, multi, rp, &ex);
    if (st) return st;
  }
  ResidentPlan plan;
  if (resident) plan = plan_resident(g, algo, mode, variant, multi, rp);
  double host_relax_ms = -1.0;
  if (rep) I2_CK(cudaEventRecord(g->ev0, s));
  if (resident) {
    const cudaError_t e = launch_resident(g, plan, multi, rp, s);
    if (e != cudaSuccess) {  // refused: one launch per iteration, for good where the device has no such launch
      if (e == cudaErrorNotSupported) g->resident_ok = false;
      resident = false;
      st = build_exec(g, algo, mode, variant, multi, rp, &ex);
      if (st) return st;
    }
  }
  if (graph_loop && !resident) {
    st = launch_exec(g, ex, rp, s);
    if (st) return st;
  } else if (!graph_loop) {
    st = prepare_run(g, s, rp);
    if (st) return st;
    st = run_host_loop(g, s, algo, multi, &host_relax_ms);
    if (st) return st;
  }
  if (rep) I2_CK(cudaEventRecord(g->ev1, s));
  I2_CK(cudaGetLastError());
  // Without a report the call stays asynchronous on the stream.
  if (!rep && graph_loop) return I2_OK;
  return fill_report(g, s, algo, rep, host_relax_ms, host_out);
}

bool graph_known_symmetric(const i2_graph* g) { return g && g->gs.symmetric == 1; }

int graph_adopt(int nodes, int edges, int* d_nindex, int* d_nlist, int* d_eweight, int symmetric, i2_graph** out) {
  i2_graph* g = new i2_graph();
  g->owns = true;
  g->d_nindex = d_nindex;
  g->d_nlist = d_nlist;
  g->d_eweight = d_eweight;
  g->g.nodes = nodes;
  g->g.edges = edges;
  g->g.nindex = d_nindex;
  g->g.nlist = d_nlist;
  g->g.eweight = d_eweight;
  int st = finish_setup(g);
  if (st) {
    free_graph_state(g);
    delete g;
    return st;
  }
  g->gs.symmetric = symmetric;
  *out = g;
  return I2_OK;
}

int graph_copy_result(i2_graph* g, int* host_out, const i2_opts* opts) {
  cudaStream_t s = (opts && opts->stream) ? (cudaStream_t)opts->stream : g->stream;
  I2_CK(cudaMemcpyAsync(host_out, g->dist, sizeof(int) * (size_t)g->g.nodes, cudaMemcpyDeviceToHost, s));
  I2_CK(cudaStreamSynchronize(s));
  return I2_OK;
}

// Per-iteration sweep: along the trajectory of `follow` (a variant, or the
// heuristic when negative), save the state before each launch, time every
// allowed variant from that state (best of `reps`), restore, and advance.
static int sweep(i2_graph* g, int algo, int src, int follow, int reps, i2_iter_record* recs, float* times, int cap,
                 int* nout) {
  I2_CK(cudaSetDevice(g->device));
  int st = ensure_workspace(g);
  if (st) return st;
  st = ensure_symmetry(g);
  if (st) return st;
  st = ensure_sp(g);  // every style is timed, the edge sweep too
  if (st) return st;
  const long long V = g->g.nodes;
  if (!g->snap_dist) {
    I2_CK(dev_alloc(&g->snap_dist, sizeof(int) * V));
    I2_CK(dev_alloc(&g->snap_bm, sizeof(unsigned) * 3ull * g->bm_words));
  }
  cudaStream_t s = g->stream;
  // a followed style runs as a switch to itself: the states that the other
  // styles are timed from are those of a run whose style may change
  const int mode = follow == I2_AUTO_LEARNED ? 2 : (follow < 0 ? 1 : 3);
  RunParams rp = make_params(g, algo, mode, follow < 0 ? 0 : follow, src, 1, 0);
  rp.then_variant = rp.fixed_variant;
  st = prepare_run(g, s, rp);
  if (st) return st;
  Ctx c = make_ctx(g);
  KernelFn ff = fill_kernel(algo);
  ff<<<grid_for(ff, 8), kBlock, 0, s>>>(c);
  seed_kernel(algo)<<<1, kBlock, 0, s>>>(c);
  const int allowed = allowed_mask(g, algo);
  Ctl snap;
  int it = 0;
  // Styles are timed through the dispatch kernel, the one the selectors run.
  KernelFn dk = dispatch_kernel(algo, wide_selector(g));
  const int dgrid = grid_for(dk, g->blocks_per_sm);
  while (it < cap) {
    I2_CK(cudaMemcpyAsync(g->h_ctl, g->ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s));
    I2_CK(cudaStreamSynchronize(s));
    snap = *g->h_ctl;
    if (!snap.go || (snap.status & kStatusIterCap)) break;
    if (snap.uf_phase) {  // the trajectory took union-find: its compress launch is not a choice
      dk<<<dgrid, kBlock, 0, s>>>(c);
      I2_CK(cudaGetLastError());
      continue;
    }
    I2_CK(cudaMemcpyAsync(g->snap_dist, g->dist, sizeof(int) * V, cudaMemcpyDeviceToDevice, s));
    I2_CK(cudaMemcpyAsync(g->snap_bm, g->bm[0], sizeof(unsigned) * 3ull * g->bm_words, cudaMemcpyDeviceToDevice, s));
    for (int v = 0; v < kNumVariants; ++v) {
      float best = -1.f;
      if ((allowed >> v) & 1) {
        for (int r = 0; r < std::max(1, reps); ++r) {
          *g->h_ctl = snap;
          g->h_ctl->variant = v;
          I2_CK(cudaMemcpyAsync(g->ctl, g->h_ctl, sizeof(Ctl), cudaMemcpyHostToDevice, s));
          I2_CK(cudaMemcpyAsync(g->dist, g->snap_dist, sizeof(int) * V, cudaMemcpyDeviceToDevice, s));
          I2_CK(cudaMemcpyAsync(g->bm[0], g->snap_bm, sizeof(unsigned) * 3ull * g->bm_words, cudaMemcpyDeviceToDevice, s));
          I2_CK(cudaEventRecord(g->ev0, s));
          dk<<<dgrid, kBlock, 0, s>>>(c);
          if (v == kUnionFind) {  // its later launches belong to it
            dk<<<dgrid, kBlock, 0, s>>>(c);
            dk<<<dgrid, kBlock, 0, s>>>(c);
          }
          I2_CK(cudaEventRecord(g->ev1, s));
          I2_CK(cudaEventSynchronize(g->ev1));
          float ms = 0.f;
          I2_CK(cudaEventElapsedTime(&ms, g->ev0, g->ev1));
          // The launches' own device time (their iteration records), without the
          // launch latency that the resident traversal does not pay.
          const int nrec = v == kUnionFind ? 3 : 1;
          if (snap.iter + nrec <= g->rec_cap) {
            IterRec r[3];
            I2_CK(cudaMemcpy(r, g->recs + snap.iter, sizeof(IterRec) * nrec, cudaMemcpyDeviceToHost));
            ms = 0.f;
            for (int j = 0; j < nrec; ++j) ms += (float)r[j].t_ns * 1e-6f;
          }
          if (best < 0.f || ms < best) best = ms;
        }
        best *= 1e6f;  // ns
      }
      times[(size_t)it * kNumVariants + v] = best;
    }
    *g->h_ctl = snap;
    I2_CK(cudaMemcpyAsync(g->ctl, g->h_ctl, sizeof(Ctl), cudaMemcpyHostToDevice, s));
    I2_CK(cudaMemcpyAsync(g->dist, g->snap_dist, sizeof(int) * V, cudaMemcpyDeviceToDevice, s));
    I2_CK(cudaMemcpyAsync(g->bm[0], g->snap_bm, sizeof(unsigned) * 3ull * g->bm_words, cudaMemcpyDeviceToDevice, s));
    dk<<<dgrid, kBlock, 0, s>>>(c);
    I2_CK(cudaGetLastError());
    if (snap.iter < g->rec_cap)
      I2_CK(cudaMemcpyAsync(&recs[it], g->recs + snap.iter, sizeof(IterRec), cudaMemcpyDeviceToHost, s));
    ++it;
  }
  I2_CK(cudaStreamSynchronize(s));
  *nout = it;
  g->last_iters = it;
  return I2_OK;
}

// True when [p, p + bytes) lies inside one device (or managed) allocation of
// the current context. Host pointers, pinned or not, are refused: a kernel
// given one would fault or read the wrong memory. So is device memory of
// another GPU: kernels launched on the current device would read it through a
// peer mapping, or fault where there is none.
typedef int (*MemGetAddressRangeFn)(unsigned long long*, size_t*, unsigned long long);

int graph_device_csr(const i2_graph* g, int* nodes, int* edges, const int** nindex, const int** nlist,
                     const int** eweight) {
  if (!g) return I2_ERR_ARG;
  *nodes = g->g.nodes;
  *edges = g->g.edges;
  *nindex = g->g.nindex;
  *nlist = g->g.nlist;
  *eweight = g->g.eweight;
  return I2_OK;
}

bool device_range_ok(const void* p, size_t bytes) {
  if (bytes == 0) return true;
  if (!p) return false;
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (a.type != cudaMemoryTypeDevice && a.type != cudaMemoryTypeManaged) return false;
  if (a.type == cudaMemoryTypeDevice) {
    int cur = -1;
    if (cudaGetDevice(&cur) != cudaSuccess || a.device != cur) {
      cudaGetLastError();
      return false;
    }
  }
  static MemGetAddressRangeFn range_fn = nullptr;
  static bool looked = false;
  if (!looked) {
    looked = true;
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuMemGetAddressRange", &fn, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      range_fn = (MemGetAddressRangeFn)fn;
    cudaGetLastError();
  }
  if (!range_fn) return true;  // type check only
  unsigned long long base = 0;
  size_t size = 0;
  if (range_fn(&base, &size, (unsigned long long)(uintptr_t)p) != 0) return false;
  return (unsigned long long)(uintptr_t)p + bytes <= base + size;
}

}  // namespace i2

// ---------------------------------------------------------------------------
// C ABI.

extern "C" {

const char* i2_status_string(int status) {
  switch (status) {
    case I2_OK: return "ok";
    case I2_ERR_ARG: return "invalid argument";
    case I2_ERR_IO: return "file i/o error";
    case I2_ERR_FORMAT: return "malformed graph";
    case I2_ERR_NOMEM: return "out of memory";
    case I2_ERR_CUDA: return "cuda error";
    case I2_ERR_NO_DEVICE: return "no cuda device";
    case I2_ERR_UNSUPPORTED: return "variant not supported on this graph";
    case I2_ERR_ITER_CAP: return "iteration cap reached";
    case I2_ERR_OVERFLOW: return "int32 limit exceeded";
    case I2_ERR_CAPACITY: return "graph exceeds the fixed scratch of i2_run_noalloc";
    case I2_ERR_STALL: return "a resident traversal's barrier wait ran out of time";
  }
  return "unknown status";
}

const char* i2_variant_name(int v) {
  static const char* names[] = {"vp_thread", "vp_warp", "vp_cta", "vp_block",
                                "pull_frontier", "pull_topo", "edge_topo", "push_topo", "union_find"};
  if (v == I2_AUTO_HEURISTIC) return "auto_heuristic";
  if (v == I2_AUTO_LEARNED) return "auto_learned";
  if (v < 0 || v >= kNumVariants) return "invalid";
  return names[v];
}

int i2_version(void) { return 100; }

int i2_device_count(void) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

static int upload_common(i2_graph* g) {
  int st = finish_setup(g);
  if (st) {
    free_graph_state(g);
    delete g;
  }
  return st;
}

// The shape of the CSR is checked on the host; its entries (monotone nindex,
// nlist in range) on the device right after the copy, before any other kernel
// reads them: a host pass over nlist costs about as much as copying it. The
// adjacency and the weights go over two streams (two copy engines).
int i2_graph_upload(const i2_eclgraph* h, i2_graph** out) {
  if (!h || !out) return I2_ERR_ARG;
  *out = nullptr;
  if (h->nodes < 1 || h->edges < 0) return I2_ERR_FORMAT;
  if (!h->nindex || (h->edges > 0 && !h->nlist)) return I2_ERR_ARG;
  if (h->nindex[0] != 0 || h->nindex[h->nodes] != h->edges) return I2_ERR_FORMAT;
  if (i2_device_count() < 1) return I2_ERR_NO_DEVICE;
  i2_graph* g = new i2_graph();
  g->owns = true;
  const size_t nn = (size_t)h->nodes + 1, ne = (size_t)h->edges + 4;
  DevPool* pool = dev_pool();
  if (!pool) {
    delete g;
    return I2_ERR_CUDA;
  }
  cudaStream_t s1 = pool->copy[0], s2 = pool->copy[1];
  int* bad = nullptr;
  int hbad = 0;
  cudaError_t e = dev_alloc(&g->d_nindex, sizeof(int) * nn);
  if (e == cudaSuccess) e = dev_alloc(&g->d_nlist, sizeof(int) * ne);
  if (e == cudaSuccess && h->eweight) e = dev_alloc(&g->d_eweight, sizeof(int) * ne);
  if (e == cudaSuccess) e = dev_alloc(&bad, sizeof(int));
  if (e == cudaSuccess) e = cudaMemsetAsync(bad, 0, sizeof(int), s1);
  if (e == cudaSuccess) e = cudaMemcpyAsync(g->d_nindex, h->nindex, sizeof(int) * nn, cudaMemcpyHostToDevice, s1);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(g->d_nlist, h->nlist, sizeof(int) * h->edges, cudaMemcpyHostToDevice, s1);
  if (e == cudaSuccess && h->eweight)
    e = cudaMemcpyAsync(g->d_eweight, h->eweight, sizeof(int) * h->edges, cudaMemcpyHostToDevice, s2);
  g->g.nodes = h->nodes;
  g->g.edges = h->edges;
  g->g.nindex = g->d_nindex;
  g->g.nlist = g->d_nlist;
  g->g.eweight = g->d_eweight;
  if (e == cudaSuccess) {
    k_validate<<<4 * sm_count(), 256, 0, s1>>>(g->g, bad);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, s1);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s1);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s2);
  dev_free(bad);
  if (e != cudaSuccess || hbad) {
    cudaGetLastError();
    free_graph_state(g);
    delete g;
    return e != cudaSuccess ? cuda_status(e) : I2_ERR_FORMAT;
  }
  int st = upload_common(g);
  if (st) return st;
  *out = g;
  return I2_OK;
}

int i2_graph_hub(i2_graph* g, int* v) {
  if (!g || !v) return I2_ERR_ARG;
  I2_CK(cudaSetDevice(g->device));
  *v = g->hub;  // found with the degree statistics
  return I2_OK;
}

int i2_graph_sp(i2_graph* g, const int** sp_dev, int* sp_host) {
  if (!g || (!sp_dev && !sp_host)) return I2_ERR_ARG;
  I2_CK(cudaSetDevice(g->device));
  int st = ensure_sp(g);
  if (st) return st;
  if (sp_dev) *sp_dev = g->d_sp;
  if (sp_host && g->g.edges > 0)
    I2_CK(cudaMemcpy(sp_host, g->d_sp, sizeof(int) * (size_t)g->g.edges, cudaMemcpyDeviceToHost));
  return I2_OK;
}

int i2_graph_wrap_device(const i2_eclgraph* d, i2_graph** out) {
  if (!d || !out || d->nodes < 1 || d->edges < 0 || !d->nindex || (d->edges > 0 && !d->nlist)) return I2_ERR_ARG;
  *out = nullptr;
  if (i2_device_count() < 1) return I2_ERR_NO_DEVICE;
  if (!device_range_ok(d->nindex, sizeof(int) * ((size_t)d->nodes + 1)) ||
      !device_range_ok(d->nlist, sizeof(int) * (size_t)d->edges) ||
      (d->eweight && !device_range_ok(d->eweight, sizeof(int) * (size_t)d->edges)))
    return I2_ERR_ARG;
  i2_graph* g = new i2_graph();
  g->owns = false;
  g->d_nindex = d->nindex;
  g->d_nlist = d->nlist;
  g->d_eweight = d->eweight;
  g->g.nodes = d->nodes;
  g->g.edges = d->edges;
  g->g.nindex = d->nindex;
  g->g.nlist = d->nlist;
  g->g.eweight = d->eweight;
  // Validate before any kernel indexes through the arrays.
  int* bad = nullptr;
  int hbad = 0;
  cudaError_t e = dev_alloc(&bad, sizeof(int));
  if (e == cudaSuccess) e = cudaMemset(bad, 0, sizeof(int));
  if (e == cudaSuccess) {
    k_validate<<<4 * sm_count(), 256>>>(g->g, bad);
    e = cudaMemcpy(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost);
  }
  dev_free(bad);
  if (e != cudaSuccess) {
    cudaGetLastError();
    delete g;
    return cuda_status(e);
  }
  if (hbad) {
    delete g;
    return I2_ERR_FORMAT;
  }
  int st = upload_common(g);
  if (st) return st;
  *out = g;
  return I2_OK;
}

int i2_graph_size(const i2_graph* g, int* nodes, int* edges) {
  if (!g || !nodes || !edges) return I2_ERR_ARG;
  *nodes = g->g.nodes;
  *edges = g->g.edges;
  return I2_OK;
}

int i2_graph_degree(const i2_graph* g, int v, int* deg) {
  if (!g || !deg || v < 0 || v >= g->g.nodes) return I2_ERR_ARG;
  int pair[2];
  I2_CK(cudaMemcpy(pair, g->g.nindex + v, sizeof(pair), cudaMemcpyDeviceToHost));
  *deg = pair[1] - pair[0];
  return I2_OK;
}

int i2_graph_info_get(const i2_graph* g, i2_graph_info* out) {
  if (!g || !out) return I2_ERR_ARG;
  if (g->gs.symmetric < 0) {
    cudaSetDevice(g->device);
    const int st = ensure_symmetry(const_cast<i2_graph*>(g));
    if (st) return st;
  }
  out->nodes = g->gs.nodes;
  out->edges = g->gs.edges;
  out->maxdeg = g->gs.maxdeg;
  out->nheavy = g->gs.nheavy;
  out->wmin = g->gs.wmin;
  out->symmetric = g->gs.symmetric;
  out->has_weights = g->g.eweight != nullptr;
  out->avgdeg = g->gs.avgdeg;
  out->degcv = g->gs.degcv;
  return I2_OK;
}

int i2_graph_download(const i2_graph* g, i2_eclgraph* out) {
  if (!g || !out) return I2_ERR_ARG;
  int st = i2_alloc_eclgraph(g->g.nodes, g->g.edges, g->g.eweight ? 1 : 0, out);
  if (st) return st;
  cudaError_t e = cudaMemcpy(out->nindex, g->g.nindex, sizeof(int) * ((size_t)g->g.nodes + 1), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(out->nlist, g->g.nlist, sizeof(int) * (size_t)g->g.edges, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && g->g.eweight)
    e = cudaMemcpy(out->eweight, g->g.eweight, sizeof(int) * (size_t)g->g.edges, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) {
    cudaGetLastError();
    i2_free_eclgraph(out);
    return cuda_status(e);
  }
  return I2_OK;
}

int i2_graph_tune(i2_graph* g, int heavy_threshold, int blocks_per_sm, int smem_carveout) {
  if (!g || heavy_threshold < 0 || blocks_per_sm < 0 || blocks_per_sm > 32) return I2_ERR_ARG;
  if (smem_carveout < -1 || smem_carveout > 100) return I2_ERR_ARG;
  if (g_carveout.exchange(smem_carveout) != smem_carveout) ++g_carveout_set;
  I2_CK(cudaSetDevice(g->device));
  if (g->stream) I2_CK(cudaStreamSynchronize(g->stream));
  drop_execs(g);
  if (blocks_per_sm) g->blocks_per_sm = blocks_per_sm;
  if (heavy_threshold && heavy_threshold != g->heavy) {
    g->heavy = std::max(32, heavy_threshold);
    // the heavy lists are sized by the number of heavy vertices
    dev_free(g->heavy_base);
    g->heavy_base = nullptr;
    for (int k = 0; k < 3; ++k) {
      g->hwl[k] = nullptr;
      g->htoff[k] = nullptr;
    }
    int st = compute_stats(g);
    if (st) return st;
    if (g->ws_ready) {
      st = alloc_heavy(g);
      if (st) return st;
    }
  }
  if (g->twin) return i2_graph_tune(g->twin, heavy_threshold, blocks_per_sm, smem_carveout);
  return I2_OK;
}

int i2_graph_synth_weights(i2_graph* g) {
  if (!g) return I2_ERR_ARG;
  if (g->g.eweight) return I2_OK;
  I2_CK(cudaSetDevice(g->device));
  int* w = nullptr;
  I2_CK(dev_alloc(&w, sizeof(int) * ((size_t)g->g.edges + 4)));
  k_synth_weights<<<8 * sm_count(), 256, 0, g->stream>>>(g->g, w);
  I2_CK(cudaStreamSynchronize(g->stream));
  g->d_eweight = w;
  g->owns_weights = true;
  g->g.eweight = w;
  g->g.vec_ok = ((((uintptr_t)g->g.nlist) & 15) == 0 && (((uintptr_t)w) & 15) == 0) ? 1 : 0;
  drop_execs(g);
  const int st = compute_stats(g);
  if (st || !g->twin) return st;
  // the weights are a function of the original IDs: renumber again
  return i2_graph_reorder(g, I2_ORDER_DEGREE);
}

int i2_graph_free(i2_graph* g) {
  if (!g) return I2_ERR_ARG;
  cudaSetDevice(g->device);
  if (g->stream) cudaStreamSynchronize(g->stream);
  free_graph_state(g);
  delete g;
  return I2_OK;
}

int i2_graph_reorder(i2_graph* g, int order) {
  if (!g || (order != I2_ORDER_NONE && order != I2_ORDER_DEGREE)) return I2_ERR_ARG;
  I2_CK(cudaSetDevice(g->device));
  if (g->stream) I2_CK(cudaStreamSynchronize(g->stream));
  if (g->twin) {
    i2_graph_free(g->twin);
    g->twin = nullptr;
    dev_free(g->d_inv);
    g->d_inv = nullptr;
    g->h_inv.clear();
    g->h_inv.shrink_to_fit();
    g->last_on_twin = false;
  }
  // nothing to renumber without edges: traversals stay on the original
  if (order == I2_ORDER_NONE || g->g.edges == 0) return I2_OK;
  i2_graph* twin = nullptr;
  int* inv = nullptr;
  int st = degree_ordered_copy(g, &twin, &inv);
  if (st) return st;
  std::vector<int> h(g->g.nodes);
  const cudaError_t e = cudaMemcpy(h.data(), inv, sizeof(int) * h.size(), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) {
    i2_graph_free(twin);
    dev_free(inv);
    return cuda_status(e);
  }
  // the copy launches like the original (settings of i2_graph_tune; the
  // heavy lists are sized for the threshold by the tune call)
  st = i2_graph_tune(twin, g->heavy, g->blocks_per_sm, g_carveout.load());
  if (st) {
    i2_graph_free(twin);
    dev_free(inv);
    return st;
  }
  g->twin = twin;
  g->d_inv = inv;
  g->h_inv.swap(h);
  return I2_OK;
}

int i2_trim_device_memory(void) {
  if (i2_device_count() < 1) return I2_ERR_NO_DEVICE;
  return dev_trim();
}

static int run_host_out(i2_graph* g, int algo, int src, int* out, const i2_opts* opts, i2_report* rep) {
  if (!out) return I2_ERR_ARG;
  int st = run_traversal(g, algo, src, nullptr, 0, opts, rep, out);
  if (st && st != I2_ERR_ITER_CAP) return st;
  if (g->staged) return st;  // the result came with the report
  cudaStream_t s = (opts && opts->stream) ? (cudaStream_t)opts->stream : g->stream;
  I2_CK(cudaMemcpyAsync(out, g->dist, sizeof(int) * (size_t)g->g.nodes, cudaMemcpyDeviceToHost, s));
  I2_CK(cudaStreamSynchronize(s));
  return st;
}

int i2_bfs(i2_graph* g, int src, int* dist, const i2_opts* opts, i2_report* rep) {
  return run_host_out(g, I2_BFS, src, dist, opts, rep);
}
int i2_sssp(i2_graph* g, int src, int* dist, const i2_opts* opts, i2_report* rep) {
  return run_host_out(g, I2_SSSP, src, dist, opts, rep);
}
int i2_cc(i2_graph* g, int* label, const i2_opts* opts, i2_report* rep) {
  return run_host_out(g, I2_CC, 0, label, opts, rep);
}

int i2_mis(i2_graph* g, int* status, const i2_opts* opts, i2_report* rep) {
  return run_host_out(g, I2_MIS, 0, status, opts, rep);
}

int i2_run_device(i2_graph* g, int algo, int src, int* out_dev, const i2_opts* opts, i2_report* rep) {
  int st = run_traversal(g, algo, (algo == I2_CC || algo == I2_MIS) ? 0 : src, nullptr, 0, opts, rep);
  if (st && st != I2_ERR_ITER_CAP) return st;
  if (out_dev) {
    cudaStream_t s = (opts && opts->stream) ? (cudaStream_t)opts->stream : g->stream;
    I2_CK(cudaMemcpyAsync(out_dev, g->dist, sizeof(int) * (size_t)g->g.nodes, cudaMemcpyDeviceToDevice, s));
  }
  return st;
}

int i2_get_records(const i2_graph* g, i2_iter_record* out, int cap, int* n) {
  if (!g || !out || !n || cap < 0) return I2_ERR_ARG;
  if (g->last_on_twin && g->twin) return i2_get_records(g->twin, out, cap, n);
  if (!g->ws_ready) {
    *n = 0;
    return I2_OK;
  }
  const int m = std::min(std::min(g->last_iters, g->rec_cap), cap);
  if (m > 0) I2_CK(cudaMemcpy(out, g->recs, sizeof(IterRec) * m, cudaMemcpyDeviceToHost));
  *n = m;
  return I2_OK;
}

int i2_sweep(i2_graph* g, int algo, int src, int follow, int reps, i2_iter_record* recs, float* times, int cap,
             int* n) {
  if (!g || !recs || !times || !n || cap < 1 || algo < I2_BFS || algo > I2_CC) return I2_ERR_ARG;
  if (follow >= kNumVariants || follow < I2_AUTO_LEARNED) return I2_ERR_ARG;
  if (algo != I2_CC && (src < 0 || src >= g->g.nodes)) return I2_ERR_ARG;
  if (algo == I2_SSSP && !g->g.eweight) return I2_ERR_ARG;
  if (follow >= 0) {
    I2_CK(cudaSetDevice(g->device));
    int st = ensure_symmetry(g);
    if (st) return st;
    st = ensure_sp(g);
    if (st) return st;
    if (!((allowed_mask(g, algo) >> follow) & 1)) return I2_ERR_UNSUPPORTED;
  }
  return sweep(g, algo, src, follow, reps, recs, times, cap, n);
}

int i2_mlp_param_count(void) { return kParams; }

int i2_mlp_set_params(const float* params, int count) { return mlp_install(params, count); }

}  // extern "C"

// ---------------------------------------------------------------------------
// Traversal that allocates nothing.
//
// Some callers cannot allocate device memory at the moment they run a query:
// their process's device memory is already held by another allocator (for
// example a framework's caching allocator that reserved the GPU), their query
// loop cannot afford cudaMalloc/cudaFree, which synchronise the device, or
// their query must not be able to fail with out-of-memory. i2_run_noalloc
// serves them: the caller passes the CSR arrays and the output array (all in
// device memory), and every piece of scratch the traversal needs (frontier
// lists, their edge offsets, the frontier bitmaps and the control block) lives
// in one fixed-size device array defined in this file. That array is part of
// the library image: every GPU that loads the library holds it (about 3 MB)
// until the process exits. Graphs above kNoAllocMaxNodes vertices are refused.

namespace i2 {

constexpr int kNoAllocMaxNodes = 1 << 17;  // 131072 vertices
constexpr int kNoAllocWords = kNoAllocMaxNodes / 32;

// Layout of the scratch array (offsets in bytes, each 256-byte aligned).
constexpr size_t kNoAllocAlign(size_t x) { return (x + 255) & ~(size_t)255; }
constexpr size_t kNaWl = 0;
constexpr size_t kNaWoff = kNaWl + kNoAllocAlign(3ull * kNoAllocMaxNodes * sizeof(int));
constexpr size_t kNaBm = kNaWoff + kNoAllocAlign(3ull * kNoAllocMaxNodes * sizeof(unsigned));
constexpr size_t kNaHeavy = kNaBm + kNoAllocAlign(3ull * kNoAllocWords * sizeof(unsigned));
constexpr size_t kNaCtl = kNaHeavy + 256;
constexpr size_t kNaBad = kNaCtl + kNoAllocAlign(sizeof(Ctl));
constexpr size_t kNoAllocBytes = kNaBad + 256;

}  // namespace i2

// The scratch itself. In host code this name is only a host-side stand-in:
// its device address is obtained with cudaGetSymbolAddress (per device).
static __device__ __align__(256) unsigned char g_noalloc_scratch[i2::kNoAllocBytes];

namespace i2 {

static std::mutex g_noalloc_mu;
static unsigned char* g_noalloc_dev[64] = {nullptr};

// Device address of the scratch on the current device; looked up on the first
// call per device.
static int noalloc_scratch(unsigned char** out) {
  int dev = 0;
  I2_CK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return I2_ERR_ARG;
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_dev[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return cuda_status(e);
    }
    g_noalloc_dev[dev] = static_cast<unsigned char*>(p);
  }
  *out = g_noalloc_dev[dev];
  return I2_OK;
}

}  // namespace i2

extern "C" int i2_run_noalloc(int algo, const i2_eclgraph* dev, int src, int* dist_dev, void* stream,
                              int* iterations) {
  using namespace i2;
  if (algo < I2_BFS || algo > I2_CC || !dev || !dist_dev) return I2_ERR_ARG;
  if (dev->nodes < 1 || dev->edges < 0 || !dev->nindex || (dev->edges > 0 && !dev->nlist)) return I2_ERR_ARG;
  if (dev->nodes > kNoAllocMaxNodes) return I2_ERR_CAPACITY;
  if (algo != I2_CC && (src < 0 || src >= dev->nodes)) return I2_ERR_ARG;
  if (algo == I2_SSSP && !dev->eweight) return I2_ERR_ARG;
  if (i2_device_count() < 1) return I2_ERR_NO_DEVICE;
  const int* w = algo == I2_SSSP ? dev->eweight : nullptr;
  if (!device_range_ok(dev->nindex, sizeof(int) * ((size_t)dev->nodes + 1)) ||
      !device_range_ok(dev->nlist, sizeof(int) * (size_t)dev->edges) ||
      (w && !device_range_ok(w, sizeof(int) * (size_t)dev->edges)) ||
      !device_range_ok(dist_dev, sizeof(int) * (size_t)dev->nodes))
    return I2_ERR_ARG;
  unsigned char* base = nullptr;
  int st = noalloc_scratch(&base);
  if (st) return st;
  cudaStream_t s = (cudaStream_t)stream;
  Ctl* ctl = reinterpret_cast<Ctl*>(base + kNaCtl);
  int* bad = reinterpret_cast<int*>(base + kNaBad);

  Ctx c{};
  c.g.nodes = dev->nodes;
  c.g.edges = dev->edges;
  c.g.nindex = dev->nindex;
  c.g.nlist = dev->nlist;
  c.g.eweight = w;
  c.g.sp = nullptr;
  c.g.vec_ok = ((((uintptr_t)dev->nlist) & 15) == 0 && (((uintptr_t)w) & 15) == 0) ? 1 : 0;
  c.gs.nodes = dev->nodes;
  c.gs.edges = dev->edges;
  c.gs.wmin = 1;
  c.gs.avgdeg = (float)dev->edges / (float)dev->nodes;
  c.dist = dist_dev;
  for (int k = 0; k < 3; ++k) {
    c.wl[k] = reinterpret_cast<int*>(base + kNaWl) + (size_t)k * kNoAllocMaxNodes;
    c.woff[k] = reinterpret_cast<unsigned*>(base + kNaWoff) + (size_t)k * kNoAllocMaxNodes;
    c.bm[k] = reinterpret_cast<unsigned*>(base + kNaBm) + (size_t)k * kNoAllocWords;
    // the heavy lists stay empty: the threshold is above every degree
    c.hwl[k] = reinterpret_cast<int*>(base + kNaHeavy);
    c.htoff[k] = reinterpret_cast<unsigned*>(base + kNaHeavy + 128);
  }
  c.ctl = ctl;
  c.recs = nullptr;
  c.rec_cap = 0;
  c.heavy = INT_MAX;
  c.bm_words = (dev->nodes + 31) / 32;
  c.mlp = nullptr;
  c.srcs = nullptr;
  c.use_loop = 0;

  // Reject malformed arrays before any traversal kernel indexes through them.
  int hbad = 0;
  I2_CK(cudaMemsetAsync(bad, 0, sizeof(int), s));
  k_validate<<<4 * sm_count(), 256, 0, s>>>(c.g, bad);
  // negative weights: refused like the allocating entry points refuse them
  if (w) k_negative_weights<<<4 * sm_count(), 256, 0, s>>>(w, dev->edges, bad);
  I2_CK(cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, s));
  I2_CK(cudaStreamSynchronize(s));
  if (hbad & 7) return I2_ERR_FORMAT;
  if (hbad & 8) return I2_ERR_UNSUPPORTED;

  // The scratch keeps the previous call's contents: the bitmaps must start at
  // zero (k_reset rewrites the control block, k_fill the output).
  RunParams rp{};
  rp.algo = algo;
  rp.mode = 0;
  rp.fixed_variant = kVPCta;
  rp.allowed = 1 << kVPCta;
  rp.src = algo == I2_CC ? 0 : src;
  rp.nsrc = 1;
  rp.iter_cap = dev->nodes + 2;
  I2_CK(cudaMemsetAsync(c.bm[0], 0, sizeof(unsigned) * 3ull * kNoAllocWords, s));
  k_reset<<<1, 32, 0, s>>>(ctl, rp);
  KernelFn ff = fill_kernel(algo);
  ff<<<grid_for(ff, 8), kBlock, 0, s>>>(c);
  seed_kernel(algo)<<<1, kBlock, 0, s>>>(c);
  KernelFn fn = relax_kernel(algo, 0, kVPCta, false, false);
  const int grid = grid_for(fn, 8);
  Ctl h;
  for (;;) {
    I2_CK(cudaMemcpyAsync(&h, ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s));
    I2_CK(cudaStreamSynchronize(s));
    if (slot_size(h.slot[h.iter % 3].packed) == 0 || (h.status & kStatusIterCap)) break;
    fn<<<grid, kBlock, 0, s>>>(c);
    I2_CK(cudaGetLastError());
  }
  if (iterations) *iterations = h.iter;
  return (h.status & kStatusIterCap) ? I2_ERR_ITER_CAP : I2_OK;
}
