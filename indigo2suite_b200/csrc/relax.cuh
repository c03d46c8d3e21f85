// Relaxation kernels of the B200 engine: one persistent, grid-stride kernel per
// (algorithm, variant). Each launch performs exactly one iteration of the
// frontier contract described in common.cuh.
//
// Reference styles these variants re-create (file names under codes/cuda/):
//   kVPThread  ~ *_V_Data_Push_*_Thread_*   (e.g. BFS ..._Atomic_Thread_..._NonDup.cu)
//   kVPWarp    ~ *_V_Data_Push_*_Warp_*     (BFS_CUDA_V_Data_Push_..._Warp_..._NonDup.cu:62-84)
//   kVPBlock   ~ *_V_Data_Push_*_Block_*    (BFS_CUDA_V_Data_Push_..._Block_..._Dup.cu:62-83)
//   kVPCta     ~ *_E_Data_Push_*            (SSSP_CUDA_E_Data_Push_..._NonDup.cu:63-82): one thread per
//                                           frontier edge, the edges split evenly over the grid
//   kPullFrontier / kPullTopo ~ *_V_{Data,Topo}_Pull_* (BFS ..._V_Topo_Pull_..._Warp_...cu:57-79,
//                                           CC_CUDA_V_Topo_Pull_..._Warp_...cu:59-78)
//   kEdgeTopo  ~ *_E_Topo_Push_*            (BFS_CUDA_E_Topo_Push_..._Thread_...cu:57-72)
//   kPushTopo  ~ *_V_Topo_Push_*            (BFS_CUDA_V_Topo_Push_..._Thread_...cu:56-79)
// The B200 versions differ in mechanism, not in fixed point:
//  * frontier appends are staged per block in shared memory and published with
//    one packed 64-bit atomic per flush, which also yields each entry's offset
//    in the frontier's edge space (the reference appends with one atomicAdd per
//    vertex, BFS_..._Warp_..._NonDup.cu:78);
//  * duplicates are filtered by a frontier bitmap (the reference uses a time[]
//    stamp array, :77);
//  * each thread issues the dist[] loads of several neighbours before any of
//    their atomicMin operations, so that several misses are in flight per thread;
//  * adjacency is read with 128-bit loads where aligned, and the frontier's
//    heavy vertices are cut into tiles that any block may take.
#pragma once
#include <cooperative_groups.h>
#include <cooperative_groups/reduce.h>
#include <cooperative_groups/scan.h>
#include <cub/block/block_scan.cuh>
#include <type_traits>
#include "common.cuh"
#include "list_walk.h"

namespace i2 {

namespace cg = cooperative_groups;

constexpr int kScanItems = kQueue / kBlock;                 // staged entries per thread in a flush
// Edges per lane of the edge-balanced tile (measured beside I2_EB_MIN_BLOCKS).
#ifndef I2_EB_EDGES
#define I2_EB_EDGES 2
#endif
constexpr int kEdgesPerThread = I2_EB_EDGES;                // edge-balanced variant
constexpr int kTileEdges = kBlock * kEdgesPerThread;        // edges per edge-balanced tile

typedef cub::BlockScan<int, kBlock> BlockScanT;

// Loads of the graph's adjacency (nlist, eweight, sp): each entry is read
// about once per iteration, so it is loaded with an evict-first policy, which
// keeps the randomly accessed, L2-sized arrays (values, bitmaps, frontier
// lists, nindex) resident in L2 instead of the streamed lines. On RMAT-22 this
// measured 3-7% faster for BFS, SSSP and CC than the read-only path.
// I2_STREAM_LOADS: 0 read-only path without a hint, 1 evict-first (default),
// 2 explicit L2 policies: adjacency evict-first, not allocated in L1 (measured
// within 1% of 1 on RMAT-22 BFS, SSSP and CC and on a 2048² grid).
#ifndef I2_STREAM_LOADS
#define I2_STREAM_LOADS 1
#endif
#if I2_STREAM_LOADS == 2
__device__ __forceinline__ unsigned long long l2_evict_first() {
  unsigned long long pol;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ int ld_adj(const int* p) {
  int v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.b32 %0, [%1], %2;"
               : "=r"(v) : "l"(p), "l"(l2_evict_first()));
  return v;
}
__device__ __forceinline__ int4 ld_adj(const int4* p) {
  int4 v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.b32 {%0, %1, %2, %3}, [%4], %5;"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p), "l"(l2_evict_first()));
  return v;
}
#else
template <typename T>
__device__ __forceinline__ T ld_adj(const T* p) {
#if I2_STREAM_LOADS
  return __ldcs(p);
#else
  return __ldg(p);
#endif
}
#endif

// Frontier statistics of one thread's pushes; kept in registers and reduced
// once per block at the end of the launch.
struct Acc {
  int maxdeg;
  int mindist;
  int visited;
  int fmin;  // smallest value put on a far pile
};

__device__ __forceinline__ void acc_init(Acc& a) {
  a.maxdeg = 0;
  a.mindist = kInf;
  a.visited = 0;
  a.fmin = kInf;
}

// Per-block staging of pushes into the next frontier.
struct Stage {
  int q[kQueue];    // vertices
  int qd[kQueue];   // their degrees
  int hq[kHQueue];  // heavy vertices
  int ht[kHQueue];  // their tile counts
  int n;
  int hn;
  unsigned long long base;
  unsigned long long hbase;
  int chunk;
  int last;
  int j0;
  int m;
  Acc red[kBlock / kWarp];
  typename BlockScanT::TempStorage scan;
};

__device__ __forceinline__ void stage_init(Stage& s) {
  if (threadIdx.x == 0) {
    s.n = 0;
    s.hn = 0;
    s.last = 0;
  }
}

__device__ __forceinline__ int heavy_tiles(int deg) { return (int)(((unsigned)deg + kHeavyTile - 1) / kHeavyTile); }

// Block-wide reduction of the per-thread statistics into s.red[0] (thread 0).
// S is any shared struct with `Acc red[kBlock / kWarp]` and `int last`.
template <typename S>
__device__ __forceinline__ void acc_reduce(Acc a, S& s) {
  a.maxdeg = __reduce_max_sync(0xffffffffu, a.maxdeg);
  a.mindist = __reduce_min_sync(0xffffffffu, a.mindist);
  a.visited = __reduce_add_sync(0xffffffffu, a.visited);
  a.fmin = __reduce_min_sync(0xffffffffu, a.fmin);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s.red[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
      s.red[0].maxdeg = max(s.red[0].maxdeg, s.red[w].maxdeg);
      s.red[0].mindist = min(s.red[0].mindist, s.red[w].mindist);
      s.red[0].visited += s.red[w].visited;
      s.red[0].fmin = min(s.red[0].fmin, s.red[w].fmin);
    }
  }
}

// Append (v, deg) or (v, tiles) to a list without the staging queue: used only
// when a round produces more pushes than the shared queue holds. The threads
// that overflow together share one packed atomic.
__device__ __forceinline__ void direct_append(unsigned long long* packed, int* list, unsigned* off, int v, int w) {
  cg::coalesced_group g = cg::coalesced_threads();
  const int pre = cg::exclusive_scan(g, w);
  const int tot = cg::reduce(g, w, cg::plus<int>());
  unsigned long long base = 0;
  if (g.thread_rank() == 0) base = atomicAdd(packed, ((unsigned long long)g.size() << 32) | (unsigned)tot);
  base = g.shfl(base, 0);
  const int pos = (int)(base >> 32) + (int)g.thread_rank();
  list[pos] = v;
  off[pos] = (unsigned)(base & 0xffffffffu) + (unsigned)pre;
}

// Append v (degree deg) to far pile p; the threads that append together share
// one atomic. False when the pile is full (the size counter may then pass the
// capacity: readers clamp it).
__device__ __forceinline__ bool pile_append(const Ctx& c, int p, int v, int deg) {
  cg::coalesced_group g = cg::coalesced_threads();
  unsigned base = 0;
  if (g.thread_rank() == 0) base = atomicAdd(&c.ctl->psize[p], (unsigned)g.size());
  base = g.shfl(base, 0);
  const unsigned pos = base + g.thread_rank();
  if (pos >= c.pile_cap || pos < base) return false;
  c.pile[p][pos] = v;
  c.pdeg[p][pos] = deg;
  return true;
}

// Per-block distance histograms of the budgeted near/far ordering (shared
// memory; h null when off): h[0..kHistBins) for the next frontier (every near
// push adds the vertex's degree to the bin of its value, (val - fbase) >> shift
// clamped to the bins), h[kHistBins..) for the far pile (every new pile entry,
// relative to pbase). The block adds its bins to the device histograms once
// per launch.
struct Hists {
  unsigned* h;
  int fbase;
  int pbase;
  int shift;
};

__device__ __forceinline__ int hist_bin(int val, int base, int shift) {
  const long long off = ((long long)val - (long long)base) >> shift;
  return (int)(off < 0 ? 0 : (off >= kHistBins ? kHistBins - 1 : off));
}

__device__ __forceinline__ void hist_near(const Hists& hs, int val, int deg) {
  atomicAdd(&hs.h[hist_bin(val, hs.fbase, hs.shift)], (unsigned)deg);
}

__device__ __forceinline__ void hist_far(const Hists& hs, int val, int deg) {
  atomicAdd(&hs.h[kHistBins + hist_bin(val, hs.pbase, hs.shift)], (unsigned)deg);
}

// Defer v (new value val, at or above the threshold) to the current far pile.
// The pile's bitmap keeps one live entry per vertex: a vertex already on the
// pile only lowers the pile's minimum. Vertices without edges are never
// deferred. With a warp stage the entry is staged (published by warp_publish
// with one atomic per flush); without one it is appended at once. False when
// the pile is full: the caller then pushes v into the next frontier, which is
// always valid. With the edge budget (hs) new entries are histogrammed.
struct WarpStage;
__device__ __forceinline__ bool stage_far(const Ctx& c, int pile, WarpStage* ws, int v, int deg);

__device__ __forceinline__ bool defer_vertex(const Ctx& c, Acc& a, int pile, int v, int val, WarpStage* ws,
                                             const Hists* hs) {
  const unsigned bit = 1u << (v & 31);
  unsigned* w = &c.fbm[v >> 5];
  if (*(volatile unsigned*)w & bit) {
    a.fmin = min(a.fmin, val);
    return true;
  }
  if (atomicOr(w, bit) & bit) {
    a.fmin = min(a.fmin, val);
    return true;
  }
  const int deg = c.g.nindex[v + 1] - c.g.nindex[v];
  if (deg == 0) {
    atomicAnd(w, ~bit);
    return true;
  }
  if (!stage_far(c, pile, ws, v, deg)) {
    atomicAnd(w, ~bit);
    return false;
  }
  a.fmin = min(a.fmin, val);
  if (hs) hist_far(*hs, val, deg);
  return true;
}

// A near push of v supersedes v's pile entry, if any (its bit is cleared, so
// the entry is dropped when the pile is next read). Needed where the
// threshold may fall (the edge budget): there a pile entry cannot be told
// stale from its value alone.
__device__ __forceinline__ void unpile(const Ctx& c, int v) {
  const unsigned bit = 1u << (v & 31);
  unsigned* w = &c.fbm[v >> 5];
  if (*(volatile unsigned*)w & bit) atomicAnd(w, ~bit);
}

// Record vertex v (degree deg >= 1) in the next frontier. The bitmap bit is
// already set, and the frontier minimum already updated, by the caller.
__device__ __forceinline__ void stage_entry(const Ctx& c, Stage& s, Acc& a, int nxt, int v, int deg) {
  a.maxdeg = max(a.maxdeg, deg);
  int p = atomicAdd(&s.n, 1);
  if (p < kQueue) {
    s.q[p] = v;
    s.qd[p] = deg;
  } else {
    direct_append(&c.ctl->slot[nxt].packed, c.wl[nxt], c.woff[nxt], v, deg);
  }
  if (deg >= c.heavy) {
    const int t = heavy_tiles(deg);
    p = atomicAdd(&s.hn, 1);
    if (p < kHQueue) {
      s.hq[p] = v;
      s.ht[p] = t;
    } else {
      direct_append(&c.ctl->slot[nxt].hpacked, c.hwl[nxt], c.htoff[nxt], v, t);
    }
  }
}

// Push after a successful atomicMin (old > val). The frontier minimum is
// lowered on every improvement, including repeat improvements of a vertex that
// is already in the next frontier, so it is a true lower bound of the values
// the next iteration reads. A plain read of the bitmap word skips the atomic
// for vertices already pushed in this launch (bits of the next frontier are
// only set during the launch, so a set bit that is read is never stale).
// Vertices without edges leave the frontier at once.
__device__ __forceinline__ void push_vertex(const Ctx& c, Stage& s, Acc& a, int nxt, int v, int val, int old) {
  if (old == kInf) a.visited++;
  a.mindist = min(a.mindist, val);
  const unsigned bit = 1u << (v & 31);
  unsigned* w = &c.bm[nxt][v >> 5];
  if (*(volatile unsigned*)w & bit) return;
  if (atomicOr(w, bit) & bit) return;
  const int deg = c.g.nindex[v + 1] - c.g.nindex[v];
  if (deg == 0) {
    atomicAnd(w, ~bit);
    return;
  }
  stage_entry(c, s, a, nxt, v, deg);
}

// Exclusive scan of up to kHQueue ints in shared memory by warp 0.
__device__ __forceinline__ int warp_scan_heavy(Stage& s, int hn) {
  constexpr int kPer = kHQueue / kWarp;
  const int lane = threadIdx.x & 31;
  int loc[kPer];
  int sum = 0;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int j = lane * kPer + i;
    loc[i] = sum;
    sum += j < hn ? s.ht[j] : 0;
  }
  int incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  const int excl = incl - sum;
  const int tot = __shfl_sync(0xffffffffu, incl, 31);
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int j = lane * kPer + i;
    if (j < hn) s.ht[j] = excl + loc[i];
  }
  return tot;
}

// Publish the staged pushes of this block (block-uniform call): one packed
// atomic reserves positions and edge offsets for all staged entries.
__device__ __forceinline__ void stage_flush(const Ctx& c, Stage& s, int nxt) {
  __syncthreads();
  const int n = min(s.n, kQueue);
  const int hn = min(s.hn, kHQueue);
  __syncthreads();  // every thread has read the counters before anyone changes them
  if (n == 0 && hn == 0) return;
  const int t = threadIdx.x;
  int d[kScanItems];
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    const int j = t * kScanItems + i;
    d[i] = j < n ? s.qd[j] : 0;
  }
  int tot = 0;
  BlockScanT(s.scan).ExclusiveSum(d, d, tot);
  if (hn && t < 32) {
    const int htot = warp_scan_heavy(s, hn);
    if (t == 0) s.hbase = atomicAdd(&c.ctl->slot[nxt].hpacked, ((unsigned long long)hn << 32) | (unsigned)htot);
  }
  if (t == 0) {
    if (n) s.base = atomicAdd(&c.ctl->slot[nxt].packed, ((unsigned long long)n << 32) | (unsigned)tot);
    s.n = 0;
    s.hn = 0;
  }
  __syncthreads();
  if (n) {
    const int b = (int)(s.base >> 32);
    const unsigned eb = (unsigned)(s.base & 0xffffffffu);
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
      const int j = t * kScanItems + i;
      if (j < n) {
        c.wl[nxt][b + j] = s.q[j];
        c.woff[nxt][b + j] = eb + (unsigned)d[i];
      }
    }
  }
  if (hn) {
    const int b = (int)(s.hbase >> 32);
    const unsigned tb = (unsigned)(s.hbase & 0xffffffffu);
    for (int j = t; j < hn; j += blockDim.x) {
      c.hwl[nxt][b + j] = s.hq[j];
      c.htoff[nxt][b + j] = tb + (unsigned)s.ht[j];
    }
  }
  __syncthreads();
}

// Relax up to R candidate edges of this thread. All dist[] loads are issued
// before any atomicMin. A value read before another thread lowered it is only
// larger, which can cost an unneeded atomic but never skips an improvement.
template <int ALG, int R>
__device__ __forceinline__ void relax_batch(const Ctx& c, Stage& s, Acc& a, int nxt, const int* du, const int* nv,
                                            const int* wv, const bool* ok) {
  int cand[R], cur[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    cand[r] = ok[r] ? Op<ALG>::cand(du[r], wv[r]) : kInf;
    cur[r] = ok[r] ? c.dist[nv[r]] : kInf;
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (cand[r] < cur[r]) {
      const int old = atomicMin(&c.dist[nv[r]], cand[r]);
      if (cand[r] < old) push_vertex(c, s, a, nxt, nv[r], cand[r], old);
    }
  }
}

// Relax CSR entries [lo, hi) of one source with value du. The calling group has
// gsize threads and this thread is `lane` in it. Aligned 16-byte units of nlist
// (and eweight) are read with one 128-bit load; a unit that would reach past
// the end of the arrays is read element by element.
template <int ALG>
__device__ __forceinline__ void relax_range(const Ctx& c, Stage& s, Acc& a, int nxt, int du, int lo, int hi, int lane,
                                            int gsize) {
  const int* __restrict__ nl = c.g.nlist;
  const int* __restrict__ ew = c.g.eweight;
  const int dus[4] = {du, du, du, du};
  if (c.g.vec_ok && hi - lo >= 8) {
    // 64-bit index arithmetic: edges may come within a few units of INT_MAX
    const long long q0 = lo >> 2;
    const long long q1 = ((long long)hi + 3) >> 2;
    for (long long q = q0 + lane; q < q1; q += gsize) {
      const long long k0 = q << 2;
      int nv[4], wv[4] = {0, 0, 0, 0};
      bool ok[4];
      if (k0 + 3 < c.g.edges) {
        const int4 x = ld_adj(reinterpret_cast<const int4*>(nl + k0));
        nv[0] = x.x; nv[1] = x.y; nv[2] = x.z; nv[3] = x.w;
        if (Op<ALG>::kWeighted) {
          const int4 y = ld_adj(reinterpret_cast<const int4*>(ew + k0));
          wv[0] = y.x; wv[1] = y.y; wv[2] = y.z; wv[3] = y.w;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) ok[r] = k0 + r >= lo && k0 + r < hi;
      } else {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const long long k = k0 + r;
          ok[r] = k >= lo && k < hi;
          nv[r] = ok[r] ? nl[k] : 0;
          if (Op<ALG>::kWeighted) wv[r] = ok[r] ? ew[k] : 0;
        }
      }
      relax_batch<ALG, 4>(c, s, a, nxt, dus, nv, wv, ok);
    }
  } else {
    for (long long k0 = lo + (long long)lane * 4; k0 < hi; k0 += (long long)gsize * 4) {
      int nv[4], wv[4] = {0, 0, 0, 0};
      bool ok[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const long long k = k0 + r;
        ok[r] = k < hi;
        nv[r] = ok[r] ? ld_adj(nl + k) : 0;
        if (Op<ALG>::kWeighted) wv[r] = ok[r] ? ld_adj(ew + k) : 0;
      }
      relax_batch<ALG, 4>(c, s, a, nxt, dus, nv, wv, ok);
    }
  }
}

// Last j in [0, n) with off[j] <= x (off[0] == 0 <= x).
__device__ __forceinline__ int owner_search(const unsigned* off, int n, unsigned x) {
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    const int mid = lo + ((hi - lo) >> 1);
    if (off[mid] <= x) lo = mid; else hi = mid;
  }
  return lo;
}

// Warp-cooperative version for global arrays (warp 0 calls it; every lane gets
// the result): each round probes 32 evenly spaced positions, so the range
// shrinks 32-fold per round of parallel loads instead of 2-fold per dependent load.
__device__ __forceinline__ int owner_search_warp(const unsigned* off, int n, unsigned x) {
  const int lane = threadIdx.x & 31;
  int lo = 0, hi = n;  // off[lo] <= x, answer in [lo, hi)
  while (hi - lo > 32) {
    const long long span = hi - lo;
    const int p = lo + (int)((span * lane) / 32);
    const unsigned ballot = __ballot_sync(0xffffffffu, off[p] <= x);
    const int last = 31 - __clz(ballot);  // lane 0 always qualifies (p == lo)
    const int nlo = lo + (int)((span * last) / 32);
    const int nhi = last == 31 ? hi : lo + (int)((span * (last + 1)) / 32);
    lo = nlo;
    hi = nhi;
  }
  const int p = lo + lane;
  const unsigned ballot = __ballot_sync(0xffffffffu, p < hi && off[p] <= x);
  return lo + 31 - __clz(ballot);
}

// Flush only when the staging queue is at least half full (block-uniform).
__device__ __forceinline__ void stage_flush_if_half(const Ctx& c, Stage& s, int nxt) {
  __syncthreads();
  const bool full = s.n >= kQueue / 2 || s.hn >= kHQueue / 2;
  __syncthreads();
  if (full) stage_flush(c, s, nxt);
}

// Contiguous share [lo, hi) of [0, total) for this block among `nb` blocks.
__device__ __forceinline__ void block_share(unsigned total, int nb, unsigned* lo, unsigned* hi) {
  *lo = (unsigned)(((unsigned long long)total * blockIdx.x) / nb);
  *hi = (unsigned)(((unsigned long long)total * (blockIdx.x + 1)) / nb);
}

// Heavy frontier vertices: their adjacency is cut into tiles of kHeavyTile
// entries. Each block takes a contiguous share of the tile sequence, finds the
// vertex of its first tile once, and walks forward.
template <int ALG>
__device__ void heavy_path(const Ctx& c, const CtlHead& S, Stage& s, Acc& a, int cur, int nxt, int active) {
  const unsigned long long hp = S.slot[cur].hpacked;
  const int nh = slot_size(hp);
  const unsigned ntiles = slot_edges(hp);
  if (ntiles == 0) return;
  unsigned t0, t1;
  block_share(ntiles, active, &t0, &t1);
  if (t0 >= t1) return;  // uniform
  const unsigned* toff = c.htoff[cur];
  if (threadIdx.x < 32) {
    const int j = owner_search_warp(toff, nh, t0);
    if (threadIdx.x == 0) s.j0 = j;
  }
  __syncthreads();
  int j = s.j0;
  for (unsigned t = t0; t < t1; ++t) {
    while (j + 1 < nh && toff[j + 1] <= t) ++j;
    const int u = c.hwl[cur][j];
    const int du = c.dist[u];
    const int beg = c.g.nindex[u];
    const int end = c.g.nindex[u + 1];
    const int lo = beg + (int)(t - toff[j]) * kHeavyTile;
    const int hi = end - lo > kHeavyTile ? lo + kHeavyTile : end;  // lo + kHeavyTile may pass INT_MAX
    if (Op<ALG>::valid(du)) relax_range<ALG>(c, s, a, nxt, du, lo, hi, threadIdx.x, blockDim.x);
    stage_flush_if_half(c, s, nxt);
  }
}

// Clear the bitmap of F_{i-1} (slot old): by entries when it is small, by
// words otherwise. Spread over the launch's `active` blocks.
__device__ __forceinline__ void clear_old(const Ctx& c, const CtlHead& S, int old, int active) {
  const int n = slot_size(S.slot[old].packed);
  unsigned* bm = c.bm[old];
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long stride = (long long)active * blockDim.x;
  if ((long long)n * 4 > c.bm_words) {
    for (long long w = tid; w < c.bm_words; w += stride) bm[w] = 0u;
  } else {
    const int* wl = c.wl[old];
    for (long long j = tid; j < n; j += stride) bm[wl[j] >> 5] = 0u;
  }
}

template <class H>
static __device__ __forceinline__ void finish_iteration(const Ctx& c, H& S, int i, int cur, int nxt, int old);

// Copy the head of the control block to (or from) shared memory: one coalesced
// access, from L2 (other blocks wrote it). Block-uniform; the caller synchronises.
__device__ __forceinline__ void load_head(const Ctx& c, CtlHead& S) {
  if (threadIdx.x < kHeadWords)
    reinterpret_cast<unsigned*>(&S)[threadIdx.x] =
        __ldcg(reinterpret_cast<const unsigned*>(static_cast<const CtlHead*>(c.ctl)) + threadIdx.x);
}
__device__ __forceinline__ void store_head(const Ctx& c, const CtlHead& S) {
  if (threadIdx.x < kHeadWords)
    __stcg(reinterpret_cast<unsigned*>(static_cast<CtlHead*>(c.ctl)) + threadIdx.x,
           reinterpret_cast<const unsigned*>(&S)[threadIdx.x]);
}

// Count this block into `done` (thread 0, after the block's writes and a block
// barrier): they are visible to the block that finishes the iteration.
__device__ __forceinline__ unsigned arrive(const Ctx& c) {
  unsigned t;
  asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(t) : "l"(&c.ctl->done) : "memory");
  return t;
}

// Blocks of a launch that take part in it. Blocks at or above this index
// return at once, so a small frontier does not pay for the whole grid; the
// clearing of F_{i-1} is work too. Full sweeps pass `need` = gridDim.x.
__device__ __forceinline__ int active_blocks(const Ctx& c, const CtlHead& S, int old, long long need) {
  const int n_old = slot_size(S.slot[old].packed);
  const long long clear = ((long long)n_old * 4 > c.bm_words) ? ((long long)c.bm_words + 8191) / 8192
                                                                : ((long long)n_old + 2047) / 2048;
  long long a = need > clear ? need : clear;
  if (a < 1) a = 1;
  if (a > gridDim.x) a = gridDim.x;
  return (int)a;
}

// Common epilogue: publish block statistics and let the last block finish the
// iteration. Every block of the launch, active or not, counts into `done`, so
// the iteration advances only after every block has read its state.
template <class H, typename Sh>
__device__ __forceinline__ bool block_epilogue(const Ctx& c, H& S, Sh& s, const Acc& a, int i, int cur, int nxt,
                                               int old) {
  acc_reduce(a, s);
  if (threadIdx.x == 0) {
    const Acc& r = s.red[0];
    Slot& sl = c.ctl->slot[nxt];
    if (r.maxdeg) atomicMax(&sl.maxdeg, r.maxdeg);
    if (r.mindist != kInf) atomicMin(&sl.mindist, r.mindist);
    if (r.visited) atomicAdd((unsigned long long*)&c.ctl->visited, (unsigned long long)r.visited);
    // far pushes of a relax or trim launch go onto pile pcur, a move's onto the other
    if (r.fmin != kInf) atomicMin(&c.ctl->pmin[S.split == 1 ? 1 - S.pcur : S.pcur], r.fmin);
    s.last = (arrive(c) == gridDim.x - 1);
  }
  __syncthreads();
  const bool last = s.last;
  if (last) finish_iteration(c, S, i, cur, nxt, old);
  return last;  // this block finished the iteration
}

// Epilogue of a block with no work in this launch.
template <class H, typename Sh>
__device__ __forceinline__ bool idle_epilogue(const Ctx& c, H& S, Sh& s, int i, int cur, int nxt, int old) {
  if (threadIdx.x == 0) s.last = (arrive(c) == gridDim.x - 1);
  __syncthreads();
  const bool last = s.last;
  if (last) finish_iteration(c, S, i, cur, nxt, old);
  return last;  // this block finished the iteration
}

// The launch's start time is taken by block 0, which the scheduler dispatches
// first; the last block reads it after every block has finished.
__device__ __forceinline__ void block_prologue(const Ctx& c) {
  if (blockIdx.x == 0 && threadIdx.x == 0) c.ctl->tstart = globaltimer();
}

// ---------------------------------------------------------------------------
// Data-driven push, vertex granularity: thread, warp or block per frontier
// vertex. Heavy vertices are skipped here and taken by the heavy path.

template <int ALG, int VAR, class H>
__device__ __forceinline__ bool body_push(const Ctx& c, H& S, Stage& s) {
  block_prologue(c);
  const int i = S.iter;
  const int cur = i % 3, nxt = (i + 1) % 3, old = (i + 2) % 3;
  const int n = slot_size(S.slot[cur].packed);
  const int per = VAR == kVPThread ? kBlock : (VAR == kVPWarp ? kBlock / kWarp : 1);
  const int active = active_blocks(c, S, old, ((long long)n + per - 1) / per + slot_edges(S.slot[cur].hpacked));
  if (blockIdx.x >= active) {
    return idle_epilogue(c, S, s, i, cur, nxt, old);
  }
  stage_init(s);
  Acc a;
  acc_init(a);
  clear_old(c, S, old, active);
  __syncthreads();
  const int* wl = c.wl[cur];

  for (;;) {
    if (threadIdx.x == 0) s.chunk = atomicAdd(&c.ctl->chunk, per);
    __syncthreads();
    const int base = s.chunk;
    if (base >= n) break;  // uniform
    if (VAR == kVPThread) {
      const int idx = base + threadIdx.x;
      if (idx < n) {
        const int u = wl[idx];
        const int beg = c.g.nindex[u], end = c.g.nindex[u + 1];
        const int du = c.dist[u];
        if (end - beg < c.heavy && Op<ALG>::valid(du)) relax_range<ALG>(c, s, a, nxt, du, beg, end, 0, 1);
      }
    } else if (VAR == kVPWarp) {
      const int idx = base + threadIdx.x / kWarp;
      if (idx < n) {
        const int u = wl[idx];
        const int beg = c.g.nindex[u], end = c.g.nindex[u + 1];
        const int du = c.dist[u];
        if (end - beg < c.heavy && Op<ALG>::valid(du))
          relax_range<ALG>(c, s, a, nxt, du, beg, end, threadIdx.x % kWarp, kWarp);
      }
    } else {
      const int u = wl[base];
      const int beg = c.g.nindex[u], end = c.g.nindex[u + 1];
      const int du = c.dist[u];
      if (end - beg < c.heavy && Op<ALG>::valid(du))
        relax_range<ALG>(c, s, a, nxt, du, beg, end, threadIdx.x, blockDim.x);
    }
    stage_flush_if_half(c, s, nxt);
  }
  heavy_path<ALG>(c, S, s, a, cur, nxt, active);
  stage_flush(c, s, nxt);
  return block_epilogue(c, S, s, a, i, cur, nxt, old);
}

// ---------------------------------------------------------------------------
// Edge-balanced push: the frontier's edges [0, edges) are split into one
// contiguous share per warp of the grid (equal edges, hence equal work). A warp
// finds the frontier entry holding its first edge once (warp-cooperative
// search) and walks its share in warp tiles of kWarpTile edges: it loads the
// entries overlapping the tile into its own slice of shared memory, and each
// lane relaxes kEdgesPerThread consecutive edges. Warps never wait for each
// other: each stages its pushes in its own queue and publishes them with a
// warp scan and one packed atomic. No vertex is too big or too small: work is
// split by edges, as in the reference's edge-centric codes.
constexpr int kWarpTile = kWarp * kEdgesPerThread;  // edges per warp tile
// Warp queue capacity; a tile queues at most kWarpTile vertices, and the queue
// is resolved when the next tile's might not fit. 192 rather
// than 256: the 5 KB less shared memory per block is L1 for the random value
// and bitmap reads (RMAT-22 SSSP 4% faster; 128 loses on grids).
#ifndef I2_WARP_QUEUE
#define I2_WARP_QUEUE 192
#endif
constexpr int kWarpQueue = I2_WARP_QUEUE;
static_assert(kWarpQueue % kWarp == 0 && kWarpTile <= kWarpQueue, "a tile's vertices must fit");
constexpr int kWarpsPerBlock = kBlock / kWarp;

struct WarpStage {
  unsigned off[kWarpTile + kWarp];
  int beg[kWarpTile];
  int du[kWarpTile];
  int q[kWarpQueue];
  int qd[kWarpQueue];
  int n;
};

// Stage a push into the warp's queue (heavy entries go straight to their list).
__device__ __forceinline__ void warp_stage_entry(const Ctx& c, WarpStage& ws, Acc& a, int nxt, int v, int deg) {
  a.maxdeg = max(a.maxdeg, deg);
  const int p = atomicAdd(&ws.n, 1);
  if (p < kWarpQueue) {
    ws.q[p] = v;
    ws.qd[p] = deg;
  } else {
    direct_append(&c.ctl->slot[nxt].packed, c.wl[nxt], c.woff[nxt], v, deg);
  }
  if (deg >= c.heavy) direct_append(&c.ctl->slot[nxt].hpacked, c.hwl[nxt], c.htoff[nxt], v, heavy_tiles(deg));
}

// Stage a far-pile entry of the near/far ordering: kept in the warp's queue
// as ~v (negative) beside its degree, and published by warp_publish<true>.
// Without room in the queue it is appended at once.
__device__ __forceinline__ bool stage_far(const Ctx& c, int pile, WarpStage* ws, int v, int deg) {
  const int p = atomicAdd(&ws->n, 1);
  if (p < kWarpQueue) {
    ws->q[p] = ~v;
    ws->qd[p] = deg;
    return true;
  }
  return pile_append(c, pile, v, deg);
}

// Publish the warp's resolved queue entries [0, n) (warp-uniform call): q[j] a
// vertex and qd[j] its degree, 0 where the entry was dropped. One packed atomic
// reserves positions and edge offsets in the next frontier for all of them.
// DEFER: negative entries (~v) are far-pile entries; they go onto the current
// pile with one more atomic. Far entries that find the pile full join the next
// frontier. Lane l owns the entries l, l + 32, ...
template <bool DEFER = false>
__device__ __forceinline__ void warp_publish(const Ctx& c, WarpStage& ws, int nxt, int n, int pile) {
  constexpr int kPer = kWarpQueue / kWarp;
  const int lane = threadIdx.x & 31;
  if constexpr (DEFER) {
    int nf = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int j = lane + i * kWarp;
      nf += (j < n && ws.q[j] < 0 && ws.qd[j] > 0) ? 1 : 0;
    }
    int fincl = nf;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, fincl, o);
      if (lane >= o) fincl += y;
    }
    const int ftot = __shfl_sync(0xffffffffu, fincl, 31);
    if (ftot) {
      const int p = pile;
      unsigned pb = 0;
      if (lane == 0) pb = atomicAdd(&c.ctl->psize[p], (unsigned)ftot);
      pb = __shfl_sync(0xffffffffu, pb, 0);
      unsigned k = pb + (unsigned)(fincl - nf);
      for (int i = 0; i < kPer; ++i) {
        const int j = lane + i * kWarp;
        if (j < n && ws.q[j] < 0 && ws.qd[j] > 0) {
          const int v = ~ws.q[j];
          if (k < c.pile_cap && k >= pb) {
            c.pile[p][k] = v;
            c.pdeg[p][k] = ws.qd[j];
          } else {  // pile full: the vertex joins the next frontier instead
            const unsigned bit = 1u << (v & 31);
            atomicAnd(&c.fbm[v >> 5], ~bit);
            if (!(atomicOr(&c.bm[nxt][v >> 5], bit) & bit)) {
              ws.q[j] = v;
              if (ws.qd[j] >= c.heavy)
                direct_append(&c.ctl->slot[nxt].hpacked, c.hwl[nxt], c.htoff[nxt], v, heavy_tiles(ws.qd[j]));
            }
          }
          ++k;
        }
      }
      __syncwarp();
    }
  }
  // frontier entries: count and degree prefix in one 64-bit scan
  unsigned long long sum = 0;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int j = lane + i * kWarp;
    if (j < n && (!DEFER || ws.q[j] >= 0) && ws.qd[j] > 0) sum += (1ull << 32) | (unsigned)ws.qd[j];
  }
  unsigned long long incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  unsigned long long base = 0;
  if (lane == 31 && incl) base = atomicAdd(&c.ctl->slot[nxt].packed, incl);
  base = __shfl_sync(0xffffffffu, base, 31) + incl - sum;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int j = lane + i * kWarp;
    if (j < n && (!DEFER || ws.q[j] >= 0) && ws.qd[j] > 0) {
      c.wl[nxt][slot_size(base)] = ws.q[j];
      c.woff[nxt][slot_size(base)] = slot_edges(base);
      base += (1ull << 32) | (unsigned)ws.qd[j];
    }
  }
  __syncwarp();
}

// Resolve and publish the warp's queue of n lowered vertices (warp-uniform
// call). An entry is a vertex whose value a relaxation lowered; the frontier
// bitmap decides here, for up to kPart entries per lane at once, whether it is
// pushed, so the chain of dependent bitmap read, atomicOr and degree reads is
// paid once per queue and not for each edge of every tile that lowers a value
// (ER 2M SSSP 1,651 -> 1,558 us, RMAT-22 SSSP 2,314 -> 2,205, grid 2000^2 BFS
// 2,580 -> 2,337, a batch of 32 graphs 6,476 -> 5,952).
// BFS (visited counted here; level `val`): entries may repeat.
// DEFER: negative entries (~v) are values at or above the threshold, bound for
// the far pile; qd holds the values. One whose vertex has meanwhile fallen
// below the threshold is dropped: the fall queued it as near.
// A vertex without edges keeps its bitmap bit and is dropped: it has nothing
// to relax in any style, and the bit keeps its visit counted once.
template <int ALG, bool DEFER>
__device__ __forceinline__ void warp_resolve(const Ctx& c, WarpStage& ws, Acc& a, int nxt, int n, int thr,
                                             const Hists& hs, int pile) {
  constexpr int kPer = kWarpQueue / kWarp;
  constexpr int kPart = 3;
  static_assert(kPer % kPart == 0, "whole parts");
  const int lane = threadIdx.x & 31;
  __syncwarp();
  for (int part = 0; part < kPer && part * kWarp < n; part += kPart) {
    int v[kPart], deg[kPart];
    unsigned w[kPart];
    bool live[kPart], far[kPart];
#pragma unroll
    for (int r = 0; r < kPart; ++r) {
      const int j = (part + r) * kWarp + lane;
      const int e = j < n ? ws.q[j] : 0;
      live[r] = j < n;
      far[r] = DEFER && e < 0;
      v[r] = far[r] ? ~e : e;
      unsigned* word = (far[r] ? c.fbm : c.bm[nxt]) + (v[r] >> 5);
      w[r] = live[r] ? *(volatile unsigned*)word : ~0u;
      if (DEFER && far[r] && live[r] && *(volatile int*)&c.dist[v[r]] < thr) {
        live[r] = false;
        w[r] = ~0u;
      }
    }
#pragma unroll
    for (int r = 0; r < kPart; ++r) {
      const unsigned bit = 1u << (v[r] & 31);
      deg[r] = 0;
      if (!(w[r] & bit)) {
        deg[r] = c.g.nindex[v[r] + 1] - c.g.nindex[v[r]];
        w[r] = atomicOr((far[r] ? c.fbm : c.bm[nxt]) + (v[r] >> 5), bit);
      }
    }
#pragma unroll
    for (int r = 0; r < kPart; ++r) {
      const unsigned bit = 1u << (v[r] & 31);
      const int j = (part + r) * kWarp + lane;
      const bool won = live[r] && !(w[r] & bit);
      if (ALG == kBFS && won) a.visited++;
      if (DEFER && live[r]) {
        const int val = ws.qd[j];
        if (far[r]) {
          if (won && deg[r] == 0) {
            atomicAnd(&c.fbm[v[r] >> 5], ~bit);  // never on the pile
          } else {
            a.fmin = min(a.fmin, val);
            if (won && hs.h) hist_far(hs, val, deg[r]);
          }
        } else {
          if (hs.h) unpile(c, v[r]);
          if (won && deg[r] && hs.h) hist_near(hs, val, deg[r]);
        }
      }
      if (won && deg[r] && !far[r]) {
        a.maxdeg = max(a.maxdeg, deg[r]);
        if (deg[r] >= c.heavy)
          direct_append(&c.ctl->slot[nxt].hpacked, c.hwl[nxt], c.htoff[nxt], v[r], heavy_tiles(deg[r]));
      }
      if (j < n) ws.qd[j] = won ? deg[r] : 0;
    }
  }
  warp_publish<DEFER>(c, ws, nxt, n, pile);
}

// Relax this lane's candidate edges and queue the vertices whose values fell:
// all dist[] loads first, then all atomicMins, then the queue (its length qn
// is warp-uniform and returned). BFS runs level by level in every style, so an
// unreached neighbour takes the level with a plain store (every writer of the
// iteration writes the same one). CC lowers a label many times in an iteration
// (all vertices relax at once), so a vertex that the next frontier's bitmap
// already holds is not queued again (ER 2M: 1,095 -> 931 us; for SSSP the read
// costs more than it saves, 2%).
template <int ALG, bool DEFER>
__device__ __forceinline__ int warp_relax_batch(const Ctx& c, WarpStage& ws, Acc& a, int nxt, const int* du,
                                                const int* nv, const int* wv, const bool* ok, int thr, int qn) {
  int cand[kEdgesPerThread], old[kEdgesPerThread];
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int r = 0; r < kEdgesPerThread; ++r) {
    cand[r] = ok[r] ? Op<ALG>::cand(du[r], wv[r]) : kInf;
    old[r] = ok[r] ? c.dist[nv[r]] : kInf;
  }
#pragma unroll
  for (int r = 0; r < kEdgesPerThread; ++r) {
    if (ALG == kBFS) {
      if (cand[r] < old[r]) c.dist[nv[r]] = cand[r];
    } else if (cand[r] < old[r]) {
      old[r] = atomicMin(&c.dist[nv[r]], cand[r]);
    }
  }
  bool queue[kEdgesPerThread];
#pragma unroll
  for (int r = 0; r < kEdgesPerThread; ++r) {
    queue[r] = cand[r] < old[r];
    if (ALG == kCC && queue[r]) {
      a.mindist = min(a.mindist, cand[r]);
      queue[r] = !((*(volatile unsigned*)&c.bm[nxt][nv[r] >> 5] >> (nv[r] & 31)) & 1u);
    }
  }
#pragma unroll
  for (int r = 0; r < kEdgesPerThread; ++r) {
    const unsigned m = __ballot_sync(0xffffffffu, queue[r]);
    if (queue[r]) {
      const int p = qn + __popc(m & ((1u << lane) - 1u));
      const bool far = DEFER && cand[r] >= thr;
      ws.q[p] = far ? ~nv[r] : nv[r];
      if (DEFER) ws.qd[p] = cand[r];
      if (ALG != kBFS && old[r] == kInf) a.visited++;
      if (!far) a.mindist = min(a.mindist, cand[r]);
    }
    qn += __popc(m);
  }
  return qn;
}

struct EpiStage {
  Acc red[kBlock / kWarp];
  int last;
};

// Resident blocks per SM that the edge-balanced kernels are compiled for: 5
// leaves them 48 registers, no spills but 56 bytes in the near/far form (6: 40
// registers, 192 bytes there). ER 2M SSSP 1,318 us (6 blocks 1,367; 4 blocks
// 1,323), RMAT-22 near/far 2,007 (2,238; 2,057), RMAT-25 ordered 16,213
// (17,455; 17,664); 3 edges per lane at 5 and 4 blocks 1,396 and 1,342, 2,025
// and 1,967, 16,288 and 16,608.
#ifndef I2_EB_MIN_BLOCKS
#define I2_EB_MIN_BLOCKS 5
#endif
// ... and the other fixed styles' kernels, and the wide forms. The other styles at
// 5 blocks, us, against 6: ER 2 x 10^6 vp_warp SSSP 6,877 / 6,000, RMAT-18 vp_block
// CC 1,518 / 840, RMAT-20 push_topo SSSP 11,440 / 10,500.
#ifndef I2_FIXED_MIN_BLOCKS
#define I2_FIXED_MIN_BLOCKS 6
#endif
// ... and union-find's: the most that it is launched with (style_blocks).
#ifndef I2_UF_MIN_BLOCKS
#define I2_UF_MIN_BLOCKS 6
#endif
// Resident blocks per SM that the selectors' kernels (every style in one
// kernel) are compiled for: 4 leaves them 64 registers, where 6 (40 registers)
// spilled 160-224 bytes per thread. Held-out RMAT/ER/grid graphs
// of 2^18 and 2^20 vertices, geomean time against 6: BFS 0.90, SSSP 0.97-0.98,
// CC 0.97-0.98 for both selectors (5 blocks: 0.93-0.98); grid 4096² BFS 0.92.
// On RMAT-26 the heuristic BFS took 1.21x as long at 4 blocks (its pull
// iterations over 2^26 vertices need the warps), so graphs of
// kWideSelectorNodes vertices or more get the selector kernel compiled for
// I2_FIXED_MIN_BLOCKS.
#ifndef I2_SEL_MIN_BLOCKS
#define I2_SEL_MIN_BLOCKS 4
#endif

struct EBShared {
  EpiStage s;
  WarpStage wss[kWarpsPerBlock];
};

// Near/far ordering: the per-block distance histogram of the edge budget.
static_assert(kHistBins == kBlock, "one histogram bin per thread");
struct EBSharedFar : EBShared {
  unsigned hist[2 * kHistBins];  // next frontier, far pile
};

template <bool DEFER>
using EBSharedT = typename std::conditional<DEFER, EBSharedFar, EBShared>::type;

// Budgeted near/far ordering, start of a launch (block-uniform): clear the
// block's histograms. End of a launch: add them to the device histograms.
__device__ __forceinline__ void block_hist_begin(unsigned* h) {
  h[threadIdx.x] = 0u;
  h[kHistBins + threadIdx.x] = 0u;
  __syncthreads();
}

__device__ __forceinline__ void block_hist_end(const unsigned* h, unsigned long long* dst) {
  __syncthreads();
  const unsigned x = h[threadIdx.x], y = h[kHistBins + threadIdx.x];
  if (x) atomicAdd(&dst[threadIdx.x], (unsigned long long)x);
  if (y) atomicAdd(&dst[kHistBins + threadIdx.x], (unsigned long long)y);
}

// Publish a split launch's staged entries once there are `least` of them
// (warp-uniform call).
__device__ __forceinline__ void split_flush(const Ctx& c, WarpStage& ws, int nxt, int least, int pile) {
  __syncwarp();
  const int n = min(ws.n, kWarpQueue);
  __syncwarp();
  if (n < least) return;
  warp_publish<true>(c, ws, nxt, n, pile);
  if ((threadIdx.x & 31) == 0) ws.n = 0;
  __syncwarp();
}

// Launches of the SSSP near/far ordering other than relaxations (Ctl::split):
//  1 move: F_i is empty, the pile is not, and the threshold has just risen
//    from T0 to T. Each live pile entry with a distance below T moves into
//    F_{i+1}; one at or above T moves onto the other pile. Fixed step: an entry
//    whose distance is below T0 was lowered after it was deferred by a push
//    that put it into a frontier (values only fall and the threshold only
//    rises), so it has been relaxed with that distance and is dropped. Edge
//    budget: an entry is live while its fbm bit is set (a near push clears it)
//    and dead entries are dropped; the first copy of a vertex that moves clears
//    the bit, so it moves once; the kept entries are histogrammed anew (base T)
//    for the next move.
//  3 trim (edge budget): F_i carries more than twice the budget and the
//    threshold has just fallen to T; entries below T move into F_{i+1}, the
//    others onto the pile (nothing is relaxed).
// The loop is block-uniform: a block appends the entries it keeps with one
// atomic per pass (a single pile counter takes every block's appends).
template <class H>
__device__ __forceinline__ bool body_split(const Ctx& c, H& S, EBSharedFar& sh, int i, int cur, int nxt, int old) {
  __shared__ int s_keep[kWarpsPerBlock];
  __shared__ unsigned s_kbase;
  EpiStage& s = sh.s;
  const int mode = S.split;
  const bool budget = S.delta < 0;
  const int p = S.pcur;
  const unsigned long long P = S.slot[cur].packed;
  // F_i's entries first (a trim's input, or what an early move carries), then
  // the pile's (a move)
  const unsigned nf = (unsigned)slot_size(P);
  const unsigned n = nf + (mode == 1 ? min(S.psize[p], c.pile_cap) : 0u);
  const int T = S.threshold, T0 = S.prev_threshold;
  const Hists hs = budget ? Hists{sh.hist, S.hbase, S.pbase, S.hshift} : Hists{};
  const int active = active_blocks(c, S, old, ((long long)n + kBlock - 1) / kBlock);
  if (blockIdx.x >= active) {
    return idle_epilogue(c, S, s, i, cur, nxt, old);
  }
  if (threadIdx.x == 0) s.last = 0;
  Acc a;
  acc_init(a);
  if (budget) block_hist_begin(sh.hist);
  clear_old(c, S, old, active);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  WarpStage& ws = sh.wss[wid];
  if (lane == 0) ws.n = 0;
  __syncwarp();
  const int* pv = c.pile[p];
  const int* pd = c.pdeg[p];
  // kR entries per thread and pass (L2-coherent loads: other blocks wrote
  // these arrays in earlier iterations). kR = 4 measured no faster on RMAT-22
  // moves and slower on trims (fewer blocks share a small frontier).
  constexpr int kR = 1;
  const unsigned stride = (unsigned)active * kBlock * kR;
  for (unsigned base = blockIdx.x * kBlock * kR; base < n; base += stride) {
    int v[kR], d[kR], deg[kR];
    unsigned fw[kR];
    bool in[kR], front[kR];
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const unsigned j = base + (unsigned)r * kBlock + threadIdx.x;
      in[r] = j < n;
      front[r] = j < nf;
      v[r] = in[r] ? (front[r] ? __ldcg(&c.wl[cur][j]) : __ldcg(&pv[j - nf])) : 0;
      deg[r] = 0;
      if (in[r]) {
        if (front[r]) {
          const unsigned w1 = j + 1 < nf ? __ldcg(&c.woff[cur][j + 1]) : slot_edges(P);
          deg[r] = (int)(w1 - __ldcg(&c.woff[cur][j]));
        } else {
          deg[r] = __ldcg(&pd[j - nf]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      fw[r] = in[r] && !front[r] ? __ldcg(&c.fbm[v[r] >> 5]) : 0u;
      d[r] = in[r] ? __ldcg(&c.dist[v[r]]) : 0;
    }
    bool keep[kR];
    int nkeep = 0;
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      keep[r] = false;
      if (!in[r]) continue;
      const unsigned bit = 1u << (v[r] & 31);
      if (front[r]) {  // a frontier entry: below T it stays near, else it goes onto the pile
        if (d[r] >= T && defer_vertex(c, a, p, v[r], d[r], &ws, budget ? &hs : nullptr)) {
          // on the pile
        } else if (!(atomicOr(&c.bm[nxt][v[r] >> 5], bit) & bit)) {
          a.mindist = min(a.mindist, d[r]);
          if (budget) hist_near(hs, d[r], deg[r]);
          warp_stage_entry(c, ws, a, nxt, v[r], deg[r]);
        }
      } else if (budget) {  // a pile entry (move), live while its fbm bit is set
        if (fw[r] & bit) {
          if (d[r] < T) {
            if ((atomicAnd(&c.fbm[v[r] >> 5], ~bit) & bit) && !(atomicOr(&c.bm[nxt][v[r] >> 5], bit) & bit)) {
              a.mindist = min(a.mindist, d[r]);
              hist_near(hs, d[r], deg[r]);
              warp_stage_entry(c, ws, a, nxt, v[r], deg[r]);
            }
          } else {
            keep[r] = true;
            a.fmin = min(a.fmin, d[r]);
            hist_far(hs, d[r], deg[r]);
          }
        }
      } else if (d[r] < T) {  // fixed step
        atomicAnd(&c.fbm[v[r] >> 5], ~bit);
        if (d[r] >= T0) {
          atomicOr(&c.bm[nxt][v[r] >> 5], bit);
          a.mindist = min(a.mindist, d[r]);
          warp_stage_entry(c, ws, a, nxt, v[r], deg[r]);
        }
      } else {
        keep[r] = true;
        a.fmin = min(a.fmin, d[r]);
      }
      nkeep += keep[r] ? 1 : 0;
    }
    if (mode == 1) {  // kept entries onto the other pile: one atomic per block pass
      int incl = nkeep;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) s_keep[wid] = incl;
      __syncthreads();
      if (threadIdx.x == 0) {
        int t = 0;
        for (int w = 0; w < kWarpsPerBlock; ++w) {
          const int x = s_keep[w];
          s_keep[w] = t;
          t += x;
        }
        s_kbase = t ? atomicAdd(&c.ctl->psize[1 - p], (unsigned)t) : 0u;
      }
      __syncthreads();
      unsigned pos = s_kbase + (unsigned)s_keep[wid] + (unsigned)(incl - nkeep);
#pragma unroll
      for (int r = 0; r < kR; ++r) {
        if (keep[r]) {
          if (pos < c.pile_cap) {  // kept entries <= pile entries <= capacity
            c.pile[1 - p][pos] = v[r];
            c.pdeg[1 - p][pos] = deg[r];
          }
          ++pos;
        }
      }
      __syncthreads();  // s_keep and s_kbase are rewritten by the next pass
    }
    split_flush(c, ws, nxt, kWarpQueue - kR * kWarp, p);
  }
  split_flush(c, ws, nxt, 1, p);
  if (budget) block_hist_end(sh.hist, c.hist);
  __syncthreads();
  return block_epilogue(c, S, s, a, i, cur, nxt, old);
}

// DEFER: SSSP near/far ordering (pushes at or above the threshold go onto the
// far pile, and split launches refill the frontier from it).
// LONG: tiles that lie inside one entry skip the offsets, the search and the
// entry reads (the kernels of skewed graphs, where most edges are a hub's;
// elsewhere the test costs 1%). us: RMAT-22 near/far 1,957 -> 1,931, RMAT-25
// ordered 13,525 -> 13,204, CC RMAT 4 x 10^6 1,843 -> 1,741. Reading the next
// such tile's adjacency ahead made it 6-9% slower (spills). What is left is the
// neighbours' random value reads, one L1 or L2 sector an edge.
template <int ALG, bool DEFER = false, bool LONG = false, class H>
__device__ __forceinline__ bool body_edge_balanced(const Ctx& c, H& S, EBSharedT<DEFER>& sh) {
  static_assert(!DEFER || ALG == kSSSP, "near/far ordering is for SSSP");
  EpiStage& s = sh.s;
  block_prologue(c);
  const int i = S.iter;
  const int cur = i % 3, nxt = (i + 1) % 3, old = (i + 2) % 3;
  if constexpr (DEFER) {
    if (S.split) return body_split(c, S, sh, i, cur, nxt, old);
  }
  const int thr = DEFER ? S.threshold : kInf;
  Hists hs{};
  if constexpr (DEFER) {
    if (S.delta < 0) hs = Hists{sh.hist, S.hbase, S.pbase, S.hshift};
  }
  const unsigned long long P = S.slot[cur].packed;
  const int n = slot_size(P);
  const unsigned total = slot_edges(P);
  const int active = active_blocks(c, S, old, ((long long)total + kWarpTile * kWarpsPerBlock - 1) /
                                              (kWarpTile * kWarpsPerBlock));
  if (blockIdx.x >= active) {
    return idle_epilogue(c, S, s, i, cur, nxt, old);
  }
  if (threadIdx.x == 0) s.last = 0;
  Acc a;
  acc_init(a);
  if (DEFER && hs.h) block_hist_begin(hs.h);
  clear_old(c, S, old, active);
  const int lane = threadIdx.x & 31;
  WarpStage& ws = sh.wss[threadIdx.x >> 5];
  int qn = 0;  // queued vertices of this warp
  const int* wl = c.wl[cur];
  const unsigned* woff = c.woff[cur];
  const int* __restrict__ nl = c.g.nlist;
  const int* __restrict__ ew = c.g.eweight;
  // Only as many warps as there are warp tiles take part, so a small frontier
  // is not spread over (and searched by) every warp of the grid.
  const unsigned long long gw = (unsigned long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  const unsigned long long need = ((unsigned long long)total + kWarpTile - 1) / kWarpTile;
  const unsigned long long nw = need < (unsigned long long)active * kWarpsPerBlock
                                    ? (need > 0 ? need : 1)
                                    : (unsigned long long)active * kWarpsPerBlock;
  const unsigned W0 = gw < nw ? (unsigned)((total * gw) / nw) : 0u;
  const unsigned W1 = gw < nw ? (unsigned)((total * (gw + 1)) / nw) : 0u;
  if (W0 < W1) {
    int j = owner_search_warp(woff, n, W0);  // entry holding edge W0
    // the entry that the last tile ended in, where it fills the next tile too:
    // its end, its vertex, and its adjacency's place relative to the edge space
    unsigned lend = 0;
    int lv = 0, lbase = 0;
    for (unsigned e0 = W0; e0 < W1; e0 += kWarpTile) {
      const unsigned e1 = min(W1, e0 + kWarpTile);
      int du[kEdgesPerThread], nv[kEdgesPerThread], wv[kEdgesPerThread];
      bool ok[kEdgesPerThread];
      if (LONG && e1 <= lend) {  // warp-uniform
        const int d = ALG == kBFS ? i : __ldcg(&c.dist[lv]);  // may have fallen since the last tile
        const unsigned b = (unsigned)lbase + e0 + (unsigned)lane;
#pragma unroll
        for (int r = 0; r < kEdgesPerThread; ++r) {
          ok[r] = e0 + lane + r * kWarp < e1;
          nv[r] = ok[r] ? ld_adj(nl + b + r * kWarp) : 0;
          wv[r] = Op<ALG>::kWeighted && ok[r] ? ld_adj(ew + b + r * kWarp) : 0;
          du[r] = d;
        }
#pragma unroll
        for (int r = 0; r < kEdgesPerThread; ++r) ok[r] = ok[r] && Op<ALG>::valid(d);
        if (e1 == lend) ++j;
      } else {
        // offsets of the entries from j on, 32 at a time, until one reaches e1;
        // each batch's vertex ids are loaded with its offsets, and the adjacency
        // start and value of the entries inside the tile right after
        int m = 0;
        for (;;) {
          const int jj = j + m + lane;
          const bool in = jj < n;
          const unsigned w = in ? woff[jj] : total;
          const int v = in ? wl[jj] : 0;
          ws.off[m + lane] = w;
          const int below = __popc(__ballot_sync(0xffffffffu, w < e1));
          if (lane < below) {  // offsets ascend: the entries below e1 are a prefix
            ws.beg[m + lane] = c.g.nindex[v];
            if (ALG != kBFS) ws.du[m + lane] = c.dist[v];
          }
          m += below;
          if (below < kWarp) break;
        }
        __syncwarp();
        const unsigned x0 = e0 + (unsigned)lane * kEdgesPerThread;
        int o = x0 < e1 ? owner_search(ws.off, m, x0) : 0;
#pragma unroll
        for (int r = 0; r < kEdgesPerThread; ++r) {
          const unsigned x = x0 + r;
          ok[r] = x < e1;
          nv[r] = 0;
          wv[r] = 0;
          du[r] = kInf;
          if (ok[r]) {
            while (x >= ws.off[o + 1]) ++o;
            const int e = ws.beg[o] + (int)(x - ws.off[o]);
            nv[r] = ld_adj(nl + e);
            if (Op<ALG>::kWeighted) wv[r] = ld_adj(ew + e);
            du[r] = ALG == kBFS ? i : ws.du[o];  // BFS: F_i is level i
            ok[r] = Op<ALG>::valid(du[r]);
          }
        }
        // the next tile starts at e1: its first entry is the last one with offset <= e1
        lend = ws.off[m];
        if (lend == e1) {
          j += m;
        } else {
          j += m - 1;
          if (LONG && lend >= e1 + kWarpTile) {
            lv = wl[j];
            lbase = ws.beg[m - 1] - (int)ws.off[m - 1];
          } else {
            lend = 0;
          }
        }
      }
      qn = warp_relax_batch<ALG, DEFER>(c, ws, a, nxt, du, nv, wv, ok, thr, qn);
      __syncwarp();
      if (qn > kWarpQueue - kWarpTile) {  // the next tile's might not fit
        warp_resolve<ALG, DEFER>(c, ws, a, nxt, qn, thr, hs, DEFER ? S.pcur : 0);
        qn = 0;
      }
    }
  }
  if (qn) warp_resolve<ALG, DEFER>(c, ws, a, nxt, qn, thr, hs, DEFER ? S.pcur : 0);
  if (DEFER && hs.h) block_hist_end(hs.h, c.hist);
  __syncthreads();
  return block_epilogue(c, S, s, a, i, cur, nxt, old);
}

// ---------------------------------------------------------------------------
// Bitmap-gated topology sweep: thread per vertex, light vertices only; heavy
// frontier vertices take the shared heavy path.
template <int ALG, class H>
__device__ __forceinline__ bool body_push_topo(const Ctx& c, H& S, Stage& s) {
  block_prologue(c);
  stage_init(s);
  Acc a;
  acc_init(a);
  const int i = S.iter;
  const int cur = i % 3, nxt = (i + 1) % 3, old = (i + 2) % 3;
  const int active = gridDim.x;  // topology sweeps use the whole grid
  clear_old(c, S, old, active);
  __syncthreads();
  const unsigned* bmc = c.bm[cur];
  const int V = c.g.nodes;
  for (long long base = (long long)blockIdx.x * kBlock; base < V; base += (long long)gridDim.x * kBlock) {
    const int v = (int)base + threadIdx.x;
    if ((unsigned)v < (unsigned)V && ((bmc[v >> 5] >> (v & 31)) & 1u)) {  // v may pass INT_MAX
      const int beg = c.g.nindex[v];
      const int end = c.g.nindex[v + 1];
      const int du = c.dist[v];
      if (end - beg < c.heavy && Op<ALG>::valid(du)) relax_range<ALG>(c, s, a, nxt, du, beg, end, 0, 1);
    }
    stage_flush_if_half(c, s, nxt);
  }
  heavy_path<ALG>(c, S, s, a, cur, nxt, active);
  stage_flush(c, s, nxt);
  return block_epilogue(c, S, s, a, i, cur, nxt, old);
}

// ---------------------------------------------------------------------------
// Edge-centric sweep over all CSR entries, gated by the source's frontier bit.
template <int ALG, class H>
__device__ __forceinline__ bool body_edge_topo(const Ctx& c, H& S, Stage& s) {
  block_prologue(c);
  stage_init(s);
  Acc a;
  acc_init(a);
  const int i = S.iter;
  const int cur = i % 3, nxt = (i + 1) % 3, old = (i + 2) % 3;
  const int active = gridDim.x;  // topology sweeps use the whole grid
  clear_old(c, S, old, active);
  __syncthreads();
  const unsigned* bmc = c.bm[cur];
  const int E = c.g.edges;
  const long long units = ((long long)E + 3) >> 2;
  const int* __restrict__ sp = c.g.sp;
  const int* __restrict__ nl = c.g.nlist;
  const int* __restrict__ ew = c.g.eweight;
  for (long long base = (long long)blockIdx.x * kBlock; base < units; base += (long long)gridDim.x * kBlock) {
    const long long q = base + threadIdx.x;
    if (q < units) {
      const long long k0 = q << 2;
      int su[4], nv[4], wv[4] = {0, 0, 0, 0}, du[4];
      bool ok[4];
      if (c.g.vec_ok && k0 + 3 < E) {
        const int4 x = ld_adj(reinterpret_cast<const int4*>(sp + k0));
        su[0] = x.x; su[1] = x.y; su[2] = x.z; su[3] = x.w;
        const int4 y = ld_adj(reinterpret_cast<const int4*>(nl + k0));
        nv[0] = y.x; nv[1] = y.y; nv[2] = y.z; nv[3] = y.w;
        if (Op<ALG>::kWeighted) {
          const int4 z = ld_adj(reinterpret_cast<const int4*>(ew + k0));
          wv[0] = z.x; wv[1] = z.y; wv[2] = z.z; wv[3] = z.w;
        }
      } else {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const long long k = k0 + r;
          su[r] = (k < E) ? sp[k] : -1;
          nv[r] = (k < E) ? nl[k] : 0;
          if (Op<ALG>::kWeighted) wv[r] = (k < E) ? ew[k] : 0;
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int u = su[r];
        ok[r] = u >= 0 && ((bmc[u >> 5] >> (u & 31)) & 1u);
        du[r] = ok[r] ? c.dist[u] : kInf;
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) ok[r] = ok[r] && Op<ALG>::valid(du[r]);
      relax_batch<ALG, 4>(c, s, a, nxt, du, nv, wv, ok);
    }
    stage_flush_if_half(c, s, nxt);
  }
  stage_flush(c, s, nxt);
  return block_epilogue(c, S, s, a, i, cur, nxt, old);
}

// ---------------------------------------------------------------------------
// Pull variants (symmetric graphs only). Thread per destination vertex; a warp
// covers 32 consecutive vertices, i.e. exactly one bitmap word, so the next
// frontier's bitmap is written with one plain store per warp. dist[v] is only
// written by v's own thread, so no atomics are needed on it.
template <int ALG, bool FRONTIER, class H>
__device__ __forceinline__ bool body_pull(const Ctx& c, H& S, Stage& s) {
  block_prologue(c);
  stage_init(s);
  Acc a;
  acc_init(a);
  const int i = S.iter;
  const int cur = i % 3, nxt = (i + 1) % 3, old = (i + 2) % 3;
  const int active = gridDim.x;  // every vertex is visited
  clear_old(c, S, old, active);
  __syncthreads();
  const unsigned* bmc = c.bm[cur];
  const int V = c.g.nodes;
  const int* __restrict__ nl = c.g.nlist;
  const int* __restrict__ ew = c.g.eweight;
  const int fmin = S.slot[cur].mindist;
  // Where the style may change between iterations BFS stays level by level (the
  // edge-balanced push takes F_i for level i), so a neighbour reached in this
  // iteration waits. A run of this style alone uses it at once: it recomputes
  // every vertex until none falls, so levels reached early and too large are
  // corrected. It takes fewer iterations where neighbours are visited late in a
  // sweep (RMAT-18 4-5 instead of 5, grid 1024^2 without long edges 1,793 of 2,045).
  // One test of the neighbour's value covers this and an unreached neighbour: with
  // a second one the loop's loads are no longer issued together (RMAT-18, an
  // iteration of the hub's thread 1,450 instead of 1,082 us).
  const bool by_level = ALG == kBFS && !FRONTIER && S.mode != 0;
  const int last = by_level ? i : kInf - 1;  // values above it are no use to BFS
  // Smallest candidate any frontier vertex can produce.
  const int bound = FRONTIER ? (fmin == kInf ? kInf : Op<ALG>::cand(fmin, c.gs.wmin)) : INT_MIN;
  for (long long base = (long long)blockIdx.x * kBlock; base < V; base += (long long)gridDim.x * kBlock) {
    const int v = (int)base + threadIdx.x;
    bool improved = false;
    int best = kInf, dv = kInf, deg = 0;
    if ((unsigned)v < (unsigned)V) {  // v may pass INT_MAX
      dv = c.dist[v];
      best = dv;
      if (!FRONTIER || dv > bound) {
        const int beg = c.g.nindex[v];
        const int end = c.g.nindex[v + 1];
        deg = end - beg;
        for (int k = beg; k < end; ++k) {
          const int u = ld_adj(nl + k);
          if (FRONTIER && !((bmc[u >> 5] >> (u & 31)) & 1u)) continue;
          const int du = c.dist[u];
          if (ALG == kBFS && !FRONTIER ? du > last : !Op<ALG>::valid(du)) continue;
          const int cd = Op<ALG>::cand(du, Op<ALG>::kWeighted ? ld_adj(ew + k) : 0);
          if (cd < best) {
            best = cd;
            if (FRONTIER && best == bound) break;
          }
        }
        if (best < dv) {
          c.dist[v] = best;
          improved = true;
        }
      }
    }
    // A warp covers one whole bitmap word; lane 0's vertex lies in it.
    const unsigned word = __ballot_sync(0xffffffffu, improved);
    if ((threadIdx.x & 31) == 0 && word) c.bm[nxt][v >> 5] = word;
    if (improved) {
      if (dv == kInf) a.visited++;
      a.mindist = min(a.mindist, best);
      stage_entry(c, s, a, nxt, v, deg);
    }
    stage_flush_if_half(c, s, nxt);
  }
  stage_flush(c, s, nxt);
  return block_epilogue(c, S, s, a, i, cur, nxt, old);
}

// ---------------------------------------------------------------------------
// Kernels: one per (algorithm, style) for fixed-style runs, and one dispatch
// kernel per algorithm for the selectors, whose blocks branch on the style
// chosen at the end of the previous iteration (one kernel node per iteration
// instead of a conditional SWITCH node).

// ---------------------------------------------------------------------------
// Union-find CC (kUnionFind; CC on symmetric graphs only). The labels are read
// as parent pointers: every label is a vertex of the same component with an ID
// no larger than the vertex's own (true of the initial labels and of every
// label propagation writes), so following labels ends at a vertex that is its
// own label, a root. The hook launch links, for every edge, the roots of its
// two ends, always the larger root below the smaller one with a compare-and-
// swap on the larger (which succeeds only while it is still a root). The
// smallest ID of a component is therefore never linked and ends as the root of
// the whole component; the compress launch sets every label to its root. The
// result is the minimum-ID labelling that label propagation converges to,
// reached from any propagation state in three launches (below).

// Reads of parents may be served from this SM's L1 and so be stale: a stale
// parent is still an ancestor (links are never undone), and a vertex wrongly
// seen as a root only makes the linking compare-and-swap fail and return its
// true parent, from which the climb continues (ancestors only decrease, so it
// ends). Cached loads matter: the ancestors near a component's root are read by
// most vertices, and L2 would serialise on them.

// Root of x; each step points the visited vertex at its grandparent (path
// halving: any ancestor is a valid label, and a vertex that is not a root never
// becomes one again, so these plain writes cannot undo a link).
__device__ __forceinline__ int uf_find(int* p, int x) {
  for (;;) {
    const int px = p[x];
    if (px == x) return x;
    const int ppx = p[px];
    if (ppx != px) p[x] = ppx;
    x = ppx;
  }
}

// Link the roots of a and b, the larger below the smaller.
__device__ __forceinline__ void uf_union(int* p, int a, int b) {
  int ra = uf_find(p, a), rb = uf_find(p, b);
  while (ra != rb) {
    if (ra < rb) {
      const int t = ra;
      ra = rb;
      rb = t;
    }
    const int seen = atomicCAS(&p[ra], ra, rb);
    if (seen == ra) return;
    ra = uf_find(p, seen);  // ra was linked meanwhile: continue from its root
    rb = uf_find(p, rb);
  }
}

// The same without finding the roots first (the link step of Sutton et al.,
// "Optimizing parallel graph connectivity computation via subgraph sampling",
// IPDPS 2018, with the path halved on the way and an early end where the larger's
// parent is the smaller): pa and pb are ancestors of a and b; climb from the
// larger of the two until the ancestors meet or the larger is a root, which is
// then linked below the smaller. Two vertices whose parents are the same are done
// after those two reads. Returns an ancestor of both.
__device__ __forceinline__ int uf_climb(int* p, int pa, int pb) {
  while (pa != pb) {
    const int high = max(pa, pb), low = min(pa, pb);
    int ph = p[high];
    if (ph == low) return low;
    if (ph == high) {
      ph = atomicCAS(&p[high], high, low);
      if (ph == high) return low;
    }
    pa = p[ph];
    pb = p[low];
    if (pa != ph) p[high] = pa;  // halve the path (high is no root)
  }
  return pa;
}

// Link vertex v with u, pv being v's parent as last seen, by climbing, and put
// both (where they are no roots) below the ancestor found. Returns it or pv.
__device__ __forceinline__ int uf_link(int* p, int v, int pv, int u, int pu) {
  const int low = uf_climb(p, pv, pu);
  if (pu != u && low < pu) p[u] = low;
  if (pv != v && low < pv) p[v] = low;
  return min(pv, low);
}

// Link the ends of an edge, by climbing or by their roots.
__device__ __forceinline__ void uf_edge(int* p, int v, int u, bool climb) {
  if (climb) uf_climb(p, p[v], p[u]);
  else if (u != v) uf_union(p, v, u);
}

// List length from which launch 1 gives a vertex to the whole block. (One thread
// per vertex left the hubs outside the largest tree, as in a batch of RMAT
// graphs, to one thread each: 23 graphs of 10^3 to 10^6 vertices 16,181 us, now
// 751.) From 512 / 2,048 / 8,192 entries, us: that batch 680 / 751 / 852, 23 RMAT
// graphs 774 / 829 / 1,118, 48 graphs of up to 10^5 vertices 325 / 367 / 379;
// single RMAT graphs the same.
constexpr int kUfBlockDegree = 2048;

// Neighbours each vertex is linked with before the largest tree is sampled.
constexpr int kAfforestLinks = 2;
constexpr int kAfforestSamples = 1024;

// Root of x with coherent loads (the sampling after the first hook launch).
__device__ __forceinline__ int uf_find_fresh(int* p, int x) {
  for (;;) {
    const int px = *(volatile int*)&p[x];
    if (px == x) return x;
    x = px;
  }
}

// Boyer-Moore majority pairs (candidate, count) merge like single votes: a
// majority element of the union survives the merge of the parts' pairs.
__device__ __forceinline__ void vote_merge(int& cand, int& cnt, int c2, int n2) {
  if (c2 == cand) cnt += n2;
  else if (n2 > cnt) { cand = c2; cnt = n2 - cnt; }
  else cnt -= n2;
}

// Called by the whole last block of the first hook launch (kBlock threads):
// the roots of kAfforestSamples vertices spread over the graph, and the root
// held by a majority of them (Boyer-Moore vote, per thread, then merged across
// lanes and warps), taken as the largest tree. Any root would keep the result
// correct; the vote only decides how many vertices the second hook launch can
// skip. Registers and 64 bytes of shared memory: this runs in the epilogue of
// every relax kernel, whose shared-memory size sets the L1 left to it.
__device__ __forceinline__ void uf_sample_giant(const Ctx& c, CtlHead& S) {
  __shared__ int wc[kBlock / kWarp], wn[kBlock / kWarp];
  const int V = c.g.nodes;
  int cand = -1, cnt = 0;
  for (int k = threadIdx.x; k < kAfforestSamples; k += blockDim.x)
    vote_merge(cand, cnt, V > 0 ? uf_find_fresh(c.dist, (int)((unsigned)mis_priority(k) % (unsigned)V)) : 0, 1);
  for (int o = 16; o > 0; o >>= 1) {
    const int c2 = __shfl_down_sync(0xffffffffu, cand, o);
    const int n2 = __shfl_down_sync(0xffffffffu, cnt, o);
    vote_merge(cand, cnt, c2, n2);
  }
  if ((threadIdx.x & 31) == 0) {
    wc[threadIdx.x >> 5] = cand;
    wn[threadIdx.x >> 5] = cnt;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) vote_merge(cand, cnt, wc[w], wn[w]);
    S.uf_giant = cand;
  }
  __syncthreads();
}

// Three launches (CtlHead::uf_phase): (0) link every vertex with its first
// kAfforestLinks neighbours, after which the last block samples the largest
// tree; (1) link the remaining neighbours of every vertex whose root is not
// that tree's (an edge from a skipped vertex to a vertex outside the tree is
// linked from the other end, and an edge inside the tree changes nothing);
// (2) set every label to its root. Links put the larger root below the
// smaller one whatever the order, so the roots are the components' minimum
// IDs, as in a single pass over all edges (sampling scheme of Sutton et al.,
// "Optimizing parallel graph connectivity computation via subgraph sampling",
// IPDPS 2018). On graphs with a giant component the second launch skips most
// edges.
// Order and links (CtlHead::uf_step). On graphs of average degree 6 or more
// (RMAT, ER: neighbours all over the ID range) warps take chunks of 32
// consecutive vertices spread over the whole graph (chunk k * uf_step mod
// chunks, a step near the golden section) and link by climbing. On sparser
// ones (grids, road networks: neighbours close by, trees as deep as the graph
// is long) they take them in ascending order and link roots, whose finds
// flatten the paths that the next vertices walk. Launch 0, us, links spread /
// ascending: RMAT-22 104-121 / 222-333, ER 4M 163-170 / 296-345, grid 4096^2
// 900-1,120 / 455, grid 1000^2 96-139 / 85-92. The whole traversal against one
// order (grid-stride, finds) with a frontier built by the fill: RMAT-22 442 ->
// 231, ER 4M 487 -> 270, RMAT-20 272 -> 221, ER 600,000 248 -> 169, grid 4096^2
// 1,380 -> 666, grid 1000^2 191 -> 158. Bound by the latency of dependent
// parent reads.
template <int ALG, class H>
__device__ __forceinline__ bool body_union(const Ctx& c, H& S, Stage& s) {
  block_prologue(c);
  stage_init(s);
  Acc a;
  acc_init(a);
  const int i = S.iter;
  const int cur = i % 3, nxt = (i + 1) % 3, old = (i + 2) % 3;
  int* p = c.dist;
  const int V = c.g.nodes;
  const int* __restrict__ nl = c.g.nlist;
  const int* __restrict__ ni = c.g.nindex;
  const int phase = S.uf_phase;
  const int giant = S.uf_giant;
  const bool climb = S.uf_step != 1;
  const int lane = threadIdx.x & 31;
  const unsigned chunks = ((unsigned)V + kWarp - 1) / kWarp;
  const unsigned nw = gridDim.x * kWarpsPerBlock;
  const unsigned w0 = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  unsigned at = (unsigned)(((unsigned long long)w0 * S.uf_step) % chunks);
  const unsigned step = (unsigned)(((unsigned long long)nw * S.uf_step) % chunks);
  __syncthreads();  // stage_init
  int top = giant;  // the largest tree's root once every link is made
  if (phase == 2)
    for (int px; (px = p[top]) != top;) top = px;
  for (unsigned k = w0; k < chunks; k += nw) {
    const unsigned v = at * kWarp + lane;
    at += step;
    if (at >= chunks) at -= chunks;
    const bool in = v < (unsigned)V;
    if (phase == 0) {
      if (!in) continue;
      const unsigned b = ni[v], e = ni[v + 1];
      int u[kAfforestLinks], pu[kAfforestLinks];
#pragma unroll
      for (int r = 0; r < kAfforestLinks; ++r) u[r] = b + r < e ? ld_adj(nl + b + r) : (int)v;
      int pv = p[v];
#pragma unroll
      for (int r = 0; r < kAfforestLinks; ++r) pu[r] = climb ? p[u[r]] : 0;
#pragma unroll
      for (int r = 0; r < kAfforestLinks; ++r) {
        if (climb) pv = uf_link(p, (int)v, pv, u[r], pu[r]);
        else if (u[r] != (int)v) uf_union(p, (int)v, u[r]);
      }
    } else if (phase == 1) {
      unsigned b = 0, e = 0;
      if (in) {
        b = (unsigned)ni[v] + kAfforestLinks;
        e = ni[v + 1];
      }
      if (b < e) {
        int x = (int)v;
        for (int px; x != giant && (px = p[x]) != x;) x = px;
        if (x == giant) {
          if (p[v] != giant && (int)v != giant) p[v] = giant;
          e = b;
        }
      }
      // short lists by their thread, longer ones by the warp, the hubs' by the block
      int left = b < e ? (int)(e - b) : 0;
      if (left > kUfBlockDegree) {
        const int q = atomicAdd(&s.hn, 1);
        if (q < kHQueue) {
          s.hq[q] = (int)v;
          left = 0;
        }
      }
      if (left > 0 && left <= kWarp) {
        walk_list(b, e, 0, 1, [&](unsigned j) { uf_edge(p, (int)v, ld_adj(nl + j), climb); });
        left = 0;
      }
      for (unsigned todo = __ballot_sync(0xffffffffu, left > 0); todo; todo &= todo - 1) {
        const int l = __ffs(todo) - 1;
        const int wv = __shfl_sync(0xffffffffu, (int)v, l);
        const unsigned wb = __shfl_sync(0xffffffffu, b, l), we = __shfl_sync(0xffffffffu, e, l);
        walk_list(wb, we, lane, kWarp, [&](unsigned j) { uf_edge(p, wv, ld_adj(nl + j), climb); });
      }
    } else if (in) {
      // compress: read-only finds (a shortening write could replace a finished
      // label with an intermediate ancestor), each thread writing its own label
      const int pv = p[v];
      int x = pv;
      for (int px; x != giant && x != top && (px = p[x]) != x;) x = px;
      if (x == giant) x = top;
      if (x != pv) p[v] = x;
    }
  }
  if (phase == 1) {
    __syncthreads();
    const int nh = min(s.hn, kHQueue);
    for (int q = 0; q < nh; ++q) {
      const int hv = s.hq[q];
      walk_list((unsigned)ni[hv] + kAfforestLinks, ni[hv + 1], threadIdx.x, kBlock,
                [&](unsigned j) { uf_edge(p, hv, ld_adj(nl + j), climb); });
    }
  }
  return block_epilogue(c, S, s, a, i, cur, nxt, old);
}

// ---------------------------------------------------------------------------
// Maximal independent set (kMIS; one style). A frontier entry is an undecided
// vertex v with a cursor into its adjacency: every neighbour before the cursor
// is known not to block v (it does not outrank v, or it is out). An iteration
// moves the cursor on to the first neighbour that outranks v and is undecided,
// and v waits there; one that is in the set makes v out; past the end v joins
// the set and writes its neighbours out, which the waiting ones find when their
// turn comes. Decisions depend only on outranking vertices, whose decisions are
// final, so the set is the greedy one in decreasing rank whatever the order of
// the updates; a vertex in the set outranks all its undecided neighbours, and
// those that outrank it are out already, so its writes are right without
// looking.
//
// Each adjacency list is scanned once over the whole run and mostly not past
// its second entry (a random neighbour outranks v half the time), so the work
// is far below the graph's edges: random status reads bound it. One thread
// scans the first kMisProbe entries, a warp goes on, and lists of
// kMisBlockDegree entries or more take the whole block after the warps are done.
// The first iteration takes every vertex without a list (building one was 60 of
// 195 us on RMAT 3 x 10^5), and each warp stages its own waiting vertices. RMAT
// with 1,000,003 vertices 2,625-3,129 -> 396-587 us, ER 10^6 796 -> 175, grid
// 10^6 699 -> 119; the form before, a warp per vertex that rescanned the list in
// every iteration, left a hub to one warp (2,122 us of its first iteration).
enum { kMisNone, kMisWait, kMisJoin, kMisLeave, kMisMore };  // what an iteration finds for a vertex
// Entries a thread scans (or writes) by itself: 8 / 16 / 32, us: RMAT-22 1,902 /
// 1,776 / 1,730, RMAT 1,000,003 394 / 396 / 411, ER 10^6 180 / 174 / 173, ER with 64
// entries a vertex 235 / 233 / 242.
constexpr int kMisProbe = 16;
// Entries from which the whole block does: 512, 2,048 and 8,192 within 1% on the
// same graphs (after the first iteration few long lists are scanned far).
constexpr int kMisBlockDegree = 2048;

// Outcome of `count` (<= 4) consecutive entries from k on, loaded together:
// bit r of *wait: entry r outranks v and is undecided; returns whether one
// that outranks v is in the set.
__device__ __forceinline__ bool mis_probe(const Ctx& c, int v, int pv, const unsigned* k, int count, unsigned* wait) {
  volatile int* st = c.dist;
  const int* __restrict__ nl = c.g.nlist;
  int u[4], su[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) u[r] = r < count ? ld_adj(nl + k[r]) : v;
#pragma unroll
  for (int r = 0; r < 4; ++r)
    su[r] = (u[r] != v && mis_outranks(u[r], mis_priority(u[r]), v, pv)) ? (int)st[u[r]] : (int)kMisOut;
  unsigned w = 0;
  bool in = false;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    in |= su[r] == kMisIn;
    w |= su[r] == kMisUndecided ? 1u << r : 0u;
  }
  *wait = w;
  return in;
}

// Publish a warp's n staged waiting vertices (warp-uniform call): q the
// vertices, cur their cursors, `left` the lane's share of their entries still
// to scan.
__device__ __forceinline__ void mis_flush(const Ctx& c, const int* q, const int* cur, int n, int left, int nxt) {
  __syncwarp();
  const int lane = threadIdx.x & 31;
  left = __reduce_add_sync(0xffffffffu, left);
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(&c.ctl->slot[nxt].packed, ((unsigned long long)n << 32) | (unsigned)left);
  const int b = slot_size(__shfl_sync(0xffffffffu, base, 0));
  for (int j = lane; j < n; j += kWarp) {
    c.wl[nxt][b + j] = q[j];
    c.woff[nxt][b + j] = (unsigned)cur[j];
  }
  __syncwarp();
}

template <class H>
__device__ __forceinline__ bool body_mis(const Ctx& c, H& S, Stage& s) {
  block_prologue(c);
  const int i = S.iter;
  const int cur = i % 3, nxt = (i + 1) % 3, old = (i + 2) % 3;
  // the first iteration may take every vertex, without a list (a vertex without
  // neighbours joins the set at once)
  const bool all = i == 0 && S.whole;
  const int n = all ? c.g.nodes : slot_size(S.slot[cur].packed);
  const int active = (int)min((long long)gridDim.x, ((long long)n + kBlock - 1) / kBlock);
  if (blockIdx.x >= active) return idle_epilogue(c, S, s, i, cur, nxt, old);
  stage_init(s);
  Acc a;
  acc_init(a);
  __syncthreads();
  const int* wl = c.wl[cur];
  const unsigned* cursor = c.woff[cur];
  volatile int* st = c.dist;
  const int* __restrict__ nl = c.g.nlist;
  const int lane = threadIdx.x & 31;
  // each warp stages its waiting vertices; no warp waits for another
  constexpr int kStage = kQueue / kWarpsPerBlock;
  int* const wq = s.q + (threadIdx.x >> 5) * kStage;
  int* const wcur = s.qd + (threadIdx.x >> 5) * kStage;
  int qn = 0, qleft = 0;
  for (long long base = (long long)blockIdx.x * kBlock; base < n; base += (long long)active * kBlock) {
    const long long idx = base + threadIdx.x;
    int state = kMisNone, v = 0, pv = 0;
    unsigned k = 0, end = 0;
    if (idx < n) {
      v = all ? (int)idx : wl[idx];
      state = kMisMore;
      if (st[v] != kMisUndecided) {  // a neighbour joined the set meanwhile
        state = kMisNone;
        a.visited++;
      } else {
        k = i == 0 ? (unsigned)c.g.nindex[v] : cursor[idx];
        end = c.g.nindex[v + 1];
        pv = mis_priority(v);
        for (int t = 0; t < kMisProbe && state == kMisMore; t += 4) {
          const int cnt = min(4, (int)(end - k));
          const unsigned ks[4] = {k, k + 1, k + 2, k + 3};
          unsigned w = 0;
          if (cnt <= 0) {
            state = kMisJoin;
          } else if (mis_probe(c, v, pv, ks, cnt, &w)) {
            state = kMisLeave;
          } else if (w) {
            k += __ffs(w) - 1;
            state = kMisWait;
          } else {
            k += cnt;
          }
        }
        if (state == kMisMore && k >= end) state = kMisJoin;
      }
    }
    // longer lists: the block's (deferred to after the pass), else the warp's
    bool mine = state == kMisMore;
    if (mine && (int)(end - k) >= kMisBlockDegree) {
      const int p = atomicAdd(&s.hn, 1);
      if (p < kHQueue) {
        s.hq[p] = v;
        s.ht[p] = (int)k;
        state = kMisNone;
        mine = false;
      }
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, mine); todo; todo &= todo - 1) {
      const int l = __ffs(todo) - 1;
      const int wv = __shfl_sync(0xffffffffu, v, l), wpv = __shfl_sync(0xffffffffu, pv, l);
      const unsigned we = __shfl_sync(0xffffffffu, end, l);
      unsigned wk = __shfl_sync(0xffffffffu, k, l);
      int out = kMisJoin;
      for (; wk < we; wk += 4 * kWarp) {
        unsigned ks[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) ks[r] = wk + r * kWarp + lane;
        const int cnt = window_share(wk, we, lane, kWarp);
        unsigned w = 0;
        const bool in = mis_probe(c, wv, wpv, ks, cnt, &w);
        if (__any_sync(0xffffffffu, in)) {
          out = kMisLeave;
          break;
        }
        const int first = __reduce_min_sync(0xffffffffu, w ? (__ffs(w) - 1) * kWarp + lane : INT_MAX);
        if (first != INT_MAX) {
          wk += first;
          out = kMisWait;
          break;
        }
      }
      if (lane == l) {
        state = out;
        k = wk;
      }
    }
    if (state == kMisLeave) {
      st[v] = kMisOut;
      a.visited++;
    }
    // joined: neighbours are out
    bool wide = false;
    if (state == kMisJoin) {
      st[v] = kMisIn;
      a.visited++;
      const unsigned b = c.g.nindex[v];
      if (end - b <= kMisProbe) {
        walk_list(b, end, 0, 1, [&](unsigned j) {
          const int u = ld_adj(nl + j);
          if (u != v) st[u] = kMisOut;
        });
      } else {
        k = b;
        wide = true;
      }
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, wide); todo; todo &= todo - 1) {
      const int l = __ffs(todo) - 1;
      const int wv = __shfl_sync(0xffffffffu, v, l);
      const unsigned wb = __shfl_sync(0xffffffffu, k, l), we = __shfl_sync(0xffffffffu, end, l);
      walk_list(wb, we, lane, kWarp, [&](unsigned j) {
        const int u = ld_adj(nl + j);
        if (u != wv) st[u] = kMisOut;
      });
    }
    // waiting vertices into the warp's queue
    const unsigned waiting = __ballot_sync(0xffffffffu, state == kMisWait);
    if (state == kMisWait) {
      const int p = qn + __popc(waiting & ((1u << lane) - 1u));
      wq[p] = v;
      wcur[p] = (int)k;
      qleft += (int)(end - k);
    }
    qn += __popc(waiting);
    if (qn > kStage - kWarp) {
      mis_flush(c, wq, wcur, qn, qleft, nxt);
      qn = 0;
      qleft = 0;
    }
  }
  if (qn) mis_flush(c, wq, wcur, qn, qleft, nxt);
  __syncthreads();
  // the lists for the whole block
  const int nb = min(s.hn, kHQueue);
  for (int x = 0; x < nb; ++x) {
    const int bv = s.hq[x], bpv = mis_priority(bv);
    const unsigned be = c.g.nindex[bv + 1];
    unsigned bk = s.ht[x];
    int out = kMisJoin;
    for (; bk < be; bk += 4 * kBlock) {
      if (threadIdx.x == 0) {
        s.j0 = INT_MAX;
        s.chunk = 0;
      }
      __syncthreads();
      unsigned ks[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) ks[r] = bk + r * kBlock + threadIdx.x;
      const int t = threadIdx.x;
      const int cnt = window_share(bk, be, t, kBlock);
      unsigned w = 0;
      if (mis_probe(c, bv, bpv, ks, cnt, &w)) s.chunk = 1;
      if (w) atomicMin(&s.j0, (__ffs(w) - 1) * kBlock + t);
      __syncthreads();
      const int found = s.chunk, first = s.j0;
      __syncthreads();  // read before the next step resets them
      if (found) {
        out = kMisLeave;
        break;
      }
      if (first != INT_MAX) {
        bk += first;
        out = kMisWait;
        break;
      }
    }
    if (out == kMisJoin) {
      walk_list(c.g.nindex[bv], be, threadIdx.x, kBlock, [&](unsigned j) {
        const int u = ld_adj(nl + j);
        if (u != bv) st[u] = kMisOut;
      });
    }
    if (threadIdx.x == 0) {
      if (out == kMisWait) {
        const unsigned long long p =
            atomicAdd(&c.ctl->slot[nxt].packed, (1ull << 32) | (be - bk));
        c.wl[nxt][slot_size(p)] = bv;
        c.woff[nxt][slot_size(p)] = bk;
      } else {
        st[bv] = out == kMisJoin ? kMisIn : kMisOut;
        a.visited++;
      }
    }
  }
  __syncthreads();
  return block_epilogue(c, S, s, a, i, cur, nxt, old);
}

// ---------------------------------------------------------------------------
// Kernel wrappers, one launch per iteration. H: what the end of an iteration may
// have to do (common.cuh); with the selector's network in it the pull kernels
// took 69-78 registers and lost the fourth block per SM (BFS pull_frontier,
// launched per iteration, us, before / with the network / FixedHead: RMAT-20
// 1,132 / 1,464 / 1,059, grid 6000^2 83.7 / 108 / 81.8 ms). pull_topo, whose time on
// hubs is one thread's list, needs the 64 registers of the 4 blocks to issue its
// loads together: left to itself the compiler takes 54 (RMAT-20 BFS 23.6 ms).
template <int ALG, int VAR, class H>
__global__ void __launch_bounds__(kBlock) relax_push(const __grid_constant__ Ctx c) {
  __shared__ Stage s;
  __shared__ H S;
  load_head(c, S);
  __syncthreads();
  body_push<ALG, VAR>(c, S, s);
}

template <int ALG, class H, bool LONG = false>
__global__ void __launch_bounds__(kBlock, LONG ? I2_FIXED_MIN_BLOCKS : I2_EB_MIN_BLOCKS)
    relax_edge_balanced(const __grid_constant__ Ctx c) {
  __shared__ EBShared sh;
  __shared__ H S;
  load_head(c, S);
  __syncthreads();
  body_edge_balanced<ALG, false, LONG>(c, S, sh);
}

static __global__ void __launch_bounds__(kBlock, I2_FIXED_MIN_BLOCKS) relax_mis(const __grid_constant__ Ctx c) {
  __shared__ Stage s;
  __shared__ FixedHead S;
  load_head(c, S);
  __syncthreads();
  body_mis(c, S, s);
}

// Edge-balanced SSSP push with near/far ordering (Ctl::delta != 0).
static __global__ void __launch_bounds__(kBlock, I2_EB_MIN_BLOCKS) relax_near_far(const __grid_constant__ Ctx c) {
  __shared__ EBSharedFar sh;
  __shared__ FixedHead S;
  load_head(c, S);
  __syncthreads();
  body_edge_balanced<kSSSP, true>(c, S, sh);
}

template <int ALG, class H>
__global__ void __launch_bounds__(kBlock) relax_push_topo(const __grid_constant__ Ctx c) {
  __shared__ Stage s;
  __shared__ H S;
  load_head(c, S);
  __syncthreads();
  body_push_topo<ALG>(c, S, s);
}

template <int ALG, class H>
__global__ void __launch_bounds__(kBlock) relax_edge_topo(const __grid_constant__ Ctx c) {
  __shared__ Stage s;
  __shared__ H S;
  load_head(c, S);
  __syncthreads();
  body_edge_topo<ALG>(c, S, s);
}

template <int ALG, class H>
__global__ void __launch_bounds__(kBlock, I2_UF_MIN_BLOCKS) relax_union(const __grid_constant__ Ctx c) {
  __shared__ Stage s;
  __shared__ H S;
  load_head(c, S);
  __syncthreads();
  body_union<ALG>(c, S, s);
}

template <int ALG, bool FRONTIER, class H>
__global__ void __launch_bounds__(kBlock, 4) relax_pull(const __grid_constant__ Ctx c) {
  __shared__ Stage s;
  __shared__ H S;
  load_head(c, S);
  __syncthreads();
  body_pull<ALG, FRONTIER>(c, S, s);
}

template <bool DEFER = false>
union AnyShared {
  Stage st;
  EBSharedT<DEFER> eb;
};

// ---------------------------------------------------------------------------
// Resident traversal: one launch runs the iterations one after another, the
// grid meeting at a barrier where separate launches would meet at a kernel
// boundary. The block that finishes an iteration (the last one to count into
// `done`) has already advanced the control block when it bumps bar_gen, which
// releases the others. Every wait is bounded by Ctl::stall_ns: a block that
// waits longer sets kStatusStall and leaves, and every other block leaves at
// its next wait, so the launch always ends. All blocks must be resident at
// once, which the cooperative launch guarantees.
// Data written in one iteration is read by other blocks in the next, so the
// bodies read the frontier lists, bitmaps and values with coherent loads only
// (the read-only path is used for the graph arrays alone).

// Thread 0 of a block: wait until bar_gen has moved past `gen`. False once the
// wait has run out (status kStatusStall) or another block has given up. The
// polls are plain reads of one line; the fence after them orders what follows
// (an acquire in every poll would drop the L1 of the SM's working blocks).
__device__ __forceinline__ bool grid_wait(const Ctx& c, unsigned gen, unsigned long long limit) {
  const unsigned long long t0 = globaltimer();
  Ctl* ctl = c.ctl;
  bool ok = true;
  for (unsigned k = 1;; ++k) {
    unsigned g, st;
    asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(g), "=r"(st) : "l"(&ctl->bar_gen) : "memory");
    if (st & kStatusStall) ok = false;
    if (g != gen || !ok) break;
    if (k >= 256) __nanosleep(100);
    if ((k & 63) == 0 && globaltimer() - t0 > limit) {
      atomicOr(&ctl->status, kStatusStall);
      ok = false;
      break;
    }
  }
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
  return ok;
}

template <int ALG, int VAR, bool DEFER, bool LONG, class H>
__device__ __forceinline__ bool run_body(const Ctx& c, H& S, AnyShared<DEFER>& sh) {
  if constexpr (ALG == kMIS) {
    return body_mis(c, S, sh.st);  // one style
  } else {
    const int v = VAR >= 0 ? VAR : S.variant;
    switch (v) {
      case kVPThread: return body_push<ALG, kVPThread>(c, S, sh.st);
      case kVPWarp: return body_push<ALG, kVPWarp>(c, S, sh.st);
      case kVPCta: return body_edge_balanced<ALG, DEFER, LONG>(c, S, sh.eb);
      case kVPBlock: return body_push<ALG, kVPBlock>(c, S, sh.st);
      case kPullFrontier: return body_pull<ALG, true>(c, S, sh.st);
      case kPullTopo: return body_pull<ALG, false>(c, S, sh.st);
      case kEdgeTopo: return body_edge_topo<ALG>(c, S, sh.st);
      case kUnionFind:
        if constexpr (ALG == kCC) return body_union<ALG>(c, S, sh.st);
        [[fallthrough]];  // not allowed for BFS/SSSP
      default: return body_push_topo<ALG>(c, S, sh.st);
    }
  }
}

// VAR >= 0: that style every iteration; VAR < 0: the style picked for each
// iteration by the previous one (heuristic or learned selector). WIDE: the form
// for more resident blocks (selectors: the largest graphs; edge-balanced push:
// graphs of skewed degrees, with long tiles too).
template <int VAR, bool WIDE>
constexpr int kResidentMinBlocks = WIDE                ? I2_FIXED_MIN_BLOCKS
                                   : VAR < 0           ? I2_SEL_MIN_BLOCKS
                                   : VAR == kVPCta     ? I2_EB_MIN_BLOCKS
                                   : VAR == kUnionFind ? I2_UF_MIN_BLOCKS
                                                       : I2_FIXED_MIN_BLOCKS;
template <int ALG, int VAR, bool DEFER = false, bool WIDE = false, int MINB = kResidentMinBlocks<VAR, WIDE>>
__global__ void __launch_bounds__(kBlock, MINB) relax_resident(const __grid_constant__ Ctx c) {
  __shared__ AnyShared<DEFER> sh;
  // the selectors' form for more blocks runs on the largest graphs only
  static_assert(kWideSelectorNodes > kMaxTrainedNodes, "no network in the wide forms");
  using Pick = typename std::conditional<WIDE, RuleHead, SelectHead>::type;
  __shared__ typename std::conditional<(VAR < 0), Pick, FixedHead>::type S;
  constexpr bool LONG = DEFER || (VAR == kVPCta && WIDE);  // skewed graphs' forms
  // thread 0's: barrier generation, whether to go on, the test hook (kept in
  // shared memory: the bodies have no register to spare)
  __shared__ unsigned s_gen;
  __shared__ int s_ok, s_hold;
  load_head(c, S);
  if (threadIdx.x == 0) {
    s_ok = !(*(volatile int*)&c.ctl->status & kStatusStall);
    s_gen = *(volatile unsigned*)&c.ctl->bar_gen;  // no iteration ends before every block arrives
    s_hold = c.ctl->hold;
  }
  __syncthreads();
  // Blocks of this traversal have given up already, before this one began: it
  // leaves and says so, like a block whose wait ran out. (With a bare return here
  // nvcc 12.9 keeps the kernel's parameters in registers across the loop and
  // spills them in the bodies: 88 instead of 56 bytes in the near/far form, 92
  // instead of 24 in vp_thread's.)
  if (!s_ok) {
    if (threadIdx.x == 0) atomicOr(&c.ctl->status, kStatusStall);
    return;
  }
  for (;;) {
    if (run_body<ALG, VAR, DEFER, LONG>(c, S, sh) && !s_hold) {
      // this block advanced S and wrote it back (every thread a word)
      __syncthreads();
      if (threadIdx.x == 0)
        asm volatile("red.add.release.gpu.global.u32 [%0], 1;" ::"l"(&c.ctl->bar_gen) : "memory");
    } else {
      if (threadIdx.x == 0) s_ok = grid_wait(c, s_gen, S.stall_ns);
      __syncthreads();
      if (!s_ok) break;
      load_head(c, S);
    }
    if (threadIdx.x == 0) {
      ++s_gen;
      s_hold = 0;  // the hook withholds the first release only
    }
    __syncthreads();
    if (!S.go) break;
  }
}

template <int ALG, bool WIDE = false>
__global__ void __launch_bounds__(kBlock, WIDE ? I2_FIXED_MIN_BLOCKS : I2_SEL_MIN_BLOCKS)
    relax_dispatch(const __grid_constant__ Ctx c) {
  __shared__ AnyShared<> sh;
  __shared__ typename std::conditional<WIDE, RuleHead, SelectHead>::type S;
  load_head(c, S);
  __syncthreads();
  switch (S.variant) {
    case kVPThread: body_push<ALG, kVPThread>(c, S, sh.st); break;
    case kVPWarp: body_push<ALG, kVPWarp>(c, S, sh.st); break;
    case kVPCta: body_edge_balanced<ALG>(c, S, sh.eb); break;
    case kVPBlock: body_push<ALG, kVPBlock>(c, S, sh.st); break;
    case kPullFrontier: body_pull<ALG, true>(c, S, sh.st); break;
    case kPullTopo: body_pull<ALG, false>(c, S, sh.st); break;
    case kEdgeTopo: body_edge_topo<ALG>(c, S, sh.st); break;
    case kUnionFind:
      if constexpr (ALG == kCC) {
        body_union<ALG>(c, S, sh.st);
        break;
      }
      [[fallthrough]];  // not allowed for BFS/SSSP
    default: body_push_topo<ALG>(c, S, sh.st); break;
  }
}

}  // namespace i2
