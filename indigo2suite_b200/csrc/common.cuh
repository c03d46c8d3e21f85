// Shared device-side definitions of the B200 relaxation engine.
//
// The engine computes the same fixed points as the Indigo2 suite's BFS, SSSP and
// CC codes: BFS levels (codes/cuda/bfs-cuda/*, relax `atomicMin(&dist[dst], s+1)`,
// e.g. BFS_CUDA_V_Data_Push_..._Warp_..._NonDup.cu:73-79), SSSP distances with
// int32 weights (SSSP_CUDA_E_Data_Push_..._NonDup.cu:72-73) and CC minimum-ID
// labels (CC_CUDA_E_Data_Push_..._NonDup.cu:68-71). All values are int32 and
// INT_MAX marks an unreached vertex, as in include/bfs_vertex_cuda.h:46.
//
// Frontier contract shared by every variant (so a selector may switch variant
// at any iteration without changing the result):
//   at the start of iteration i, F_i is stored in slot s = i % 3 as
//     wl[s][0..size)     its vertices (those of degree >= 1),
//     woff[s][0..size)   the exclusive prefix sum of their degrees, so that
//                        the frontier's edges form one index space [0, edges),
//     hwl[s][0..hsize)   the subset of degree >= the heavy threshold, with
//     htoff[s][0..hsize) the exclusive prefix of their tile counts,
//     bm[s]              a bitmap with the bits of F_i set. Other bits may be
//                        set too, of vertices without edges only, and may
//                        outlive their iteration: the edge-balanced push leaves
//                        the bit of such a vertex it lowers, which keeps its
//                        visit counted once, and a slot cleared by its list
//                        never sees it. Readers that relax from the bitmap find
//                        no edges there; the list never holds such a vertex;
//   every vertex outside F_i has already relaxed all of its out-edges against
//   the current dist[]. Iteration i propagates at least F_i and builds F_{i+1}
//   in slot (i+1) % 3 from every vertex whose value it lowered. It also clears
//   slot (i+2) % 3 (F_{i-1}), which no variant reads during iteration i.
// SSSP near/far ordering (Ctl::delta != 0) relaxes the contract in one way: a
// lowered vertex whose new distance is at or above the current threshold goes
// onto the far pile instead of F_{i+1}. The traversal ends when both F_{i+1}
// and the pile are empty. Only the edge-balanced push defers; every other
// variant pushes all lowered vertices into F_{i+1}, which is always valid.
#pragma once
#include <cstdint>
#include <climits>
#include <cuda_runtime.h>

namespace i2 {

constexpr int kInf = INT_MAX;
constexpr int kBlock = 256;          // threads per block for all relax kernels
constexpr int kWarp = 32;
constexpr int kQueue = 2048;         // per-block shared staging queue (light)
constexpr int kHQueue = 128;         // per-block shared staging queue (heavy)
constexpr int kHeavyTile = 2048;     // edges per tile of a heavy vertex
constexpr int kMaxVariants = 16;
constexpr int kFeatures = 16;        // selector input width
constexpr int kHidden = 64;          // selector hidden width (two layers)
constexpr int kHistBins = 256;       // distance histogram of the budgeted near/far ordering

enum Algo { kBFS = 0, kSSSP = 1, kCC = 2, kMIS = 3 };

// Maximal independent set: status per vertex, the reference's undecided /
// included / excluded (include/mis_vertex_cuda.h:52-54), and the priority its
// CUDA codes give vertex v (hash(v + 712313887) read as int, e.g.
// MIS_CUDA_V_Data_Pull_Determ_..._Thread.cu:51; the hash is a published
// integer mixing function: two rounds of xor-shift by 16 and multiply by
// 0x45d9f3b, then a final xor-shift). Neighbour u outranks v when its
// priority is larger, or equal with a larger ID (:70).
constexpr int kMisUndecided = 0;
constexpr int kMisIn = 1;
constexpr int kMisOut = 2;

__device__ __forceinline__ int mis_priority(int v) {
  unsigned x = (unsigned)v + 712313887u;
  x = ((x >> 16) ^ x) * 0x45d9f3bu;
  x = ((x >> 16) ^ x) * 0x45d9f3bu;
  return (int)((x >> 16) ^ x);
}

__device__ __forceinline__ bool mis_outranks(int u, int pu, int v, int pv) {
  return pu > pv || (pu == pv && u > v);
}

enum Variant {
  kVPThread = 0,     // vertex push, data-driven, thread per frontier vertex
  kVPWarp = 1,       // vertex push, data-driven, warp per frontier vertex, 128-bit loads
  kVPCta = 2,        // edge-balanced push: block-scan of a frontier chunk, thread per edge
  kVPBlock = 3,      // vertex push, data-driven, block per frontier vertex
  kPullFrontier = 4, // pull from neighbours that are in the frontier bitmap (bottom-up)
  kPullTopo = 5,     // topology-driven pull over all vertices and all neighbours
  kEdgeTopo = 6,     // edge-centric sweep over all CSR entries gated by the bitmap
  kPushTopo = 7,     // topology sweep of the frontier bitmap, thread per vertex
  kUnionFind = 8,    // CC only: union-find over all edges (hook launch, then compress launch)
  kNumVariants = 9
};

// Device view of a CSR graph in the ECLgraph layout (include/ECLgraph.h:44-50).
struct DGraph {
  int nodes;
  int edges;
  const int* __restrict__ nindex;   // nodes + 1
  const int* __restrict__ nlist;    // edges
  const int* __restrict__ eweight;  // edges (SSSP only)
  const int* __restrict__ sp;       // edges: source vertex of each CSR entry (edge sweeps only)
  int vec_ok;                       // 1 when nlist/eweight bases are 16-byte aligned
};

// Whole-graph statistics used by the selector and the pull bound.
struct GStats {
  int nodes;
  int edges;
  int maxdeg;
  int nheavy;       // vertices with degree >= heavy threshold
  int linked;       // vertices with edges
  int first;        // the smallest of them (kInf: none)
  int wmin;         // minimum edge weight (1 for BFS)
  int symmetric;    // 1 when every (u,v,w) has a (v,u,w) partner
  float avgdeg;
  float degcv;      // coefficient of variation of the degree distribution
  float wmean;      // mean edge weight (1 for BFS)
};

// Statistics of one frontier buffer, accumulated while it is built. Entries
// and edges share one 64-bit word (entries << 32 | edges) so that a single
// atomicAdd hands out consistent positions in wl[] and offsets in woff[]; a
// frontier holds each vertex at most once, so edges <= E < 2^31 never carries
// into the entry count. The heavy list pairs entries with tiles the same way.
struct alignas(128) Slot {    // a line of its own: every flush adds to `packed`
  unsigned long long packed;  // entries << 32 | edges
  unsigned long long hpacked; // heavy entries << 32 | heavy tiles
  int maxdeg;
  int mindist;                // smallest value pushed into this frontier
};

__host__ __device__ __forceinline__ int slot_size(unsigned long long p) { return (int)(p >> 32); }
__host__ __device__ __forceinline__ unsigned slot_edges(unsigned long long p) { return (unsigned)(p & 0xffffffffu); }

// Control block of a traversal. Its head is the state of the current iteration.
// Every block copies the head to shared memory in one coalesced read when the
// iteration begins and takes all its decisions from the copy; the block that
// finishes the iteration reads it once more (now with the accumulated counts),
// advances it in shared memory and writes it back. (Read field by field from
// global memory, the chain of dependent L2 reads cost about 8 us per iteration
// between the last relaxation and the next start: grid 2000^2 BFS, 117
// iterations, took 2,337 us and takes 1,735; SSSP on RMAT with 3,001 vertices,
// 11 iterations, 213 and 163.)
// Fields that blocks change with atomics during an iteration lie on lines of
// their own behind the state; in the copy they are only good where this
// iteration does not change them (slot[cur], slot[old], the pile that a move
// reads).
struct CtlHead {
  int iter;                 // index of the next relax launch
  int iter_cap;
  int variant;              // variant to run at the next launch
  int mode;                 // 0 fixed, 1 heuristic, 2 learned, 3 fixed switch (then_at)
  int fixed_variant;
  int allowed;              // bitmask of variants allowed on this graph
  int src;                  // source vertex (BFS/SSSP)
  int nsrc;                 // number of sources (batched runs)
  int algo;
  int sel_n;                // frontier entries at the last selector evaluation
  unsigned sel_e;           // frontier edges at the last selector evaluation
  int sel_iter;             // iteration of the last selector evaluation
  // SSSP near/far ordering (delta != 0 only): relax iterations push values at
  // or above `threshold` onto far pile `pcur` instead of the next frontier;
  // when the next frontier is empty and the pile is not, the next launch is a
  // split (split = 1): the threshold rises and the pile's entries below it
  // move into the next frontier, the others onto the other pile.
  //  * delta > 0 (fixed step): the threshold rises to max(threshold, pmin) + delta.
  //  * delta < 0 (edge budget B = -delta): the threshold is set so that about
  //    B edges lie below it, from distance histograms (weighted by degree)
  //    that the launches keep of the next frontier and of the pile: a move
  //    takes the pile's B-edge quantile, and when a frontier carries more than
  //    2B edges the threshold drops to its B-edge quantile and a trim launch
  //    (split = 3) moves the entries at or above it onto the pile. A pile
  //    entry is live while its bit in fbm is set: a near push of the vertex
  //    clears it.
  int delta;
  int threshold;
  int prev_threshold;       // threshold before the last rise
  int split;                // 0 relax, 1 move from the pile, 3 trim the frontier
  int hshift;               // histogram bin width 2^hshift (budget)
  int hbase;                // frontier histogram base of the current launch (budget)
  int pbase;                // pile histogram base (budget)
  int pcur;                 // current far pile
  int uf_phase;             // union-find CC: 1 after the hook launch (the compress launch follows)
  int uf_giant;             // union-find CC: root of the sampled largest tree
  int whole;                // the first iteration takes every vertex, without a frontier list (union-find CC, MIS)
  unsigned uf_step;         // union-find CC: order of the vertices (body_union)
  int then_at;              // mode 3: iteration from which then_variant runs
  int then_variant;
  int go;                   // 1 while another iteration follows
  int hold;                 // test hook: the first release is withheld
  unsigned long long stall_ns;  // longest wait at the barrier before giving up
  unsigned long long relax_ns;  // sum of relax launch durations
  float feat[kFeatures];    // features of the frontier the next launch consumes
  Slot slot[3];
  // counts of the traversal, added to once per block
  alignas(128) long long visited;  // vertices reached so far
  unsigned long long tstart;// start of the current launch (globaltimer ns)
  unsigned psize[2];        // entries of the far piles
  int pmin[2];              // lower bound of the values on each pile
  int chunk;                // dynamic work counter of the current launch
  alignas(128) unsigned done;  // blocks finished in the current launch
};
// A block's copy of the head, by what the end of an iteration may have to do:
// pick the next style, by the network too (SelectHead) or by the rule and fixed
// switches alone (RuleHead: graphs larger than any the network was trained on,
// where it is never asked), or stay with the one style (FixedHead). The
// network's weights are loaded up front, so its code sets a kernel's registers.
struct SelectHead : CtlHead {
  static constexpr bool kSelect = true, kNetwork = true;
};
struct RuleHead : CtlHead {
  static constexpr bool kSelect = true, kNetwork = false;
};
struct FixedHead : CtlHead {
  static constexpr bool kSelect = false, kNetwork = false;
};
constexpr int kHeadWords = sizeof(CtlHead) / 4;
static_assert(kHeadWords <= kBlock, "one word of the head per thread");

struct Ctl : CtlHead {
  // Resident launches (one launch runs every iteration, the grid meeting at
  // a barrier between them): the waiting blocks poll this line alone.
  alignas(128) unsigned bar_gen;  // barrier generation, bumped once per iteration
  int status;               // error bits, see kStatus*
  int hist[kMaxVariants];   // launches per variant
  unsigned long long reached[2];  // reached vertices and the sum of their degrees (k_reached)
};

// Where the selectors take union-find for CC, before the first iteration, on
// symmetric graphs: 2^19 vertices or more, or an average degree below 6. The line
// was drawn for an earlier union-find, to which propagation was up to 1.7x faster
// on RMAT and ER of 2^18 vertices with higher degrees. With links by climbing and
// blocks by the graph's size, union-find by name is the faster one below the line
// too (us, union-find / what the selectors run: RMAT-12 46 / 95, RMAT-16 111 / 129,
// RMAT-18 114 / 185, ER 60,000 128 / 183, ER 300,000 122 / 250): the line has not
// been moved. Above it, against the edge-balanced push: RMAT-22 186 / 1,894, ER
// 2 x 10^6 199 / 949, grid 4096^2 654 / 36,000 (pull_topo 31,764).
__host__ __device__ inline bool union_find_pays(long long nodes, float avgdeg) {
  return nodes >= (1LL << 19) || avgdeg < 6.f;
}

// Graphs on which the selectors' kernel is compiled for
// I2_FIXED_MIN_BLOCKS resident blocks per SM rather than I2_SEL_MIN_BLOCKS (relax.cuh).
constexpr long long kWideSelectorNodes = 1LL << 25;

enum : int {
  kStatusIterCap = 1,
  kStatusOverflow = 2,
  kStatusStall = 4,  // a resident launch's barrier wait ran out of time
};

// One record per relax launch: the frontier it consumed and its duration.
struct IterRec {
  int iter;
  int variant;
  int size;
  int hsize;
  unsigned long long edges;
  int maxdeg;
  int mindist;
  long long visited;
  unsigned long long t_ns;
  float feat[kFeatures];
  int kind;                 // Ctl::split of the launch: 0 relax, 1 move, 3 trim
  int threshold;            // near/far threshold of the launch (INT_MAX: none)
  unsigned pile;            // far-pile entries after the launch
  int pad;
};

// Everything a relax kernel needs, passed by value.
struct Ctx {
  DGraph g;
  GStats gs;
  int* dist;
  int* wl[3];
  unsigned* woff[3];
  int* hwl[3];
  unsigned* htoff[3];
  int* pile[2];             // far piles (SSSP near/far ordering), vertices
  int* pdeg[2];             // their degrees
  unsigned pile_cap;        // entries per pile
  unsigned* fbm;            // bit set: vertex is on the current far pile
  unsigned long long* hist; // 2 x kHistBins edge counts: [0] next frontier, [1] pile
  unsigned* bm[3];
  Ctl* ctl;
  IterRec* recs;
  int rec_cap;
  int heavy;                // degree threshold of the heavy list
  int bm_words;             // words per bitmap
  const float* mlp;         // selector weights (device), may be null
  const int* srcs;          // batched sources (device), may be null
  unsigned long long loop_h;   // cudaGraphConditionalHandle of the while node
  int use_loop;
};

__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Relaxation operators: candidate value for dst from source value du along CSR entry k.
template <int ALG>
struct Op;

template <>
struct Op<kBFS> {
  static __device__ __forceinline__ bool valid(int du) { return du != kInf; }
  static __device__ __forceinline__ int cand(int du, int /*w*/) { return du + 1; }
  static constexpr bool kWeighted = false;
};
template <>
struct Op<kSSSP> {
  static __device__ __forceinline__ bool valid(int du) { return du != kInf; }
  static __device__ __forceinline__ int cand(int du, int w) { return du + w; }
  static constexpr bool kWeighted = true;
};
template <>
struct Op<kCC> {
  static __device__ __forceinline__ bool valid(int) { return true; }
  static __device__ __forceinline__ int cand(int du, int) { return du; }
  static constexpr bool kWeighted = false;
};

}  // namespace i2
