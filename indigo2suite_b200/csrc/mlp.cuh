// Learned style selector: layout of the MLP parameter blob, the feature vector,
// and the block-level inference routine used inside the relax kernels' epilogue.
//
// Network: x (16 features) -> standardise with (mu, sd) -> 64 ReLU -> 64 ReLU -> 9
// outputs, one predicted log2 launch time (ns) per variant. The selector picks
// the allowed variant with the smallest prediction. Weights are stored
// [in][out] so that, for a fixed input, consecutive outputs are consecutive in memory.
#pragma once
#include "common.cuh"

namespace i2 {

static_assert(kBlock == 4 * 64, "mlp_forward_block assumes 256 threads");

constexpr int kOut = kNumVariants;
constexpr int kOffMu = 0;
constexpr int kOffSd = kOffMu + kFeatures;
constexpr int kOffW1 = kOffSd + kFeatures;
constexpr int kOffB1 = kOffW1 + kFeatures * kHidden;
constexpr int kOffW2 = kOffB1 + kHidden;
constexpr int kOffB2 = kOffW2 + kHidden * kHidden;
constexpr int kOffW3 = kOffB2 + kHidden;
constexpr int kOffB3 = kOffW3 + kHidden * kOut;
constexpr int kParams = kOffB3 + kOut;

// Feature k of a frontier about to be consumed (one lane per feature). All are finite and O(1..30).
// The features that grow with the graph (frontier size and edges, largest
// degrees, vertex and CSR-entry counts) are clamped to the largest values of
// the training sweep (graphs of up to 2^21 vertices, 2^25.9 CSR entries,
// degree 2^16.7): a larger graph is read as the largest one trained on
// instead of extrapolating the network. The iteration index is clamped to 64
// (frontiers reach their steady state by then).
constexpr float kCapLogV = 21.f;     // log2 vertices
constexpr long long kMaxTrainedNodes = 1LL << 21;  // the largest training graph's vertices
constexpr float kCapLogE = 26.f;     // log2 CSR entries (frontier edges too)
constexpr float kCapLogDeg = 17.f;   // log2 degree
__device__ __forceinline__ float frontier_feature(int k, const GStats& gs, int algo, int iter, int size, int hsize,
                                                  unsigned long long edges, int maxdeg, long long visited) {
  const float fs = (float)size + (float)hsize;
  const float fe = (float)edges;
  const float V = (float)gs.nodes;
  const float E = (float)gs.edges > 0.f ? (float)gs.edges : 1.f;
  switch (k) {
    case 2: return fs / V;
    case 3: return fe / E;
    case 6: return (float)visited / V;
    case 13: return algo == kSSSP ? 1.f : 0.f;
    case 14: return algo == kCC ? 1.f : 0.f;
    case 15: return fs > 0.f ? (float)hsize / fs : 0.f;
  }
  // the others are logarithms (one log2f for the lanes that need one)
  float x = 1.f, lo = -3.0e38f, hi = 3.0e38f;
  switch (k) {
    case 0: x = 1.f + fs; hi = kCapLogV; break;
    case 1: x = 1.f + fe; hi = kCapLogE; break;
    case 4: x = 1.f + fe / fmaxf(1.f, fs); break;
    case 5: x = 1.f + (float)maxdeg; hi = kCapLogDeg; break;
    case 7: x = 1.f + fminf((float)iter, 64.f); break;
    case 8: x = V; lo = 16.f; hi = kCapLogV; break;
    case 9: x = 1.f + (float)gs.edges; lo = 17.f; hi = kCapLogE; break;
    case 10: x = 1.f + gs.avgdeg; break;
    case 11: x = 1.f + (float)gs.maxdeg; hi = kCapLogDeg; break;
    case 12: x = 1.f + gs.degcv; break;
  }
  return fminf(fmaxf(log2f(x), lo), hi);
}

// Block-cooperative forward pass for a block of kBlock (256) threads. Each
// hidden unit is computed by 4 threads (partial dot products reduced with
// shuffles) and each output by one warp. Every weight that a thread uses in
// any layer is loaded before the first layer (about 40 independent loads, one
// L2 latency), so that the layers themselves only wait on shared memory: the
// pass stands between two iterations of a resident traversal, and three layers
// of dependent loads cost it about 2.5 us. x and y live in shared memory; h1
// and h2 are shared scratch.
__device__ __forceinline__ void mlp_forward_block(const float* __restrict__ P, const float* x, float* h1,
                                                  float* h2, float* y) {
  constexpr int kIn1 = kFeatures / 4, kIn2 = kHidden / 4, kIn3 = kHidden / kWarp, kWarps = kBlock / kWarp;
  static_assert(kOut <= 2 * kWarps, "two outputs per warp at most");
  const int t = threadIdx.x;
  const int j = t >> 2;  // hidden unit
  const int q = t & 3;   // quarter of its inputs
  const int lane = t & 31, wid = t >> 5;
  float mu[kIn1], sd[kIn1], w1[kIn1], w2[kIn2], w3[2][kIn3], b3[2];
#pragma unroll
  for (int i = 0; i < kIn1; ++i) {
    const int k = q * kIn1 + i;
    mu[i] = P[kOffMu + k];
    sd[i] = P[kOffSd + k];
    w1[i] = P[kOffW1 + k * kHidden + j];
  }
  const float b1 = P[kOffB1 + j], b2 = P[kOffB2 + j];
#pragma unroll
  for (int i = 0; i < kIn2; ++i) w2[i] = P[kOffW2 + (q * kIn2 + i) * kHidden + j];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int o = min(wid + r * kWarps, kOut - 1);
#pragma unroll
    for (int i = 0; i < kIn3; ++i) w3[r][i] = P[kOffW3 + (lane * kIn3 + i) * kOut + o];
    b3[r] = P[kOffB3 + o];
  }
  float acc = 0.f;
#pragma unroll
  for (int i = 0; i < kIn1; ++i) acc = fmaf((x[q * kIn1 + i] - mu[i]) / sd[i], w1[i], acc);
  acc += __shfl_xor_sync(0xffffffffu, acc, 1);
  acc += __shfl_xor_sync(0xffffffffu, acc, 2);
  if (q == 0) h1[j] = fmaxf(acc + b1, 0.f);
  __syncthreads();
  acc = 0.f;
#pragma unroll
  for (int i = 0; i < kIn2; ++i) acc = fmaf(h1[q * kIn2 + i], w2[i], acc);
  acc += __shfl_xor_sync(0xffffffffu, acc, 1);
  acc += __shfl_xor_sync(0xffffffffu, acc, 2);
  if (q == 0) h2[j] = fmaxf(acc + b2, 0.f);
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int o = wid + r * kWarps;
    acc = 0.f;
#pragma unroll
    for (int i = 0; i < kIn3; ++i) acc = fmaf(h2[lane * kIn3 + i], w3[r][i], acc);
    for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
    if (lane == 0 && o < kOut) y[o] = acc + b3[r];
  }
  __syncthreads();
}

}  // namespace i2
