// Kernel tables: the bodies of relax_fn, dispatch_fn and resident_fn
// (engine.h). Each is instantiated for one algorithm per translation unit.
#pragma once
#include "engine.h"
#include "mlp.cuh"
#include "relax.cuh"
#include "iteration.cuh"

namespace i2 {

template <int ALG, class H>
KernelFn relax_fn_of(int v) {
  switch (v) {
    case kVPThread: return relax_push<ALG, kVPThread, H>;
    case kVPWarp: return relax_push<ALG, kVPWarp, H>;
    case kVPCta: return relax_edge_balanced<ALG, H>;
    case kVPBlock: return relax_push<ALG, kVPBlock, H>;
    case kPullFrontier: return relax_pull<ALG, true, H>;
    case kPullTopo: return relax_pull<ALG, false, H>;
    case kEdgeTopo: return relax_edge_topo<ALG, H>;
    case kPushTopo: return relax_push_topo<ALG, H>;
    case kUnionFind:
      if constexpr (ALG == kCC) return relax_union<ALG, H>;
      return nullptr;
  }
  return nullptr;
}

template <int ALG>
KernelFn relax_fn(int v, bool select, bool wide) {
  if (select) return relax_fn_of<ALG, SelectHead>(v);
  // the wide form spills here; BFS, whose tiles do least, does not gain (RMAT-20,
  // us, wide / not: BFS 297 / 285, SSSP 736 / 732, CC 521 / 547; RMAT-25 in degree
  // order, ms: 8.4 / 8.2, 17.8 / 18.8, 22.2 / 24.3)
  if constexpr (ALG != kBFS)
    if (v == kVPCta && wide) return relax_edge_balanced<ALG, FixedHead, true>;
  return relax_fn_of<ALG, FixedHead>(v);
}

template <int ALG>
KernelFn dispatch_fn(bool wide) {
  return wide ? relax_dispatch<ALG, true> : relax_dispatch<ALG>;
}

template <int ALG>
KernelFn resident_fn(int v, bool wide) {
  switch (v) {
    case kVPThread: return relax_resident<ALG, kVPThread>;
    case kVPWarp: return relax_resident<ALG, kVPWarp>;
    case kVPCta: return wide ? relax_resident<ALG, kVPCta, false, true> : relax_resident<ALG, kVPCta>;
    case kVPBlock: return relax_resident<ALG, kVPBlock>;
    case kPullFrontier: return relax_resident<ALG, kPullFrontier>;
    case kPullTopo: return relax_resident<ALG, kPullTopo>;
    case kEdgeTopo: return relax_resident<ALG, kEdgeTopo>;
    case kPushTopo: return relax_resident<ALG, kPushTopo>;
    case kUnionFind:
      if constexpr (ALG == kCC) return relax_resident<ALG, kUnionFind>;
      return nullptr;
  }
  // per-iteration pick
  return wide ? relax_resident<ALG, -1, false, true> : relax_resident<ALG, -1>;
}

}  // namespace i2
