// SSSP kernels that run a whole traversal in one launch.
#include "kernels.cuh"

namespace i2 {

template KernelFn resident_fn<kSSSP>(int, bool);
KernelFn near_far_launch();  // relax_sssp.cu
KernelFn near_far_kernel(bool resident) { return resident ? (KernelFn)relax_resident<kSSSP, kVPCta, true> : near_far_launch(); }

}  // namespace i2
