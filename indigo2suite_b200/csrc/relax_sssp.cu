// SSSP kernels launched once per iteration (every style, and the selectors' dispatch).
#include "kernels.cuh"

namespace i2 {

template KernelFn relax_fn<kSSSP>(int, bool, bool);
template KernelFn dispatch_fn<kSSSP>(bool);
KernelFn near_far_launch() { return relax_near_far; }

}  // namespace i2
