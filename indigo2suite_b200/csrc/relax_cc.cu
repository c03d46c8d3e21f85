// CC kernels launched once per iteration (every style, and the selectors' dispatch).
#include "kernels.cuh"

namespace i2 {

template KernelFn relax_fn<kCC>(int, bool, bool);
template KernelFn dispatch_fn<kCC>(bool);

}  // namespace i2
