// BFS kernels launched once per iteration (every style, and the selectors' dispatch).
#include "kernels.cuh"

namespace i2 {

template KernelFn relax_fn<kBFS>(int, bool, bool);
template KernelFn dispatch_fn<kBFS>(bool);

}  // namespace i2
