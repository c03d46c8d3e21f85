// BFS kernels that run a whole traversal in one launch.
#include "kernels.cuh"

namespace i2 {

template KernelFn resident_fn<kBFS>(int, bool);

}  // namespace i2
