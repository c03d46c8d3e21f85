// Maximal independent set kernels (one style).
#include "kernels.cuh"

namespace i2 {

KernelFn mis_kernel(bool resident) { return resident ? (KernelFn)relax_resident<kMIS, kVPWarp> : relax_mis; }

}  // namespace i2
