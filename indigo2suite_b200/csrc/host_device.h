// Functions shared by kernels and host code (and host tests).
#pragma once

#ifdef __CUDACC__
#define I2_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define I2_HOST_DEVICE inline
#endif
