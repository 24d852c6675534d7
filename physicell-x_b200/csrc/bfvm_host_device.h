// bfvm_host_device.h -- for the kernels' plain index arithmetic, which CPU tests
// compile without CUDA.
#pragma once

#ifdef __CUDACC__
#define BFVM_HD __host__ __device__ __forceinline__
#else
#define BFVM_HD inline
#endif
