// CUDA's keywords and built-in names for a plain C++ compiler, so that the body
// of a kernel whose threads work alone can be run on the CPU, thread by thread.
#pragma once
#define __CUDACC__ 1  // the kernels' own declarations too
#define __host__
#define __device__
#define __global__ static
#define __forceinline__ inline
#define __noinline__
#define __launch_bounds__(...)
#define __grid_constant__
#define __restrict__ __restrict
#define __shared__
struct uint3 {
  unsigned x, y, z;
};
static uint3 threadIdx, blockIdx, blockDim{1, 1, 1}, gridDim{1, 1, 1};
inline void __syncthreads() {}
