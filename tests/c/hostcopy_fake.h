// What csrc/hostcopy.cu needs of the device side, for a host compiler.
#pragma once
#include <cuda_runtime.h>

#undef __global__
#undef __launch_bounds__
#undef __grid_constant__
#define __global__ static
#define __launch_bounds__(...)
#define __grid_constant__
static struct { unsigned x, y; } blockIdx, blockDim, gridDim, threadIdx;
