// The double of the plain FP64 kernels: the built-in type's values, bit for
// bit, from cheaper instructions on this part.
//
// Additions and products are issued as fused multiply-adds with a neutral
// third operand held in a register: one rounding of the same exact value (a * 1
// and the zero added are exact; the zero is -0, which keeps a product's zero
// sign).  Measured on a GB300, a warp's DADD or DMUL - and a DFMA with an
// immediate or constant-bank operand - holds its sub-partition's FP64 pipe for
// 81 cycles, a DFMA with three register operands for 64.  Division, reciprocal
// and square root run on the integer pipe (exact64.cuh).
//
// Plain FP64 step with this type, whole pass: 3D 128^3 MLAU + WCNS4 79.4 ->
// 56.5 ms, 2D 512^2 LHLLD + WCNS4 5.72 -> 4.31 ms.
#pragma once

#include "exact64.cuh"
#include "point.cuh"

namespace mlau {

// Zero that the compiler cannot see through, for constants that have to sit
// in registers.
__device__ __forceinline__ uint32_t opaque_zero()
{
    uint32_t z;
    asm("mov.u32 %0, %%total_smem_size;" : "=r"(z));
    return z >> 24;  // an SM's shared memory is below 16 MB
}
__device__ __forceinline__ double ed_one()
{
    return __hiloint2double((int)(0x3ff00000u + opaque_zero()), 0);
}
__device__ __forceinline__ double ed_minus_zero()
{
    return __hiloint2double((int)(0x80000000u + opaque_zero()), 0);
}

struct ed {
    double v;
    ed() = default;
    MLAU_HD constexpr ed(double x) : v(x) {}
    MLAU_HD constexpr ed(int x) : v(x) {}
};

MLAU_HD ed operator+(ed a, ed b)
{
#ifdef __CUDA_ARCH__
    return __fma_rn(a.v, ed_one(), b.v);
#else
    return a.v + b.v;
#endif
}
MLAU_HD ed operator-(ed a, ed b)
{
#ifdef __CUDA_ARCH__
    return __fma_rn(-b.v, ed_one(), a.v);
#else
    return a.v - b.v;
#endif
}
MLAU_HD ed operator*(ed a, ed b)
{
#ifdef __CUDA_ARCH__
    return __fma_rn(a.v, b.v, ed_minus_zero());
#else
    return a.v * b.v;
#endif
}
MLAU_HD ed operator/(ed a, ed b) { return x64::div(a.v, b.v); }
MLAU_HD ed operator-(ed a) { return -a.v; }
MLAU_HD ed operator+(ed a) { return a; }
MLAU_HD ed &operator+=(ed &a, ed b) { return a = a + b; }
MLAU_HD ed &operator-=(ed &a, ed b) { return a = a - b; }
MLAU_HD ed &operator*=(ed &a, ed b) { return a = a * b; }
MLAU_HD ed &operator/=(ed &a, ed b) { return a = a / b; }
MLAU_HD bool operator>(ed a, ed b) { return a.v > b.v; }
MLAU_HD bool operator>=(ed a, ed b) { return a.v >= b.v; }
MLAU_HD bool operator<(ed a, ed b) { return a.v < b.v; }
MLAU_HD bool operator<=(ed a, ed b) { return a.v <= b.v; }
MLAU_HD bool operator==(ed a, ed b) { return a.v == b.v; }
MLAU_HD bool operator!=(ed a, ed b) { return a.v != b.v; }

template <> MLAU_HD ed tsqrt<ed>(ed x) { return x64::sqrt(x.v); }
template <> MLAU_HD ed tabs<ed>(ed x) { return fabs(x.v); }
template <> MLAU_HD ed trcp<ed>(ed x) { return x64::rcp(x.v); }
template <> MLAU_HD ed thalf_over<ed>(ed x) { return x64::half_over(x.v); }
template <> MLAU_HD ed tsqrt_two<ed>() { return 0x1.6a09e667f3bcdp+0; }
template <> MLAU_HD ed tsqrt_half<ed>() { return 0x1.6a09e667f3bcdp-1; }
template <> MLAU_HD ed tdiv24<ed>(ed x) { return x64::div24(x.v); }


}  // namespace mlau
