// 27 (e2 - e1) - (e3 - e0) of four FP32 edge EMFs as a double, the stencil of
// the 4th-order CT curl.  In doubles it takes four operations of the FP64 pipe (64 cycles
// each per warp and SM sub-partition), 24 of the some 40 of an updated cell,
// which bounded that kernel.  The values are integers times a common power of
// two, so here the sum is formed exactly in 64 bits on the integer pipe and
// rounded once.  While the exponents of the non-zero values are within 23 of
// each other every difference and product of the double form is exact too and
// it also rounds once: the results are the same.  Outside that, and for
// infinities, NaN and subnormals, the double form decides.
#pragma once

#include "exact64.cuh"

namespace mlau {

X64 uint32_t f32_bits(float f)
{
#ifdef __CUDA_ARCH__
    return __float_as_uint(f);
#else
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
#endif
}
// 1 << s, 0 for s outside 0 .. 31
X64 uint32_t pow2_or0(int s)
{
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm("shl.b32 %0, 1, %1;" : "=r"(r) : "r"(s));  // clamps
    return r;
#else
    return (uint32_t)s < 32 ? 1u << s : 0u;
#endif
}
X64 int clz64(uint64_t v)
{
#ifdef __CUDA_ARCH__
    return __clzll((long long)v);
#else
    return v ? __builtin_clzll(v) : 64;
#endif
}

static X64_SLOW double emf_diff4_slow(float e0, float e1, float e2, float e3)
{
    return 27.0 * ((double)e2 - (double)e1) - ((double)e3 - (double)e0);
}

X64 double emf_diff4(const float e[4])
{
    const int c[4] = {1, -27, 27, -1};
    uint32_t u[4], t[4], top = 24u << 23, bad = 0;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int n = 0; n < 4; n++) {
        u[n] = f32_bits(e[n]);
        t[n] = u[n] & 0x7f800000u;
        top = t[n] > top ? t[n] : top;
    }
    const uint32_t low = top - (23u << 23);  // exponent of the common unit
    int64_t v = 0;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int n = 0; n < 4; n++) {
        const uint32_t p = pow2_or0((int32_t)(t[n] - low) >> 23);
        const int32_t m = (int32_t)((u[n] & 0x7fffffu) | 0x800000u);
        v += (int64_t)(m * ((int32_t)u[n] < 0 ? -c[n] : c[n])) * (int64_t)(int32_t)p;
        bad |= p ? 0u : u[n] << 1;  // a value left out that is not zero
    }
    bad |= top >= (255u << 23) ? 1u : 0u;
    if (bad) return emf_diff4_slow(e[0], e[1], e[2], e[3]);
    const uint64_t a = v < 0 ? (uint64_t)-v : (uint64_t)v;
    const int lz = clz64(a);
    const uint64_t w = a << (lz & 63);
    const uint32_t h = (uint32_t)(w >> 32), l = (uint32_t)w;
    // the leading bit of a counts 2^(63 - lz + (low >> 23) - 150)
    const uint32_t ex = (uint32_t)(63 - lz + 1023 - 150 - 1) + (low >> 23);
    const double r = x64::round_pack(h >> 11, (h << 21) | (l >> 11), l << 21,
                                     (ex << 20) + ((uint32_t)(v >> 32) & 0x80000000u));
    return v ? r : 0.0;
}

}  // namespace mlau
