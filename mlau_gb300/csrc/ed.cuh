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


// a * b on the integer pipe.
static X64_SLOW double mul_pipe(double a, double b) { return a * b; }
MLAU_HD ed imul(ed a, ed b)
{
    uint32_t bad = x64::off_wide(a.v) | x64::off_wide(b.v);
    double r = x64::mul(a.v, b.v, bad);
    if (bad) r = mul_pipe(a.v, b.v);
    return r;
}
// a 2^P, and k a for a small odd k
template <int P> MLAU_HD ed iscale(ed a)
{
    double r = x64::scale<P>(a.v);
    constexpr double c = P >= 0 ? (double)(1 << (P >= 0 ? P : 0)) : 1.0 / (double)(1 << (P < 0 ? -P : 0));
    if (x64::off_wide(a.v)) r = mul_pipe(a.v, c);
    return r;
}
MLAU_HD ed ihalf(ed a) { return iscale<-1>(a); }
template <int K> MLAU_HD ed imulk(ed a)
{
    double r = x64::mulk<K>(a.v);
    if (x64::off_wide(a.v)) r = mul_pipe(a.v, (double)K);
    return r;
}

template <> MLAU_HD ed thalf<ed>(ed x) { return ihalf(x); }
template <> MLAU_HD ed tsixteenth<ed>(ed x) { return iscale<-4>(x); }
template <> MLAU_HD ed t9<ed>(ed x) { return imulk<9>(x); }
template <> MLAU_HD ed t27<ed>(ed x) { return imulk<27>(x); }
template <> MLAU_HD bool tzero<ed>(ed x) { return ((x64::hi32(x.v) << 1) | x64::lo32(x.v)) == 0; }

// Comparisons (81 cycles each on the FP64 pipe) on the values' bits.  An
// infinity or NaN among the operands takes the pipe's.
MLAU_HD bool ed_special(uint32_t h, uint32_t g)
{
    const uint32_t a = h << 1, b = g << 1;
    return (a > b ? a : b) >= 0xffe00000u;
}
static X64_SLOW bool ge_pipe(double a, double b) { return a >= b; }
MLAU_HD bool ed_ge(ed a, ed b)
{
    const uint32_t ha = x64::hi32(a.v), hb = x64::hi32(b.v);
    const int32_t sa = (int32_t)ha >> 31, sb = (int32_t)hb >> 31;
    const int32_t ka = (int32_t)ha ^ (sa & 0x7fffffff), kb = (int32_t)hb ^ (sb & 0x7fffffff);
    bool r = ka > kb || (ka == kb && (x64::lo32(a.v) ^ (uint32_t)sa) >= (x64::lo32(b.v) ^ (uint32_t)sb));
    if (ed_special(ha, hb)) r = ge_pipe(a.v, b.v);
    return r;
}
template <> MLAU_HD ed vmax<ed>(ed a, ed b) { return ed_ge(a, b) ? a : b; }
template <> MLAU_HD ed vmin<ed>(ed a, ed b) { return ed_ge(a, b) ? b : a; }

static X64_SLOW double minmod_pipe(double a, double b) { return minmod<double>(a, b); }
static X64_SLOW double minmod3_pipe(double a, double b, double c) { return minmod3<double>(a, b, c); }
// the operand of smaller magnitude where the signs agree, else 0
template <> MLAU_HD ed minmod<ed>(ed a, ed b)
{
    const uint32_t ha = x64::hi32(a.v), hb = x64::hi32(b.v);
    const uint32_t ma = ha & 0x7fffffffu, mb = hb & 0x7fffffffu;
    double r = (ma < mb || (ma == mb && x64::lo32(a.v) < x64::lo32(b.v))) ? a.v : b.v;
    if ((ha ^ hb) >> 31) r = 0.0;
    if (ed_special(ha, hb)) r = minmod_pipe(a.v, b.v);
    return r;
}
template <> MLAU_HD ed minmod3<ed>(ed a, ed b, ed c)
{
    const uint32_t hc = x64::hi32(c.v);
    double r = minmod(minmod(a, b), c).v;
    if (ed_special(x64::hi32(a.v), x64::hi32(b.v)) || ed_special(hc, hc)) r = minmod3_pipe(a.v, b.v, c.v);
    return r;
}

// The 4th-order linear face value 1/320 (9 f0 - 56 f1 + 234 f2 + 144 f3 - 11 f4)
// of lin_l, products on the integer pipe (56 = 8 x 7, 234 = 2 x 117 and 144 =
// 16 x 9: the powers of two ride on the sums), the four sums on the FP64 pipe.
static __device__ __noinline__ double lin4_pipe(double f0, double f1, double f2, double f3, double f4)
{
    return lin_l<double>(4, f0, f1, f2, f3, f4);
}
__device__ __forceinline__ ed lin4_ed(double f0, double f1, double f2, double f3, double f4)
{
    using namespace x64;
    const uint32_t z = opaque_zero();
    auto K = [&](uint32_t h) { return __hiloint2double((int)(h + z), 0); };
    uint32_t bad = off_wide(f0) | off_wide(f1) | off_wide(f2) | off_wide(f3) | off_wide(f4);
    double s = __fma_rn(K(0xc0200000u), mulk<7>(f1), mulk<9>(f0));  // -8
    s = __fma_rn(K(0x40000000u), mulk<117>(f2), s);                 // 2
    s = __fma_rn(K(0x40300000u), mulk<9>(f3), s);                   // 16
    s = __fma_rn(-mulk<11>(f4), K(0x3ff00000u), s);
    double r = mul(s, 0.003125, bad);
    if (bad) r = lin4_pipe(f0, f1, f2, f3, f4);
    return r;
}
template <> MLAU_HD ed lin_l<ed>(int odr, ed f0, ed f1, ed f2, ed f3, ed f4)
{
#ifdef __CUDA_ARCH__
    odr = lin_odr(odr);
    if (odr == 4) return lin4_ed(f0.v, f1.v, f2.v, f3.v, f4.v);
    const double four = __hiloint2double((int)(0x40100000u + opaque_zero()), 0);
    const double two = __hiloint2double((int)(0x40000000u + opaque_zero()), 0);
    if (odr == 2) return iscale<-2>(ed(__fma_rn(four, f2.v, -f1.v)) + f3);
    if (odr == 3) return iscale<-3>(ed(__fma_rn(two, imulk<3>(f2).v, -f1.v)) + imulk<3>(f3));
#endif
    return f2;
}
template <> MLAU_HD ed lin_r<ed>(int odr, ed f0, ed f1, ed f2, ed f3, ed f4)
{
    return lin_l<ed>(odr, f4, f3, f2, f1, f0);
}

}  // namespace mlau
