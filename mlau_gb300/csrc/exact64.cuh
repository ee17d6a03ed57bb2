// Reciprocal, division, square root and product of doubles, correctly rounded
// (round to nearest even), computed on the integer and FP32 pipes.
//
// Why: this part's FP64 pipe takes 64 cycles per warp instruction in each SM
// sub-partition (2 lanes per cycle per SM), and CUDA's own FP64 division,
// reciprocal and square root run on it: measured 577 / 362 / 602 cycles per
// warp, while the integer and FP32 pipes beside it are idle.  The functions
// here take 132 / 79 / 121 cycles of issue slots (latency 257 / 203 / 237
// against 607 / 388 / 645), leave the FP64 pipe to the additions and products,
// and return the same bits, so the plain FP64 kernels keep the reference's
// values.
//
// Method: significands as 53-bit integers.  An FP32 reciprocal (square root)
// seed, one Newton step whose residual is formed exactly modulo 2^64, and a
// correction from the next exact residual give the quotient to well below a
// unit; the correctly rounded result follows unless that lies within the
// correction's error of a midpoint between two doubles (about one reciprocal in
// 2^15, one root in 2^13), where the pipe's own operation decides.  Division
// instead makes two quotient digits (32 and 29 bits) and settles the last unit by
// its exact remainder.  Operands whose magnitude is outside 2^-255 .. 2^256, zeros,
// infinities and NaN also take the pipe's operation.  The seeds may be off by
// 2 units in the last place (CUDA states at most 1 for rcp.approx, 2^-22.9 for
// rsqrt.approx); tests/test_exact64.py tries them perturbed.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#include <cuda_runtime.h>
#define X64 __host__ __device__ __forceinline__
// the rarely run pipe operations stay out of line
#define X64_SLOW __host__ __device__ __noinline__
#else
#define X64 inline
#define X64_SLOW inline
#endif

namespace mlau {
namespace x64 {

X64 uint32_t hi32(double x)
{
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2hiint(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return (uint32_t)(u >> 32);
#endif
}
X64 uint32_t lo32(double x)
{
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2loint(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return (uint32_t)u;
#endif
}
X64 double make(uint32_t h, uint32_t l)
{
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)h, (int)l);
#else
    const uint64_t u = ((uint64_t)h << 32) | l;
    double x;
    memcpy(&x, &u, 8);
    return x;
#endif
}
X64 float as_f(uint32_t u)
{
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float f;
    memcpy(&f, &u, 4);
    return f;
#endif
}
X64 uint32_t as_u(float f)
{
#ifdef __CUDA_ARCH__
    return __float_as_uint(f);
#else
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
#endif
}
// (hi:lo) << s, upper word; s in [0, 31]
X64 uint32_t shfl_(uint32_t lo, uint32_t hi, int s)
{
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, s);
#else
    return s ? (hi << s) | (lo >> (32 - s)) : hi;
#endif
}
// (hi:lo) >> s, lower word; s in [0, 31]
X64 uint32_t shfr_(uint32_t lo, uint32_t hi, int s)
{
#ifdef __CUDA_ARCH__
    return __funnelshift_r(lo, hi, s);
#else
    return s ? (lo >> s) | (hi << (32 - s)) : lo;
#endif
}
X64 uint64_t wide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }

// The host's seeds are exact to half a unit; MLAU_X64_SEED_ULPS (a function
// call in a test) moves them.
#ifndef MLAU_X64_SEED_ULPS
#define MLAU_X64_SEED_ULPS 0
#endif
X64 float seed_rcp(float x)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return as_f(as_u((float)(1.0 / (double)x)) + MLAU_X64_SEED_ULPS);
#endif
}
X64 float seed_rsqrt(float x)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return as_f(as_u((float)(1.0 / std::sqrt((double)x))) + MLAU_X64_SEED_ULPS);
#endif
}

// Zero exactly for exponent fields 768..1279 (magnitudes 2^-255 to 2^256, any
// sign): the integer path's operands, whose products and quotients are normal.
X64 uint32_t off_range(uint32_t h) { return (h + 0x50000000u) & 0x60000000u; }
X64 uint32_t off_range(uint32_t h, uint32_t g)
{
    return ((h + 0x50000000u) | (g + 0x50000000u)) & 0x60000000u;
}

// Operands of the products below: zero, or exponent field 512..1535 (off_wide
// is zero exactly for these).  Sums and products of such values that pass
// through a computation stay normal as long as every product's result passes
// too (its field cannot wrap around into the range), so a computation checks
// its inputs once and its products by their results.
X64 uint32_t off_field(uint32_t h) { return (h + 0x60000000u) & 0x40000000u; }
X64 uint32_t off_wide(double x)
{
    const uint32_t h = hi32(x);
    return ((h << 1) | lo32(x)) == 0 ? 0u : off_field(h);
}

// Significand's upper word, without the implicit bit for a zero.
X64 uint32_t sig_hi(uint32_t h)
{
    const uint32_t e = h & 0x7ff00000u;
    return (h & 0xfffffu) | (e < 0x100000u ? e : 0x100000u);
}

// Round (h:l | m as a fraction of 2^32 below l) to nearest even and add the
// sign and exponent word e.
X64 double round_pack(uint32_t h, uint32_t l, uint32_t m, uint32_t e)
{
#ifdef __CUDA_ARCH__
    asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %2, %3;\n\taddc.cc.u32 %0, %0, 0;\n\t"
        "addc.u32 %1, %1, %4;\n\t}"
        : "+r"(l), "+r"(h)
        : "r"(m), "r"(0x7fffffffu + (l & 1u)), "r"(e));
    return make(h, l);
#else
    const uint64_t c = ((uint64_t)m + 0x7fffffffu + (l & 1u)) >> 32;
    const uint64_t v = (((uint64_t)h << 32) | l) + c;
    return make((uint32_t)(v >> 32) + e, (uint32_t)v);
#endif
}

// 106-bit product w of two 53-bit significands (upper half p11, then w1, w0),
// normalised and rounded; sg: the sum of the operands' sign and exponent words.
X64 double norm_round(uint64_t p11, uint32_t w1, uint32_t w0, uint32_t sg)
{
    const uint32_t w3 = (uint32_t)(p11 >> 32), w2 = (uint32_t)p11, t = w3 >> 9, s = 12u - t;
    uint32_t h = shfl_(w2, w3, (int)s), l = shfl_(w1, w2, (int)s), m = shfl_(w0, w1, (int)s);
    const uint32_t e = sg + (t << 20) - (1024u << 20);
    // up when m > half, or m = half and something below it or an odd l: the
    // carry of (m : v) + 0x7fffffff:ffffffff
    const uint32_t v = w0 | (l & 1u);
#ifdef __CUDA_ARCH__
    asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %3, 0xffffffff;\n\taddc.cc.u32 t, %2, 0x7fffffff;\n\t"
        "addc.cc.u32 %0, %0, 0;\n\taddc.u32 %1, %1, %4;\n\t}"
        : "+r"(l), "+r"(h)
        : "r"(m), "r"(v), "r"(e));
    return make(h, l);
#else
    const uint64_t c = ((uint64_t)m + 0x7fffffffu + (v ? 1u : 0u)) >> 32;
    const uint64_t r = (((uint64_t)h << 32) | l) + c;
    return make((uint32_t)(r >> 32) + e, (uint32_t)r);
#endif
}
X64 double norm_product(uint64_t p11, uint32_t w1, uint32_t w0, uint32_t sg, uint32_t &bad)
{
    const double r = norm_round(p11, w1, w0, sg);
    const uint32_t rh = hi32(r);
    const bool zero = (uint32_t)(p11 >> 32) == 0;
    bad |= zero ? 0u : off_field(rh);
    return make(zero ? sg & 0x80000000u : rh, lo32(r));
}

// a * b and a * a of operands in 2^-255 .. 2^256, zero excluded
X64 double mul_nz(double a, double b, uint32_t &bad)
{
    const uint32_t ah = hi32(a), al = lo32(a), bh = hi32(b), bl = lo32(b);
    const uint32_t ma = (ah & 0xfffffu) | 0x100000u, mb = (bh & 0xfffffu) | 0x100000u;
    const uint64_t p00 = wide(al, bl);
    const uint64_t p01 = wide(ma, bl) + (wide(al, mb) + (p00 >> 32));  // below 2^55
    const uint64_t p11 = wide(ma, mb) + (p01 >> 32);
    bad |= off_range(ah, bh);
    return norm_round(p11, (uint32_t)p01, (uint32_t)p00, (ah & 0xfff00000u) + (bh & 0xfff00000u));
}
X64 double sqr_nz(double a, uint32_t &bad)
{
    const uint32_t ah = hi32(a), al = lo32(a), ma = (ah & 0xfffffu) | 0x100000u;
    const uint64_t p00 = wide(al, al);
    const uint64_t p01 = wide(al, 2u * ma) + (p00 >> 32);
    const uint64_t p11 = wide(ma, ma) + (p01 >> 32);
    bad |= off_range(ah);
    return norm_round(p11, (uint32_t)p01, (uint32_t)p00, (ah & 0x7ff00000u) << 1);
}

X64 double mul(double a, double b, uint32_t &bad)
{
    const uint32_t ah = hi32(a), al = lo32(a), bh = hi32(b), bl = lo32(b);
    const uint32_t ma = sig_hi(ah), mb = sig_hi(bh);
    const uint64_t p00 = wide(al, bl);
    const uint64_t p01 = wide(ma, bl) + (wide(al, mb) + (p00 >> 32));  // below 2^55
    const uint64_t p11 = wide(ma, mb) + (p01 >> 32);
    return norm_product(p11, (uint32_t)p01, (uint32_t)p00, (ah & 0xfff00000u) + (bh & 0xfff00000u), bad);
}

X64 double sqr(double a, uint32_t &bad)
{
    const uint32_t ah = hi32(a), al = lo32(a), ma = sig_hi(ah);
    const uint64_t p00 = wide(al, al);
    const uint64_t p01 = wide(al, 2u * ma) + (p00 >> 32);
    const uint64_t p11 = wide(ma, ma) + (p01 >> 32);
    return norm_product(p11, (uint32_t)p01, (uint32_t)p00, (ah & 0x7ff00000u) << 1, bad);
}

// k * a for an odd integer k in [3, 255]
template <int K> X64 double mulk(double a)
{
    constexpr int B = K < 4 ? 2 : K < 8 ? 3 : K < 16 ? 4 : K < 32 ? 5 : K < 64 ? 6 : K < 128 ? 7 : 8;
    // K << (11 - B) brings the 53-bit significand's product to bit 63 or 62
    constexpr uint32_t KS = (uint32_t)K << (11 - B);
    const uint32_t ah = hi32(a), al = lo32(a), ma = sig_hi(ah);
    const uint64_t p0 = wide(al, KS);
    const uint32_t xl = (uint32_t)p0, xh = ma * KS + (uint32_t)(p0 >> 32);
    // significand = X >> (11 - s), s = 1 where bit 63 is clear
    const uint32_t t = 10u + (xh >> 31);
    const uint32_t h = xh >> t, l = shfr_(xl, xh, (int)t), f = xl << (32u - t);
    const uint32_t e = (ah & 0xfff00000u) + (t << 20) + ((uint32_t)(B - 12) << 20);
    const double r = round_pack(h, l, f, e);
    return make(xh == 0 ? ah : hi32(r), lo32(r));
}

// a * 2^P, exact
template <int P> X64 double scale(double a)
{
    const uint32_t h = hi32(a);
    return make((h & 0x7ff00000u) ? h + ((uint32_t)P << 20) : h, lo32(a));
}

// Reciprocal seed of the 53-bit significand (mh:ml) in [2^52, 2^53): Y0 in
// [2^23, 2^24) with Y0 ~ 2^76 / B, and e1 = (B Y0 - 2^76) >> 24.
X64 void rcp_seed(uint32_t mh, uint32_t ml, uint32_t &Y0, int32_t &e1)
{
    const float x = as_f(0x3f800000u | (shfl_(ml, mh, 3) & 0x7fffffu));
    // y in (0.49, 1.01): its distance to 1 - 2^-22, added to a power of two's
    // significand, reads as an integer without a test of y's own exponent
    const float y = seed_rcp(x) + (1.0f - 0x1p-22f);
    Y0 = 2u * as_u(y) - (2u * 0x3f800000u - 4u);
    const uint64_t p = wide(ml, Y0);
    const uint32_t eh = mh * Y0 + (uint32_t)(p >> 32);
    e1 = (int32_t)shfr_((uint32_t)p, eh, 24);
}

// The FP64 pipe's own results, for the few lanes the integer path leaves.
static X64_SLOW double rcp_hw(double x) { return 1.0 / x; }
static X64_SLOW double div_hw(double a, double b) { return a / b; }
static X64_SLOW double sqrt_hw(double x) { return ::sqrt(x); }

// bad: nonzero where the pipe's operation has to decide
X64 double rcp_fast(double x, uint32_t &bad)
{
    const uint32_t ah = hi32(x), ml = lo32(x);
    const uint32_t mh = (ah & 0xfffffu) | 0x100000u;
    uint32_t Y0;
    int32_t e1;
    rcp_seed(mh, ml, Y0, e1);
    // Q1 ~ 2^105 / B to 2^-44: Y0 2^29 - (Y0 e1 >> 23)
    const uint64_t Q1 = ((uint64_t)Y0 << 29) - (uint64_t)(((int64_t)(int32_t)Y0 * e1) >> 23);
    const uint32_t qh = (uint32_t)(Q1 >> 32), ql = (uint32_t)Q1;
    // R = 2^105 - B Q1 (|R| < 2^61, exact modulo 2^64); r ~ R / 2^32
    const uint64_t p = wide(ml, ql);
    const uint32_t rh = (uint32_t)(p >> 32) + ml * qh + mh * ql;
    const int32_t r = (int32_t)~rh;
    // correction R Q1 / 2^105, 18 fraction bits
    const int32_t P = (int32_t)(((int64_t)r * (int32_t)shfr_(ql, qh, 23)) >> 32);
    const int32_t T = P + (1 << 17);
    const uint64_t Q = Q1 + (uint64_t)(int64_t)(T >> 18);
    bad |= off_range(ah) | ((((uint32_t)T + 4u) & 0x3ffffu) <= 8u ? 1u : 0u);
    const uint32_t e = (2044u << 20) - (ah & 0x7ff00000u) + (ah & 0x80000000u);
    return make((uint32_t)(Q >> 32) + e, (uint32_t)Q);
}

X64 double rcp(double x)
{
    uint32_t bad = 0;
    double q = rcp_fast(x, bad);
    if (bad) q = rcp_hw(x);
    return q;
}


// 0.5 / x
X64 double half_over(double x)
{
    const double r = rcp(x);
    // 1 / x a normal number above 2^-1021: the halving is exact
    const uint32_t h = hi32(r), e = (h >> 20) & 0x7ffu;
    return e - 2u < 2044u ? make(h - 0x100000u, lo32(r)) : div_hw(0.5, x);
}

// x / 24: the significand's quotient by 3 (no ties: the remainder is a third
// of a unit or two), then the exponent.
X64 double div24(double x)
{
    const uint32_t ah = hi32(x), al = lo32(x);
    const uint32_t mh = (ah & 0xfffffu) | 0x100000u;
    // N = B 2^s with N / 3 in [2^52, 2^53): s = 1 from 1.5 on, else 2
    const uint32_t s = mh >= 0x180000u ? 1u : 2u;
    const uint32_t nh = shfl_(al, mh, (int)s), nl = (al << s) + 1u;  // N + 1: round to nearest
    const uint32_t qh = nh / 3u, ql = nl / 3u;
    const uint32_t t = (nh - 3u * qh) + (nl - 3u * ql);
    const uint64_t Q = (((uint64_t)qh << 32) | ql) + (uint64_t)(nh - 3u * qh) * 0x55555555u + (t >= 3u ? 1u : 0u);
    // x / 24 = Q 2^-s 2^-3 in units of x's significand
    const uint32_t e = (ah & 0xfff00000u) - ((4u + s) << 20);
    double q = make((uint32_t)(Q >> 32) + e, (uint32_t)Q);
    if (off_range(ah)) q = div_hw(x, 24.0);
    return q;
}

X64 double div_fast(double a, double b, uint32_t &bad)
{
    const uint32_t ah = hi32(a), al = lo32(a), bh = hi32(b), ml = lo32(b);
    const uint32_t na = (ah & 0xfffffu) | 0x100000u, mh = (bh & 0xfffffu) | 0x100000u;
    uint32_t Y0;
    int32_t e1;
    rcp_seed(mh, ml, Y0, e1);
    // Y1 ~ 2^84 / B, 2 to 5 units low
    const uint32_t Y1 = (Y0 << 8) - (uint32_t)(int32_t)(((int64_t)(int32_t)Y0 * e1) >> 44) - 3u;
    // first digit, low: (A / B) 2^31 - d1 in (0, 12)
    const uint32_t d1 = (uint32_t)(wide(shfl_(al, na, 11), Y1) >> 32) - 3u;
    // R1 = A 2^31 - B d1
    const uint64_t pb = wide(ml, d1);
    const uint32_t ph = (uint32_t)(pb >> 32) + mh * d1;
    const uint64_t R1 = (((uint64_t)shfr_(al, na, 1) << 32) | (al << 31)) -
                        (((uint64_t)ph << 32) | (uint32_t)pb);
    // second digit: (A / B) 2^31 = d1 + P / 2^58
    const uint32_t r = shfr_((uint32_t)R1, (uint32_t)(R1 >> 32), 25);
    const uint64_t P = wide(r, Y1 >> 1);
    // quotient significand: (A / B) 2^52, or 2^53 where A < B
    const bool lt = na < mh || (na == mh && al < ml);
    const int sh = lt ? 22 : 21;
    const uint32_t d2 = ((uint32_t)(P >> 32) + (1u << (25 - sh))) >> (26 - sh);
    const uint64_t Q = ((uint64_t)d1 << sh) + d2;
    // remainder A 2^(31+sh) - B Q = R1 2^sh - B d2, exact modulo 2^64
    const uint64_t pd = wide(ml, d2);
    const uint64_t R2 = (R1 << sh) - (((uint64_t)((uint32_t)(pd >> 32) + mh * d2) << 32) | (uint32_t)pd);
    const int64_t B = (int64_t)(((uint64_t)mh << 32) | ml), t = 2 * (int64_t)R2;
    const uint64_t Qr = Q + (t > B ? 1u : 0u) - (t < -B ? 1u : 0u);
    const uint32_t e = (ah & 0x7ff00000u) - (bh & 0x7ff00000u) + ((lt ? 1021u : 1022u) << 20) +
                       ((ah ^ bh) & 0x80000000u);
    bad |= off_range(ah, bh);
    return make((uint32_t)(Qr >> 32) + e, (uint32_t)Qr);
}

X64 double div(double a, double b)
{
    uint32_t bad = 0;
    double q = div_fast(a, b, bad);
    if (bad) q = div_hw(a, b);
    return q;
}

X64 double sqrt_fast(double x, uint32_t &bad)
{
    const uint32_t ah = hi32(x), al = lo32(x);
    // x = X 2^(2k - 52), X = B or 2 B in [2^52, 2^54)
    const uint32_t odd = (~ah >> 20) & 1u, o23 = odd << 23;
    // xh + xl = X / 2^52 in [1, 4): the top 24 bits, the rest (23 bits of it)
    const float xh = as_f((o23 + 0x3f800000u) | (shfl_(al, ah, 3) & 0x7fffffu));
    const float xl = as_f((o23 + 0x34000000u) | ((al & 0x1fffffffu) >> 6)) - as_f(o23 + 0x34000000u);
    float y = seed_rsqrt(xh);
    y = fmaf(0.5f * y, fmaf(-xh * y, y, 1.0f), y);
    const float s1 = fminf(fmaxf(xh * y, 1.0f), 0x1.fffffep0f);
    // sqrt = s1 + c, |c| < 2^-21: C = c 2^52
    const float r1 = fmaf(-s1, s1, xh) + xl;
#ifdef __CUDA_ARCH__
    const int32_t C = __float2int_rn(r1 * (y * 0x1p51f));
#else
    const int32_t C = (int32_t)std::lrintf(r1 * (y * 0x1p51f));
#endif
    const uint64_t S2 = ((uint64_t)((as_u(s1) & 0x7fffffu) | 0x800000u) << 29) + (uint64_t)(int64_t)C;
    const uint32_t sh = (uint32_t)(S2 >> 32), sl = (uint32_t)S2;
    // R = X 2^52 - S2^2 (|R| < 2^63, exact modulo 2^64); r = floor(R / 2^32)
    const uint64_t p = wide(sl, sl);
    const uint32_t ph = (uint32_t)(p >> 32) + 2u * sh * sl;
    const int32_t r = (int32_t)((al << (20 + odd)) - ph - ((uint32_t)p != 0 ? 1u : 0u));
    // correction R / (2 S2) = r Y / 2^52 with Y = y 2^31, 20 fraction bits
    const uint32_t yb = as_u(y) < 0x3f7fffffu ? as_u(y) : 0x3f7fffffu;
    const int32_t P = (int32_t)(((int64_t)r * (int32_t)(((yb & 0x7fffffu) | 0x800000u) << 7)) >> 32);
    const int32_t T = P + (1 << 19);
    const uint64_t S = S2 + (uint64_t)(int64_t)(T >> 20);
    const uint32_t e = (((ah + 0x100000u) >> 1) & 0x7ff00000u) + (510u << 20);
    // positive, mid-range and not near a midpoint
    bad |= (ah + 0x50000000u) >> 29 == 4u && (((uint32_t)T + 64u) & 0xfffffu) > 128u ? 0u : 1u;
    return make((uint32_t)(S >> 32) + e, (uint32_t)S);
}

X64 double sqrt(double x)
{
    uint32_t bad = 0;
    double q = sqrt_fast(x, bad);
    if (bad) q = sqrt_hw(x);
    return q;
}

}  // namespace x64

}  // namespace mlau
