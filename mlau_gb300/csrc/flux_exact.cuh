// Riemann fluxes of the plain FP64 kernels on both pipes: the values of
// riemann<double> (point.cuh) for MLAU, LHLLD and HLLD.
//
// What bounds a face: written for the FP64 pipe alone, MLAU's 113 sums, 182
// products, 23 quotients and roots and some 25 comparisons kept that pipe 94 %
// busy with issue slots 13 % used.  Here the sums and some 40 products stay on
// it; the other products, the quotients and roots run as integer sequences
// (exact64.cuh), comparisons look at the values' bits, products by powers of
// two move exponents, and weights that are 0 or 1 become selections (which can
// change the sign of a zero, no value).  A reciprocal or root whose rounding is
// undecided (one in 2^15, 2^13) is settled by the pipe on the spot: collected instead,
// one lane in a warp of some 600 evaluations sent the whole face through
// riemann<double>, and every small launch waited for such a warp (200 x 120
// cells, fluxes of a step 139 -> 83 us; 128^3 8.9 -> 7.7 ms).  `bad` collects
// products outside the integer path's range and values that are not finite;
// such a face is evaluated again with the products on the pipe, and by
// riemann<double> if that is not enough.
//
// The new bound is instruction supply: integer products make the code long
// (some 35 instructions each), and beyond the instruction caches a sub-partition
// gets about one instruction per two cycles.  The two sides and the two
// tangential components therefore share code in loops of two with their values
// in shared memory, and blocks have 256 threads, two per SM (of 128 threads,
// four per SM, 1.1 ms more; products out of line 1.3, all unrolled 6.9 more).
//
// Face fluxes of a 128^3 step: MLAU 15.5 -> 7.7 ms.
#pragma once

#include "ed.cuh"

namespace mlau {

// Operations of one flux evaluation.  Sums run on the FP64 pipe, quotients and
// roots as integer sequences.  PIPE = false: products are integer sequences too,
// and `bad` collects every input and product outside the integer path's range
// (zero apart).  PIPE = true, for grids that leave the pipes idle and wait on
// instructions instead, and for magnitudes beyond that range: products stay on
// the FP64 pipe, one instruction each.  Either way `bad` is zero only if every
// value that was compared is finite, so comparisons can be made on the values'
// bits.
template <bool PIPE> struct FxOpsT {
    uint32_t bad = 0;
    double one, mz;
    __device__ __forceinline__ FxOpsT() : one(ed_one()), mz(ed_minus_zero()) {}

    static __device__ __forceinline__ uint32_t hi(double x) { return x64::hi32(x); }
    static __device__ __forceinline__ uint32_t lo(double x) { return x64::lo32(x); }
    static __device__ __forceinline__ bool zero(double x) { return ((hi(x) << 1) | lo(x)) == 0; }
    // an input: zero or in range
    __device__ __forceinline__ double in(double x)
    {
        if constexpr (!PIPE) bad |= x64::off_wide(x);
        return x;
    }
    // a value about to be compared: finite
    __device__ __forceinline__ void cmp(double x)
    {
        if constexpr (PIPE) bad |= (hi(x) << 1) >= 0xffe00000u ? 1u : 0u;
    }
    __device__ __forceinline__ double add(double a, double b) const { return __fma_rn(a, one, b); }
    __device__ __forceinline__ double sub(double a, double b) const { return __fma_rn(-b, one, a); }
    // on the FP64 pipe; the operands are looked at elsewhere
    __device__ __forceinline__ double hmul(double a, double b) const { return __fma_rn(a, b, mz); }
    __device__ __forceinline__ double mul(double a, double b)
    {
        return PIPE ? hmul(a, b) : x64::mul(a, b, bad);
    }
    __device__ __forceinline__ double sqr(double a) { return PIPE ? hmul(a, a) : x64::sqr(a, bad); }
    template <int P> __device__ __forceinline__ double scale(double a) const
    {
        constexpr double c = P >= 0 ? (double)(1 << (P >= 0 ? P : 0)) : 1.0 / (double)(1 << (P < 0 ? -P : 0));
        return PIPE ? hmul(a, c) : x64::scale<P>(a);
    }
    // an undecided rounding or an operand out of range is settled where it occurs;
    // results that are not finite hand the face over
    __device__ __forceinline__ double finite(double r)
    {
        bad |= (hi(r) << 1) >= 0xffe00000u ? 1u : 0u;
        return r;
    }
    __device__ __forceinline__ double rcp(double a) { return finite(x64::rcp(a)); }
    // a may be zero
    __device__ __forceinline__ double div(double a, double b)
    {
        const bool z = zero(a);
        const double r = finite(x64::div(z ? 1.0 : a, b));
        return z ? x64::make((hi(a) ^ hi(b)) & 0x80000000u, 0) : r;
    }
    __device__ __forceinline__ double sqrt(double a)
    {
        const bool z = zero(a);
        const double r = finite(x64::sqrt(z ? 1.0 : a));
        return z ? a : r;
    }
    static __device__ __forceinline__ double abs(double a) { return x64::make(hi(a) & 0x7fffffffu, lo(a)); }
    __device__ __forceinline__ bool positive(double a)
    {
        cmp(a);
        return PIPE ? (int32_t)hi(a) > 0 || (hi(a) == 0 && lo(a) != 0) : (int32_t)hi(a) > 0;
    }
    __device__ __forceinline__ bool ge(double a, double b)
    {
        cmp(a);
        cmp(b);
        const int32_t ha = (int32_t)hi(a), hb = (int32_t)hi(b), sa = ha >> 31, sb = hb >> 31;
        const int32_t ka = ha ^ (sa & 0x7fffffff), kb = hb ^ (sb & 0x7fffffff);
        return ka > kb || (ka == kb && (lo(a) ^ (uint32_t)sa) >= (lo(b) ^ (uint32_t)sb));
    }
    // a > b for a >= 0 and a constant b > 0
    __device__ __forceinline__ bool above(double a, double b)
    {
        cmp(a);
        return hi(a) > hi(b) || (hi(a) == hi(b) && lo(a) > lo(b));
    }
    __device__ __forceinline__ double max(double a, double b) { return ge(a, b) ? a : b; }
    __device__ __forceinline__ double min(double a, double b) { return ge(a, b) ? b : a; }
    __device__ __forceinline__ double max0(double a)
    {
        cmp(a);
        return (int32_t)hi(a) < 0 ? 0.0 : a;
    }
    __device__ __forceinline__ double min0(double a)
    {
        cmp(a);
        return (int32_t)hi(a) < 0 ? a : 0.0;
    }
    static __device__ __forceinline__ double flip(double a, uint32_t sign) { return x64::make(hi(a) ^ sign, lo(a)); }
};

static __device__ __noinline__ void flux_mlau_pipe(const double *L, const double *R, double bn, double gamma,
                                                   double dv0, double dv1, double *f)
{
    flux_mlau<double>(L, R, bn, gamma, dv0, dv1, f);
}

// A face's shared scratch: ROWS values per side, one column per thread.
enum { FX_ROI, FX_PT, FX_HN, FX_CF2, FX_CC2, FX_BF, FX_FF, FX_SV, FX_RS, FX_DV, FX_DB = FX_DV + 2,
       FX_V2 = FX_DB + 2, FX_B2 = FX_V2 + 2, FX_ROWS = FX_B2 + 2 };
// rows used again once their first value is spent
enum { FX_SCI = FX_CF2, FX_SRO = FX_CC2, FX_FB = FX_BF, FX_FV = FX_FF };

// IN(s, n): variable n of the left (s = 0) and right (1) state;
// dv: the ND shock sensors, of which the smallest counts.  The two sides, and
// the two tangential components, run through the same code in loops of two:
// written out twice it overflows the instruction cache.
template <int ND, int NT, bool PIPE, class LOAD>
__device__ __forceinline__ bool flux_mlau_core(LOAD IN, double (*rows)[NT], double bnc, double gamma, double dv0,
                                               const double dv[ND], double f[7])
{
    FxOpsT<PIPE> o;
    const int t = threadIdx.x;
    auto W = [&](int s, int k) -> double & { return rows[s * FX_ROWS + k][t]; };
    double dv1 = dv[0];
#pragma unroll
    for (int n = 0; n < ND; n++) {
        o.in(dv[n]);
        if (n) dv1 = o.min(dv1, dv[n]);
    }
    const double EPS = 1e-8;
    o.in(dv0);
    o.in(bnc);
    o.in(gamma);
    const double gm1i = o.rcp(gamma - 1.0);
    const double bnc2 = o.sqr(bnc);
    const uint32_t sgn = o.positive(bnc) ? 0u : 0x80000000u;
    const double bnca = o.flip(bnc, sgn);
    // each side: energy, enthalpy, fast and "cc" speeds squared
#pragma unroll 1
    for (int s = 0; s < 2; s++) {
        const double ro = o.in(IN(s, 0)), bt = o.in(IN(s, 4)), bu = o.in(IN(s, 5)), pr = o.in(IN(s, 6));
        const double roi = o.rcp(ro);
        const double v2 = o.add(o.add(o.sqr(o.in(IN(s, 1))), o.sqr(o.in(IN(s, 2)))), o.sqr(o.in(IN(s, 3))));
        const double pm = o.scale<-1>(o.add(o.sqr(bt), o.sqr(bu)));
        const double pt = o.add(pr, pm);
        const double en = o.add(o.add(o.mul(pr, gm1i), pm), o.mul(v2, o.scale<-1>(ro)));
        const double ca2 = o.mul(bnc2, roi), pb = o.mul(o.scale<1>(pm), roi);
        W(s, FX_ROI) = roi;
        W(s, FX_PT) = pt;
        W(s, FX_HN) = o.mul(o.add(en, pt), roi);
        double c2 = o.mul(o.mul(pr, gamma), roi);
#pragma unroll 1
        for (int q = 0; q < 2; q++) {
            const double cb2 = o.add(o.add(c2, ca2), pb);
            W(s, q ? FX_CC2 : FX_CF2) =
                o.scale<-1>(o.add(cb2, o.sqrt(o.abs(o.sub(o.sqr(cb2), o.mul(o.scale<2>(c2), ca2))))));
            c2 = v2;
        }
    }
    const double rol = IN(0, 0), vnl = IN(0, 1), ror = IN(1, 0), vnr = IN(1, 1);
    const double cfn = o.sqrt(o.max(W(0, FX_CF2), W(1, FX_CF2)));
    const double cfni = o.rcp(cfn);
    const double sl = o.min0(o.sub(o.min(vnl, vnr), cfn));
    const double sr = o.max0(o.add(o.max(vnl, vnr), cfn));
    double theta = o.div(o.sub(cfn, o.min0(dv0)), o.sub(cfn, o.min0(dv1)));
    theta = o.min(1.0, theta);
    theta = o.sqr(o.sqr(theta));
    const double cfmod = o.sqrt(o.max(W(0, FX_CC2), W(1, FX_CC2)));
    // Mach polynomials (the right side's mirror the left's), wave - flow speed
#pragma unroll 1
    for (int s = 0; s < 2; s++) {
        const uint32_t sp = s ? 0x80000000u : 0u;
        const double ro = IN(s, 0), vn = IN(s, 1), m = o.mul(vn, cfni);
        const double m2 = o.sub(o.sqr(m), o.one), q = o.scale<-2>(o.sqr(o.add(m, o.flip(o.one, sp))));
        const double a = o.mul(o.mul(o.mul(m, 0.1875), m2), m2);
        const bool sup = o.above(o.abs(m), 1.0);
        const double bf = o.add(o.mul(q, o.sub(2.0, o.flip(m, sp))), o.flip(a, sp));
        const double ff = o.flip(o.add(q, o.scale<-3>(o.sqr(m2))), sp);
        const double on = o.positive(o.flip(m, sp)) ? 1.0 : 0.0;
        W(s, FX_BF) = sup ? on : bf;
        W(s, FX_FF) = sup ? (on != 0.0 ? m : 0.0) : ff;
        const double sv = o.sub(s ? sr : sl, vn);
        W(s, FX_SV) = sv;
        W(s, FX_RS) = o.mul(sv, ro);
    }
    const double ptl = W(0, FX_PT), ptr = W(1, FX_PT), bfl = W(0, FX_BF), bfr = W(1, FX_BF);
    const double rsum = o.add(rol, ror);
    const double mnc = o.add(W(0, FX_FF), W(1, FX_FF));
    double mflux = o.mul(mnc, cfn);
    mflux = o.sub(mflux, o.div(o.mul(o.mul(o.mul(o.max0(o.sub(o.one, o.abs(mnc))), theta), cfni),
                                     o.sub(ptr, ptl)), rsum));
    const int up = o.positive(mflux) ? 0 : 1;  // the upwind side
    mflux = o.mul(mflux, IN(up, 0));
    double ptot = o.add(o.hmul(bfl, ptl), o.hmul(bfr, ptr));
    ptot = o.sub(ptot, o.mul(o.mul(o.mul(o.scale<-2>(o.mul(bfl, bfr)), rsum), cfmod), o.sub(vnr, vnl)));
    ptot = o.sub(ptot, o.hmul(o.hmul(o.scale<-1>(o.sub(o.one, o.mul(cfmod, cfni))),
                                     o.sub(o.add(bfl, bfr), o.one)), o.add(ptl, ptr)));
    const double snc = up ? sr : sl;
    const double vndnm = o.add(mflux, W(up, FX_RS));
    const bool has = o.above(o.abs(vndnm), EPS) && !o.zero(snc);
    const double vq = o.div(o.mul(mflux, snc), has ? vndnm : 1.0);
    const double vnc = has ? vq : IN(up, 1);
    // each side's star state
#pragma unroll 1
    for (int s = 0; s < 2; s++) {
        const double sc = o.sub(s ? sr : sl, vnc), sci = o.rcp(sc);
        const double rhd = o.sub(o.mul(W(s, FX_RS), sc), bnc2);
        const bool on = o.above(o.abs(rhd), EPS);
        const double gq = o.div(o.sub(vnc, IN(s, 1)), on ? rhd : 1.0), g = on ? gq : 0.0;
        const double c = o.mul(W(s, FX_SV), sci);
        W(s, FX_SCI) = sci;
        W(s, FX_SRO) = o.sqrt(o.mul(c, IN(s, 0)));
#pragma unroll 1
        for (int p = 0; p < 2; p++) {
            const double b = IN(s, 4 + p);
            const double d = o.hmul(o.hmul(-bnc, b), g), e = o.hmul(o.hmul(o.hmul(bnc2, b), g), sci);
            W(s, FX_DV + p) = d;
            W(s, FX_DB + p) = e;
            W(s, FX_V2 + p) = o.add(d, IN(s, 2 + p));
            W(s, FX_B2 + p) = o.add(e, o.hmul(b, c));
        }
    }
    const double srol = W(0, FX_SRO), sror = W(1, FX_SRO);
    const double sroi = o.rcp(o.add(srol, sror));
    auto clip = [&](double x) { return o.flip(o.min(o.max0(x), bnca), sgn); };
#pragma unroll 1
    for (int s = 0; s < 2; s++) {
        const uint32_t sp = s ? 0x80000000u : 0u;
        const double own = s ? sror : srol, oth = s ? srol : sror;
        W(s, FX_FB) = clip(o.mul(o.add(bnca, o.flip(o.mul(vnc, oth), sp)), o.mul(own, sroi)));
        W(s, FX_FV) = clip(o.mul(o.add(bnca, o.flip(o.div(mflux, oth), sp)), o.mul(oth, sroi)));
    }
    const double bnsrv = o.max0(o.sub(bnca, o.mul(up ? -vnc : vnc, up ? sror : srol)));
    const double ccb = o.mul(bnsrv, sroi);
    const double ccv = o.mul(o.mul(srol, sror), ccb);
    const double flb = W(0, FX_FB), frb = W(1, FX_FB), flv = W(0, FX_FV), frv = W(1, FX_FV);
    const double roi = W(up, FX_ROI);
    double vb1 = 0.0, vb2 = 0.0, vb3 = 0.0;
#pragma unroll 1
    for (int p = 0; p < 2; p++) {
        const double v2l = W(0, FX_V2 + p), v2r = W(1, FX_V2 + p), b2l = W(0, FX_B2 + p), b2r = W(1, FX_B2 + p);
        const double vs = IN(up, 2 + p), bs = IN(up, 4 + p);
        double nv = o.add(o.add(o.hmul(flb, v2l), o.hmul(frb, v2r)), o.hmul(ccb, o.sub(b2r, b2l)));
        double nb = o.add(o.add(o.hmul(flv, b2l), o.hmul(frv, b2r)), o.hmul(ccv, o.sub(v2r, v2l)));
        nv = o.sub(nv, o.hmul(vnc, W(up, FX_DB + p)));
        nb = o.sub(nb, o.hmul(mflux, W(up, FX_DV + p)));
        const double fv = o.sub(o.mul(mflux, vs), nb), fb = o.sub(o.mul(o.mul(mflux, bs), roi), nv);
        W(0, FX_DV + p) = fv;
        W(0, FX_DB + p) = fb;
        const double w1 = o.mul(vs, bs), w2 = o.mul(up ? v2r : v2l, up ? b2r : b2l);
        const double w3 = o.mul(o.add(o.mul(fv, vnc), o.mul(fb, bnc)), o.add(o.mul(fv, bnc), o.mul(fb, mflux)));
        vb1 = p ? o.add(vb1, w1) : w1;
        vb2 = p ? o.add(vb2, w2) : w2;
        vb3 = p ? o.add(vb3, w3) : w3;
    }
    const double rv = o.sqr(o.sub(o.mul(mflux, vnc), bnc2));
    const bool on = o.above(rv, EPS * EPS);
    vb3 = o.div(vb3, on ? rv : 1.0);
    vb3 = on ? vb3 : 0.0;
    const double nvb = o.add(o.mul(o.mul(bnca, o.sub(o.mul(snc, vb2), o.mul(vnc, vb1))), W(up, FX_SCI)),
                             o.hmul(bnsrv, o.sub(vb3, vb2)));
    f[0] = mflux;
    f[1] = o.sub(o.add(o.mul(mflux, IN(up, 1)), ptot), o.scale<-1>(bnc2));
    f[2] = W(0, FX_DV);
    f[3] = W(0, FX_DV + 1);
    f[4] = W(0, FX_DB);
    f[5] = W(0, FX_DB + 1);
    f[6] = o.sub(o.mul(mflux, W(up, FX_HN)), o.flip(nvb, sgn));
    return o.bad != 0;
}

// Faces the integer path hands over: first with the products on the FP64 pipe,
// which take any magnitude, then all of it.
template <int NT>
__device__ __noinline__ void flux_mlau_over(const double *c, double (*rows)[NT], double bnc, double gamma, double dv0,
                                          double dv1, double *f)
{
    const double dv[1] = {dv1};
    if (flux_mlau_core<1, NT, true>([&](int s, int n) { return c[7 * s + n]; }, rows, bnc, gamma, dv0, dv, f))
        flux_mlau_pipe(c, c + 7, bnc, gamma, dv0, dv1, f);
}

template <int ND, int NT, class LOAD>
__device__ __forceinline__ void flux_mlau_ed(LOAD IN, double (*rows)[NT], double bnc, double gamma, double dv0,
                                             const double dv[ND], double f[7])
{
    if (flux_mlau_core<ND, NT, false>(IN, rows, bnc, gamma, dv0, dv, f)) {
        double c[14], g[7];
#pragma unroll
        for (int n = 0; n < 7; n++) {
            c[n] = IN(0, n);
            c[7 + n] = IN(1, n);
        }
        double d1 = vmin(dv[0], dv[ND > 1 ? 1 : 0]);
        if constexpr (ND == 4) d1 = vmin(d1, vmin(dv[2], dv[3]));
        flux_mlau_over<NT>(c, rows, bnc, gamma, dv0, d1, g);
#pragma unroll
        for (int n = 0; n < 7; n++) f[n] = g[n];
    }
}


template <bool LOWDISS>
static __device__ __noinline__ void flux_hlld_pipe(const double *L, const double *R, double bn, double gamma,
                                                   double dv0, double dv1, double *f)
{
    flux_hlld<double, LOWDISS>(L, R, bn, gamma, dv0, dv1, f);
}

enum { HX_PT, HX_EN, HX_VB, HX_CF2, HX_CC2, HX_V2, HX_B2 = HX_V2 + 2, HX_ROWS = HX_B2 + 2 };
enum { HX_RO2 = HX_PT, HX_RRO = HX_VB, HX_VB2 = HX_CF2, HX_EN2 = HX_EN };

template <bool LOWDISS, int ND, int NT, bool PIPE, class LOAD>
__device__ __forceinline__ bool flux_hlld_core(LOAD IN, double (*rows)[NT], double bnc, double gamma, double dv0,
                                               const double dv[ND], double f[7])
{
    FxOpsT<PIPE> o;
    const int t = threadIdx.x;
    auto W = [&](int s, int k) -> double & { return rows[s * HX_ROWS + k][t]; };
    double dv1 = dv[0];
    if constexpr (LOWDISS) {
#pragma unroll
        for (int n = 0; n < ND; n++) {
            o.in(dv[n]);
            if (n) dv1 = o.min(dv1, dv[n]);
        }
        o.in(dv0);
    }
    o.in(bnc);
    o.in(gamma);
    const double EPS = 1e-8;
    const double gm1i = o.rcp(gamma - 1.0);
    const double bnc2 = o.sqr(bnc);
    const uint32_t sgn = o.positive(bnc) ? 0u : 0x80000000u;
    const double bnca = o.abs(bnc);
#pragma unroll 1
    for (int s = 0; s < 2; s++) {
        const double ro = o.in(IN(s, 0)), bt = o.in(IN(s, 4)), bu = o.in(IN(s, 5)), pr = o.in(IN(s, 6));
        const double vt = o.in(IN(s, 2)), vu = o.in(IN(s, 3));
        const double roi = o.rcp(ro);
        const double v2 = o.add(o.add(o.sqr(o.in(IN(s, 1))), o.sqr(vt)), o.sqr(vu));
        const double pm = o.scale<-1>(o.add(o.sqr(bt), o.sqr(bu)));
        W(s, HX_PT) = o.add(pr, pm);
        W(s, HX_EN) = o.add(o.add(o.hmul(pr, gm1i), pm), o.hmul(v2, o.scale<-1>(ro)));
        W(s, HX_VB) = o.add(o.hmul(vt, bt), o.hmul(vu, bu));
        const double ca2 = o.mul(bnc2, roi), pb = o.mul(o.scale<1>(pm), roi);
        double c2 = o.mul(o.mul(pr, gamma), roi);
#pragma unroll 1
        for (int q = 0; q < (LOWDISS ? 2 : 1); q++) {
            const double cb2 = o.add(o.add(c2, ca2), pb);
            W(s, q ? HX_CC2 : HX_CF2) =
                o.scale<-1>(o.add(cb2, o.sqrt(o.abs(o.sub(o.sqr(cb2), o.mul(o.scale<2>(c2), ca2))))));
            c2 = v2;
        }
    }
    const double vnl = IN(0, 1), vnr = IN(1, 1), ptl = W(0, HX_PT), ptr = W(1, HX_PT);
    // a root is monotonic: the larger of the two roots is the root of the larger
    const double cmax = o.sqrt(o.max(W(0, HX_CF2), W(1, HX_CF2)));
    const double sl = o.min0(o.sub(o.min(vnl, vnr), cmax));
    const double sr = o.max0(o.add(o.max(vnl, vnr), cmax));
    const double slvl = o.sub(sl, vnl), srvr = o.sub(sr, vnr);
    const double rsl = o.mul(IN(0, 0), slvl), rsr = o.mul(IN(1, 0), srvr);
    const double drsvi = o.rcp(o.sub(rsr, rsl));
    const double mom = o.sub(o.mul(rsr, vnr), o.mul(rsl, vnl));
    const double dpt = o.sub(ptr, ptl);
    const double cross = o.sub(o.mul(rsr, ptl), o.mul(rsl, ptr)), dvn = o.sub(vnr, vnl);
    double vnc, ptc;
    if constexpr (LOWDISS) {
        double theta = o.div(o.sub(cmax, o.min0(dv0)), o.sub(cmax, o.min0(dv1)));
        theta = o.min(1.0, theta);
        theta = o.sqr(o.sqr(theta));
        vnc = o.mul(o.sub(mom, o.mul(theta, dpt)), drsvi);
        const double mcc = o.min(1.0, o.div(o.sqrt(o.max(W(0, HX_CC2), W(1, HX_CC2))), cmax));
        const double phi = o.mul(mcc, o.sub(2.0, mcc));
        ptc = o.mul(o.add(cross, o.mul(o.mul(o.mul(phi, rsr), rsl), dvn)), drsvi);
    } else {
        vnc = o.mul(o.add(o.sub(mom, ptr), ptl), drsvi);
        ptc = o.mul(o.add(cross, o.mul(o.mul(rsr, rsl), dvn)), drsvi);
    }
#pragma unroll 1
    for (int s = 0; s < 2; s++) {
        const double sv = s ? srvr : slvl, rs = s ? rsr : rsl, vn = s ? vnr : vnl, pt = s ? ptr : ptl;
        const double sc = o.sub(s ? sr : sl, vnc);
        const double ro2 = o.div(rs, sc);
        const double rhd = o.sub(o.mul(rs, sc), bnc2);
        const bool on = o.above(o.abs(rhd), EPS);
        const double rhdi = o.rcp(on ? rhd : 1.0);
        const double gv = o.mul(o.mul(o.sub(vn, vnc), bnc), rhdi);
        const double gb = o.mul(o.sub(o.mul(rs, sv), bnc2), rhdi);
        double vb2 = 0.0;
#pragma unroll 1
        for (int p = 0; p < 2; p++) {
            const double v = IN(s, 2 + p), b = IN(s, 4 + p);
            const double x = on ? o.add(v, o.mul(gv, b)) : v, y = on ? o.mul(gb, b) : b;
            const double xy = o.mul(x, y);
            W(s, HX_V2 + p) = x;
            W(s, HX_B2 + p) = y;
            vb2 = p ? o.add(vb2, xy) : xy;
        }
        const double e = o.add(o.add(o.sub(o.hmul(sv, W(s, HX_EN)), o.hmul(pt, vn)), o.hmul(ptc, vnc)),
                               o.hmul(bnc, o.sub(W(s, HX_VB), vb2)));
        W(s, HX_EN2) = o.div(o.in(e), sc);
        W(s, HX_RO2) = ro2;
        W(s, HX_RRO) = o.sqrt(ro2);
        W(s, HX_VB2) = vb2;
    }
    const double ql = W(0, HX_RRO), qr = W(1, HX_RRO);
    const double qi = o.rcp(o.add(qr, ql)), qq = o.mul(qr, ql);
    const int up = o.positive(vnc) ? 0 : 1;
    const bool outl = o.positive(o.sub(vnc, o.div(bnca, ql))), outr = !o.positive(o.add(vnc, o.div(bnca, qr)));
    const bool mid = !outl && !outr;
    double vu[2], bu[2], vb3 = 0.0, vbu = 0.0;
#pragma unroll 1
    for (int p = 0; p < 2; p++) {
        const double v2l = W(0, HX_V2 + p), v2r = W(1, HX_V2 + p), b2l = W(0, HX_B2 + p), b2r = W(1, HX_B2 + p);
        const double v3 = o.mul(o.in(o.add(o.add(o.mul(qr, v2r), o.mul(ql, v2l)), o.flip(o.sub(b2r, b2l), sgn))), qi);
        const double b3 = o.mul(o.in(o.add(o.add(o.mul(ql, b2r), o.mul(qr, b2l)),
                                           o.flip(o.mul(qq, o.sub(v2r, v2l)), sgn))), qi);
        const double w3 = o.mul(v3, b3);
        vb3 = p ? o.add(vb3, w3) : w3;
        const double v = mid ? v3 : (outl ? v2l : v2r), b = mid ? b3 : (outl ? b2l : b2r);
        const double w = o.mul(v, b);
        vbu = p ? o.add(vbu, w) : w;
        vu[0] = vu[1];
        vu[1] = v;
        bu[0] = bu[1];
        bu[1] = b;
    }
    // energy of the state at the face: a star state, corrected in the middle
    const int sd = mid ? up : (outl ? 0 : 1);
    double en = W(sd, HX_EN2);
    const double cor = o.hmul(sd ? qr : ql, o.sub(W(sd, HX_VB2), vb3));
    if (mid) en = o.sub(en, o.flip(cor, sgn ^ (sd ? 0x80000000u : 0u)));
    const double rou = W(up, HX_RO2), rv = o.mul(rou, vnc);
    f[0] = rv;
    f[1] = o.sub(o.add(o.mul(rv, vnc), ptc), o.scale<-1>(bnc2));
    f[2] = o.sub(o.hmul(o.hmul(rou, vu[0]), vnc), o.hmul(bnc, bu[0]));
    f[3] = o.sub(o.hmul(o.hmul(rou, vu[1]), vnc), o.hmul(bnc, bu[1]));
    f[4] = o.sub(o.hmul(bu[0], vnc), o.hmul(bnc, vu[0]));
    f[5] = o.sub(o.hmul(bu[1], vnc), o.hmul(bnc, vu[1]));
    f[6] = o.sub(o.hmul(o.add(en, ptc), vnc), o.hmul(bnc, vbu));
    return o.bad != 0;
}

// Faces the integer path hands over: first with the products on the FP64 pipe,
// which take any magnitude, then all of it.
template <bool LOWDISS, int NT>
__device__ __noinline__ void flux_hlld_over(const double *c, double (*rows)[NT], double bnc, double gamma, double dv0,
                                          double dv1, double *f)
{
    const double dv[1] = {dv1};
    if (flux_hlld_core<LOWDISS, 1, NT, true>([&](int s, int n) { return c[7 * s + n]; }, rows, bnc, gamma, dv0, dv, f))
        flux_hlld_pipe<LOWDISS>(c, c + 7, bnc, gamma, dv0, dv1, f);
}

template <bool LOWDISS, int ND, int NT, class LOAD>
__device__ __forceinline__ void flux_hlld_ed(LOAD IN, double (*rows)[NT], double bnc, double gamma, double dv0,
                                             const double dv[ND], double f[7])
{
    if (flux_hlld_core<LOWDISS, ND, NT, false>(IN, rows, bnc, gamma, dv0, dv, f)) {
        double c[14], g[7];
#pragma unroll
        for (int n = 0; n < 7; n++) {
            c[n] = IN(0, n);
            c[7 + n] = IN(1, n);
        }
        double d1 = vmin(dv[0], dv[ND > 1 ? 1 : 0]);
        if constexpr (ND == 4) d1 = vmin(d1, vmin(dv[2], dv[3]));
        flux_hlld_over<LOWDISS, NT>(c, rows, bnc, gamma, dv0, d1, g);
#pragma unroll
        for (int n = 0; n < 7; n++) f[n] = g[n];
    }
}

// shared memory of a block of NT threads
template <int WHICH, int NT> constexpr size_t fx_smem()
{
    return sizeof(double) * 2 * (WHICH == FLUX_MLAU ? (int)FX_ROWS : (int)HX_ROWS) * NT;
}

// riemann (point.cuh) of one face.
template <int WHICH, int ND, int NT, class LOAD>
__device__ __forceinline__ void riemann_ed(LOAD IN, double (*rows)[NT], double bn, double gamma, double dv0,
                                           const double dv[ND], double f[7])
{
    if constexpr (WHICH == FLUX_MLAU) flux_mlau_ed<ND, NT>(IN, rows, bn, gamma, dv0, dv, f);
    else flux_hlld_ed<WHICH == FLUX_LHLLD, ND, NT>(IN, rows, bn, gamma, dv0, dv, f);
}

}  // namespace mlau
