// Characteristic WCNS4 reconstruction of one cell for the plain FP64 kernels:
// the values of reconst_full / reconst_alfven with wcns4_lr (point.cuh), bit
// for bit, with the work split between the FP64 pipe and the integer pipes.
//
// What bounds it: the FP64 pipe, 64 cycles per warp instruction and
// sub-partition.  Of the 92 products and 41 sums of one field's wcns4_lr the
// sums stay on that pipe, those with a product by 2, 4 or 0.25 as one operation
// (exact scalings); the other products and the five reciprocals run as integer
// instructions (exact64.cuh: 51 / 45 / 24 / 75 cycles for a b, a a, k a, 1 / x),
// in the issue slots the FP64 pipe leaves idle, and so do the products of the
// projections.  The seven fields, the three smoothness indicators and the two
// sides go through loops over a shared-memory scratch and rotating registers:
// unrolled, the code outgrows the instruction caches.  One flag collects the
// operands outside the integer path's range; such a lane evaluates the field on
// the FP64 pipe alone.  Undecided reciprocals are settled on the spot, and
// differences that vanish (uniform on one side of a jump) stay on the integer
// path: its products by zero cost 0.7 % here and save the lanes of a shock tube
// the other path (1D, 2048 cells, a step 90 -> 71 us).  Five equal values (a
// uniform region) take constants.
//
// Reconstruction of a 3D 128^3 step (9 launches): WCNS4 34.0 ms on the FP64 pipe
// alone, 20.5 with the WCNS4 products moved, 16.7 with the projections' (FP64 pipe
// 85 % busy, issue slots 46 %), 15.9 as it stands; MUSCL 9.3 -> 5.2 ms (three-point stencils project
// three points only).  Block shapes (threads x blocks per SM) for 3D, at 16.7:
// 256 x 3; 256 x 2 16.9, 128 x 5 17.3, 384 x 1 18.9 ms; the 2D grids' few waves
// prefer 128 x 5 (512^2: 1.19 against 1.22 ms).
#pragma once

#include "ed.cuh"

namespace mlau {

// wcns4_lr on the FP64 pipe.
static __device__ __noinline__ double2 wcns4_pipe(double f0, double f1, double f2, double f3, double f4)
{
    double2 r;
    wcns4_lr<double>(f0, f1, f2, f3, f4, r.x, r.y);
    return r;
}

// Constants that stay in registers (a constant operand slows the FP64 pipe).
struct ConstReg {
    uint32_t z;
    __device__ __forceinline__ ConstReg() : z(opaque_zero()) {}
    __device__ __forceinline__ double operator()(double c) const
    {
        return __hiloint2double((int)((uint32_t)__double2hiint(c) + z), (int)((uint32_t)__double2loint(c) + z));
    }
};

// A stencil of five equal values c != 0: the weights are constants.
static __device__ __noinline__ double2 wcns4_const(double c)
{
    constexpr double S = 1.0 / 1e-40, A = 0.075 * S, M = 0.65 * S, C = 0.275 * S;
    constexpr double rl = 1.0 / (A + M + C), rr = 1.0 / (C + M + A);
    constexpr double l0 = A * rl, l1 = M * rl, l2 = 1.0 - l0 - l1;
    constexpr double r0 = C * rr, r1 = M * rr, r2 = 1.0 - r0 - r1;
    const double c3 = 3.0 * c, c6 = 6.0 * c;
    const double pa = c3 - 10.0 * c + 15.0 * c, pb = -c + c6 + c3, pc = c3 + c6 - c;
    return make_double2(0.125 * (l0 * pa + l1 * pb + l2 * pc), 0.125 * (r2 * pa + r1 * pb + r0 * pc));
}

// (value at i+1/2 from the left, at i-1/2 from the right) of one field.  A
// product by a power of two is exact, so 3 f2 serves 6 f2, and 0.25 p p is a
// quarter of the rounded p p; the operands' range excludes the underflow that
// would tell them apart.
__device__ __forceinline__ double2 wcns4_ed(double f0, double f1, double f2, double f3, double f4)
{
    using namespace x64;
    const uint32_t h2 = hi32(f2), l2 = lo32(f2);
    if ((((hi32(f0) ^ h2) | (hi32(f1) ^ h2)) | ((hi32(f3) ^ h2) | (hi32(f4) ^ h2)) |
         ((lo32(f0) ^ l2) | (lo32(f1) ^ l2)) | ((lo32(f3) ^ l2) | (lo32(f4) ^ l2))) == 0)
        return (h2 << 1 | l2) == 0 ? make_double2(0.0, 0.0) : wcns4_const(f2);
    const ConstReg K;
    uint32_t bad = off_wide(f0) | off_wide(f1) | off_wide(f2) | off_wide(f3) | off_wide(f4);
    const double one = K(1.0), m4 = K(-4.0), m2 = K(-2.0), p2 = K(2.0), q4 = K(0.25), eps = K(1e-40);
    auto add = [&](double a, double b) { return __fma_rn(a, one, b); };
    auto sub = [&](double a, double b) { return __fma_rn(-b, one, a); };
    auto times = [&](double a, double b) { return mul_nz(a, b, bad); };
    const double t0 = mulk<3>(f0), t1 = mulk<3>(f1), t2 = mulk<3>(f2), t3 = mulk<3>(f3), t4 = mulk<3>(f4);
    const double f15 = mulk<15>(f2);
    // the three smoothness indicators, then their inverse squares
    double p = add(__fma_rn(m4, f1, f0), t2), q = add(__fma_rn(m2, f1, f0), f2);
    double p1 = sub(f1, f3), q1 = add(__fma_rn(m2, f2, f1), f3);
    double p2_ = add(__fma_rn(m4, f3, f4), t2), q2 = add(__fma_rn(m2, f3, f4), f2);
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
#pragma unroll 1
    for (int n = 0; n < 3; n++) {
        const double s = __fma_rn(q4, sqr(p, bad), mul(mul(13. / 12., q, bad), q, bad));
        const double g = rcp(add(sqr(s, bad), eps));
        s0 = s1;
        s1 = s2;
        s2 = g;
        p = p1;
        q = q1;
        p1 = p2_;
        q1 = q2;
    }
    // candidate stencils of the left (+1/2) and right (-1/2) value, in the
    // order of their sum: the left weights stencil 0 first, the right stencil 2
    double x0 = add(__fma_rn(m2, mulk<5>(f1), t0), f15), x1 = add(__fma_rn(p2, t2, -f1), t3);
    double x2 = sub(__fma_rn(p2, t3, t2), f4);
    const double y0 = add(__fma_rn(m2, mulk<5>(f3), t4), f15), y1 = add(__fma_rn(p2, t2, -f3), t1);
    const double y2 = sub(__fma_rn(p2, t1, t2), f0);
    const double m1 = times(0.65, s1);
    double c0 = 0.075, c2 = 0.275;
    double2 r;
#pragma unroll 1
    for (int n = 0; n < 2; n++) {
        const double w0 = times(c0, s0);
        const double d = rcp(add(add(w0, m1), times(c2, s2)));
        const double a = times(w0, d), b = times(m1, d), c = sub(sub(one, a), b);
        const double v = add(add(mul(n ? c : a, x0, bad), mul(b, x1, bad)), mul(n ? a : c, x2, bad));
        r.x = r.y;
        r.y = scale<-3>(v);
        x0 = y0;
        x1 = y1;
        x2 = y2;
        c0 = 0.275;
        c2 = 0.075;
    }
    if (bad) r = wcns4_pipe(f0, f1, f2, f3, f4);
    return r;
}


// One thread's part of a block's shared scratch: 35 rows of NT doubles.
template <int NT> struct RecScratch {
    double (*w)[NT];
    int t;
    __device__ __forceinline__ double &operator()(int n, int m) const { return w[5 * n + m][t]; }
};

// reconst_full / reconst_alfven (point.cuh).  Q(k, m): variable k at stencil
// point m; full: the full system; PUT(s, n, u): variable n of the value at i+1/2
// from the left (s = 0) and at i-1/2 from the right (s = 1).  W4: WCNS4; else
// the code odr, whose stencil is three points (one point for first order).
// KEEP: hold the full system in registers between projection and
// back-projection, else form it again (kernels where it is rare and registers
// are short).
template <bool W4, int NT, bool KEEP = false, class LOAD, class STORE>
__device__ __forceinline__ void reconst_ed(int odr, LOAD Q, bool full, ed bn, ed gamma,
                                                 const RecScratch<NT> &W, STORE PUT)
{
    unsigned nz[7] = {0, 0, 0, 0, 0, 0, 0};
    auto column = [&](int m, ed c[7]) {
#pragma unroll
        for (int k = 0; k < 7; k++) {
            const double x = Q(k, m);
            c[k] = x;
            nz[k] |= (x64::hi32(x) << 1) | x64::lo32(x);
        }
    };
    ed by, bz, icf2, isroh;
    const int m0 = W4 ? 0 : (odr == 1 ? 2 : 1), m1 = 4 - m0;
    if constexpr (!W4) {  // the points outside count for the zero guard only
#pragma unroll
        for (int k = 1; k <= 5; k++)
            for (int m = 0; m < 5; m++)
                if (m < m0 || m > m1) nz[k] |= (x64::hi32(Q(k, m)) << 1) | x64::lo32(Q(k, m));
    }
    Eigen7<ed> E;
    if (full) {
        ed c[7];
        column(2, c);
        eigen_full<ed>(c[0], c[1], bn, c[4], c[5], c[6], gamma, E);
#pragma unroll 1
        for (int m = m0; m <= m1; m++) {
            ed wm[7];
            column(m, c);
            proj_full<ed>(E, c[0], c[1], c[2], c[3], c[4], c[5], c[6], wm);
#pragma unroll
            for (int n = 0; n < 7; n++) W(n, m) = wm[n].v;
        }
    } else {
        ed c[7];
        column(2, c);
        by = c[4];
        bz = c[5];
        const ed ro = c[0], iro = trcp(ro);
        const ed cs2 = gamma * c[6] * iro;
        const ed ca2 = bn * bn * iro;
        const ed ct2 = (by * by + bz * bz) * iro;
        const ed cb2 = cs2 + ca2 + ct2;
        const ed cf2 = ed(0.5) * (cb2 + tsqrt(tabs(cb2 * cb2 - ed(4.0) * cs2 * ca2)));
        const ed sro = tsqrt(ro);
        isroh = thalf_over(sro);
        icf2 = trcp(cf2);
#pragma unroll 1
        for (int m = m0; m <= m1; m++) {
            column(m, c);
            const ed r = c[0], b1 = c[4], b2 = c[5], p = c[6];
            const ed y1 = imul(by, b1), z2 = imul(bz, b2);
            W(0, m) = c[1].v;
            W(1, m) = (imul(cf2, r) - y1 - z2 - p).v;
            W(2, m) = (y1 + z2 + p).v;
            const ed sy = imul(sro, c[2]), sz = imul(sro, c[3]);
            W(3, m) = (sy + b1).v;
            W(4, m) = (sy - b1).v;
            W(5, m) = (sz + b2).v;
            W(6, m) = (sz - b2).v;
        }
    }
#pragma unroll 1
    for (int n = 0; n < 7; n++) {
        if constexpr (W4) {
            const double2 v = wcns4_ed(W(n, 0), W(n, 1), W(n, 2), W(n, 3), W(n, 4));
            W(n, 0) = v.x;
            W(n, 1) = v.y;
        } else {
            const double c = W(n, 2), a = odr == 1 ? c : W(n, 1), b = odr == 1 ? c : W(n, 3);
            const ed f[5] = {a, a, c, b, b};
            ed l, r;
            rec_lr(odr, f, l, r);
            W(n, 0) = l.v;
            W(n, 1) = r.v;
        }
    }
#pragma unroll 1
    for (int s = 0; s < 2; s++) {
        ed w[7], u[7];
#pragma unroll
        for (int n = 0; n < 7; n++) w[n] = W(n, s);
        if (full) {
            if constexpr (!KEEP) eigen_full<ed>(Q(0, 2), Q(1, 2), bn, Q(4, 2), Q(5, 2), Q(6, 2), gamma, E);
            back_full<ed>(E, w, u);
        } else {
            const ed byh = ihalf(by), bzh = ihalf(bz);
            u[0] = imul(icf2, w[1]) + imul(icf2, w[2]);
            u[1] = w[0];
            u[2] = imul(isroh, w[3]) + imul(isroh, w[4]);
            u[3] = imul(isroh, w[5]) + imul(isroh, w[6]);
            u[4] = ihalf(w[3]) - ihalf(w[4]);
            u[5] = ihalf(w[5]) - ihalf(w[6]);
            u[6] = w[2] - imul(byh, w[3]) + imul(byh, w[4]) - imul(bzh, w[5]) + imul(bzh, w[6]);
        }
#pragma unroll
        for (int k = 1; k <= 5; k++)
            if (nz[k] == 0) u[k] = 0.0;
#pragma unroll
        for (int k = 0; k < 7; k++) PUT(s, k, u[k].v);
    }
}

template <int NT> constexpr size_t rec_smem() { return sizeof(double) * 35 * NT; }

}  // namespace mlau
