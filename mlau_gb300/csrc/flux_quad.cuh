// One face's MLAU, LHLLD or HLLD flux on four lanes, for grids too small to fill
// the FP64 pipes: lane bit 0 is the side (0 left, 1 right), bit 1 the tangential
// component.  A warp's FP64 instruction holds its sub-partition's pipe for 64
// cycles however many lanes take part, so formulas that are the same for both
// sides or both components are evaluated once, on the lanes side by side, and
// exchanged by shuffles; what joins them is evaluated on all four.  Sums that
// meet across lanes have two terms, whose order does not matter.  Values and
// the hand-over to riemann<double> as in flux_exact.cuh.
#pragma once

#include "flux_exact.cuh"

namespace mlau {

struct Quad {
    int side, comp;
    unsigned mask;
    __device__ __forceinline__ double other(double v) const { return __shfl_xor_sync(mask, v, 1); }
    __device__ __forceinline__ double comp2(double v) const { return __shfl_xor_sync(mask, v, 2); }
    // a difference right - left of a quantity held per side
    __device__ __forceinline__ double diff(const FxOpsT<true> &o, double v) const
    {
        const double w = other(v);
        return side ? o.sub(v, w) : o.sub(w, v);
    }
    // the quantity of side s
    __device__ __forceinline__ double from(int s, double v) const
    {
        const double w = other(v);
        return s == side ? v : w;
    }
    __device__ __forceinline__ bool any(uint32_t bad) const
    {
        bad |= __shfl_xor_sync(mask, bad, 1);
        return (bad | __shfl_xor_sync(mask, bad, 2)) != 0;
    }
};

// IN(s, n): variable n of side s; dv0, dv1 as calc_flux_*.  Lane (side 0,
// component c) returns f[2 + c] in ft and f[4 + c] in fb; every lane f[0], f[1]
// and f[6] in f0, f1, f6.
template <class LOAD>
__device__ __forceinline__ void flux_mlau_quad(LOAD IN, const Quad &Q, double bnc, double gamma, double dv0,
                                               double dv1, double &f0, double &f1, double &ft, double &fb,
                                               double &f6)
{
    FxOpsT<true> o;
    const int side = Q.side, comp = Q.comp;
    const uint32_t sp = side ? 0x80000000u : 0u;
    const double EPS = 1e-8;
    o.in(dv0);
    o.in(dv1);
    o.in(bnc);
    o.in(gamma);
    const double ro = o.in(IN(side, 0)), vn = o.in(IN(side, 1)), pr = o.in(IN(side, 6));
    const double v = o.in(IN(side, 2 + comp)), b = o.in(IN(side, 4 + comp));
    const double gm1i = o.rcp(gamma - 1.0), roi = o.rcp(ro);
    const double bnc2 = o.sqr(bnc);
    const uint32_t sgn = o.positive(bnc) ? 0u : 0x80000000u;
    const double bnca = o.flip(bnc, sgn);
    const double vv = o.sqr(v), bb = o.sqr(b), vvo = Q.comp2(vv), bbo = Q.comp2(bb);
    const double v2 = o.add(o.add(o.sqr(vn), comp ? vvo : vv), comp ? vv : vvo);
    const double pm = o.scale<-1>(o.add(bb, bbo));
    const double pt = o.add(pr, pm);
    const double en = o.add(o.add(o.mul(pr, gm1i), pm), o.mul(v2, o.scale<-1>(ro)));
    const double hn = o.mul(o.add(en, pt), roi);
    const double ca2 = o.mul(bnc2, roi), pb = o.mul(o.scale<1>(pm), roi);
    // component 0: the fast speed, component 1: the "cc" speed
    const double cs = o.mul(o.mul(pr, gamma), roi), c2 = comp ? v2 : cs;
    const double cb2 = o.add(o.add(c2, ca2), pb);
    const double cw = o.scale<-1>(o.add(cb2, o.sqrt(o.abs(o.sub(o.sqr(cb2), o.mul(o.scale<2>(c2), ca2))))));
    const double root = o.sqrt(o.max(cw, Q.other(cw))), rooto = Q.comp2(root);
    const double cfn = comp ? rooto : root, cfmod = comp ? root : rooto;
    const double cfni = o.rcp(cfn);
    const double vno = Q.other(vn);
    const double sl = o.min0(o.sub(o.min(vn, vno), cfn)), sr = o.max0(o.add(o.max(vn, vno), cfn));
    double theta = o.div(o.sub(cfn, o.min0(dv0)), o.sub(cfn, o.min0(dv1)));
    theta = o.min(1.0, theta);
    theta = o.sqr(o.sqr(theta));
    const double m = o.mul(vn, cfni), m2 = o.sub(o.sqr(m), o.one);
    const double q = o.scale<-2>(o.sqr(o.add(m, o.flip(o.one, sp))));
    const double a = o.mul(o.mul(o.mul(m, 0.1875), m2), m2);
    const bool sup = o.above(o.abs(m), 1.0);
    double bf = o.add(o.mul(q, o.sub(2.0, o.flip(m, sp))), o.flip(a, sp));
    double ff = o.flip(o.add(q, o.scale<-3>(o.sqr(m2))), sp);
    const double away = o.positive(o.flip(m, sp)) ? 1.0 : 0.0;
    bf = sup ? away : bf;
    ff = sup ? (away != 0.0 ? m : 0.0) : ff;
    const double sv = o.sub(side ? sr : sl, vn), rs = o.mul(sv, ro);
    const double rsum = o.add(ro, Q.other(ro)), bfo = Q.other(bf);
    const double mnc = o.add(ff, Q.other(ff));
    double mflux = o.mul(mnc, cfn);
    mflux = o.sub(mflux, o.div(o.mul(o.mul(o.mul(o.max0(o.sub(o.one, o.abs(mnc))), theta), cfni),
                                     Q.diff(o, pt)), rsum));
    const int up = o.positive(mflux) ? 0 : 1;
    mflux = o.mul(mflux, Q.from(up, ro));
    const double bp = o.mul(bf, pt);
    double ptot = o.add(bp, Q.other(bp));
    ptot = o.sub(ptot, o.mul(o.mul(o.mul(o.scale<-2>(o.mul(bf, bfo)), rsum), cfmod), Q.diff(o, vn)));
    ptot = o.sub(ptot, o.mul(o.mul(o.scale<-1>(o.sub(o.one, o.mul(cfmod, cfni))),
                                   o.sub(o.add(bf, bfo), o.one)), o.add(pt, Q.other(pt))));
    const double snc = up ? sr : sl;
    const double vndnm = o.add(mflux, Q.from(up, rs)), vnu = Q.from(up, vn);
    const bool has = o.above(o.abs(vndnm), EPS) && !o.zero(snc);
    const double vq = o.div(o.mul(mflux, snc), has ? vndnm : 1.0), vnc = has ? vq : vnu;
    const double sc = o.sub(side ? sr : sl, vnc), sci = o.rcp(sc);
    const double rhd = o.sub(o.mul(rs, sc), bnc2);
    const bool on = o.above(o.abs(rhd), EPS);
    const double gq = o.div(o.sub(vnc, vn), on ? rhd : 1.0), g = on ? gq : 0.0;
    const double c = o.mul(sv, sci);
    const double sro = o.sqrt(o.mul(c, ro)), oth = Q.other(sro);
    const double d = o.mul(o.mul(-bnc, b), g), e = o.mul(o.mul(o.mul(bnc2, b), g), sci);
    const double vs = o.add(d, v), bs = o.add(e, o.mul(b, c));
    const double sroi = o.rcp(o.add(sro, oth));
    auto clip = [&](double x) { return o.flip(o.min(o.max0(x), bnca), sgn); };
    const double wb = clip(o.mul(o.add(bnca, o.flip(o.mul(vnc, oth), sp)), o.mul(sro, sroi)));
    const double wv = clip(o.mul(o.add(bnca, o.flip(o.div(mflux, oth), sp)), o.mul(oth, sroi)));
    const double bnsrv = o.max0(o.sub(bnca, o.mul(up ? -vnc : vnc, Q.from(up, sro))));
    const double ccb = o.mul(bnsrv, sroi), ccv = o.mul(o.mul(sro, oth), ccb);
    const double pv = o.mul(wb, vs), pq = o.mul(wv, bs);
    double nv = o.add(o.add(pv, Q.other(pv)), o.mul(ccb, Q.diff(o, bs)));
    double nb = o.add(o.add(pq, Q.other(pq)), o.mul(ccv, Q.diff(o, vs)));
    nv = o.sub(nv, o.mul(vnc, Q.from(up, e)));
    nb = o.sub(nb, o.mul(mflux, Q.from(up, d)));
    const double vu = Q.from(up, v), bu = Q.from(up, b);
    ft = o.sub(o.mul(mflux, vu), nb);
    fb = o.sub(o.mul(o.mul(mflux, bu), Q.from(up, roi)), nv);
    const double w1 = o.mul(vu, bu), w2 = o.mul(Q.from(up, vs), Q.from(up, bs));
    const double w3 = o.mul(o.add(o.mul(ft, vnc), o.mul(fb, bnc)), o.add(o.mul(ft, bnc), o.mul(fb, mflux)));
    const double vb1 = o.add(w1, Q.comp2(w1)), vb2 = o.add(w2, Q.comp2(w2));
    double vb3 = o.add(w3, Q.comp2(w3));
    const double rv = o.sqr(o.sub(o.mul(mflux, vnc), bnc2));
    const bool ok = o.above(rv, EPS * EPS);
    vb3 = o.div(vb3, ok ? rv : 1.0);
    vb3 = ok ? vb3 : 0.0;
    const double nvb = o.add(o.mul(o.mul(bnca, o.sub(o.mul(snc, vb2), o.mul(vnc, vb1))), Q.from(up, sci)),
                             o.mul(bnsrv, o.sub(vb3, vb2)));
    f0 = mflux;
    f1 = o.sub(o.add(o.mul(mflux, vnu), ptot), o.scale<-1>(bnc2));
    f6 = o.sub(o.mul(mflux, Q.from(up, hn)), o.flip(nvb, sgn));
    if (Q.any(o.bad)) {
        double t[14], f[7];
#pragma unroll
        for (int n = 0; n < 7; n++) {
            t[n] = IN(0, n);
            t[7 + n] = IN(1, n);
        }
        flux_mlau_pipe(t, t + 7, bnc, gamma, dv0, dv1, f);
        f0 = f[0];
        f1 = f[1];
        ft = comp ? f[3] : f[2];
        fb = comp ? f[5] : f[4];
        f6 = f[6];
    }
}

template <bool LOWDISS, class LOAD>
__device__ __forceinline__ void flux_hlld_quad(LOAD IN, const Quad &Q, double bnc, double gamma, double dv0,
                                               double dv1, double &f0, double &f1, double &ft, double &fb,
                                               double &f6)
{
    FxOpsT<true> o;
    const int side = Q.side, comp = Q.comp;
    const double EPS = 1e-8;
    if constexpr (LOWDISS) {
        o.in(dv0);
        o.in(dv1);
    }
    o.in(bnc);
    o.in(gamma);
    const double ro = o.in(IN(side, 0)), vn = o.in(IN(side, 1)), pr = o.in(IN(side, 6));
    const double v = o.in(IN(side, 2 + comp)), b = o.in(IN(side, 4 + comp));
    const double gm1i = o.rcp(gamma - 1.0), roi = o.rcp(ro);
    const double bnc2 = o.sqr(bnc);
    const uint32_t sgn = o.positive(bnc) ? 0u : 0x80000000u;
    const double vv = o.sqr(v), bb = o.sqr(b), vvo = Q.comp2(vv), bbo = Q.comp2(bb), vbc = o.mul(v, b);
    const double v2 = o.add(o.add(o.sqr(vn), comp ? vvo : vv), comp ? vv : vvo);
    const double pm = o.scale<-1>(o.add(bb, bbo)), vb = o.add(vbc, Q.comp2(vbc));
    const double pt = o.add(pr, pm);
    const double en = o.add(o.add(o.mul(pr, gm1i), pm), o.mul(v2, o.scale<-1>(ro)));
    const double ca2 = o.mul(bnc2, roi), pb = o.mul(o.scale<1>(pm), roi);
    const double cs = o.mul(o.mul(pr, gamma), roi), c2 = (LOWDISS && comp) ? v2 : cs;
    const double cb2 = o.add(o.add(c2, ca2), pb);
    const double cw = o.scale<-1>(o.add(cb2, o.sqrt(o.abs(o.sub(o.sqr(cb2), o.mul(o.scale<2>(c2), ca2))))));
    const double root = o.sqrt(o.max(cw, Q.other(cw))), rooto = Q.comp2(root);
    const double cmax = comp ? rooto : root, croot = comp ? root : rooto;
    const double vno = Q.other(vn);
    const double sl = o.min0(o.sub(o.min(vn, vno), cmax)), sr = o.max0(o.add(o.max(vn, vno), cmax));
    const double sw = side ? sr : sl, sv = o.sub(sw, vn), rs = o.mul(ro, sv);
    const double drsvi = o.rcp(Q.diff(o, rs)), mom = Q.diff(o, o.mul(rs, vn));
    const double pto = Q.other(pt), rso = Q.other(rs);
    const double cross = Q.diff(o, o.mul(rs, pto)), dvn = Q.diff(o, vn);
    const double rsl = side ? rso : rs, rsr = side ? rs : rso;
    double vnc, ptc;
    if constexpr (LOWDISS) {
        double theta = o.div(o.sub(cmax, o.min0(dv0)), o.sub(cmax, o.min0(dv1)));
        theta = o.min(1.0, theta);
        theta = o.sqr(o.sqr(theta));
        vnc = o.mul(o.sub(mom, o.mul(theta, Q.diff(o, pt))), drsvi);
        const double mcc = o.min(1.0, o.div(croot, cmax));
        const double phi = o.mul(mcc, o.sub(2.0, mcc));
        ptc = o.mul(o.add(cross, o.mul(o.mul(o.mul(phi, rsr), rsl), dvn)), drsvi);
    } else {
        const double ptl = side ? pto : pt, ptr = side ? pt : pto;
        vnc = o.mul(o.add(o.sub(mom, ptr), ptl), drsvi);
        ptc = o.mul(o.add(cross, o.mul(o.mul(rsr, rsl), dvn)), drsvi);
    }
    const double sc = o.sub(sw, vnc), ro2 = o.div(rs, sc);
    const double rhd = o.sub(o.mul(rs, sc), bnc2);
    const bool on = o.above(o.abs(rhd), EPS);
    const double rhdi = o.rcp(on ? rhd : 1.0);
    const double gv = o.mul(o.mul(o.sub(vn, vnc), bnc), rhdi);
    const double gb = o.mul(o.sub(o.mul(rs, sv), bnc2), rhdi);
    const double x = on ? o.add(v, o.mul(gv, b)) : v, y = on ? o.mul(gb, b) : b;
    const double xy = o.mul(x, y), vb2 = o.add(xy, Q.comp2(xy));
    const double e = o.add(o.add(o.sub(o.mul(sv, en), o.mul(pt, vn)), o.mul(ptc, vnc)),
                           o.mul(bnc, o.sub(vb, vb2)));
    const double en2 = o.div(o.in(e), sc);
    const double rro = o.sqrt(ro2), oth = Q.other(rro);
    const double qi = o.rcp(o.add(rro, oth)), qq = o.mul(rro, oth);
    const double al = o.div(o.abs(bnc), rro), alo = Q.other(al);
    const int up = o.positive(vnc) ? 0 : 1;
    const bool outl = o.positive(o.sub(vnc, side ? alo : al)), outr = !o.positive(o.add(vnc, side ? al : alo));
    const bool mid = !outl && !outr;
    const double px = o.mul(rro, x), py = o.mul(oth, y);
    const double v3 = o.mul(o.in(o.add(o.add(px, Q.other(px)), o.flip(Q.diff(o, y), sgn))), qi);
    const double b3 = o.mul(o.in(o.add(o.add(py, Q.other(py)), o.flip(o.mul(qq, Q.diff(o, x)), sgn))), qi);
    const double w3 = o.mul(v3, b3), vb3 = o.add(w3, Q.comp2(w3));
    const int sd = mid ? up : (outl ? 0 : 1);
    const double xs = Q.from(sd, x), ys = Q.from(sd, y);
    const double vu = mid ? v3 : xs, bu = mid ? b3 : ys;
    const double w = o.mul(vu, bu), vbu = o.add(w, Q.comp2(w));
    double es = Q.from(sd, en2);
    const double cor = o.mul(Q.from(sd, rro), o.sub(Q.from(sd, vb2), vb3));
    if (mid) es = o.sub(es, o.flip(cor, sgn ^ (sd ? 0x80000000u : 0u)));
    const double rou = Q.from(up, ro2), rv = o.mul(rou, vnc);
    f0 = rv;
    f1 = o.sub(o.add(o.mul(rv, vnc), ptc), o.scale<-1>(bnc2));
    ft = o.sub(o.mul(o.mul(rou, vu), vnc), o.mul(bnc, bu));
    fb = o.sub(o.mul(bu, vnc), o.mul(bnc, vu));
    f6 = o.sub(o.mul(o.add(es, ptc), vnc), o.mul(bnc, vbu));
    if (Q.any(o.bad)) {
        double t[14], f[7];
#pragma unroll
        for (int n = 0; n < 7; n++) {
            t[n] = IN(0, n);
            t[7 + n] = IN(1, n);
        }
        flux_hlld_pipe<LOWDISS>(t, t + 7, bnc, gamma, dv0, dv1, f);
        f0 = f[0];
        f1 = f[1];
        ft = comp ? f[3] : f[2];
        fb = comp ? f[5] : f[4];
        f6 = f[6];
    }
}

}  // namespace mlau
