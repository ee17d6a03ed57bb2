// Device helpers shared by the plain FP64 step kernels (1D, 2D, 3D).
#pragma once

#include "sim.cuh"
#include "point.cuh"
#include "ed.cuh"

namespace mlau {
namespace {

constexpr int TPB = 128;

struct Box {
    int lo0, lo1, lo2, e0, e1, e2;
    __device__ __forceinline__ bool decode(long long t, int &i, int &j, int &k) const
    {
        long long tot = (long long)e0 * e1 * e2;
        if (t >= tot) return false;
        int a = (int)(t % e0);
        long long r = t / e0;
        int b = (int)(r % e1);
        int c = (int)(r / e1);
        i = lo0 + a;
        j = lo1 + b;
        k = lo2 + c;
        return true;
    }
    __host__ __device__ long long count() const { return (long long)e0 * e1 * e2; }
};

struct Dims {
    int nx, ny, nz, ox, oy, oz;
    __device__ __forceinline__ long long at(int i, int j, int k) const
    {
        return (long long)nx * ((long long)ny * k + j) + i;
    }
};

// ---------------------------------------------------------------------------
// Alfven-upwind weight of one edge from the 4 surrounding cells, summed in
// the reference's order (s-P-Q, s-P, s-Q, s); face B averaged with the cell
// offset oa (first axis) and ob (second axis).  mhd_fd_ct_3d.c:277-289.
__device__ __forceinline__ double ct_weight(const double *va, const double *vb, const double *ro,
                                            const double *ba, const double *bbf, long long s,
                                            long long P, long long Q, long long oa, long long ob)
{
    const ed eps = 1e-6;
    auto sum4 = [&](const double *f) { return ed(f[s - P - Q]) + f[s - P] + f[s - Q] + f[s]; };
    ed a = iscale<-2>(sum4(va));
    ed c = iscale<-2>(sum4(vb));
    ed rc = iscale<-2>(sum4(ro));
    rc = trcp(tsqrt(rc));
    const ed fa = ihalf(ed(ba[s - oa]) + ba[s]);
    const ed fb = ihalf(ed(bbf[s - ob]) + bbf[s]);
    a = tabs(a) + tabs(imul(fa, rc));
    c = tabs(c) + tabs(imul(fb, rc));
    return ((a + ed(0.5 * 1e-6)) / (a + c + eps)).v;
}

// One edge contribution: sgn*0.5*((ul0+ur0) + w*(ul1+ur1)) with ul from the
// linear interpolation centred one edge below and ur centred on the edge.
__device__ __forceinline__ ed emf_part(const double *fu, const double *fc, ed w, double sgn,
                                       long long c, long long st, int odr)
{
    auto l = [&](const double *f) {
        return lin_l<ed>(odr, f[c - 3 * st], f[c - 2 * st], f[c - st], f[c], f[c + st]);
    };
    auto r = [&](const double *f) {
        return lin_r<ed>(odr, f[c - 2 * st], f[c - st], f[c], f[c + st], f[c + 2 * st]);
    };
    const ed e = ihalf((l(fu) + r(fu)) + w * (l(fc) + r(fc)));
    return sgn < 0.0 ? -e : e;
}

inline void rk_coef(int nrk, int stage, double &a, double &b)
{
    const double t[3][2] = {{0.0, 1.0},
                            {0.5 + (nrk - 2) * 0.25, 0.5 - (nrk - 2) * 0.25},
                            {1. / 3., 2. / 3.}};
    a = t[stage][0];
    b = t[stage][1];
}

}  // namespace
}  // namespace mlau
