// Plain FP64 1D step: one SSP-RK step of 1D MHD (7 variables, constant Bx),
// the GPU form of 1D/SERIAL/shock/mhd_fd4c_1d.c:60-271 with either the
// characteristic open boundary of 1D/SERIAL/shock/openbc1d_mhd.c:21-175
// (applied once, at stage 0, between the fluxes and the update) or the
// periodic boundary of 1D/SERIAL/wave (prdc_1d after each stage).
// Compiled with --fmad=false: bit-for-bit the reference's arithmetic.
//
// State slots: 0 ro, 1 mx, 2 my, 3 mz, 4 en, 6 by, 7 bz (slot 5 unused).
//
// One launch per RK stage (k_stage1).  A 1D grid holds a few thousand cells, so
// what bounds a step is the chain of dependent operations a cell runs through
// (75 cycles for each FP64 sum or product, and 64 of its sub-partition's FP64
// pipe for a warp however few lanes are active) and what separates kernels:
// launches, loads and stores.  A block therefore takes a tile of 16 cells from
// primitives to the updated state, with everything between in shared memory,
// and spreads each cell over lanes: reconstruction 8 lanes per cell, fluxes 4
// per face (flux_quad.cuh), update 7 per cell.  Neighbouring tiles overlap by
// the stencil (14 new cells of 16 at 2nd order, 12 at 4th).  Stages read one
// buffer and write another - the state itself last - so that no block
// overwrites what a neighbour reads; U^n stays in the state until then.
//
// One step, RK3, against separate kernels for primitives, reconstruction, fluxes,
// boundary and update: 2048 cells MLAU + MUSCL 104 -> 60 us, LHLLD 100 -> 51 us,
// MLAU + WCNS4 136 -> 97 us; 16384 cells MLAU + MUSCL 319 -> 164 us.  Products stay
// FP64 instructions here, unlike in the 2D and 3D kernels: with one or two warps
// to a sub-partition the 30 instructions of an integer product cost more than
// the pipe's 64 cycles (2048 cells: 87 us with integer products).
#include "stencil.cuh"
#include "rec_exact.cuh"
#include "flux_quad.cuh"

namespace mlau {
namespace {

constexpr int T1D = 128;           // threads of a block
constexpr int RLANES = 8;          // lanes of a reconstructed cell
constexpr int NR = T1D / RLANES;   // cells a tile reconstructs
constexpr int NP = NR + 4;         // cells it reads

struct Stage1 {
    const double *src[8], *u0[8];  // state read, U^n
    double *dst[8];                // state written
    int nx, off, odr, eig, periodic, open, first, ntiles, no;  // no: new cells per tile
    double ra, rb, bx, dtdx, gamma;
};

__device__ __constant__ const int kSlot1[7] = {0, 1, 2, 3, 6, 7, 4};  // ro, mx, my, mz, by, bz, en

// Primitives (ro, vx, vy, vz, by, bz, pr) of cell s.
__device__ __forceinline__ void prim1(const double *const u[8], int s, double bx, double gamma, ed p[7])
{
    const ed ro = u[0][s], by = u[6][s], bz = u[7][s], en = u[4][s];
    const ed iro = trcp(ro);
    const ed vx = u[1][s] * iro, vy = u[2][s] * iro, vz = u[3][s] * iro;
    const ed v2 = vx * vx + vy * vy + vz * vz;
    const ed b2 = ed(bx) * bx + by * by + bz * bz;
    p[0] = ro;
    p[1] = vx;
    p[2] = vy;
    p[3] = vz;
    p[4] = by;
    p[5] = bz;
    p[6] = ed(gamma - 1) * (en - thalf(ro * v2 + b2));
}

// Left eigenvector n (Ln[k] = L[n][k]) and entry n of every right
// eigenvector (Rc[k] = R[k][n], the back-projection's coefficients of output
// n) from a dense fill, selected with unrolled predicated moves so that the
// 7x7 matrices stay in registers and their constant entries fold away;
// eigenvalue n into *lam.
template <class FILL>
__device__ __forceinline__ void eig_row(FILL fill, int n, ed Ln[7], ed Rc[7], ed *lam)
{
    ed al[7], L[7][7], R[7][7];
    fill(al, L, R);
#pragma unroll
    for (int k = 0; k < 7; k++) {
        Ln[k] = L[0][k];
        Rc[k] = R[k][0];
    }
    *lam = al[0];
#pragma unroll
    for (int j = 1; j < 7; j++) {
#pragma unroll
        for (int k = 0; k < 7; k++) {
            Ln[k] = (n == j) ? L[j][k] : Ln[k];
            Rc[k] = (n == j) ? R[k][j] : Rc[k];
        }
        *lam = (n == j) ? al[j] : *lam;
    }
}

// sum of c[k] v[k], in the header's order
__device__ __forceinline__ ed dot7(const ed c[7], const ed v[7])
{
    return c[0] * v[0] + c[1] * v[1] + c[2] * v[2] + c[3] * v[3] + c[4] * v[4] + c[5] * v[5] + c[6] * v[6];
}

// openbc1d_mhd (1D/SERIAL/shock/openbc1d_mhd.c:21-175): 8 lanes per side of one
// block.  Lane r (0..6) projects both cells on characteristic field r and
// applies its outflow condition; the back-projection of primitive r follows
// the dense 7-term sums of the header, with the fields exchanged by shuffles;
// the ghost cells of the side (all the same state) go to dst.
__device__ void openbc1(const Stage1 &a)
{
    if (threadIdx.x >= 16) return;
    const int r = threadIdx.x & 7, side = threadIdx.x >> 3, n = r < 7 ? r : 6;
    const int sgn = side ? -1 : 1;
    const int si = side ? (a.nx - a.off - 1) : a.off, so = si - sgn;
    ed q[2][7];
    prim1(a.src, si, a.bx, a.gamma, q[0]);
    prim1(a.src, so, a.bx, a.gamma, q[1]);
    ed m[7];
#pragma unroll
    for (int k = 0; k < 7; k++) m[k] = thalf(q[0][k] + q[1][k]);
    ed Ln[7], Rc[7], lam;
    eig_row([&](ed *l, ed (*L)[7], ed (*R)[7]) {
        eigen_st_dense<ed>(m[0], m[1], 0.0, 0.0, ed(0.5) * (ed(a.bx) + a.bx), m[4], m[5], m[6], a.gamma, l,
                           L, R); }, n, Ln, Rc, &lam);
    const ed w0 = dot7(Ln, q[0]), w1 = dot7(Ln, q[1]);
    const ed c = ed(sgn) * lam;
    const ed w = (c > ed(0)) ? w1 : (ed(1) + c * a.dtdx) * w1 - c * a.dtdx * w0;
    ed wv[7], p[7];
#pragma unroll
    for (int k = 0; k < 7; k++) wv[k] = __shfl_sync(0xffffu, w.v, k, 8);
    const ed pn = dot7(Rc, wv);
#pragma unroll
    for (int k = 0; k < 7; k++) p[k] = __shfl_sync(0xffffu, pn.v, k, 8);
    // conserved ghost state, in the reference's order of operations
    const ed v2 = p[1] * p[1] + p[2] * p[2] + p[3] * p[3];
    const ed b2 = ed(a.bx) * a.bx + p[4] * p[4] + p[5] * p[5];
    const ed u[7] = {p[0], p[1] * p[0], p[2] * p[0], p[3] * p[0], p[4], p[5],
                     p[6] / (a.gamma - 1.0) + ed(0.5) * (p[0] * v2 + b2)};
    const int g0 = side ? a.nx - a.off : 0;
    if (r >= 7) return;
    double v = u[0].v;
#pragma unroll
    for (int k = 1; k < 7; k++) v = (r == k) ? u[k].v : v;
    for (int j = 0; j < a.off; j++) a.dst[kSlot1[r]][g0 + j] = v;
}

// One RK stage.  WHICH: Riemann solver; W4: WCNS4, else the code odr.
template <int WHICH, bool W4>
__global__ void __launch_bounds__(T1D) k_stage1(const __grid_constant__ Stage1 a)
{
    __shared__ double P[7][NP], M2[NP], UL[7][NR], UR[7][NR], F[7][NR];
    const int tid = threadIdx.x, nx = a.nx, off = a.off;
    if ((int)blockIdx.x == a.ntiles) {  // first stage of an open boundary
        openbc1(a);
        return;
    }
    const int o0 = off + blockIdx.x * a.no;  // first new cell
    const int c0 = o0 - (NR - a.no) / 2;     // first reconstructed cell
    // the state this thread updates, asked for early
    const int lane = tid & 7, uj = tid >> 3, ui = o0 + uj;
    const bool upd = lane < 7 && uj < a.no && ui < nx - off;
    const int us = kSlot1[lane < 7 ? lane : 6];
    const double su = upd ? a.src[us][ui] : 0.0, s0 = upd ? a.u0[us][ui] : 0.0;
    if (tid < NP) {
        const int s = min(c0 - 2 + tid, nx - 1);
        ed p[7];
        prim1(a.src, s, a.bx, a.gamma, p);
#pragma unroll
        for (int k = 0; k < 7; k++) P[k][tid] = p[k].v;
        const ed c2 = ed(a.gamma) * p[6] / p[0];
        M2[tid] = ((p[1] * p[1] + p[2] * p[2] + p[3] * p[3]) / c2).v;
    }
    __syncthreads();
    // Face states (:133-186): full characteristic system where any of the
    // three central cells has sonic Mach^2 >= 1, Alfven + entropy elsewhere.
    // Lane n of a cell projects the stencil on field n, interpolates it and
    // back-projects output n (lane 7 repeats 6), with the dense 7-term sums of
    // include/mhd_eigen.h (:455-684) in its order.
    {
        const int r = tid / RLANES, n = lane < 7 ? lane : 6;
        ed q[7];
#pragma unroll
        for (int k = 0; k < 7; k++) q[k] = P[k][r + 2];
        ed Ln[7], Rc[7], lam;
        if (vmax(M2[r + 1], vmax(M2[r + 2], M2[r + 3])) >= 1.0) {
            if (a.eig == EIG_MIYOSHI)
                eig_row([&](ed *l, ed (*L)[7], ed (*R)[7]) {
                    eigen_mi_dense<ed>(q[0], q[1], q[2], q[3], a.bx, q[4], q[5], q[6], a.gamma, l, L, R); },
                    n, Ln, Rc, &lam);
            else
                eig_row([&](ed *l, ed (*L)[7], ed (*R)[7]) {
                    eigen_st_dense<ed>(q[0], q[1], q[2], q[3], a.bx, q[4], q[5], q[6], a.gamma, l, L, R); },
                    n, Ln, Rc, &lam);
        } else {
            eig_row([&](ed *l, ed (*L)[7], ed (*R)[7]) {
                eigen_ae_dense<ed>(q[0], q[1], q[2], q[3], a.bx, q[4], q[5], q[6], a.gamma, l, L, R); },
                n, Ln, Rc, &lam);
        }
        // the stencil is three points but for WCNS4
        ed w[5];
#pragma unroll
        for (int m = W4 ? 0 : 1; m < (W4 ? 5 : 4); m++) {
            ed x[7];
#pragma unroll
            for (int k = 0; k < 7; k++) x[k] = P[k][r + m];
            w[m] = dot7(Ln, x);
        }
        ed wl, wr;
        if constexpr (W4) {
            const double2 v = wcns4_ed(w[0].v, w[1].v, w[2].v, w[3].v, w[4].v);
            wl = v.x;
            wr = v.y;
        } else {
            w[0] = w[1];
            w[4] = w[3];
            rec_lr(a.odr, w, wl, wr);
        }
        const int g0 = (tid & 31) & ~(RLANES - 1);
        ed fl[7], fr[7];
#pragma unroll
        for (int k = 0; k < 7; k++) {
            fl[k] = __shfl_sync(0xffffffffu, wl.v, g0 + k);
            fr[k] = __shfl_sync(0xffffffffu, wr.v, g0 + k);
        }
        ed ul = dot7(Rc, fl), ur = dot7(Rc, fr);
        // exact-zero guard (mhd_eigen.h:516-529): output n of a field that is
        // zero across the stencil
        bool zero = n >= 1 && n <= 5;
#pragma unroll
        for (int m = 0; m < 5; m++) zero = zero && tzero(ed(P[n][r + m]));
        if (zero) {
            ul = 0.0;
            ur = 0.0;
        }
        if (lane < 7) {
            UL[n][r] = ul.v;
            UR[n][r] = ur.v;
        }
    }
    __syncthreads();
    // face j between cells j - 1 and j of the tile
    if constexpr (WHICH == FLUX_ROE) {
        if (tid >= 1 && tid < NR) {
            ed L[7], R[7], f[7];
#pragma unroll
            for (int n = 0; n < 7; n++) {
                L[n] = UL[n][tid - 1];
                R[n] = UR[n][tid];
            }
            flux_roe<ed>(L, R, a.bx, a.gamma, f);
#pragma unroll
            for (int n = 0; n < 7; n++) F[n][tid] = f[n].v;
        }
    } else if (tid < 4 * NR) {
        const int j = max(tid >> 2, 1);
        const Quad Q{tid & 1, (tid >> 1) & 1, 0xffffffffu};
        auto IN = [&](int s, int n) { return s ? UR[n][j] : UL[n][j - 1]; };
        const double dv0 = (ed(P[1][j + 2]) - P[1][j + 1]).v;
        double f0, f1, ft, fb, f6;
        if constexpr (WHICH == FLUX_MLAU)
            flux_mlau_quad(IN, Q, a.bx, a.gamma, dv0, 0.0, f0, f1, ft, fb, f6);
        else
            flux_hlld_quad<WHICH == FLUX_LHLLD>(IN, Q, a.bx, a.gamma, dv0, 0.0, f0, f1, ft, fb, f6);
        if (Q.side == 0 && tid >= 4) {
            F[2 + Q.comp][j] = ft;
            F[4 + Q.comp][j] = fb;
            if (Q.comp == 0) {
                F[0][j] = f0;
                F[1][j] = f1;
                F[6][j] = f6;
            }
        }
    }
    __syncthreads();
    // Update (:220-255); with periodic boundaries each cell also writes its
    // ghost images (prdc_1d, 1D/SERIAL/wave/prdc_1d.c).  Flux order (ro, mx,
    // my, mz, by, bz, en).
    if (upd) {
        const int j = ui - c0;
        const double *fx = F[lane];
        const ed dd = fdiff<ed>(a.odr, fx[max(j - 1, 1)], fx[j], fx[j + 1], fx[min(j + 2, NR - 1)]);
        const double out = (ed(a.ra) * s0 + ed(a.rb) * (ed(su) - a.dtdx * dd)).v;
        a.dst[us][ui] = out;
        const int N = nx - 2 * off;
        if (a.periodic) {
            if (ui < 2 * off) a.dst[us][ui + N] = out;
            if (ui >= N) a.dst[us][ui - N] = out;
        }
    }
    // an open boundary's ghost cells keep the first stage's state
    if (a.open && !a.first) {
        const int side = blockIdx.x == 0 ? 0 : 1;
        if (blockIdx.x == 0 || (int)blockIdx.x == a.ntiles - 1)
            for (int t = tid; t < 7 * off; t += T1D) {
                const int v = kSlot1[t / off], g = t % off;
                if (side == 0) a.dst[v][g] = a.src[v][g];
                if ((int)blockIdx.x == a.ntiles - 1) a.dst[v][nx - off + g] = a.src[v][nx - off + g];
            }
    }
}

template <bool W4> const void *stage_kernel1(int flux)
{
    switch (flux) {
    case FLUX_MLAU: return (const void *)k_stage1<FLUX_MLAU, W4>;
    case FLUX_LHLLD: return (const void *)k_stage1<FLUX_LHLLD, W4>;
    case FLUX_HLLD: return (const void *)k_stage1<FLUX_HLLD, W4>;
    default: return (const void *)k_stage1<FLUX_ROE, W4>;
    }
}

}  // namespace

int plain1d_alloc(Sim *s)
{
    PlainFields &f = s->f;
    const long long n = s->g.n;
    int rc = 0;
    // the state and the two buffers the stages go through
    for (int v = 0; v < 8; v++) rc |= dalloc(s, &f.s[v], n);
    for (int v = 0; v < 7; v++) rc |= dalloc(s, &f.ul[v], n) | dalloc(s, &f.ur[v], n);
    return rc ? MLAU_ERR_NOMEM : MLAU_OK;
}

// Enqueue one 1D step on `st`: the state f.s, with f.ul and f.ur (7 arrays of nx
// each) as the buffers between the stages.
int plain1d_enqueue(const PlainFields &f, int nx, int off, int odr, int eig, int flux, int nrk, int bc,
                    double bx, double dt, double dx, double gamma, cudaStream_t st)
{
    static const int slot[7] = {0, 1, 2, 3, 6, 7, 4};
    const void *kern = odr == 4 ? stage_kernel1<true>(flux) : stage_kernel1<false>(flux);
    Stage1 a{};
    a.nx = nx;
    a.off = off;
    a.odr = odr;
    a.eig = eig;
    a.periodic = bc == MLAU_BC1D_PERIODIC;
    a.open = bc == MLAU_BC1D_OPEN;
    a.no = lin_odr(odr) > 2 ? NR - 4 : NR - 2;
    a.ntiles = (int)blocks_for(nx - 2 * off, a.no);
    a.bx = bx;
    a.dtdx = dt / dx;
    a.gamma = gamma;
    for (int k = 0; k < 7; k++) a.src[slot[k]] = a.u0[slot[k]] = f.s[slot[k]];
    for (int rk = 0; rk < nrk; rk++) {
        rk_coef(nrk, rk, a.ra, a.rb);
        a.first = rk == 0;
        const bool back = rk > 0 && rk == nrk - 1;  // a one-stage step copies back
        for (int k = 0; k < 7; k++)
            a.dst[slot[k]] = back ? f.s[slot[k]] : (rk & 1 ? f.ur[k] : f.ul[k]);
        void *args[] = {&a};
        MLAU_CUDA(cudaLaunchKernel(kern, dim3(a.ntiles + (a.open && a.first ? 1 : 0)), dim3(T1D), args, 0,
                                   st));
        for (int k = 0; k < 7; k++) a.src[slot[k]] = a.dst[slot[k]];
    }
    if (nrk == 1)
        for (int k = 0; k < 7; k++)
            MLAU_CUDA(cudaMemcpyAsync(f.s[slot[k]], f.ul[k], sizeof(double) * nx, cudaMemcpyDeviceToDevice,
                                      st));
    return MLAU_OK;
}

int plain1d_step(Sim *s, double dt)
{
    const Geometry &g = s->g;
    TimedLaunch tl(&s->timer, KK_FLUX);
    return plain1d_enqueue(s->f, g.nx, g.ox, s->odr, s->eig, s->flux, s->nrk, s->bc1d, s->bx1d, dt, g.dx,
                           s->gamma, s->stream);
}

}  // namespace mlau
