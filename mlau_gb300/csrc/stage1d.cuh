// One RK stage of the plain FP64 1D step on a tile of cells, for the single
// simulation (plain1d.cu) and the batched engine (batch1d_plain.cu).
#pragma once

#include "stencil.cuh"
#include "rec_exact.cuh"
#include "flux_quad.cuh"

namespace mlau {

constexpr int RLANES1 = 8;  // lanes of a reconstructed cell

// New cells of a tile that NT threads work on.
MLAU_HD int tile1_cells(int nt, int odr) { return nt / RLANES1 - (lin_odr(odr) > 2 ? 4 : 2); }

// What a stage is asked for; derived types add src(v), u0(v) and dst(v), the
// arrays (from cell 0) of the state read, U^n and the state written.
struct Stage1 {
    int nx, off, odr, eig, flux, periodic, open, first, no;  // no: new cells of a tile
    double ra, rb, bx, gamma;
    ed dtdx;
};

// slot of flux variable n: ro, mx, my, mz, by, bz, en
__device__ __forceinline__ int slot1(int n) { return n < 4 ? n : n == 6 ? 4 : n + 2; }

// Primitives (ro, vx, vy, vz, by, bz, pr) of cell s.
template <class STAGE> __device__ __forceinline__ void prim1(const STAGE &a, int s, ed p[7])
{
    const ed ro = a.src(0)[s], by = a.src(6)[s], bz = a.src(7)[s], en = a.src(4)[s];
    const ed iro = trcp(ro);
    const ed vx = a.src(1)[s] * iro, vy = a.src(2)[s] * iro, vz = a.src(3)[s] * iro;
    const ed v2 = vx * vx + vy * vy + vz * vz;
    const ed b2 = ed(a.bx) * a.bx + by * by + bz * bz;
    p[0] = ro;
    p[1] = vx;
    p[2] = vy;
    p[3] = vz;
    p[4] = by;
    p[5] = bz;
    p[6] = ed(a.gamma - 1) * (en - thalf(ro * v2 + b2));
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
template <class STAGE> __device__ __noinline__ void openbc1(const STAGE &a)
{
    if (threadIdx.x >= 16) return;
    const int r = threadIdx.x & 7, side = threadIdx.x >> 3, n = r < 7 ? r : 6;
    const int sgn = side ? -1 : 1;
    const int si = side ? (a.nx - a.off - 1) : a.off, so = si - sgn;
    ed q[2][7];
    prim1(a, si, q[0]);
    prim1(a, so, q[1]);
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
    for (int j = 0; j < a.off; j++) a.dst(slot1(r))[g0 + j] = v;
}

// An open boundary's ghost cells keep the first stage's state.
template <int NT, class STAGE> __device__ __forceinline__ void keep_open1(const STAGE &a, int o0)
{
    const int nx = a.nx, off = a.off;
    if (!a.open || a.first) return;
    const bool left = o0 == off, right = o0 + a.no >= nx - off;
    if (!left && !right) return;
    for (int t = threadIdx.x; t < 7 * off; t += NT) {
        const int v = slot1(t / off), g = t % off;
        if (left) a.dst(v)[g] = a.src(v)[g];
        if (right) a.dst(v)[nx - off + g] = a.src(v)[nx - off + g];
    }
}

// One RK stage of the new cells [o0, o0 + a.no) by a block of NT threads, all
// of which call: eight lanes to a reconstructed cell, four to a face.
// W4: WCNS4, else the code a.odr.
template <int NT, int WHICH, bool W4, class STAGE>
__device__ __forceinline__ void stage1_tile(const STAGE &a, int o0)
{
    constexpr int NR = NT / RLANES1;  // cells a tile reconstructs
    constexpr int NP = NR + 4;        // cells it reads
    __shared__ double P[7][NP], M2[NP], UL[7][NR], UR[7][NR], F[7][NR];
    const int tid = threadIdx.x, nx = a.nx, off = a.off;
    const int c0 = o0 - (NR - a.no) / 2;     // first reconstructed cell
    // the state this thread updates, asked for early
    const int lane = tid & 7, uj = tid >> 3, ui = o0 + uj;
    const bool upd = lane < 7 && uj < a.no && ui < nx - off;
    const int us = slot1(lane < 7 ? lane : 6);
    const double su = upd ? a.src(us)[ui] : 0.0, s0 = upd ? a.u0(us)[ui] : 0.0;
    if (tid < NP) {
        const int s = min(c0 - 2 + tid, nx - 1);
        ed p[7];
        prim1(a, s, p);
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
        const int r = tid / RLANES1, n = lane < 7 ? lane : 6;
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
        const int g0 = (tid & 31) & ~(RLANES1 - 1);
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
        a.dst(us)[ui] = out;
        const int N = nx - 2 * off;
        if (a.periodic) {
            if (ui < 2 * off) a.dst(us)[ui + N] = out;
            if (ui >= N) a.dst(us)[ui - N] = out;
        }
    }
    keep_open1<NT>(a, o0);
}

// The same with one thread to a cell or face, for loads that leave no lanes idle:
// what the lanes of a cell repeat above is done once, in the loops of
// rec_exact.cuh and flux_exact.cuh.  Tiles of NT reconstructed cells; sm: the
// block's wide1_smem<NT>() of shared memory; seen(ro, pr) is called for every
// new cell of the state read.
MLAU_HD int wide1_cells(int nt, int odr) { return nt - (lin_odr(odr) > 2 ? 4 : 2); }
template <int NT> constexpr size_t wide1_smem()
{
    return sizeof(double) * ((35 + 14 + 7) * NT + 8 * (NT + 4));
}

template <int NT, bool W4, class STAGE, class SEEN>
__device__ __forceinline__ void stage1_wide(const STAGE &a, int o0, double *sm, SEEN seen)
{
    static_assert(2 * FX_ROWS <= 35 && 2 * HX_ROWS <= 35, "flux rows exceed the scratch");
    double(*W)[NT] = (double(*)[NT])sm, (*UL)[NT] = W + 35, (*UR)[NT] = UL + 7, (*F)[NT] = UR + 7;
    double(*P)[NT + 4] = (double(*)[NT + 4])(F + 7), *M2 = P[7];
    const int t = threadIdx.x, nx = a.nx, off = a.off;
    const int c0 = o0 - (NT - a.no) / 2;  // first reconstructed cell
    for (int k = t; k < NT + 4; k += NT) {
        const int s = min(c0 - 2 + k, nx - 1);
        ed p[7];
        prim1(a, s, p);
#pragma unroll
        for (int n = 0; n < 7; n++) P[n][k] = p[n].v;
        const ed c2 = ed(a.gamma) * p[6] / p[0];
        M2[k] = ((p[1] * p[1] + p[2] * p[2] + p[3] * p[3]) / c2).v;
        if (s >= o0 && s < min(o0 + a.no, nx - off)) seen(p[0].v, p[6].v);
    }
    __syncthreads();
    // the cells beyond the last new one's stencil are of no use
    const bool live = c0 + t < nx - off + (NT - a.no) / 2;
    if (live) {
        auto Q = [&](int n, int m) { return P[n][t + m]; };
        auto PUT = [&](int s, int n, double u) { (s ? UR : UL)[n][t] = u; };
        const bool full = vmax(M2[t + 1], vmax(M2[t + 2], M2[t + 3])) >= 1.0;
        reconst_ed<W4, NT, true>(a.odr, Q, full, a.bx, a.gamma, RecScratch<NT>{W, t}, PUT);
    }
    __syncthreads();
    if (live && t > 0) {  // face between cells t - 1 and t of the tile
        auto IN = [&](int s, int n) { return s ? UR[n][t] : UL[n][t - 1]; };
        const double dv0 = (ed(P[1][t + 2]) - P[1][t + 1]).v, dv[1] = {0.0};
        double f[7];
        if (a.flux == FLUX_MLAU) {
            flux_mlau_ed<1, NT>(IN, W, a.bx, a.gamma, dv0, dv, f);
        } else if (a.flux == FLUX_LHLLD) {
            flux_hlld_ed<true, 1, NT>(IN, W, a.bx, a.gamma, dv0, dv, f);
        } else if (a.flux == FLUX_HLLD) {
            flux_hlld_ed<false, 1, NT>(IN, W, a.bx, a.gamma, dv0, dv, f);
        } else {
            ed L[7], R[7], g[7];
#pragma unroll
            for (int n = 0; n < 7; n++) {
                L[n] = IN(0, n);
                R[n] = IN(1, n);
            }
            flux_roe<ed>(L, R, a.bx, a.gamma, g);
#pragma unroll
            for (int n = 0; n < 7; n++) f[n] = g[n].v;
        }
#pragma unroll
        for (int n = 0; n < 7; n++) F[n][t] = f[n];
    }
    __syncthreads();
    const int ui = c0 + t, N = nx - 2 * off;
    if (ui >= o0 && ui < o0 + a.no && ui < nx - off) {
#pragma unroll
        for (int n = 0; n < 7; n++) {
            const int us = slot1(n);
            const double *fx = F[n];
            const ed dd = fdiff<ed>(a.odr, fx[max(t - 1, 1)], fx[t], fx[t + 1], fx[min(t + 2, NT - 1)]);
            const double out = (ed(a.ra) * a.u0(us)[ui] + ed(a.rb) * (ed(a.src(us)[ui]) - a.dtdx * dd)).v;
            a.dst(us)[ui] = out;
            if (a.periodic) {
                if (ui < 2 * off) a.dst(us)[ui + N] = out;
                if (ui >= N) a.dst(us)[ui - N] = out;
            }
        }
    }
    keep_open1<NT>(a, o0);
}

}  // namespace mlau
