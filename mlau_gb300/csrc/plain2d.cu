// Plain FP64 2D step: one SSP-RK step of ideal MHD with constrained transport,
// the GPU form of 2D/SERIAL/OTvortex/mhd_fd_ct_2d.c:91-660, with the problem's
// boundary tables (periodic, or Dirichlet / Neumann mirrors per array and
// axis as bc2d, 2D/SERIAL/OTvortex/boundary.c:18-74).
// Bz is cell-centred and advanced with the fluxes; Bx, By live on faces and
// are advanced by the curl of the corner EMF Ez.  Compiled with --fmad=false
// so the arithmetic is the reference's, bit for bit.
#include <algorithm>

#include "stencil.cuh"
#include "rec_exact.cuh"
#include "flux_exact.cuh"

namespace mlau {
namespace {

// Cell-centred B: computed at the cell itself or, in the ghost frame, at its
// boundary source times the table's sign (calc_bc then bc2d with dnxs[5..6],
// :186-200).
__global__ void __launch_bounds__(TPB)
k_prim2(PlainFields f, Dims d, Box b, int odr, double gamma, Bc2 bc, int save_u0)
{
    int i, j, k;
    if (!b.decode((long long)blockIdx.x * blockDim.x + threadIdx.x, i, j, k)) return;
    const long long sy = d.nx;
    double gx = 1.0, gy = 1.0;
    const int ix = bc_src(i, d.nx, d.ox, 0, bc.x[5], &gx), jx = bc_src(j, d.ny, d.oy, 0, bc.y[5], &gx);
    const int iy = bc_src(i, d.nx, d.ox, 0, bc.x[6], &gy), jy = bc_src(j, d.ny, d.oy, 0, bc.y[6], &gy);
    const long long wx = d.at(ix, jx, 0), wy = d.at(iy, jy, 0);
    const double *bx = f.s[5], *by = f.s[6];
    const ed cx = ed(gx) * face2cen<ed>(odr, bx[wx - 1], bx[wx], bx[wx + 1], bx[wx + 2]);
    const ed cy = ed(gy) * face2cen<ed>(odr, by[wy - sy], by[wy], by[wy + sy], by[wy + 2 * sy]);
    const long long s = d.at(i, j, 0);
    if (save_u0)  // the first stage keeps U^n
#pragma unroll
        for (int v = 0; v < 8; v++) f.u0[v][s] = f.s[v][s];
    const ed ro = f.s[0][s];
    const ed iro = trcp(ro);
    const ed vx = f.s[1][s] * iro, vy = f.s[2][s] * iro, vz = f.s[3][s] * iro;
    const ed bz = f.s[7][s];
    const ed v2 = (vx * vx + vy * vy + vz * vz);
    const ed b2 = (cx * cx + cy * cy + bz * bz);
    const ed pr = ed(gamma - 1) * (f.s[4][s] - ed(0.5) * (ro * v2 + b2));
    f.vx[s] = vx.v;
    f.vy[s] = vy.v;
    f.vz[s] = vz.v;
    f.pr[s] = pr.v;
    f.m2[s] = (v2 / (gamma * pr * iro)).v;
    f.cx[s] = cx.v;
    f.cy[s] = cy.v;
}

// Shock sensors, with the sign rules of their ghost fill (:262-271): dvx
// takes -dnxs[1] along x and +dnys[1] along y, dvy +dnxs[2] and -dnys[2].
__global__ void __launch_bounds__(TPB) k_aux2(PlainFields f, Dims d, Box b, Bc2 bc)
{
    int i, j, k;
    if (!b.decode((long long)blockIdx.x * blockDim.x + threadIdx.x, i, j, k)) return;
    const long long sy = d.nx;
    const long long s = d.at(i, j, 0);
    f.ct[0][s] = (i >= 1 && j >= 1) ? ct_weight(f.vx, f.vy, f.s[0], f.s[5], f.s[6], s, sy, 1, sy, 1)
                                    : 0.5;
    double g0 = 1.0, g1 = 1.0;
    const int i0 = bc_src(i, d.nx, d.ox, 0, -bc.x[1], &g0), j0 = bc_src(j, d.ny, d.oy, 0, bc.y[1], &g0);
    const int i1 = bc_src(i, d.nx, d.ox, 0, bc.x[2], &g1), j1 = bc_src(j, d.ny, d.oy, 0, -bc.y[2], &g1);
    const long long w0 = d.at(i0, j0, 0), w1 = d.at(i1, j1, 0);
    f.dv[0][s] = g0 * vmin((f.vx[w0 + 1] - f.vx[w0]), (f.vx[w0] - f.vx[w0 - 1]));
    f.dv[1][s] = g1 * vmin((f.vy[w1 + sy] - f.vy[w1]), (f.vy[w1] - f.vy[w1 - sy]));
}

// Sweep along x (D=0): (vn, vt, vu) = (vx, vy, vz), (bt, bu) = (cy, bz), the
// By flux is split.  Along y (D=1): (vy, vz, vx), (bz, cx), the Bx flux is split.
// Both sweeps run in one launch, side by side (blockIdx.y), so that grids of a
// few thousand cells have twice the warps to hide each other's latency (200 x 120
// cells, a step: LHLLD + MUSCL 425 -> 268 us, MLAU + WCNS4 627 -> 413; with the
// flux and weight fallbacks made local 217 and 348).  A face's
// left state lies where its flux goes.
struct Sweep2 {
    const double *vn, *vt, *vu, *cn, *ct, *cu, *bface, *dvt;
    double *ul[7], *ur[7], *ql, *qr;  // face states, central parts of the split flux
    Box rec, flux;                    // cells reconstructed, faces
    long long st;
    int split_u;  // 0: split the bt flux; 1: split the bu flux
};
struct Sweeps2 {
    Sweep2 s[2];
};

Sweeps2 make_sweeps2(const PlainFields &f, const Geometry &g)
{
    Sweeps2 S{};
    Sweep2 &x = S.s[0], &y = S.s[1];
    x = {f.vx, f.vy, f.vz, f.cx, f.cy, f.s[7], f.s[5], f.dv[1]};
    y = {f.vy, f.vz, f.vx, f.cy, f.s[7], f.cx, f.s[6], f.dv[0]};
    y.split_u = 1;
    for (int D = 0; D < 2; D++) {
        for (int n = 0; n < 7; n++) S.s[D].ul[n] = f.F[D][n];
        for (int n = 0; n < 7; n++) S.s[D].ur[n] = D ? f.ur[n] : f.ul[n];
        S.s[D].ql = f.FC[D][0];
        S.s[D].qr = D ? f.qr[0] : f.ql[0];
    }
    x.st = 1;
    y.st = g.nx;
    x.rec = {2, 0, 0, g.nx - 4, g.ny, 1};
    x.flux = {3, 0, 0, g.nx - 5, g.ny, 1};
    y.rec = {0, 2, 0, g.nx, g.ny - 4, 1};
    y.flux = {0, 3, 0, g.nx, g.ny - 5, 1};
    return S;
}

// The linear interpolation of the central part of the split tangential B flux.
__device__ __forceinline__ void rec_central2(const Sweep2 &v, long long c, int odr)
{
    const double *bt = v.split_u ? v.cu : v.ct, *vt = v.split_u ? v.vu : v.vt;
    const long long st = v.st;
    ed a5[5], t5[5];
#pragma unroll
    for (int m = 0; m < 5; m++) {
        const long long s = c + st * (m - 2);
        a5[m] = imul(bt[s], v.vn[s]);
        t5[m] = vt[s];
    }
    v.ql[c + st] = (lin_l(odr, a5[0], a5[1], a5[2], a5[3], a5[4])
                    - ed(v.bface[c + st]) * lin_l(odr, t5[0], t5[1], t5[2], t5[3], t5[4])).v;
    v.qr[c] = (lin_r(odr, a5[0], a5[1], a5[2], a5[3], a5[4])
               - ed(v.bface[c]) * lin_r(odr, t5[0], t5[1], t5[2], t5[3], t5[4])).v;
}

__global__ void __launch_bounds__(TPB)
k_rec2(PlainFields f, const __grid_constant__ Sweeps2 S, Dims d, int odr, int eig, double gamma)
{
    const Sweep2 &v = S.s[blockIdx.y];
    const long long st = v.st;
    int i, j, k;
    if (!v.rec.decode((long long)blockIdx.x * blockDim.x + threadIdx.x, i, j, k)) return;
    const long long c = d.at(i, j, 0);
    ed q[7][5];
#pragma unroll
    for (int m = 0; m < 5; m++) {
        const long long s = c + st * (m - 2);
        q[0][m] = f.s[0][s];
        q[1][m] = v.vn[s];
        q[2][m] = v.vt[s];
        q[3][m] = v.vu[s];
        q[4][m] = v.ct[s];
        q[5][m] = v.cu[s];
        q[6][m] = f.pr[s];
    }
    ed ul[7], ur[7];
    reconst_face<ed>(odr, eig, vmax(f.m2[c - st], vmax(f.m2[c], f.m2[c + st])), q, v.cn[c], gamma,
                     ul, ur);
#pragma unroll
    for (int n = 0; n < 7; n++) {
        v.ul[n][c + st] = ul[n].v;
        v.ur[n][c] = ur[n].v;
    }
    rec_central2(v, c, odr);
}

// The drivers' eigen-systems (rec_exact.cuh); W4: WCNS4, else the code odr;
// blocks of NT threads.
template <bool W4, int NT>
__global__ void __launch_bounds__(NT, 640 / NT)
k_rec2_ed(PlainFields f, const __grid_constant__ Sweeps2 S, Dims d, int odr, double gamma)
{
    extern __shared__ double rec_rows[];
    double (*w)[NT] = (double (*)[NT])rec_rows;
    const Sweep2 &v = S.s[blockIdx.y];
    const long long st = v.st;
    int i, j, k;
    if (!v.rec.decode((long long)blockIdx.x * blockDim.x + threadIdx.x, i, j, k)) return;
    const long long c = d.at(i, j, 0);
    const double *src[7] = {f.s[0], v.vn, v.vt, v.vu, v.ct, v.cu, f.pr};
    auto Q = [&](int n, int m) { return src[n][c + st * (m - 2)]; };
    const bool full = vmax(f.m2[c - st], vmax(f.m2[c], f.m2[c + st])) >= 1.0;
    auto PUT = [&](int s, int n, double u) { (s ? v.ur : v.ul)[n][s ? c : c + st] = u; };
    reconst_ed<W4, NT>(odr, Q, full, v.cn[c], gamma, RecScratch<NT>{w, (int)threadIdx.x}, PUT);
    rec_central2(v, c, W4 ? 4 : odr);
}

__global__ void __launch_bounds__(TPB)
k_flux2(PlainFields f, const __grid_constant__ Sweeps2 S, Dims d, int which, double gamma)
{
    const int D = blockIdx.y;
    const Sweep2 &v = S.s[D];
    const long long st = v.st;
    int i, j, k;
    if (!v.flux.decode((long long)blockIdx.x * blockDim.x + threadIdx.x, i, j, k)) return;
    const long long c = d.at(i, j, 0);
    ed L[7], R[7], F[7];
#pragma unroll
    for (int n = 0; n < 7; n++) {
        L[n] = v.ul[n][c];
        R[n] = v.ur[n][c];
    }
    const ed bn = ed(0.5) * (ed(v.bface[c]) + v.bface[c]);
    riemann<ed>(which, L, R, bn, gamma, (ed(v.vn[c]) - v.vn[c - st]),
                vmin(v.dvt[c - st], v.dvt[c]), F);
    const ed fc = ed(0.5) * (ed(v.ql[c]) + v.qr[c]);
    F[4 + v.split_u] -= fc;
#pragma unroll
    for (int n = 0; n < 7; n++) f.F[D][n][c] = F[n].v;
    f.FC[D][0][c] = fc.v;
}

// MLAU, LHLLD and HLLD faces on both pipes (flux_exact.cuh).
template <int WHICH, int NT>
__global__ void __launch_bounds__(NT, 512 / NT)
k_flux2_ed(PlainFields f, const __grid_constant__ Sweeps2 S, Dims d, double gamma)
{
    extern __shared__ double fx_rows[];
    const int D = blockIdx.y;
    const Sweep2 &v = S.s[D];
    const long long st = v.st;
    int i, j, k;
    if (!v.flux.decode((long long)blockIdx.x * blockDim.x + threadIdx.x, i, j, k)) return;
    const long long c = d.at(i, j, 0);
    auto IN = [&](int s, int n) { return (s ? v.ur : v.ul)[n][c]; };
    const double dv[2] = {v.dvt[c - st], v.dvt[c]};
    const double bn = (ed(0.5) * (ed(v.bface[c]) + v.bface[c])).v;
    double F[7];
    riemann_ed<WHICH, 2, NT>(IN, (double (*)[NT])fx_rows, bn, gamma, (ed(v.vn[c]) - v.vn[c - st]).v, dv, F);
    const ed fc = ihalf(ed(v.ql[c]) + v.qr[c]);
    if (v.split_u) F[5] = (F[5] - fc).v;
    else F[4] = (F[4] - fc).v;
#pragma unroll
    for (int n = 0; n < 7; n++) f.F[D][n][c] = F[n];
    f.FC[D][0][c] = fc.v;
}

// Reconstruction and fluxes of both sweeps.  Blocks are large for the sake of the
// instruction caches, which a block's warps share, and small where the grid is
// less than what the GPU holds at a time, so that it spreads evenly (200 x 120
// cells, a step of LHLLD + MUSCL: 268 us with blocks of 32, 273 of 64, 289 of 128
// and 256; 300 x 300: no difference beyond 2 %).
constexpr long long kSmall2 = 97280;  // threads: 5 reconstruction blocks of 128 on each of 152 SMs

template <int NR> void launch_rec2(Sim *s, const Sweeps2 &S, const Dims &d)
{
    const long long n = std::max(S.s[0].rec.count(), S.s[1].rec.count());
    if (s->eig != EIG_FULL)
        k_rec2<<<dim3(blocks_for(n, TPB), 2), TPB, 0, s->stream>>>(s->f, S, d, s->odr, s->eig, s->gamma);
    else if (s->odr == 4)
        k_rec2_ed<true, NR><<<dim3(blocks_for(n, NR), 2), NR, rec_smem<NR>(), s->stream>>>(s->f, S, d, 4, s->gamma);
    else
        k_rec2_ed<false, NR><<<dim3(blocks_for(n, NR), 2), NR, rec_smem<NR>(), s->stream>>>(s->f, S, d, s->odr,
                                                                                         s->gamma);
}

template <int NF> void launch_flux2(Sim *s, const Sweeps2 &S, const Dims &d)
{
    const long long n = std::max(S.s[0].flux.count(), S.s[1].flux.count());
    const dim3 g(blocks_for(n, NF), 2);
    if (s->flux == FLUX_MLAU)
        k_flux2_ed<FLUX_MLAU, NF><<<g, NF, fx_smem<FLUX_MLAU, NF>(), s->stream>>>(s->f, S, d, s->gamma);
    else if (s->flux == FLUX_LHLLD)
        k_flux2_ed<FLUX_LHLLD, NF><<<g, NF, fx_smem<FLUX_LHLLD, NF>(), s->stream>>>(s->f, S, d, s->gamma);
    else if (s->flux == FLUX_HLLD)
        k_flux2_ed<FLUX_HLLD, NF><<<g, NF, fx_smem<FLUX_HLLD, NF>(), s->stream>>>(s->f, S, d, s->gamma);
    else
        k_flux2<<<dim3(blocks_for(n, TPB), 2), TPB, 0, s->stream>>>(s->f, S, d, s->flux, s->gamma);
}

__global__ void __launch_bounds__(TPB) k_emf2(PlainFields f, Dims d, Box b, int odr)
{
    int i, j, k;
    if (!b.decode((long long)blockIdx.x * blockDim.x + threadIdx.x, i, j, k)) return;
    const long long c = d.at(i, j, 0);
    ed ez = 0.0;
    if (i >= 3 && i < d.nx - 2 && j >= 3 && j < d.ny - 2) {
        const ed w = f.ct[0][c];
        ez = (ed(0.0) + emf_part(f.F[0][4], f.FC[0][0], (ed(1.0) - w), -1.0, c, d.nx, odr))
             + emf_part(f.F[1][5], f.FC[1][0], w, +1.0, c, 1, odr);
    }
    f.e[2][c] = ez.v;
}

// RK combine + CT curl of the interior.  With periodic tables each cell also
// writes its periodic images; otherwise k_face2 and k_bc2 follow.
__global__ void __launch_bounds__(TPB)
k_update2(PlainFields f, Dims d, Box b, int odr, double ra_, double rb_, double dtdx_,
          double dtdy_, int images)
{
    const ed ra = ra_, rb = rb_, dtdx = dtdx_, dtdy = dtdy_;
    int i, j, k;
    if (!b.decode((long long)blockIdx.x * blockDim.x + threadIdx.x, i, j, k)) return;
    const long long sy = d.nx;
    const long long s = d.at(i, j, 0);
    // (ro, mx, my, mz, bz, en): state slot and flux component per direction
    const int sv[6] = {0, 1, 2, 3, 7, 4};
    const int cX[6] = {0, 1, 2, 3, 5, 6}, cY[6] = {0, 3, 1, 2, 4, 6};
    double out[8];
#pragma unroll
    for (int v = 0; v < 6; v++) {
        const double *fx = f.F[0][cX[v]], *fy = f.F[1][cY[v]];
        const ed d0 = fdiff<ed>(odr, fx[s - 1], fx[s], fx[s + 1], fx[s + 2]);
        const ed d1 = fdiff<ed>(odr, fy[s - sy], fy[s], fy[s + sy], fy[s + 2 * sy]);
        out[sv[v]] = (ra * f.u0[sv[v]][s] + rb * (ed(f.s[sv[v]][s]) - dtdx * d0 - dtdy * d1)).v;
    }
    const double *ez = f.e[2];
    {
        const ed dd = fdiff<ed>(odr, ez[s - sy], ez[s], ez[s + sy], ez[s + 2 * sy]);
        out[5] = (ra * f.u0[5][s] + rb * (ed(f.s[5][s]) - dtdy * dd)).v;
    }
    {
        const ed dd = fdiff<ed>(odr, ez[s - 1], ez[s], ez[s + 1], ez[s + 2]);
        out[6] = (ra * f.u0[6][s] + rb * (ed(f.s[6][s]) + dtdx * dd)).v;
    }
    if (!images) {
#pragma unroll
        for (int v = 0; v < 8; v++) f.s[v][s] = out[v];
        return;
    }
    const int Nx = d.nx - 2 * d.ox, Ny = d.ny - 2 * d.oy;
    int is[3] = {i, i < 2 * d.ox ? i + Nx : -1, i >= Nx ? i - Nx : -1};
    int js[3] = {j, j < 2 * d.oy ? j + Ny : -1, j >= Ny ? j - Ny : -1};
    for (int bb = 0; bb < 3; bb++) {
        if (js[bb] < 0) continue;
        for (int a = 0; a < 3; a++) {
            if (is[a] < 0) continue;
            const long long t = d.at(is[a], js[bb], 0);
#pragma unroll
            for (int v = 0; v < 8; v++) f.s[v][t] = out[v];
        }
    }
}

// The right boundary faces the CT loops also update (:593-632 run one face
// further, i < nx-xoff+1 for Bx and j < ny-yoff+1 for By); they survive the
// boundary fill only where that axis mirrors the face array.
__global__ void __launch_bounds__(TPB)
k_face2(PlainFields f, Dims d, int odr, double ra_, double rb_, double dtdx_, double dtdy_,
        int do_x, int do_y)
{
    const ed ra = ra_, rb = rb_, dtdx = dtdx_, dtdy = dtdy_;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const long long sy = d.nx;
    const double *ez = f.e[2];
    const int ny_in = d.ny - 2 * d.oy, nx_in = d.nx - 2 * d.ox;
    if (do_x && t < ny_in) {  // Bx at i = nx - xoff
        const long long s = d.at(d.nx - d.ox, d.oy + t, 0);
        const ed dd = fdiff<ed>(odr, ez[s - sy], ez[s], ez[s + sy], ez[s + 2 * sy]);
        f.s[5][s] = (ra * f.u0[5][s] + rb * (ed(f.s[5][s]) - dtdy * dd)).v;
    }
    if (do_y && t < nx_in) {  // By at j = ny - yoff
        const long long s = d.at(d.ox + t, d.ny - d.oy, 0);
        const ed dd = fdiff<ed>(odr, ez[s - 1], ez[s], ez[s + 1], ez[s + 2]);
        f.s[6][s] = (ra * f.u0[6][s] + rb * (ed(f.s[6][s]) + dtdx * dd)).v;
    }
}

// Ghost fill of the conserved arrays with the tables (:636-638): each ghost
// takes its boundary source (periodic image or mirror, composed over the two
// axes) times the signs.  Sources are interior cells or computed faces.
__global__ void __launch_bounds__(TPB) k_bc2(PlainFields f, Dims d, Box b, Bc2 bc)
{
    int i, j, k;
    if (!b.decode((long long)blockIdx.x * blockDim.x + threadIdx.x, i, j, k)) return;
    if (i >= d.ox && i < d.nx - d.ox && j >= d.oy && j < d.ny - d.oy) return;
    const long long s = d.at(i, j, 0);
#pragma unroll
    for (int v = 0; v < 8; v++) {
        double g = 1.0;
        const int si = bc_src(i, d.nx, d.ox, v == 5, bc.x[v], &g);
        const int sj = bc_src(j, d.ny, d.oy, v == 6, bc.y[v], &g);
        if (si == i && sj == j) continue;
        f.s[v][s] = g * f.s[v][d.at(si, sj, 0)];
    }
}

}  // namespace

int plain2d_alloc(Sim *s)
{
    PlainFields &f = s->f;
    const long long n = s->g.n;
    int rc = 0;
    for (int v = 0; v < 8; v++) rc |= dalloc(s, &f.s[v], n) | dalloc(s, &f.u0[v], n);
    double **singles[] = {&f.vx, &f.vy, &f.vz, &f.pr, &f.m2, &f.cx, &f.cy, &f.dv[0], &f.dv[1],
                          &f.ct[0], &f.ql[0], &f.qr[0], &f.e[2]};
    for (auto p : singles) rc |= dalloc(s, p, n);
    for (int v = 0; v < 7; v++) rc |= dalloc(s, &f.ul[v], n) | dalloc(s, &f.ur[v], n);
    for (int D = 0; D < 2; D++) {
        for (int v = 0; v < 7; v++) rc |= dalloc(s, &f.F[D][v], n);
        rc |= dalloc(s, &f.FC[D][0], n);
    }
    if (rc) return MLAU_ERR_NOMEM;
    MLAU_CUDA(cudaFuncSetAttribute(k_flux2_ed<FLUX_MLAU, 256>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fx_smem<FLUX_MLAU, 256>()));
    return MLAU_OK;
}

int plain2d_step(Sim *s, double dt)
{
    const Geometry &g = s->g;
    PlainFields &f = s->f;
    cudaStream_t st = s->stream;
    const Dims d{g.nx, g.ny, 1, g.ox, g.oy, 0};
    const Box all{0, 0, 0, g.nx, g.ny, 1};
    const Box inner{g.ox, g.oy, 0, g.nx - 2 * g.ox, g.ny - 2 * g.oy, 1};
    const double dtdx = dt / g.dx, dtdy = dt / g.dy;
    const Sweeps2 S = make_sweeps2(f, g);
    for (int rk = 0; rk < s->nrk; rk++) {
        double ra, rb;
        rk_coef(s->nrk, rk, ra, rb);
        {
            TimedLaunch tl(&s->timer, KK_PRIM);
            k_prim2<<<blocks_for(all.count(), TPB), TPB, 0, st>>>(f, d, all, s->odr, s->gamma,
                                                                  s->bc2, rk == 0);
        }
        {
            TimedLaunch tl(&s->timer, KK_AUX);
            k_aux2<<<blocks_for(all.count(), TPB), TPB, 0, st>>>(f, d, all, s->bc2);
        }
        {
            TimedLaunch tl(&s->timer, KK_REC);
            if (2 * g.n <= kSmall2) launch_rec2<32>(s, S, d);
            else launch_rec2<128>(s, S, d);
        }
        {
            TimedLaunch tl(&s->timer, KK_FLUX);
            if (2 * g.n <= kSmall2) launch_flux2<32>(s, S, d);
            else launch_flux2<256>(s, S, d);
        }
        {
            TimedLaunch tl(&s->timer, KK_EMF);
            k_emf2<<<blocks_for(all.count(), TPB), TPB, 0, st>>>(f, d, all, s->odr);
        }
        {
            TimedLaunch tl(&s->timer, KK_UPDATE);
            k_update2<<<blocks_for(inner.count(), TPB), TPB, 0, st>>>(f, d, inner, s->odr, ra, rb,
                                                                      dtdx, dtdy, !s->walls2d);
            if (s->walls2d) {
                const int n = std::max(g.nx, g.ny);
                k_face2<<<blocks_for(n, TPB), TPB, 0, st>>>(f, d, s->odr, ra, rb, dtdx, dtdy,
                                                            s->bc2.x[5] != 0, s->bc2.y[6] != 0);
                k_bc2<<<blocks_for(all.count(), TPB), TPB, 0, st>>>(f, d, all, s->bc2);
            }
        }
        MLAU_CUDA(cudaGetLastError());
    }
    return MLAU_OK;
}

}  // namespace mlau
