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
// boundary and update: 2048 cells MLAU + MUSCL 104 -> 47 us, LHLLD 100 -> 41 us,
// MLAU + WCNS4 136 -> 71 us; 16384 cells MLAU + MUSCL 319 -> 162 us.  Products stay
// FP64 instructions here, unlike in the 2D and 3D kernels: with one or two warps
// to a sub-partition the 30 instructions of an integer product cost more than
// the pipe's 64 cycles (2048 cells: 87 against 60 us, before the fallbacks were
// made local).
#include "stage1d.cuh"

namespace mlau {
namespace {

constexpr int T1D = 128;

struct SimStage1 : Stage1 {
    const double *s_[8], *u_[8];
    double *d_[8];
    __device__ __forceinline__ const double *src(int v) const { return s_[v]; }
    __device__ __forceinline__ const double *u0(int v) const { return u_[v]; }
    __device__ __forceinline__ double *dst(int v) const { return d_[v]; }
};

// One RK stage; the first stage of an open boundary has one block more.
template <int WHICH, bool W4>
__global__ void __launch_bounds__(T1D) k_stage1(const __grid_constant__ SimStage1 a, int ntiles)
{
    if ((int)blockIdx.x == ntiles) {
        openbc1(a);
        return;
    }
    stage1_tile<T1D, WHICH, W4>(a, a.off + blockIdx.x * a.no);
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
// each) as the buffers between the stages; timer: records each launch, or null.
int plain1d_enqueue(const PlainFields &f, int nx, int off, int odr, int eig, int flux, int nrk, int bc,
                    double bx, double dt, double dx, double gamma, cudaStream_t st, KernelTimer *timer)
{
    static const int slot[7] = {0, 1, 2, 3, 6, 7, 4};
    const void *kern = odr == 4 ? stage_kernel1<true>(flux) : stage_kernel1<false>(flux);
    SimStage1 a{};
    a.nx = nx;
    a.off = off;
    a.odr = odr;
    a.eig = eig;
    a.flux = flux;
    a.periodic = bc == MLAU_BC1D_PERIODIC;
    a.open = bc == MLAU_BC1D_OPEN;
    a.no = tile1_cells(T1D, odr);
    int ntiles = (int)blocks_for(nx - 2 * off, a.no);
    a.bx = bx;
    a.dtdx = dt / dx;
    a.gamma = gamma;
    for (int k = 0; k < 7; k++) a.s_[slot[k]] = a.u_[slot[k]] = f.s[slot[k]];
    for (int rk = 0; rk < nrk; rk++) {
        rk_coef(nrk, rk, a.ra, a.rb);
        a.first = rk == 0;
        const bool back = rk > 0 && rk == nrk - 1;  // a one-stage step copies back
        for (int k = 0; k < 7; k++)
            a.d_[slot[k]] = back ? f.s[slot[k]] : (rk & 1 ? f.ur[k] : f.ul[k]);
        void *args[] = {&a, &ntiles};
        {
            TimedLaunch tl(timer, KK_STAGE);
            MLAU_CUDA(cudaLaunchKernel(kern, dim3(ntiles + (a.open && a.first ? 1 : 0)), dim3(T1D), args,
                                       0, st));
        }
        for (int k = 0; k < 7; k++) a.s_[slot[k]] = a.d_[slot[k]];
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
    return plain1d_enqueue(s->f, g.nx, g.ox, s->odr, s->eig, s->flux, s->nrk, s->bc1d, s->bx1d, dt, g.dx,
                           s->gamma, s->stream, &s->timer);
}

}  // namespace mlau
