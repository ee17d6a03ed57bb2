// Batched 1D instances, plain FP64: every instance runs the stage of the
// single-instance 1D kernel (stage1d.cuh), so it advances bit for bit like
// mhd_fd4c_1d (1D/SERIAL/shock/mhd_fd4c_1d.c:60-271, open boundaries via
// openbc1d_mhd.c:21-175, or the periodic boundaries of 1D/SERIAL/wave).  As in
// 1D/SERIAL/shock/main.cpp:113-128 the time step is fixed once, from the
// initial state (cfl*dx/max(1, max|vx|+cf) over all cells); an instance retires
// after the step that reaches its end time (the last step is not clipped).
//
// 1D instances use the engine's host side (batch2d.cu) with a table of tiles
// for NT threads each: NT reconstructed cells, of which all but the stencil's
// overlap are new, and one tile more for an instance's open boundary.  A step is
// three stages with two grid barriers between them; stages read one pool and
// write another (s -> ul -> ur -> s; U^n stays in s until the last), so a tile
// needs nothing of its neighbours within a stage, and the block that finishes
// last does the step's bookkeeping.  What bounds a stage is the latency of one
// cell's chain of operations, most of it the full eigen-system where the flow is
// supersonic.  24 instances of 256 to 4096 cells, mixed solvers, 29k cells in
// all: 238 us a step with MUSCL, 345 with WCNS4; as eleven phases over arrays in
// memory, each with a barrier, 422 and 686.  The eight lanes to a cell of the
// single simulation take 536 us for this load: they repeat too much of the
// FP64 work to fill the chip with.
// State slots: 0 ro, 1 mx, 2 my, 3 mz, 4 en, 6 by, 7 bz.
//
// Each instance has its own flux, boundary, RK stage count (1-3), Bx, gamma,
// CFL number and end time; the reconstruction order is the batch's.
#include "batch2d.cuh"
#include "stage1d.cuh"

namespace mlau {
namespace {

struct BatchStage1 : Stage1 {
    double *const *s_, *const *u_, *const *d_;
    long long base;
    __device__ __forceinline__ const double *src(int v) const { return s_[v] + base; }
    __device__ __forceinline__ const double *u0(int v) const { return u_[v] + base; }
    __device__ __forceinline__ double *dst(int v) const { return d_[v] + base; }
};

// the cells a tile stands for: its new ones, with the ghosts of the instance at
// the ends
struct Cells1 { int lo, hi; };
__device__ __forceinline__ Cells1 cells_of(const BInst &I, int x0, int no)
{
    const int end = I.nx - I.off;
    return {x0 == I.off ? 0 : x0, x0 + no >= end ? I.nx : x0 + no};
}

// one-off dt of the reference 1D driver's main, at an instance's first step
__device__ void q_dt0(const BArgs &A, int nt, const BTile *tiles, int no)
{
    for (int t = blockIdx.x; t < nt; t += gridDim.x) {
        const BTile tl = tiles[t];
        BInst &I = A.inst[tl.inst];
        double vt = 0.0;
        if (!tl.open && I.active && I.steps == 0 && I.dt_fixed <= 0.0) {
            const Cells1 r = cells_of(I, tl.x0, no);
            for (int i = r.lo + threadIdx.x; i < r.hi; i += blockDim.x) {
                const long long s = I.base + i;
                const double *const *S = A.a.s;
                const double bx = I.bx;
                const double iro = 1.0 / S[0][s];
                const double vx = S[1][s] * iro, vy = S[2][s] * iro, vz = S[3][s] * iro;
                const double v2 = vx * vx + vy * vy + vz * vz;
                const double b2 = bx * bx + S[6][s] * S[6][s] + S[7][s] * S[7][s];
                const double pr = (I.gamma - 1) * (S[4][s] - 0.5 * (S[0][s] * v2 + b2));
                const double cf = sqrt((I.gamma * pr + b2) * iro);
                const double v = fabs(vx) + cf;
                vt = (v > vt) ? v : vt;  // NaN cells do not count
            }
        }
        batch_vmax(I, vt);
    }
}

// An instance's time step: fixed, or the first step's one-off dt (floor 1.0 as
// in the reference main).  The same in every block until the step's bookkeeping
// stores it.
__device__ __forceinline__ double q_dt(const BInst &I)
{
    if (I.steps != 0 || I.dt_fixed > 0.0) return I.dt_fixed;
    const double vm = __longlong_as_double((long long)I.vkey);
    const double vmax = (vm > 1.0) ? vm : 1.0;
    return I.cfl * I.dx / vmax;
}

template <int NT, bool W4>
__device__ __forceinline__ void q_stage(const BArgs &A, int nt, const BTile *tiles, int no, int rk,
                                        double *sm)
{
    for (int t = blockIdx.x; t < nt; t += gridDim.x) {
        const BTile tl = tiles[t];
        BInst &I = A.inst[tl.inst];
        if (!I.active) continue;
        if (rk >= I.nrk) {
            // a one-stage step is copied back, while others run their second
            if (rk == 1 && I.nrk == 1 && !tl.open) {
                const Cells1 r = cells_of(I, tl.x0, no);
                for (int i = r.lo + threadIdx.x; i < r.hi; i += NT)
                    for (int n = 0; n < 7; n++) {
                        const int v = slot1(n);
                        A.a.s[v][I.base + i] = A.a.ul[v][I.base + i];
                    }
            }
            continue;
        }
        if (tl.open && rk > 0) continue;
        BatchStage1 a;
        a.nx = I.nx;
        a.off = I.off;
        a.odr = A.odr;
        a.eig = EIG_FULL;
        a.flux = I.flux;
        a.periodic = I.bc == MLAU_BC1D_PERIODIC;
        a.open = I.bc == MLAU_BC1D_OPEN;
        a.first = rk == 0;
        a.no = no;
        // SSP-RK coefficients of stage rk for an nrk-stage scheme
        a.ra = (rk == 0) ? 0.0 : (rk == 1) ? 0.5 + (I.nrk - 2) * 0.25 : 1. / 3.;
        a.rb = (rk == 0) ? 1.0 : (rk == 1) ? 0.5 - (I.nrk - 2) * 0.25 : 2. / 3.;
        a.bx = I.bx;
        a.gamma = I.gamma;
        a.dtdx = ed(q_dt(I)) / I.dx;
        a.base = I.base;
        a.u_ = A.a.s;
        a.s_ = rk == 0 ? A.a.s : rk == 1 ? A.a.ul : A.a.ur;
        a.d_ = rk > 0 && rk == I.nrk - 1 ? A.a.s : rk == 1 ? A.a.ur : A.a.ul;
        if (tl.open) {
            const BatchStage1 b = a;  // out of registers on this path only
            openbc1(b);
            continue;
        }
        stage1_wide<NT, W4>(a, tl.x0, sm, [&](double ro, double pr) {
            if (rk == 0) batch_check(I, ro, pr); });
    }
}

__device__ void q_advance(const BArgs &A)
{
    for (int n = threadIdx.x; n < A.ninst; n += blockDim.x) {
        BInst &I = A.inst[n];
        if (I.active) {
            I.dt = I.dt_fixed = q_dt(I);
            I.t += I.dt;
            I.steps += 1;
            // the last step is not clipped; a bad state retires the instance
            if (I.t >= I.t_end || !(I.dt > 0.0) || I.status) {
                I.active = 0;
                atomicSub(&A.sync->active_left, 1);
            }
        }
        I.vkey = 0;
    }
}

template <int NT, bool W4> __global__ void __launch_bounds__(NT, 512 / NT)
kb_step_1d(const __grid_constant__ BArgs A)
{
    const int nt = A.sync->ntiles, no = wide1_cells(NT, A.odr);
    extern __shared__ double sm1[];
    const BTile *tl = A.sync->tiles;
    // the host sets `fresh` when some instance still needs its one-off dt;
    // every block reads it before the first barrier, block 0 clears it after
    const int fresh = *(volatile int *)&A.sync->fresh;
    if (fresh) {
        q_dt0(A, nt, tl, no);
        if (grid_barrier(A.sync, A.nblocks)) return;
        if (blockIdx.x == 0 && threadIdx.x == 0) A.sync->fresh = 0;
    }
    for (int rk = 0; rk < 3; rk++) {
        if (rk > 0 && grid_barrier(A.sync, A.nblocks)) return;
        q_stage<NT, W4>(A, nt, tl, no, rk, sm1);
    }
    if (grid_last(A.sync, A.nblocks)) q_advance(A);
}

}  // namespace

const void *batch1d_plain_kernel(int threads, int odr)
{
    if (odr == 4)
        return threads == 64    ? (const void *)kb_step_1d<64, true>
               : threads == 128 ? (const void *)kb_step_1d<128, true>
                                : (const void *)kb_step_1d<256, true>;
    return threads == 64    ? (const void *)kb_step_1d<64, false>
           : threads == 128 ? (const void *)kb_step_1d<128, false>
                            : (const void *)kb_step_1d<256, false>;
}

int batch1d_tile_cells(int threads, int odr) { return wide1_cells(threads, odr); }

size_t batch1d_smem(int threads)
{
    return threads == 64 ? wide1_smem<64>() : threads == 128 ? wide1_smem<128>() : wide1_smem<256>();
}

}  // namespace mlau
