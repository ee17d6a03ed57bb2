// The integer-path products, scalings, comparisons and limiters of csrc/ed.cuh and
// csrc/exact64.cuh, and the EMF difference of csrc/emf_diff.cuh, on the device beside
// the built-in operations.  out[k n + i] of row k, rows ROWS.. the built-in results.
#include "ed.cuh"
#include "emf_diff.cuh"

namespace {
using namespace mlau;
constexpr int ROWS = 24;

// a product of x64 with its operands checked as its users do
__device__ double nz(double a, double b)
{
    uint32_t bad = 0;
    const double r = x64::mul_nz(a, b, bad);
    return bad ? a * b : r;
}
__device__ double square(double a)
{
    uint32_t bad = x64::off_wide(a);
    const double r = x64::sqr(a, bad);
    return bad ? a * a : r;
}

__global__ void k_ops(const double *a, const double *b, const double *c, long n, double *o)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double A = a[i], B = b[i], C = c[i];
    const ed x = A, y = B, z = C;
    const double r[ROWS] = {
        imul(x, y).v, square(A), nz(A, B), imulk<3>(x).v, imulk<5>(x).v, imulk<7>(x).v, imulk<9>(x).v,
        imulk<11>(x).v, imulk<15>(x).v, imulk<27>(x).v, imulk<117>(x).v, iscale<-1>(x).v, iscale<-2>(x).v,
        iscale<-3>(x).v, iscale<-4>(x).v, iscale<1>(x).v, iscale<2>(x).v, ed_ge(x, y) ? 1.0 : 0.0,
        vmax(x, y).v, vmin(x, y).v, minmod(x, y).v, minmod3(x, y, z).v, tzero(x) ? 1.0 : 0.0,
        (x64::off_wide(A) == 0) ? 1.0 : 0.0};
    const unsigned e = (unsigned)(__double2hiint(A) >> 20) & 0x7ffu;
    const double w[ROWS] = {
        A * B, A * A, A * B, 3.0 * A, 5.0 * A, 7.0 * A, 9.0 * A, 11.0 * A, 15.0 * A, 27.0 * A, 117.0 * A,
        0.5 * A, 0.25 * A, 0.125 * A, 0.0625 * A, 2.0 * A, 4.0 * A, A >= B ? 1.0 : 0.0,
        vmax<double>(A, B), vmin<double>(A, B), minmod<double>(A, B), minmod3<double>(A, B, C),
        A == 0.0 ? 1.0 : 0.0, (A == 0.0 || (e >= 512 && e < 1536)) ? 1.0 : 0.0};
    for (int k = 0; k < ROWS; k++) {
        o[k * n + i] = r[k];
        o[(ROWS + k) * n + i] = w[k];
    }
}

__global__ void k_emf(const float4 *e, long n, double *o)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float v[4] = {e[i].x, e[i].y, e[i].z, e[i].w};
    o[i] = emf_diff4(v);
}

template <class F> int on_device(const void *in, size_t in_bytes, void *out, size_t out_bytes, F launch)
{
    char *d = nullptr;
    cudaError_t e = cudaMalloc(&d, in_bytes + out_bytes);
    if (e == cudaSuccess) e = cudaMemcpy(d, in, in_bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        launch(d, d + in_bytes);
        e = cudaMemcpy(out, d + in_bytes, out_bytes, cudaMemcpyDeviceToHost);
    }
    cudaFree(d);
    return (int)e;
}
}  // namespace

// abc: three arrays of n; out: 2 ROWS arrays of n
extern "C" int exact64_ops(const double *abc, long n, double *out)
{
    return on_device(abc, sizeof(double) * 3 * n, out, sizeof(double) * 2 * ROWS * n, [&](char *i, char *o) {
        const double *a = (const double *)i;
        k_ops<<<(unsigned)((n + 127) / 128), 128>>>(a, a + n, a + 2 * n, n, (double *)o);
    });
}
// e: n quadruples
extern "C" int emf_diff_gpu(const float *e, long n, double *out)
{
    return on_device(e, sizeof(float) * 4 * n, out, sizeof(double) * n, [&](char *i, char *o) {
        k_emf<<<(unsigned)((n + 127) / 128), 128>>>((const float4 *)i, n, (double *)o);
    });
}
