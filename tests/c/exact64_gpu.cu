// Integer-path double operations and the ed type on the device: out[k*n + i] of
// operands a[i], b[i]; k = 0..4 rcp, half_over, div, div24, sqrt; 5..7 sum,
// difference, product.  Rows 8.. hold CUDA's own results.
#include "ed.cuh"

__global__ void k_run(const double *a, const double *b, long n, double *o)
{
    using namespace mlau;
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const ed x = a[i], y = b[i];
    const ed r[8] = {trcp(x), thalf_over(x), x / y, tdiv24(x), tsqrt(x), x + y, x - y, x * y};
    const double c[8] = {1.0 / a[i], 0.5 / a[i], a[i] / b[i], a[i] / 24.0, sqrt(a[i]),
                         a[i] + b[i], a[i] - b[i], a[i] * b[i]};
    for (int k = 0; k < 8; k++) {
        o[k * n + i] = r[k].v;
        o[(8 + k) * n + i] = c[k];
    }
}

extern "C" int exact64_run(const double *a, const double *b, long n, double *out)
{
    double *d = nullptr;
    cudaError_t e = cudaMalloc(&d, sizeof(double) * 18 * n);
    if (e == cudaSuccess) e = cudaMemcpy(d, a, sizeof(double) * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + n, b, sizeof(double) * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k_run<<<(unsigned)((n + 127) / 128), 128>>>(d, d + n, n, d + 2 * n);
        e = cudaMemcpy(out, d + 2 * n, sizeof(double) * 16 * n, cudaMemcpyDeviceToHost);
    }
    cudaFree(d);
    return (int)e;
}
