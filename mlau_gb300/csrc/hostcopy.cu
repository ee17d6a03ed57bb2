// Host arrays to and from the device in one launch.
//
// A call of a driver on host arrays moves up to eight arrays each way, and a
// copy from or to pageable memory costs 2 to 10 us of the driver's time (staging
// and, to the host, waiting) before its bytes count: more than the step itself
// for small grids.  Where the GPU reaches pageable host memory through the
// host's page tables (Grace and Blackwell share them over NVLink-C2C) a kernel
// reads and writes the arrays where they are.  Eight arrays there / back, copies
// against the kernel: 2056 doubles each 23 / 66 against 11 / 10 us, 26624 79 / 74
// against 18 / 19.  Arrays above 256 KB are copied, as are device or managed
// arrays and where the GPU cannot reach host memory: the bytes count there, and
// the kernel gains less or loses (pinned arrays to the host: 213 KB 30 against
// 23 us, 0.7 MB 51 against 56, 2 MB 108 against 145; ordinary ones 3.8 MB 233
// against 266), and where another engine's steps hold the SMs, which copies do
// without, a driver's call waits for them (beside 2.4 ms steps, a 2D call with
// arrays of 0.7 / 2 MB 12 / 11 ms by copies, 22 / 28 by the kernel; 192 KB 15.8
// and 15.7).
//
// Who asks for the kernel: the 1D and 2D drivers' calls on host arrays, the engines'
// uploads and downloads and the handles' downloads, all of which return when the
// arrays have been moved.  Not the handles' uploads, which return while what is
// queued before them runs (51 kB arrays behind 39 ms of steps: 33 us; the kernel
// would have to be waited for), nor 3D drivers' calls and the MRX operators':
// beside another engine's steps each launch may wait for one of them, and two more
// cost ns_viscous_2d on 112 x 112 cells 13 ms against 6.6 by copies, a 24 x 20 x 16
// step 44 against 20 (1D 4.9 against 9.7 by ten copies, a 2D step 25 and 27).
#include "hostcopy.h"

namespace mlau {
namespace {

struct Fields8 {
    const double *src[8];
    double *dst[8];
};

constexpr long long kKernelBytes = 256 << 10;  // the largest array the kernel moves

// Array blockIdx.y, 2 NCOPY NTC doubles of it to a block; by pairs where both sides
// are aligned for it, loads first.  Blocks of one warp with 32 registers a thread:
// the engines' step kernels fill the GPU for milliseconds and leave room for one
// such block in each SM sub-partition (kb_step_split 80 registers x 6 warps of 512 x
// 32, kb_step_plain 240 x 2, kb_step_1d half of them), so that a move starts beside
// them.  With blocks of 256 threads it waited for the end of a step: 16 kB arrays
// beside a batch with 2.4 ms steps 2.4 ms, in blocks of a warp 31 to the device and
// 34 us back; alone no difference.
constexpr int NTC = 32, NCOPY = 4;
__global__ void __maxnreg__(32) k_copy8(const __grid_constant__ Fields8 a, long long n)
{
    const double *s = a.src[blockIdx.y];
    double *d = a.dst[blockIdx.y];
    if ((((unsigned long long)s | (unsigned long long)d) & 15) == 0) {
        const double2 *s2 = reinterpret_cast<const double2 *>(s);
        double2 *d2 = reinterpret_cast<double2 *>(d), v[NCOPY];
        const long long i = (long long)blockIdx.x * NTC * NCOPY + threadIdx.x;
#pragma unroll
        for (int u = 0; u < NCOPY; u++)
            if (i + u * NTC < n / 2) v[u] = s2[i + u * NTC];
#pragma unroll
        for (int u = 0; u < NCOPY; u++)
            if (i + u * NTC < n / 2) d2[i + u * NTC] = v[u];
        if (i == 0 && (n & 1)) d[n - 1] = s[n - 1];
    } else {
        const long long i = (long long)blockIdx.x * NTC * NCOPY * 2 + threadIdx.x;
        for (int u = 0; u < 2 * NCOPY; u++)
            if (i + u * NTC < n) d[i + u * NTC] = s[i + u * NTC];
    }
}

bool reaches_host_memory()
{
    int dev = 0, direct = 0, tables = 0;
    return cudaGetDevice(&dev) == cudaSuccess &&
           cudaDeviceGetAttribute(&direct, cudaDevAttrPageableMemoryAccess, dev) == cudaSuccess &&
           cudaDeviceGetAttribute(&tables, cudaDevAttrPageableMemoryAccessUsesHostPageTables, dev) ==
               cudaSuccess &&
           direct && tables;
}

// Ordinary or pinned host memory, aligned for a double.
bool host_array(const void *p)
{
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return ((unsigned long long)p & 7) == 0 &&
           (at.type == cudaMemoryTypeUnregistered || at.type == cudaMemoryTypeHost);
}

// One access by the CPU to every page of a host array before the GPU's.  An
// array that is too short or not mapped then fails here, as it does in a copy from
// pageable memory: the GPU's first access to a bad page would be a fault that takes
// the context with it.  Before a write the pages are also made present (the GPU
// would wait for each; the bytes stay as they are).  4 KB is the smallest page;
// the largest array here takes 65 accesses.
void touch(const double *p, long long n, bool write)
{
    volatile char *b = (volatile char *)p;
    const long long bytes = n * (long long)sizeof(double);
    for (long long i = 0;; i = i + 4096 < bytes ? i + 4096 : bytes - 1) {
        const char c = b[i];
        if (write) b[i] = c;
        if (i == bytes - 1) return;
    }
}

}  // namespace

int copy_fields(double *const *dev, double *const *host, int nv, long long n, bool to_host, Move how,
                cudaStream_t st)
{
    Fields8 a{};
    int m = 0;
    bool kernel = how == Move::Kernel && n > 0 && (long long)sizeof(double) * n <= kKernelBytes && nv <= 8 && reaches_host_memory();
    for (int v = 0; v < nv && kernel; v++) {
        if (!dev[v] || !host[v]) continue;
        kernel = host_array(host[v]);
        // arrays that overlap are written one after the other
        for (int w = 0; w < v && to_host; w++)
            if (dev[w] && host[w] && host[w] < host[v] + n && host[v] < host[w] + n) kernel = false;
        a.src[m] = to_host ? dev[v] : host[v];
        a.dst[m++] = to_host ? host[v] : dev[v];
    }
    if (kernel) {
        if (m == 0) return MLAU_OK;
        for (int v = 0; v < m; v++) touch(to_host ? a.dst[v] : a.src[v], n, to_host);
        const unsigned nb = blocks_for(n, 2 * NCOPY * NTC);
        // the launch's own status: an error that an earlier call left behind is not this one's
        void *args[] = {&a, &n};
        MLAU_CUDA(cudaLaunchKernel((const void *)k_copy8, dim3(nb, m), dim3(NTC), args, 0, st));
        if (to_host) MLAU_CUDA(cudaStreamSynchronize(st));
        return MLAU_OK;
    }
    for (int v = 0; v < nv; v++) {
        if (!dev[v] || !host[v]) continue;
        MLAU_CUDA(to_host ? cudaMemcpyAsync(host[v], dev[v], sizeof(double) * n, cudaMemcpyDeviceToHost, st)
                          : cudaMemcpyAsync(dev[v], host[v], sizeof(double) * n, cudaMemcpyHostToDevice, st));
    }
    if (to_host) MLAU_CUDA(cudaStreamSynchronize(st));
    return MLAU_OK;
}

}  // namespace mlau
