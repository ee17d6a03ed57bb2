// Host arrays to and from the device in one launch.
//
// A call of a driver on host arrays moves up to eight arrays each way, and a
// copy from or to pageable memory costs 2 to 10 us of the driver's time (staging
// and, to the host, waiting) before its bytes count: more than the step itself
// for small grids.  Where the GPU reaches pageable host memory through the
// host's page tables (Grace and Blackwell share them over NVLink-C2C) a kernel
// reads and writes the arrays where they are.  Eight arrays there / back, copies
// against the kernel: 2056 doubles each 23 / 66 against 11 / 10 us, 26624 79 / 74
// against 18 / 19.  The line lies where the bytes count and the kernel loses: to the
// device 4 MB (0.7 MB an array 73 against 129 us, 2 MB 98 against 174, 3.8 MB 168
// against 252, pinned 164 against 197), to the host 256 KB (pinned arrays 213 KB 23
// against 30 us, 0.7 MB 56 against 51, 2 MB 145 against 108; ordinary ones gain up
// to 2 MB, but new ones, as Sim.download makes them, wait for their pages: 64^3 3.3
// against 0.2 to 1 ms).  Larger arrays are copied, as are device or managed arrays
// and where the GPU cannot reach host memory.
//
// Who asks for the kernel: the drivers' calls on host arrays, the engines' uploads
// and downloads and the handles' downloads, all of which return when the arrays have
// been moved.  Not the handles' uploads, which return while what is queued before
// them runs (51 kB arrays behind 39 ms of steps: 33 us; the kernel would have to be
// waited for), nor the downloads of 3D drivers' calls and the MRX operators': beside
// another engine's steps it queues behind their many launches and those behind the
// steps (moves both ways by the kernel, a 24 x 20 x 16 step 44 ms beside 2.4 ms
// steps, by copies back 19.3, by copies both ways 19.6; alone 545, 610, 680 us).
#include "hostcopy.h"

namespace mlau {
namespace {

struct Fields8 {
    const double *src[8];
    double *dst[8];
};

// the largest array the kernel moves to the device, to the host
constexpr long long kKernelUp = 4 << 20, kKernelDown = 256 << 10;

// Array blockIdx.y, 2 NCOPY NTC doubles of it to a block; by pairs where both sides
// are aligned for it, loads first.  Blocks of one warp with 32 registers a thread:
// the engines' step kernels fill the GPU for milliseconds and leave room for one
// such block in each SM sub-partition (of its 512 registers a lane kb_step_split
// takes 6 x 80, kb_step_plain 2 x 216, kb_step_1d 2 x 128), so that a move starts
// beside them.  With blocks of 256 threads it waited for the end of a step: 16 kB arrays
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
// the largest array here takes 1024 accesses.
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
    bool kernel = how == Move::Kernel && n > 0 && nv <= 8 &&
                  (long long)sizeof(double) * n <= (to_host ? kKernelDown : kKernelUp) && reaches_host_memory();
    for (int v = 0; v < nv && kernel; v++) {
        if (!dev[v] || !host[v]) continue;
        kernel = host_array(host[v]);
        // arrays that overlap are written one after the other
        for (int w = 0; w < v && to_host; w++)
            if (dev[w] && host[w] && host[w] < host[v] + n && host[v] < host[w] + n) kernel = false;
        a.src[m] = to_host ? dev[v] : host[v];
        a.dst[m++] = to_host ? host[v] : dev[v];
    }
    cudaError_t e = cudaSuccess;
    if (kernel && m > 0) {
        for (int v = 0; v < m; v++) touch(to_host ? a.dst[v] : a.src[v], n, to_host);
        const unsigned nb = blocks_for(n, 2 * NCOPY * NTC);
        // the launch's own status: an error that an earlier call left behind is not this one's
        void *args[] = {&a, &n};
        e = cudaLaunchKernel((const void *)k_copy8, dim3(nb, m), dim3(NTC), args, 0, st);
    } else if (!kernel) {
        for (int v = 0; v < nv && e == cudaSuccess; v++) {
            if (!dev[v] || !host[v]) continue;
            e = to_host ? cudaMemcpyAsync(host[v], dev[v], sizeof(double) * n, cudaMemcpyDeviceToHost, st)
                        : cudaMemcpyAsync(dev[v], host[v], sizeof(double) * n, cudaMemcpyHostToDevice, st);
        }
    }
    // waited for on failure too: what is queued may read the caller's arrays (an
    // upload by the kernel) or write them
    if (to_host) {
        const cudaError_t w = cudaStreamSynchronize(st);
        if (e == cudaSuccess) e = w;
    }
    if (e != cudaSuccess) {
        set_error("host arrays %s the device: %s", to_host ? "from" : "to", cudaGetErrorString(e));
        return MLAU_ERR_CUDA;
    }
    return MLAU_OK;
}

}  // namespace mlau
