// csrc/hostcopy.cu on a fake CUDA runtime whose "device" is host memory: the
// kernel's launch copies, and notes in `launched` that it ran; `pending` is the
// error an earlier call of the caller's left behind.
#include <cstdarg>
#include <csignal>
#include <cstring>
#include <sys/mman.h>
#include <sys/wait.h>
#include <unistd.h>

#include "hostcopy_fake.h"
#include "hostcopy.cu"

static int *launched;  // shared with the children
static int copies, syncs;
static cudaError_t copy_fails = cudaSuccess;
static cudaError_t pending = cudaSuccess;

namespace mlau {
void set_error(const char *, ...) {}
}
extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 1; return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *)
{
    memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { const cudaError_t e = pending; pending = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return ""; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { syncs++; return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    copies++;
    if (copy_fails != cudaSuccess) return copy_fails;
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *, dim3 grid, dim3, void **args, size_t, cudaStream_t)
{
    ++*launched;
    const mlau::Fields8 &f = *(const mlau::Fields8 *)args[0];
    const long long n = *(const long long *)args[1];
    for (unsigned v = 0; v < grid.y; v++) memcpy(f.dst[v], f.src[v], sizeof(double) * n);
    return cudaSuccess;
}
}

static double g_dev[8 << 17];

static int move(double *host, long long n, bool to_host)
{
    double *dev[8] = {}, *h[8] = {};
    dev[3] = g_dev;
    h[3] = host;
    return mlau::copy_fields(dev, h, 8, n, to_host, mlau::Move::Kernel, nullptr);
}

static void setup()
{
    if (!launched)
        launched = (int *)mmap(nullptr, 4096, PROT_READ | PROT_WRITE, MAP_SHARED | MAP_ANONYMOUS, -1, 0);
    *launched = 0;
    copies = syncs = 0;
}

// 0: moved by the kernel although an error of another call was pending
extern "C" int pending_error_check()
{
    setup();
    static double host[100];
    for (int i = 0; i < 100; i++) host[i] = i;
    pending = cudaErrorInvalidDevice;
    const int up = move(host, 100, false);
    memset(host, 0, sizeof(host));
    const int down = move(host, 100, true);
    return up || down || host[99] != 99.0 || *launched != 2;
}

// A child moves n doubles from or to an array at the end of `pages` accessible
// pages, `shift` doubles further on, beyond which (hole: whose third page) no
// access is allowed.  Returns 0: moved; 1: the CPU's access failed and nothing was
// launched; 2: launched all the same; 3: anything else.
extern "C" int bad_array_check(int pages, long long n, int shift, int hole, int to_host)
{
    setup();
    const long pg = sysconf(_SC_PAGESIZE);
    char *m = (char *)mmap(nullptr, (pages + 1) * pg, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    mprotect(m + (hole ? 2 * pg : pages * pg), pg, PROT_NONE);
    double *host = (double *)(m + pages * pg) - n + shift;
    const pid_t pid = fork();
    if (pid == 0) {
        signal(SIGSEGV, SIG_DFL);
        signal(SIGBUS, SIG_DFL);
        _exit(move(host, n, to_host != 0) ? 9 : 0);
    }
    int st = 0;
    waitpid(pid, &st, 0);
    munmap(m, (pages + 1) * pg);
    if (WIFEXITED(st) && WEXITSTATUS(st) == 0) return *launched == 1 ? 0 : 3;
    if (!WIFSIGNALED(st) || (WTERMSIG(st) != SIGSEGV && WTERMSIG(st) != SIGBUS)) return 3;
    return *launched ? 2 : 1;
}

// a move of n doubles: 1 by the kernel, 2 by a copy
extern "C" int moved_by(long long n, int to_host)
{
    setup();
    static double host[8 << 17];
    if (move(host, n, to_host != 0)) return 0;
    return *launched == 1 && copies == 0 ? 1 : *launched == 0 && copies == 1 ? 2 : 0;
}

// A download whose copy is refused: an error, after the stream has been waited for.
extern "C" int failed_download_check()
{
    setup();
    static double host[40000];
    copy_fails = cudaErrorInvalidValue;
    const int rc = move(host, 40000, true);
    copy_fails = cudaSuccess;
    return rc == 0 || copies != 1 || syncs != 1;
}

// A download of no arrays still waits for the stream.
extern "C" int empty_download_check()
{
    setup();
    double *dev[8] = {}, *h[8] = {};
    const int rc = mlau::copy_fields(dev, h, 8, 100, true, mlau::Move::Kernel, nullptr);
    return rc != 0 || *launched || copies || syncs != 1;
}
