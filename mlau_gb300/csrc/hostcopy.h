// Host arrays to and from the device (hostcopy.cu).
#pragma once

#include "common.cuh"

namespace mlau {

// n doubles of each pair of arrays host[v], dev[v] (v < nv; either null: none), to
// the host or from it, in the order of `st`: by copies, or where it can by one
// kernel.  To the host it returns when the arrays have been written.  From the
// host, by copies, it returns as cudaMemcpyAsync does; with the kernel the caller
// leaves the arrays alone until `st` has got there.
enum class Move { Copies, Kernel };
int copy_fields(double *const *dev, double *const *host, int nv, long long n, bool to_host, Move how,
                cudaStream_t st);

}  // namespace mlau
