// Host arrays to and from the device (hostcopy.cu).
#pragma once

#include "common.cuh"

namespace mlau {

// n doubles of each pair of arrays host[v], dev[v] (v < nv; either null: none), to
// the host or from it, in the order of `st`.  wait: returns when the host arrays
// have been written, or read as far as they are ordinary memory; without it the
// caller leaves them alone until `st` has got there.
int copy_fields(double *const *dev, double *const *host, int nv, long long n, bool to_host, bool wait,
                cudaStream_t st);

}  // namespace mlau
