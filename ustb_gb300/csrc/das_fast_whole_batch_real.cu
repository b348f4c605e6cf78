// The fast path's kernels: persistent batches, real channel data.
#define USTB_SUBS 1
#include "das_fast_kernel.cuh"

template int ustb::das_dispatch<ustb::kEntReal, true, 1>(int, int, int, const Params*, const int64_t*, int, unsigned long long*, int64_t,
                                      int64_t, cudaStream_t, int);
