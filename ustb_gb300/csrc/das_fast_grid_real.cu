// The fast path's kernels: one launch per request, real channel data.
#include "das_fast_kernel.cuh"

template int ustb::das_dispatch<ustb::kEntReal, false, 2>(int, int, int, const Params*, const int64_t*, int, unsigned long long*, int64_t,
                                      int64_t, cudaStream_t, int);
