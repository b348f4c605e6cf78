// The fast path's kernels: persistent batches, complex channel data, FP32 entries.
#include "das_fast_kernel.cuh"

template int ustb::das_dispatch<ustb::kEntComplex, true, 2>(int, int, int, const Params*, const int64_t*, int, unsigned long long*, int64_t,
                                      int64_t, cudaStream_t, int);
