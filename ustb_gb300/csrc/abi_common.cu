// Error state of the C-ABI and small shared entry points.
#include <mutex>
#include <vector>

#include "common.cuh"

namespace ustb {

static thread_local std::string g_last_error;

void set_error(const char* fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_last_error = buf;
}

void clear_error() { g_last_error.clear(); }

int cuda_fail(cudaError_t e, const char* what, const char* file, int line) {
    set_error("CUDA error %s (%s) in %s at %s:%d", cudaGetErrorName(e), cudaGetErrorString(e), what,
              file, line);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();  // clear the sticky-free allocation error
        return USTB_E_OOM;
    }
    return USTB_E_CUDA;
}

int shared_limit(const void* kernel, size_t& limit) {
    struct Raised {
        const void* kernel;
        int dev;
        size_t limit;
    };
    static std::mutex mu;
    static std::vector<Raised> raised;  // at most the library's kernels, per device
    int dev = 0, optin = 0;
    USTB_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    for (const Raised& r : raised)
        if (r.kernel == kernel && r.dev == dev) {
            limit = r.limit;
            return USTB_OK;
        }
    cudaFuncAttributes fa;
    USTB_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    USTB_CUDA(cudaFuncGetAttributes(&fa, kernel));
    limit = (size_t)optin - fa.sharedSizeBytes;
    USTB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit));
    raised.push_back({kernel, dev, limit});
    return USTB_OK;
}

}  // namespace ustb

extern "C" const char* ustb_last_error(void) { return ustb::g_last_error.c_str(); }

extern "C" int ustb_abi_version(void) { return 10300; }
