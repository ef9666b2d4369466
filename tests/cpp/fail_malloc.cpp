// Preloaded by a test: cudaMalloc refuses requests above MBCG_TEST_MALLOC_LIMIT bytes (unset: none), as a device
// whose memory is nearly all taken does.
#include <cuda_runtime_api.h>
#include <dlfcn.h>

#include <cstdlib>

extern "C" cudaError_t cudaMalloc(void** p, size_t n) {
    using Fn = cudaError_t (*)(void**, size_t);
    static Fn real = reinterpret_cast<Fn>(dlsym(RTLD_NEXT, "cudaMalloc"));
    if (const char* limit = std::getenv("MBCG_TEST_MALLOC_LIMIT"))
        if (n > std::strtoull(limit, nullptr, 10)) return cudaErrorMemoryAllocation;
    return real(p, n);
}
