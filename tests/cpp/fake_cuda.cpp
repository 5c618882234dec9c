// Stands before the CUDA runtime (LD_PRELOAD) and returns errors for calls that the test asks it to refuse.
#include <dlfcn.h>

#include <cstddef>

// The runtime's own function; the library under test has loaded it by the time it calls one.
static void* runtime(const char* name) { return dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), name); }

extern "C" {

size_t fake_malloc_limit = ~(size_t)0;  // cudaMalloc of as many bytes or more fails
int fake_cooperative_error = 0;         // cudaLaunchCooperativeKernel returns this where it is not 0

int cudaMalloc(void** p, size_t n) {
    if (n >= fake_malloc_limit) return 2;  // cudaErrorMemoryAllocation
    static auto real = reinterpret_cast<int (*)(void**, size_t)>(runtime("cudaMalloc"));
    return real(p, n);
}

struct Dim {
    unsigned x, y, z;
};
int cudaLaunchCooperativeKernel(const void* fn, Dim grid, Dim block, void** args, size_t smem, void* stream) {
    if (fake_cooperative_error) return fake_cooperative_error;
    static auto real = reinterpret_cast<int (*)(const void*, Dim, Dim, void**, size_t, void*)>(
        runtime("cudaLaunchCooperativeKernel"));
    return real(fn, grid, block, args, smem, stream);
}
}
