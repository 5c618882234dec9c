// Stands before the CUDA runtime (LD_PRELOAD): returns errors for calls that the test asks it to refuse, and counts the
// bytes that cudaMalloc gave and cudaFree has not taken back.
#include <dlfcn.h>

#include <cstddef>
#include <map>
#include <mutex>

// The runtime's own function; the library under test has loaded it by the time it calls one.
static void* runtime(const char* name) { return dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), name); }
static std::mutex lock;
static std::map<void*, size_t> sizes;

extern "C" {

size_t fake_malloc_limit = ~(size_t)0;  // cudaMalloc of as many bytes or more fails
size_t fake_memory = 0;                 // bytes in use
size_t fake_memory_limit = ~(size_t)0;  // cudaMalloc beyond it fails
int fake_cooperative_error = 0;         // cudaLaunchCooperativeKernel returns this where it is not 0

int cudaMalloc(void** p, size_t n) {
    static auto real = reinterpret_cast<int (*)(void**, size_t)>(runtime("cudaMalloc"));
    std::lock_guard<std::mutex> hold(lock);
    if (n >= fake_malloc_limit || fake_memory + n > fake_memory_limit) return 2;  // cudaErrorMemoryAllocation
    const int rc = real(p, n);
    if (!rc) fake_memory += sizes[*p] = n;
    return rc;
}

int cudaFree(void* p) {
    static auto real = reinterpret_cast<int (*)(void*)>(runtime("cudaFree"));
    std::lock_guard<std::mutex> hold(lock);
    const auto it = sizes.find(p);
    if (it != sizes.end()) {
        fake_memory -= it->second;
        sizes.erase(it);
    }
    return real(p);
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
