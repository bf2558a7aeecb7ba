// Linked with the library's objects and --wrap=cudaMalloc: the allocation with the
// chosen number (counted from the last call of fake_malloc_fail) reports that the
// device is out of memory, without one being made.
#include <cuda_runtime.h>

static long number = 0, failing = -1;

extern "C" void fake_malloc_fail(long n) { number = 0; failing = n; }
extern "C" long fake_malloc_count() { return number; }
extern "C" cudaError_t __real_cudaMalloc(void** p, size_t bytes);
extern "C" cudaError_t __wrap_cudaMalloc(void** p, size_t bytes)
{
    return number++ == failing ? cudaErrorMemoryAllocation : __real_cudaMalloc(p, bytes);
}
