// cudaMalloc that fails above a limit, linked in front of the engine's objects
// (--wrap): a GPU without the memory, made on the host.
#include <cstddef>

static size_t g_limit = ~(size_t)0;

extern "C" {
int __real_cudaMalloc(void **p, size_t bytes);
int __wrap_cudaMalloc(void **p, size_t bytes) { return bytes > g_limit ? 2 /* cudaErrorMemoryAllocation */ : __real_cudaMalloc(p, bytes); }
void fake_malloc_limit(size_t bytes) { g_limit = bytes; }
}
