// A device for CPU tests of the host code: memory of a fixed size on the heap, copies at once, kernels that do nothing
// (the launch functions and the rest of the runtime are stubs that return 0).
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <new>

// host memory: requests above a size fail
static size_t g_largest = ~size_t(0);
extern "C" void fake_largest(size_t bytes) { g_largest = bytes; }
void *operator new(size_t n) {
    void *p = n <= g_largest ? std::malloc(n ? n : 1) : nullptr;
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

static size_t g_limit = ~size_t(0), g_used = 0;
static std::map<void *, size_t> g_blocks;

extern "C" {
void fake_limit(size_t bytes) { g_limit = bytes; }
size_t fake_used() { return g_used; }

cudaError_t cudaMalloc(void **p, size_t n) {
    if (n > g_limit || g_used > g_limit - n) return cudaErrorMemoryAllocation;
    *p = std::calloc(n, 1);
    if (!*p) return cudaErrorMemoryAllocation;
    g_blocks[*p] = n;
    g_used += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    auto it = g_blocks.find(p);
    if (it != g_blocks.end()) {
        g_used -= it->second;
        g_blocks.erase(it);
        std::free(p);
    }
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    *p = std::calloc(n, 1);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
    std::free(p);
    return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t) { return "fake device"; }

static int g_graphs_made = 0, g_graphs_alive = 0;
int fake_graphs_made() { return g_graphs_made; }
int fake_graphs_alive() { return g_graphs_alive; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
    *e = reinterpret_cast<cudaGraphExec_t>(static_cast<size_t>(++g_graphs_made));
    g_graphs_alive++;
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) {
    g_graphs_alive--;
    return cudaSuccess;
}
}
