#include "fake_cuda.h"

#include <dlfcn.h>
#include <pthread.h>

#include <cerrno>
#include <cstdlib>
#include <cstring>
#include <map>
#include <vector>

struct CUmemPoolHandle_st {
    size_t live = 0, held = 0, keep = 0;
};

namespace fake {
size_t budget = size_t(1) << 40;
bool threadsFail = false;
int failingRecord = 0;
namespace {
std::vector<std::function<void()>> queue;
struct Block {
    size_t bytes;
    cudaMemPool_t pool;
};
std::map<void*, Block> blocks;
std::vector<cudaMemPool_t> pools;
cudaError_t last = cudaSuccess;

// Overwrites the stack below the caller: a copy's source that was a local of a function that has returned is gone.
__attribute__((noinline)) void spoilStack() {
    char gone[1 << 16];
    std::memset(gone, 0xEE, sizeof(gone));
    asm volatile("" : : "r"(gone) : "memory");
}
void run() {
    spoilStack();
    while (!queue.empty()) {
        auto ops = std::move(queue);
        queue.clear();
        for (auto& op : ops) op();
    }
    for (auto p : pools)  // a wait returns what is above the threshold, which live blocks count against too
        if (p->live + p->held > p->keep) p->held = p->live > p->keep ? 0 : p->keep - p->live;
}
cudaError_t set(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
cudaError_t take(void** p, size_t bytes, cudaMemPool_t pool) {
    size_t reuse = pool ? (pool->held < bytes ? pool->held : bytes) : 0;
    if (used() - reuse + bytes > budget) return set(cudaErrorMemoryAllocation);
    *p = std::aligned_alloc(256, (bytes + 255) & ~size_t(255));
    std::memset(*p, 0xCD, bytes < 4096 ? bytes : 4096);
    blocks[*p] = {bytes, pool};
    if (pool) {
        pool->held -= reuse;
        pool->live += bytes;
    }
    return cudaSuccess;
}
void give(void* p) {
    auto it = blocks.find(p);
    if (it == blocks.end()) std::abort();
    if (it->second.pool) {
        it->second.pool->live -= it->second.bytes;
        it->second.pool->held += it->second.bytes;
    }
    std::memset(p, 0xDD, it->second.bytes < 4096 ? it->second.bytes : 4096);
    blocks.erase(it);
    std::free(p);
}
template <class T> cudaError_t handle(T* h) {
    *h = reinterpret_cast<T>(std::malloc(16));
    return cudaSuccess;
}
template <class T> cudaError_t dropped(T h) {
    std::free(reinterpret_cast<void*>(h));
    return cudaSuccess;
}
}  // namespace
size_t pending() { return queue.size(); }
void enqueue(std::function<void()> op) { queue.push_back(std::move(op)); }
size_t used() {
    size_t n = 0;
    for (auto& b : blocks) n += b.second.bytes;
    for (auto p : pools) n += p->held;
    return n;
}
}  // namespace fake

using namespace fake;

extern "C" {
int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
    if (threadsFail) return EAGAIN;
    using Fn = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
    static const Fn real = reinterpret_cast<Fn>(dlsym(RTLD_NEXT, "pthread_create"));
    return real(t, a, f, arg);
}

cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) { return *v = a == cudaDevAttrMultiProcessorCount ? 152 : 1, cudaSuccess; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return run(), dropped(s); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return run(), cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return dropped(e); }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return failingRecord > 0 && --failingRecord == 0 ? set(cudaErrorUnknown) : cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return set(cudaErrorNotSupported); }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return set(cudaErrorNotSupported); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return set(cudaErrorNotSupported); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return set(cudaErrorNotSupported); }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

cudaError_t cudaMalloc(void** p, size_t n) { return run(), take(p, n, nullptr); }
cudaError_t cudaFree(void* p) { return run(), p ? give(p) : void(), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = std::aligned_alloc(4096, (n + 4095) & ~size_t(4095)), cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
    *p = new CUmemPoolHandle_st;
    pools.push_back(*p);
    return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) { return p->held = 0, cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, cudaMemPoolAttr a, void* v) {
    if (a == cudaMemPoolAttrReleaseThreshold) p->keep = *static_cast<unsigned long long*>(v);
    return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t keep) {
    run();
    if (p->live + p->held > keep) p->held = p->live > keep ? 0 : keep - p->live;
    return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t) { return take(p, n, pool); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return enqueue([p] { give(p); }), cudaSuccess; }

cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    enqueue([=] { std::memcpy(d, s, n); });
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return run(), std::memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
    enqueue([=] {
        for (size_t k = 0; k < h; ++k) std::memcpy(static_cast<char*>(d) + k * dp, static_cast<const char*>(s) + k * sp, w);
    });
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    enqueue([=] { std::memset(d, v, n); });
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { return *p = const_cast<void*>(s), cudaSuccess; }
}
