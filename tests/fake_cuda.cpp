// A CUDA runtime in host memory for tests of the library's host code without a GPU: the library's own
// objects are linked against it instead of the CUDA runtime. Device memory is host memory; copies
// and fills wait in a queue until something synchronises (or the test asks), as asynchronous ones
// may; kernels do nothing but call the test's hook; any allocation or launch can be made to fail.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <deque>
#include <map>
#include <mutex>
#include <string>

namespace
{
struct Op
{
    int kind;   // 0 copy, 1 fill, 2 free
    void* dst;
    const void* src;
    size_t bytes;
    int value;
    bool pageable;   // a copy from host memory that is not page-locked
    size_t sum;      // of a copy to the device: its source when it was asked for
};
struct Block
{
    size_t bytes;
    int kind;   // 0 cudaMalloc, 1 pool, 2 page-locked
    cudaMemPool_t pool;
};

std::recursive_mutex mu;
std::deque<Op> queue;
std::map<char*, Block> blocks;
std::map<const void*, std::string> kernels;
std::map<const void*, std::pair<void*, size_t>> vars;
int badFrees = 0, changedSources = 0, failAlloc = -1, failKind = -1, failLaunch = -1, coherent = 0;
cudaError_t lastError = cudaSuccess;
int defaultPool, defaultPoolChanges = 0, pools = 0;
void (*hook)(const char*, void**) = nullptr;
dim3 cfgGrid, cfgBlock;
size_t cfgSmem;
cudaStream_t cfgStream;

typedef std::lock_guard<std::recursive_mutex> Lock;

std::map<char*, Block>::iterator holding(const void* p)
{
    auto it = blocks.upper_bound((char*)p);
    if (it == blocks.begin()) return blocks.end();
    --it;
    return (char*)p < it->first + it->second.bytes ? it : blocks.end();
}

size_t checksum(const void* p, size_t n)
{
    size_t h = 1469598103934665603ull;
    for (size_t i = 0; i < n; ++i) h = (h ^ ((const unsigned char*)p)[i]) * 1099511628211ull;
    return h;
}

void flush()
{
    while (!queue.empty())
    {
        const Op o = queue.front();
        queue.pop_front();
        if (o.sum && o.sum != checksum(o.src, o.bytes)) ++changedSources;
        if (o.kind == 0) std::memmove(o.dst, o.src, o.bytes);
        if (o.kind == 1) std::memset(o.dst, o.value, o.bytes);
        if (o.kind == 2) std::free(o.dst);
    }
}

cudaError_t done(cudaError_t e)
{
    if (e != cudaSuccess) lastError = e;
    return e;
}

cudaError_t alloc(void** p, size_t bytes, int kind, cudaMemPool_t pool)
{
    Lock l(mu);
    if (kind == failKind) return done(cudaErrorMemoryAllocation);
    if (failAlloc >= 0 && failAlloc-- == 0) return done(cudaErrorMemoryAllocation);   // *p stays as it was
    *p = std::calloc(bytes ? bytes : 1, 1);
    blocks[(char*)*p] = {bytes ? bytes : 1, kind, pool};
    return cudaSuccess;
}

cudaError_t release(void* p, int kind)
{
    Lock l(mu);
    if (!p) return cudaSuccess;
    auto it = blocks.find((char*)p);
    if (it == blocks.end() || it->second.kind != kind)
    {
        ++badFrees;
        return done(cudaErrorInvalidValue);
    }
    blocks.erase(it);
    queue.push_back({2, p, nullptr, 0, 0, false, 0});
    if (kind != 1) flush();
    return cudaSuccess;
}

cudaError_t launch(const void* f, void** args)
{
    Lock l(mu);
    if (failLaunch >= 0 && failLaunch-- == 0) return done(cudaErrorLaunchOutOfResources);
    if (hook) hook(kernels[f].c_str(), args);
    return cudaSuccess;
}
}

extern "C" {
// ------------------------------------------------------------------ what a test sets and asks
void fake_reset()
{
    Lock l(mu);
    flush();
    badFrees = changedSources = defaultPoolChanges = 0;
    failAlloc = failKind = failLaunch = -1;
    lastError = cudaSuccess;
    hook = nullptr;
    coherent = 0;
}
void fake_flush()
{
    Lock l(mu);
    flush();
}
void fake_fail_alloc(int after) { failAlloc = after; }     // the allocation that `after` others precede
void fake_fail_alloc_kind(int kind) { failKind = kind; }   // all allocations of this kind
void fake_fail_launch(int after) { failLaunch = after; }
// called for every launch with the kernel's name and the addresses of its arguments
void fake_hook(void (*f)(const char*, void**)) { hook = f; }
void fake_coherent(int on) { coherent = on; }
int fake_bad_frees() { return badFrees; }
int fake_changed_sources()   // copies whose source was written between the call and the copy
{
    fake_flush();
    return changedSources;
}
int fake_pending() { return (int)queue.size(); }
int fake_pending_pageable()
{
    Lock l(mu);
    int n = 0;
    for (const Op& o : queue) n += o.kind == 0 && o.pageable;
    return n;
}
int fake_default_pool_changes() { return defaultPoolChanges; }
int fake_pools() { return pools; }
int fake_pool_blocks(int ofDefault)   // live stream-ordered blocks (of the device's default pool alone)
{
    Lock l(mu);
    int n = 0;
    for (auto& kv : blocks) n += kv.second.kind == 1 && (!ofDefault || kv.second.pool == (cudaMemPool_t)&defaultPool);
    return n;
}
void* fake_block(size_t bytes, int kind)   // a live block of this size and kind
{
    Lock l(mu);
    for (auto& kv : blocks)
        if (kv.second.bytes == bytes && kv.second.kind == kind) return kv.first;
    return nullptr;
}

// ------------------------------------------------------------------ the runtime
cudaError_t cudaMalloc(void** p, size_t n) { return alloc(p, n, 0, nullptr); }
cudaError_t cudaFree(void* p) { return release(p, 0); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return alloc(p, n, 1, (cudaMemPool_t)&defaultPool); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t) { return alloc(p, n, 1, pool); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return release(p, 1); }
cudaError_t cudaMallocHost(void** p, size_t n) { return alloc(p, n, 2, nullptr); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return alloc(p, n, 2, nullptr); }
cudaError_t cudaFreeHost(void* p) { return release(p, 2); }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned)
{
    *d = h;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t)
{
    Lock l(mu);
    const bool in = k == cudaMemcpyHostToDevice;
    queue.push_back({0, d, s, n, 0, in && holding(s) == blocks.end(), in ? checksum(s, n) : 0});
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind)
{
    Lock l(mu);
    flush();
    std::memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t)
{
    Lock l(mu);
    queue.push_back({1, d, nullptr, n, v, false, 0});
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n)
{
    Lock l(mu);
    flush();
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t)
{
    fake_flush();
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t)
{
    fake_flush();
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t)
{
    fake_flush();
    return cudaSuccess;
}
cudaError_t cudaGetLastError()
{
    const cudaError_t e = lastError;
    lastError = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaGetDeviceCount(int* n)
{
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d)
{
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrMultiProcessorCount ? 152
         : a == cudaDevAttrPageableMemoryAccessUsesHostPageTables ? coherent
         : a == cudaDevAttrComputeCapabilityMajor ? 10
         : a == cudaDevAttrComputeCapabilityMinor ? 3
                                                  : 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int)
{
    *p = (cudaMemPool_t)&defaultPool;
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, cudaMemPoolAttr, void*)
{
    if (p == (cudaMemPool_t)&defaultPool) ++defaultPoolChanges;
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*)
{
    ++pools;
    *p = (cudaMemPool_t) new int;
    return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p)
{
    --pools;
    delete (int*)p;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned)
{
    *s = (cudaStream_t) new int;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s)
{
    delete (int*)s;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned)
{
    *e = (cudaEvent_t) new int;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e)
{
    delete (int*)e;
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t)
{
    *ms = 0.f;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g)
{
    *g = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long)
{
    *x = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphExecUpdate(cudaGraphExec_t, cudaGraph_t, cudaGraphExecUpdateResultInfo*) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t)
{
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* symbol)
{
    *p = vars[symbol].first;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* f, void** args) { return launch(f, args); }

// what the compiler's host stubs call
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, cudaStream_t s)
{
    cfgGrid = g;
    cfgBlock = b;
    cfgSmem = m;
    cfgStream = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s)
{
    *g = cfgGrid;
    *b = cfgBlock;
    *m = cfgSmem;
    *(cudaStream_t*)s = cfgStream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f)
{
    *k = (cudaKernel_t)f;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void** args, size_t, cudaStream_t)
{
    return launch((const void*)k, args);
}
void** __cudaRegisterFatBinary(void*)
{
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, void*, void*, void*, void*, int*)
{
    kernels[f] = name;
}
void __cudaRegisterVar(void**, char* v, char*, const char*, int, size_t bytes, int, int)
{
    vars[v] = {std::calloc(bytes, 1), bytes};
}
}
