// Internal state of the C-ABI runtime objects, shared by the runtime (lf_runtime.cu), the
// multi-job engine driver (lf_engine_host.cu) and the serving loop (lf_server.cu).
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <string>
#include <vector>

#include "../../../include/lavaframe_gb300.h"
#include "lf_kernels.h"

using namespace lfd;

#include "lf_guide.cuh"

namespace lfrt
{
struct EngineHost;
void engine_destroy(EngineHost* e);
lfd::guide::Net guide_net(const lf_guide* g);
int guide_tensor_path(const lf_guide* g);
}

struct lf_ctx
{
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaMemPool_t pool = nullptr;   // stream-ordered memory (pool_acquire)
    std::recursive_mutex mu;
    std::string err;
    // status words of the kernels ([0]; [1] for lf_render_noalloc, which reports its own): in mapped page-locked memory, so that reading it after a
    // synchronisation needs no copy (the kernels only write it when something went wrong)
    volatile uint32_t* h_status = nullptr;
    uint32_t* d_status = nullptr;         // its device address
    unsigned long long* d_stats = nullptr;   // [3] traversal counters
    uint32_t devErrors = 0;
    uint64_t lastStats[3] = {0, 0, 0};
    // reusable device buffers of the host-pointer ray queries
    void* scratchRays = nullptr;
    size_t scratchRaysBytes = 0;
    void* scratchOut = nullptr;
    size_t scratchOutBytes = 0;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    // pieces of the host-pointer ray queries: copy streams and one event per piece and side
    static constexpr int kMaxHostChunks = 8;
    int hostChunks = 0;                       // 0: automatic
    cudaStream_t copyIn = nullptr, copyOut = nullptr;
    cudaEvent_t chunkIn[kMaxHostChunks] = {}, chunkDone[kMaxHostChunks] = {};
    cudaEvent_t chunkStart = nullptr, chunkEnd = nullptr;
    // page-locked blocks from lf_host_alloc and their device addresses: results of host queries
    // whose output lies in one are written there by the kernels, without a copy back
    struct HostBlock
    {
        char* host;
        char* dev;
        size_t bytes;
    };
    std::vector<HostBlock> hostBlocks;
    // scratch of the binned ray queries
    uint32_t* binKeys = nullptr;
    int* binPerm = nullptr;
    size_t binCap = 0;
    uint32_t* binHist = nullptr;
    unsigned long long* binNext = nullptr;   // fetch counter and blocks done, zero between launches
    bool hostDirect = false;                 // kernels may address the host's own memory (direct_host)
    char* stage = nullptr;                   // page-locked staging block (ensure_stage)
    char* d_stage = nullptr;                 // its device address
    lfrt::EngineHost* engine = nullptr;   // multi-job engine, created on first use
    // traversal-kernel timer of the binned ray queries: one event pair per launch while on
    bool kernelTimer = false;
    std::vector<cudaEvent_t> ktEvents;     // start, stop, start, stop, ...
    size_t ktUsed = 0;                     // pairs recorded since the last read
};

struct lf_scene
{
    lf_ctx* ctx = nullptr;
    std::vector<void*> allocs;
    size_t bytes = 0;
    ShadeScene view{};
    // re-encoding metadata for instance updates
    int numRefNodes = 0;
    int topLevelIndex = 0;
    int numMeshNodes = 0;       // device records that belong to mesh levels
    std::vector<int> blasRootCode;   // per reference node index of a mesh root (code), lazily
    float4* d_nodes = nullptr;
    size_t nodeCapacity = 0;    // records allocated
    float4* d_instances = nullptr;
    ShadeInstance* d_sinst = nullptr;
    DevMaterial* d_materials = nullptr;
    int numMaterials = 0;
    std::vector<int> meshNodeMap;   // reference index -> device record (mesh levels), -1 otherwise
    float4* d_wide = nullptr;       // wide tree
    size_t wideCapacity = 0;        // wide records allocated
    float* d_refNodes = nullptr;    // the reference nodes (tie resolution)
    int* d_parent = nullptr;
    int* d_leafOfTri = nullptr;     // reference leaf of every triangle
    int* d_leafOfInst = nullptr;    // reference leaf of every instance
    int* d_instOfTri = nullptr;     // instance of the triangles merged into the instance level
    float boundsLo[3] = {0, 0, 0}, boundsHi[3] = {0, 0, 0};   // instance-level root box
};

struct lf_frame
{
    lf_ctx* ctx = nullptr;
    lf_scene* scene = nullptr;
    Params P{};
    uint32_t flags = 0;
    int W = 0, H = 0;
    int numTilesX = 1, numTilesY = 1;
    int sppBatch = 0;
    long long cap = 0;   // path slots
    float4* accum = nullptr;
    double* accum64 = nullptr;
    PathSoA ps{};
    BounceBuffers bb{};
    std::vector<void*> fixedAllocs;   // accumulation buffers and counters
    std::vector<void*> allocs;        // path state and queues (sized by the batch)
    uint64_t paths = 0;
    int lastBatchSamples = 0;
    cudaGraphExec_t graph = nullptr;
    int graphDepth = -1;
    // engine path (default): job slot in the context's engine and the per-path radiance of
    // the most recent pass ([sample][pixel] of a single-tile frame), in the allocation lastBlock
    int engineJob = -1;
    float4* lastRadiance = nullptr;
    float4* lastBlock = nullptr;
    int lastRadianceSamples = 0;
    // learned path guiding (per-batch pipeline, one sample per batch)
    lf_guide* guide = nullptr;
    float guideAlpha = 0.5f;
    int guideTrainEvery = 4;
    float guideLr = 1e-2f;
    int guideTrainCap = 1 << 20;
    int guideBatch = 16384;        // samples per Adam step
    long long guideCap = 0;        // path slots the guide buffers hold
    GuideBuffers gb{};
    std::vector<void*> guideAllocs;
    uint64_t guideSteps = 0;
    uint64_t guideSamples = 0;
    uint64_t guideBatches = 0;     // guided batches rendered (training cadence)
};

namespace lfrt
{
inline lf_status fail(lf_ctx* c, lf_status st, const std::string& msg)
{
    if (c) c->err = msg;
    return st;
}

inline lf_status cuda_fail(lf_ctx* c, cudaError_t e, const char* what)
{
    std::string m = std::string(what) + ": " + cudaGetErrorString(e);
    cudaGetLastError();   // reported here: the next launch's check must not find it again
    if (e == cudaErrorMemoryAllocation) return fail(c, LF_ERR_OOM, m);
    return fail(c, LF_ERR_CUDA, m);
}

template <class T>
inline cudaError_t dalloc(std::vector<void*>& list, size_t& bytes, T** p, size_t count)
{
    *p = nullptr;
    if (count == 0) count = 1;
    cudaError_t e = cudaMalloc((void**)p, sizeof(T) * count);
    if (e == cudaSuccess)
    {
        list.push_back(*p);
        bytes += sizeof(T) * count;
    }
    return e;
}

// Stream-ordered memory of the library's own pool of the context's device (given back with
// cudaFreeAsync).
template <class T>
inline cudaError_t pool_alloc(const lf_ctx* c, T** p, size_t bytes, cudaStream_t st)
{
    return cudaMallocFromPoolAsync((void**)p, bytes, c->pool, st);
}

inline lf_status check_device(lf_ctx* c)
{
    cudaError_t e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "stream synchronize");
    const uint32_t bits = *c->h_status;
    if (bits)
    {
        c->devErrors |= bits;
        *c->h_status = 0;
        return fail(c, LF_ERR_DEVICE, "device error bits 0x" + std::to_string(bits));
    }
    return LF_OK;
}

// Lets go of the most recent pass's radiance (in stream order).
inline void drop_last_radiance(lf_frame* f)
{
    if (f->lastBlock) cudaFreeAsync(f->lastBlock, f->ctx->stream);
    f->lastRadiance = f->lastBlock = nullptr;
    f->lastRadianceSamples = 0;
}

// Kernel parameters of one render (lf_render_params + scene facts); tile fields cover the
// whole frame unless the parameters set a tile size.
void fill_params(Params& P, const lf_render_params* p, const lf_scene* sc);

// Whether a kernel may read (or write) the caller's buffer itself. On a coherent host (Grace: the GPU
// walks the host's page tables) any memory of the process can be addressed, and what the kernel moves
// over C2C is hidden behind its work, which a copy before or after it is not. The pages are
// brought in first: that tells a range that isn't mapped (or not writable) from one that is before
// a kernel meets it - such a range takes the copy path and its errors - and fresh pages cost a third
// less than when the GPU faults them in one by one (32 MB: 0.78 ms, 1.16 faulted, 0.97 by copy).
// Buffers must be aligned for the kernel's words; on other hosts everything is copied.
bool direct_host(const lf_ctx* c, const void* p, size_t bytes, bool write, size_t align = 16);
// Inputs and results that overlap go through copies.
inline bool disjoint(const void* a, size_t na, const void* b, size_t nb)
{
    const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
    return x + na <= y || y + nb <= x;
}

// Page-locked staging of small results and queries, mapped for the kernels (c->stage, c->d_stage);
// false when there is none.
constexpr size_t kStageBytes = size_t(1) << 18;
bool ensure_stage(lf_ctx* c);
// The colour channels of n padded pixels into host memory, after the work of `st` (synchronises).
cudaError_t copy_rgb(const lf_ctx* c, cudaStream_t st, const float4* src, size_t n, float* rgb);

struct RefNode
{
    float bmin[3], bmax[3], lr[3];
};

inline float ulp_of(float x)
{
    x = std::fabs(x);
    float n = std::nextafter(x, INFINITY);
    return n - x;
}
}
