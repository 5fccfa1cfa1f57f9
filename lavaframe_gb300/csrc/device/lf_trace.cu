// Batched ray queries (ClosestHit / AnyHit as a service): ray binning and a persistent
// traversal kernel.
//
// Random rays give each lane of a warp its own path through the BVH: few lanes share an
// instruction and almost every node comes from DRAM. Three measures, none of which changes
// any per-ray result:
//  - binning: rays of large queries are counting-sorted by a key made of the Morton code of
//    their origin cell (64^3 cells over the scene box, 32^3 below kFineRays) and their direction
//    octant, so neighbouring lanes start in the same region heading the same way and share nodes
//    in L1/L2;
//  - persistent warps with dynamic fetch: warps take rays from a counter in the binned order, so
//    a warp that finished early takes more work;
//  - queries that cannot fill the GPU put fewer rays into a warp (chunk_for): with 32 rays a
//    warp runs the union of their branches, with few it runs little more than one ray's.
#include <algorithm>

#include "lf_kernels.h"

namespace lfd
{
namespace
{
constexpr unsigned kFullMask = 0xffffffffu;
constexpr int kCellBits = 6;                           // most cells per axis = 2^kCellBits
constexpr int bins_of(int cellBits) { return 1 << (3 * cellBits + 3); }   // origin Morton code + direction octant
constexpr int kScanBlock = 1024;
constexpr int kScanBlocks = bins_of(kCellBits) / kScanBlock;   // partial sums of the bin scan
static_assert(kScanBlocks >= 1 && kScanBlocks <= 2 * kScanBlock, "bin scan covers 2^10 to 2^21 bins");

// Sizes from which queries are binned. Binning costs about 20 us and two scattered passes; it pays
// once many rays share a bin, the sooner the more the geometry's cache misses cost. Closest hits in
// device memory, binned / input order, us. Up to 8k triangles (Cornell box, room, random): 2^20 rays
// 151 / 139, 162 / 155, 148 / 121, 2^21 261 / 257, 285 / 287, 258 / 220, 2^22 on the Cornell box 456 / 492.
// Up to 1.2M (Cornell 35k, room 48k, spheres 164k, random 327k): 524k rays 141 / 135, 169 / 175, 186 / 168,
// 624 / 636, 800k 189 / 189, 230 / 245, 243 / 225, 889 / 907, 2^21 415 / 446, 517 / 585, 512 / 504,
// 2148 / 2217: 2^19 lies between them (3 * 2^18 gives spheres 16 % there and takes 5 % from the
// room). Scenes larger than the L2 (1.3M, 2M, 5.2M random triangles, about 200 bytes each): 131k
// 283 / 274, -, 407 / 401, 262k 445 / 492, 495 / 534, 643 / 671, 524k 751 / 835, 779 / 935, 1047 / 1212. The
// lines are triangle counts between measured scenes; nothing between 327k and 1.3M was measured. Queries
// of host buffers have a rule of their own (direct_query), as their binning also costs the copies.
long long sort_closest(int tris)
{
    if (tris <= 1 << 13) return 1 << 21;
    return tris <= 1200000 ? 1 << 19 : 1 << 18;
}
// Occlusion queries end early and write one byte per ray, which binning scatters: 4M rays on 1.3M random
// triangles, a room, spheres and the Cornell box 4254 / 4460, 472 / 485, 1033 / 1048, 427 / 373; 16M
// rays 16.3 / 17.3, 1.89 / 1.87, 3.96 / 3.86, 1.69 / 1.44 ms.
constexpr long long kSortAny = 1 << 23;
// 64^3 cells from here on, 32^3 below: 4M rays 4.94 / 4.97 ms on the random triangles, but 1.00 / 0.94,
// 1.29 / 1.20 and 0.70 / 0.63 ms on the others; on 2^24 rays against 10.5M triangles 32^3 cells
// are 1.3 % slower.
constexpr long long kFineRays = 1 << 23;

__device__ __forceinline__ uint32_t spread3(uint32_t x)   // up to 7 bits -> every third bit
{
    x &= 127u;
    x = (x | (x << 16)) & 0x030000FFu;
    x = (x | (x << 8)) & 0x0300F00Fu;
    x = (x | (x << 4)) & 0x030C30C3u;
    x = (x | (x << 2)) & 0x09249249u;
    return x;
}

__device__ __forceinline__ uint32_t cell(float v, float lo, float inv, float top)
{
    float q = (v - lo) * inv;
    q = q < 0.f ? 0.f : (q > top ? top : q);
    return (uint32_t)q;
}

// Exclusive scan of 1024 values held one per thread (a block of 1024 threads): returns the
// thread's exclusive prefix and stores the block total in *total (shared memory).
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total)
{
    __shared__ uint32_t warpSums[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1)
    {
        const uint32_t u = __shfl_up_sync(kFullMask, incl, k);
        if (lane >= k) incl += u;
    }
    if (lane == 31) warpSums[warp] = incl;
    __syncthreads();
    if (warp == 0)
    {
        const uint32_t w = warpSums[lane];
        uint32_t wi = w;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1)
        {
            const uint32_t u = __shfl_up_sync(kFullMask, wi, k);
            if (lane >= k) wi += u;
        }
        warpSums[lane] = wi - w;
        if (lane == 31) *total = wi;
    }
    __syncthreads();
    return warpSums[warp] + incl - v;
}
}

__global__ void ray_keys_kernel(const float4* rays, long long n, float3 lo, float3 inv, float top, uint32_t* keys,
                                uint32_t* hist)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    {
        float4 o = rays[2 * i], d = rays[2 * i + 1];
        uint32_t m = (spread3(cell(o.x, lo.x, inv.x, top)) << 2) | (spread3(cell(o.y, lo.y, inv.y, top)) << 1) |
                     spread3(cell(o.z, lo.z, inv.z, top));
        uint32_t oct = (d.x < 0.f ? 4u : 0u) | (d.y < 0.f ? 2u : 0u) | (d.z < 0.f ? 1u : 0u);
        uint32_t k = (m << 3) | oct;
        keys[i] = k;
        atomicAdd(&hist[k], 1u);
    }
}

// Exclusive scan of the bins' counters: each block of 1024 scans its slice and records the slice
// total (hist[bins + block]); the last block to end scans the totals (at most two per thread), which
// the scatter adds to its slice's offsets. hist[bins + kScanBlocks] counts the blocks (zeroed with
// the bins).
__global__ void __launch_bounds__(kScanBlock) bins_scan_kernel(uint32_t* hist, int bins)
{
    __shared__ uint32_t total;
    __shared__ bool last;
    const int i = blockIdx.x * kScanBlock + threadIdx.x;
    const uint32_t v = hist[i];
    const uint32_t ex = block_exclusive_scan(v, &total);
    hist[i] = ex;
    __syncthreads();
    uint32_t* sums = hist + bins;
    if (threadIdx.x == 0)
    {
        sums[blockIdx.x] = total;
        __threadfence();
        last = atomicAdd(&sums[kScanBlocks], 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    const int t = threadIdx.x, blocks = bins / kScanBlock;
    const uint32_t a = 2 * t < blocks ? __ldcg(&sums[2 * t]) : 0u;
    const uint32_t b = 2 * t + 1 < blocks ? __ldcg(&sums[2 * t + 1]) : 0u;
    const uint32_t ex2 = block_exclusive_scan(a + b, &total);
    if (2 * t < blocks) sums[2 * t] = ex2;
    if (2 * t + 1 < blocks) sums[2 * t + 1] = ex2 + a;
}

__global__ void ray_scatter_kernel(const uint32_t* keys, long long n, uint32_t* cursor, int bins, int* perm)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    {
        const uint32_t k = keys[i];
        const uint32_t pos = cursor[bins + k / kScanBlock] + atomicAdd(&cursor[k], 1u);
        perm[pos] = (int)i;
    }
}

// Persistent closest-hit / any-hit over `n` rays taken in `perm` order (or input order).
template <bool kAny>
__global__ void __launch_bounds__(128) trace_persistent_kernel(DevScene S, const float4* rays, const int* perm,
                                                                long long n, int4* hits, uint8_t* occluded, int lights,
                                                                unsigned long long* next, uint32_t* status)
{
    TravState s;
    long long rid = -1;   // -1: needs a ray, -2: no rays left
    int light = -1;
    const int lane = threadIdx.x & 31;
    while (true)
    {
        unsigned need = __ballot_sync(kFullMask, rid == -1);
        if (need)
        {
            int leader = __ffs(need) - 1;
            unsigned long long base = 0;
            if (lane == leader) base = atomicAdd(next, (unsigned long long)__popc(need));
            base = __shfl_sync(kFullMask, base, leader);
            if (rid == -1)
            {
                unsigned long long my = base + __popc(need & ((1u << lane) - 1u));
                if (my < (unsigned long long)n)
                {
                    rid = perm ? (long long)perm[my] : (long long)my;
                    float4 o4 = rays[2 * rid], d4 = rays[2 * rid + 1];
                    v3 o(o4.x, o4.y, o4.z), d(d4.x, d4.y, d4.z);
                    float t = d4.w;
                    light = -1;
                    bool done = false;
                    if (lights)
                    {
                        if (kAny)
                            done = lights_any(S, o, d, t);
                        else
                            t = lights_closest(S, o, d, t, &light);
                    }
                    trav_init(s, S, o, d, t);
                    if (done)
                    {
                        occluded[rid] = 1;
                        rid = -1;
                    }
                }
                else
                    rid = -2;
            }
        }
        if (__all_sync(kFullMask, rid == -2)) break;
        if (rid >= 0 && trav_run<kAny>(s, S, 32))
        {
            if (kAny)
                occluded[rid] = s.hitPrim >= 0 ? 1 : 0;
            else
                hits[rid] = make_int4(__float_as_int(s.t), s.hitInst, s.hitPrim, s.hitPrim >= 0 ? -1 : light);
            if (s.err) atomicOr(status, s.err);
            rid = -1;
        }
    }
}

// Wide-tree form: each lane traces its ray to completion; warps take `chunk` rays at a time (in
// `perm` order), the first by their place in the grid and further ones from a global counter, so a
// warp that finished early takes more work. The last block to end clears the counter for the next
// launch. (Refilling single lanes as their rays end, with the traversal state kept in registers,
// measured 35 % slower: the binned rays of a warp stop sharing nodes and the refill logic spills.)
template <bool kAny>
__global__ void __launch_bounds__(128, kAny ? 8 : 7) trace_fetch_wide_kernel(DevScene S, const float4* rays, const int* perm,
                                                               long long n, int4* hits, uint8_t* occluded, int lights,
                                                               unsigned long long* next, uint32_t* status, int chunk)
{
    const int lane = threadIdx.x & 31;
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    long long base = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * chunk;
    while (base < n)
    {
        const long long my = base + lane;
        if (lane < chunk && my < n)
        {
            const long long rid = perm ? (long long)perm[my] : my;
            const float4 o4 = rays[2 * rid], d4 = rays[2 * rid + 1];
            const v3 o(o4.x, o4.y, o4.z), d(d4.x, d4.y, d4.z);
            Hit h;
            uint32_t err;
            if (kAny)
            {
                bool occ;
                err = any_hit<false>(S, o, d, d4.w, lights != 0, &occ, &h, nullptr);
                occluded[rid] = occ ? 1 : 0;
            }
            else
            {
                err = closest_hit<false>(S, o, d, d4.w, lights != 0, &h, nullptr);
                hits[rid] = make_int4(__float_as_int(h.t), h.inst, h.prim, h.light);
            }
            if (err) atomicOr(status, err);
        }
        if (n <= warps * chunk) return;   // every warp had one chunk: the counter is not used
        unsigned long long got = 0;
        if (lane == 0) got = atomicAdd(next, (unsigned long long)chunk);
        base = warps * chunk + (long long)__shfl_sync(kFullMask, got, 0);
    }
    if (n <= warps * chunk) return;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        // next[1]: blocks that have taken their last chunk; all have when the count is full
        __threadfence();
        if (atomicAdd(next + 1, 1ull) == gridDim.x - 1)
        {
            next[0] = 0;
            next[1] = 0;
        }
    }
}

namespace
{
// Rays a warp takes at a time: 32, or fewer (a power of two) while the query still has no more
// chunks than the GPU holds warps (4256 at 72 registers). A small query is a chain of dependent
// node visits, and a warp visits the union of its rays' branches: 1000 rays 37 -> 21 us in a room
// of 48k triangles, 173 -> 112 us against 1.3M random triangles, 16,000 rays 43 -> 36 and
// 197 -> 136 us. Twice or four times the warps a GPU holds lose that again (16,000 rays 145 and
// 160 us), at 130,000 rays and above 32 a warp are best.
int chunk_for(long long n, long long warps)
{
    int chunk = 1;
    while (chunk < 32 && chunk * warps < n) chunk *= 2;
    return chunk;
}

template <bool kAny>
void launch_wide(const DevScene& S, const float4* rays, const int* order, long long n, void* out, int lights, int sms,
                 unsigned long long* next, uint32_t* status, cudaStream_t st)
{
    const int perSm = occupancy_blocks_per_sm((const void*)trace_fetch_wide_kernel<kAny>, 128);
    const long long full = (long long)sms * perSm;
    const int chunk = chunk_for(n, 4 * full);
    const long long need = (n + 4ll * chunk - 1) / (4ll * chunk);
    trace_fetch_wide_kernel<kAny><<<(int)std::min(full, need), 128, 0, st>>>(
        S, rays, order, n, kAny ? nullptr : (int4*)out, kAny ? (uint8_t*)out : nullptr, lights, next, status, chunk);
}

void sort_rays(const float4* rays, long long n, const float lo[3], const float hi[3], int sms, uint32_t* keys,
               uint32_t* hist, int* perm, cudaStream_t st)
{
    const int cellBits = n >= kFineRays ? kCellBits : kCellBits - 1;
    const int bins = bins_of(cellBits), cells = 1 << cellBits;
    const float3 flo = make_float3(lo[0], lo[1], lo[2]);
    auto inv = [&](float a, float b) { return b > a ? (float)cells / (b - a) : 0.0f; };
    const float3 finv = make_float3(inv(lo[0], hi[0]), inv(lo[1], hi[1]), inv(lo[2], hi[2]));
    cudaMemsetAsync(hist, 0, sizeof(uint32_t) * ((size_t)bins + kScanBlocks + 1), st);   // bins and block count
    const int g = (int)std::min<long long>(sms * 8, (n + 255) / 256);
    ray_keys_kernel<<<g, 256, 0, st>>>(rays, n, flo, finv, (float)(cells - 1), keys, hist);
    bins_scan_kernel<<<bins / kScanBlock, kScanBlock, 0, st>>>(hist, bins);
    ray_scatter_kernel<<<g, 256, 0, st>>>(keys, n, hist, bins, perm);
}
}

int launch_trace_binned(const DevScene& S, const float4* rays, long long n, void* out, bool any, int lights,
                        const float lo[3], const float hi[3], bool binning, uint32_t* keys, uint32_t* hist, int* perm,
                        unsigned long long* next, uint32_t* status, cudaStream_t st, cudaEvent_t evStart,
                        cudaEvent_t evStop)
{
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int* order = nullptr;
    if (binning)
    {
        sort_rays(rays, n, lo, hi, sms, keys, hist, perm, st);
        order = perm;
    }
    if (S.wnodes && S.wideOn)
    {
        if (evStart) cudaEventRecord(evStart, st);
        if (any)
            launch_wide<true>(S, rays, order, n, out, lights, sms, next, status, st);
        else
            launch_wide<false>(S, rays, order, n, out, lights, sms, next, status, st);
        if (evStop) cudaEventRecord(evStop, st);
        return (int)cudaGetLastError();
    }
    int per_sm = 0;
    if (evStart) cudaEventRecord(evStart, st);
    if (any)
    {
        per_sm = occupancy_blocks_per_sm((const void*)trace_persistent_kernel<true>, 128);
        trace_persistent_kernel<true><<<sms * (per_sm > 0 ? per_sm : 1), 128, 0, st>>>(
            S, rays, order, n, nullptr, (uint8_t*)out, lights, next, status);
    }
    else
    {
        per_sm = occupancy_blocks_per_sm((const void*)trace_persistent_kernel<false>, 128);
        trace_persistent_kernel<false><<<sms * (per_sm > 0 ? per_sm : 1), 128, 0, st>>>(
            S, rays, order, n, (int4*)out, nullptr, lights, next, status);
    }
    if (evStop) cudaEventRecord(evStop, st);
    cudaMemsetAsync(next, 0, sizeof(unsigned long long), st);   // the counter is zero between launches
    return (int)cudaGetLastError();
}

bool trace_sorts(long long n, bool any, int tris) { return n >= (any ? kSortAny : sort_closest(tris)); }

int trace_bins() { return bins_of(kCellBits) + kScanBlocks + 1; }   // counters, scan partial sums, block count
}
