// Instance cull + single-pass prefix sum that allocates nothing.
//
// Some callers cannot call cudaMalloc: an engine that owns every byte of
// device memory under a fixed budget and forbids hidden allocations, a frame
// loop that must never stall (cudaMalloc can synchronise the whole device),
// or code that records work while a stream is being captured.  This entry
// point serves them: the caller passes the scene and the output sector, and
// the only scratch the kernel needs -- the look-back words of its tiles and
// the tile claim counter -- lives in a fixed array compiled into this library
// (`g_cull_scratch` below, about 8 KB, held by every GPU that loads the
// library until the process exits).
//
// Limits and rules of use:
//  - at most kNoAllocMaxTiles tiles of kCullTile instances (1,048,576
//    instances); larger calls are rejected with LH_ERR_CAPACITY;
//  - a call made outside stream capture looks up the device address of the
//    array (cudaGetSymbolAddress) with the caller's device current and keeps
//    it for that device; a call made while its stream is being captured uses
//    the address kept by the last call outside capture, so make the first
//    call on a device before any stream capture (after a cudaDeviceReset,
//    or under another context, make one call outside capture again);
//  - every call above 4,096 instances shares the one array: calls whose work overlaps on the GPU
//    (different streams, or different host threads) race on it and give
//    wrong results; serialise them;
//  - each call clears the array on its own stream before the kernel runs
//    (calls of at most 4,096 instances run in one cluster and do not use it).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <atomic>
#include <mutex>

#include "cull_phases.cuh"
#include "tma.cuh"

namespace cg = cooperative_groups;

namespace lh {
namespace {

constexpr uint32_t kCullTile = 1024, kNoAllocMaxTiles = 1024, kNoAllocMaxInstances = kCullTile * kNoAllocMaxTiles;
constexpr uint32_t kNoAllocWords = kNoAllocMaxTiles + 32;  // look-back words + the tile claim counter

// The scratch of every call.  Host code must not use `g_cull_scratch`
// directly: on the host it names a stand-in, not the device memory.
static __device__ __align__(256) unsigned long long g_cull_scratch[kNoAllocWords];

constexpr int kMaxDevices = 64;
std::mutex g_setup_mutex;
std::atomic<unsigned long long*> g_scratch_ptr[kMaxDevices];

// Same cull and ordered append as the frame's instance cull
// (cull_instances.comp:7-27 with prefix_sum.glsl:17-30): one instance per
// thread, warp scans, decoupled look-back with bounded waits.
//
// Bound, at the size of an open world (700,001 instances, 78 MB of records: a
// floor of 12 us), by HBM and by the look-back, whose 32 predecessors a step
// cross all tiles in flight: few large tiles.  A tile's records are one bulk
// copy into shared memory (115 KB, 2 blocks a SM), so no thread's 112-byte
// stride reaches the memory system, and a record is read from shared memory
// without bank conflicts (28 words a lane: the 8 lanes of a 16-byte access
// phase start 4 banks apart).  700,001 instances inside a graph: 35 us by tiles
// of 256, 33 by 512, 28 by 1,024 (4,097: 4.4, 4.9 and 5.3); a call by itself 50 to
// 52 with each thread's own loads and a look-back of one predecessor at a time, 35
// to 37.5 now.
__global__ void __launch_bounds__(kCullTile) k_cull_instances_noalloc(const Instance* instances, uint32_t n,
                                                                    const __grid_constant__ Uniforms u, uint8_t* sector,
                                                                    uint32_t capacity, uint32_t* flags_out,
                                                                    unsigned long long* scratch) {
    extern __shared__ __align__(128) unsigned char s_dynamic[];
    Instance* s_inst = reinterpret_cast<Instance*>(s_dynamic);  // [kCullTile]
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ uint64_t s_warp[kCullTile / 32];
    __shared__ uint64_t s_excl;
    __shared__ uint32_t s_tile, s_flags;
    __shared__ SidePlanes s_planes;
    uint64_t* status = reinterpret_cast<uint64_t*>(scratch);  // one word per tile
    unsigned int* claim = reinterpret_cast<unsigned int*>(scratch + kNoAllocMaxTiles);
    if (threadIdx.x == 0) {
        mbar_init(&s_bar, 1);
        mbar_init_fence();
        const uint32_t tile = atomicAdd(claim, 1u);
        s_tile = tile;
        s_flags = 0u;
        if (tile < gridDim.x) {
            const uint32_t bytes = min(n - tile * kCullTile, kCullTile) * (uint32_t)sizeof(Instance);
            mbar_expect_tx(&s_bar, bytes);
            bulk_load(s_inst, instances + (size_t)tile * kCullTile, bytes, &s_bar);
        }
        s_planes = side_planes(u.perspective);
    }
    __syncthreads();
    const uint32_t tile = s_tile;
    if (tile >= gridDim.x) return;  // another call's claims: wrong results, but none out of range
    const uint32_t i = tile * kCullTile + threadIdx.x;
    // (a copy that never lands: reported, the tile counts as empty)
    const bool landed = mbar_wait(&s_bar, 0u);
    if (!landed) atomicOr(&s_flags, LH_FLAG_TIMEOUT);
    bool keep = false;
    uint32_t nm = 0;
    if (landed && i < n) {
        const Instance& inst = s_inst[threadIdx.x];
        const MeshInfoCull mi = load_mesh_info(mesh_info_of(&inst));
        nm = mi.num_meshlets;
        keep = !cull_bounding_sphere(u.initial_view, s_planes, inst.transform, mi.bounding_sphere);
    }
    const uint64_t pay = keep ? ((1ull << 40) | nm) : 0ull;
    const uint64_t incl = warp_incl_scan(pay);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint64_t sum = lane < kCullTile / 32 ? s_warp[lane] : 0ull;
        const uint64_t own = sum;
        sum = warp_incl_scan(sum);
        if (lane < kCullTile / 32) s_warp[lane] = sum - own;
        const uint64_t run = __shfl_sync(0xFFFFFFFFu, sum, kCullTile / 32 - 1);
        const uint64_t excl = lookback_warp(status, tile, run, &s_flags);
        if (lane == 0) {
            s_excl = excl;
            if (tile == gridDim.x - 1) {
                const uint64_t total = excl + run, count = total >> 40;
                *reinterpret_cast<unsigned long long*>(sector) = (count << 32) | (uint32_t)(total & kSum40);
                if (count > capacity) s_flags |= LH_FLAG_INSTANCE_OVERFLOW;
            }
            if (s_flags && flags_out) atomicOr(flags_out, s_flags);
        }
    }
    __syncthreads();
    if (keep) {
        const uint64_t before = s_excl + s_warp[warp] + incl - pay;
        const uint32_t pos = (uint32_t)(before >> 40);
        if (pos < capacity) {
            PrefixSumValue v;
            v.index = i;
            v.sum = (uint32_t)(before & kSum40) + nm;
            reinterpret_cast<PrefixSumValue*>(sector + 8)[pos] = v;
        }
    }
    if (!landed) mbar_wait(&s_bar, 0u);  // the block does not leave a copy behind
}

// The same for at most kSmallInstances instances, by one cluster: its blocks
// pass their totals through shared memory, so nothing has to be cleared first and
// the call is one launch.  Bound by latency and, at one block, by issue (the
// square roots and divisions of 32 warps on one SM): inside a graph 1,024
// instances take 2.3 us by 8 blocks, 4.1 by one, 4.4 cleared and by tiles; 4,096
// take 3.6 and 4,097, by tiles, 5.3.  A call by itself: 4.1 us, 9.2 before.
constexpr uint32_t kSmallBlocks = 8, kSmallThreads = 512, kSmallInstances = kSmallBlocks * kSmallThreads;
__global__ void __cluster_dims__(kSmallBlocks, 1, 1) __launch_bounds__(kSmallThreads) k_cull_instances_noalloc_small(
    const Instance* instances, uint32_t n, const __grid_constant__ Uniforms u, uint8_t* sector, uint32_t capacity,
    uint32_t* flags_out) {
    __shared__ uint64_t s_warp[kSmallThreads / 32];
    __shared__ uint64_t s_block[kSmallBlocks];
    cg::cluster_group cluster = cg::this_cluster();
    cluster.barrier_arrive();  // waited for before the first access to another block's memory
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rank = blockIdx.x;
    const uint32_t i = rank * blockDim.x + threadIdx.x;
    uint64_t pay = 0;
    uint32_t nm = 0;
    if (i < n) {
        const Instance* inst = instances + i;
        lh_mat4 transform;
        const float4* src = reinterpret_cast<const float4*>(inst);
        float4* dst = reinterpret_cast<float4*>(&transform);
#pragma unroll
        for (int c = 0; c < 4; c++) dst[c] = __ldg(src + c);
        const MeshInfoCull mi = load_mesh_info(mesh_info_of(inst));
        nm = mi.num_meshlets;
        if (!cull_bounding_sphere(u.initial_view, side_planes(u.perspective), transform, mi.bounding_sphere))
            pay = (1ull << 40) | nm;
    }
    const uint64_t incl = warp_incl_scan(pay);
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    const uint64_t sums = warp_incl_scan(lane < blockDim.x / 32 ? s_warp[lane] : 0ull);
    const uint64_t own = __shfl_sync(0xffffffffu, sums, 31);
    uint64_t before = __shfl_sync(0xffffffffu, sums, warp ? warp - 1 : 0);
    before = (warp ? before : 0) + incl - pay;
    cluster.barrier_wait();
    if (threadIdx.x < kSmallBlocks) *cluster.map_shared_rank(&s_block[rank], threadIdx.x) = own;
    cluster.sync();
    uint64_t total = 0;
#pragma unroll
    for (uint32_t b = 0; b < kSmallBlocks; b++) {
        if (b == rank) before += total;
        total += s_block[b];
    }
    if (rank == 0 && threadIdx.x == 0) {
        const uint64_t count = total >> 40;
        *reinterpret_cast<unsigned long long*>(sector) = (count << 32) | (uint32_t)(total & kSum40);
        if (count > capacity && flags_out) atomicOr(flags_out, LH_FLAG_INSTANCE_OVERFLOW);
    }
    if (pay) {
        const uint32_t pos = (uint32_t)(before >> 40);
        if (pos < capacity) {
            PrefixSumValue v;
            v.index = i;
            v.sum = (uint32_t)(before & kSum40) + nm;
            reinterpret_cast<PrefixSumValue*>(sector + 8)[pos] = v;
        }
    }
}

// Device address of the scratch array on the current device.  Outside
// stream capture it is looked up on every call (cheap, host side only), so a
// device reset or another current context is picked up; during capture the
// address kept by the last call outside capture on this device is used.
lh_status scratch_for_current_device(cudaStream_t s, unsigned long long** out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return LH_ERR_CUDA;
    if (dev < 0 || dev >= kMaxDevices) return LH_ERR_UNSUPPORTED;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cs) != cudaSuccess) return LH_ERR_CUDA;
    if (cs != cudaStreamCaptureStatusNone) {
        unsigned long long* p = g_scratch_ptr[dev].load(std::memory_order_acquire);
        if (!p) return LH_ERR_UNSUPPORTED;  // no call outside capture on this device yet
        *out = p;
        return LH_OK;
    }
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    void* addr = nullptr;
    if (cudaGetSymbolAddress(&addr, g_cull_scratch) != cudaSuccess || !addr) return LH_ERR_CUDA;
    unsigned long long* p = reinterpret_cast<unsigned long long*>(addr);
    g_scratch_ptr[dev].store(p, std::memory_order_release);
    *out = p;
    return LH_OK;
}

}  // namespace
}  // namespace lh

extern "C" lh_status lh_cull_instances_noalloc(const Instance* d_instances, uint32_t n_instances,
                                               const Uniforms* host_uniforms, uint8_t* d_sector, uint32_t capacity,
                                               uint32_t* d_flags, void* stream) {
    using namespace lh;
    if (!host_uniforms || !d_sector || (n_instances && !d_instances)) return LH_ERR_INVALID_ARGUMENT;
    if (((uintptr_t)d_instances & 15) || ((uintptr_t)d_sector & 7)) return LH_ERR_INVALID_ARGUMENT;
    const uint32_t tiles = (n_instances + kCullTile - 1) / kCullTile;
    if (n_instances > kNoAllocMaxInstances) return LH_ERR_CAPACITY;  // more than 1,048,576 instances
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    unsigned long long* scratch = nullptr;
    lh_status st = scratch_for_current_device(s, &scratch);
    if (st != LH_OK) return st;
    if (n_instances && n_instances <= kSmallInstances) {
        const uint32_t per_block = (n_instances + kSmallBlocks - 1) / kSmallBlocks;
        k_cull_instances_noalloc_small<<<kSmallBlocks, (per_block + 31) & ~31u, 0, s>>>(
            d_instances, n_instances, *host_uniforms, d_sector, capacity, d_flags);
        return cudaGetLastError() == cudaSuccess ? LH_OK : LH_ERR_CUDA;
    }
    // the previous call's look-back words and claim counter must not leak in
    if (cudaMemsetAsync(scratch, 0, sizeof(unsigned long long) * kNoAllocWords, s) != cudaSuccess) return LH_ERR_CUDA;
    if (tiles == 0) {
        if (cudaMemsetAsync(d_sector, 0, 8, s) != cudaSuccess) return LH_ERR_CUDA;
        return LH_OK;
    }
    constexpr uint32_t kShared = kCullTile * (uint32_t)sizeof(Instance);
    if (cudaFuncSetAttribute(k_cull_instances_noalloc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kShared) != cudaSuccess)
        return LH_ERR_CUDA;
    k_cull_instances_noalloc<<<tiles, kCullTile, kShared, s>>>(d_instances, n_instances, *host_uniforms, d_sector, capacity,
                                                        d_flags, scratch);
    return cudaGetLastError() == cudaSuccess ? LH_OK : LH_ERR_CUDA;
}
