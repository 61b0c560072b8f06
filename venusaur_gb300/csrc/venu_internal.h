// venu_internal.h -- host-side internals shared by the library's translation units.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <string>

#include "../../include/venu.h"

namespace venu {

void set_error(const std::string& msg);
venu_status cuda_fail(cudaError_t e, const char* what);

#define VENU_CUDA(call)                                          \
    do {                                                         \
        cudaError_t _e = (call);                                 \
        if (_e != cudaSuccess) return ::venu::cuda_fail(_e, #call); \
    } while (0)

venu_status require_device();  // sm_103 device present and kernels loadable
int sm_count();

// Shared-memory carveout preference: just what `per_sm` resident blocks of
// `kernel` need (static + dynamic + the 1 KB the system reserves per block),
// so that the rest of the SM's unified memory is L1 (the node records and
// spheres stay in L1 longer: RTIOW 1080p x 256 +0.5 %, the batch engine on
// the 64-scene mix +0.3 %).
template <typename K>
cudaError_t prefer_l1(K kernel, int per_sm, size_t dyn) {
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, kernel);
    if (e != cudaSuccess) return e;
    int dev = 0, maxsm = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) != cudaSuccess) return e;
    const size_t need = (size_t)(per_sm > 1 ? per_sm : 1) * (fa.sharedSizeBytes + dyn + 1024);
    const size_t pct = (need * 100 + (size_t)maxsm - 1) / (size_t)maxsm + 1;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)(pct < 100 ? pct : 100));
}

}  // namespace venu

namespace venu {
constexpr uint32_t kTraceWords = 64;  // two for each venu_trace call of a scene that may run without allocating

// How venu_trace runs n rays: blocks of kTraceBlock threads, per_warp rays a warp
// (fewer than 32 while that puts a warp or more on every scheduler); walk: split
// as the renderer's k_traverse, the hits so far in the caller's outputs (both).
// Where the split pays (us without -> with): 1M rays on 20k spheres 636 -> 719, 2M
// on 50k 1472 -> 1512, 2M on 100k 1656 -> 1536, 2M on 200k 1740 -> 1508, 500k on
// 100k 589 -> 549, 250k on 200k 359 -> 360; and its hand-out counter, which each
// warp takes past n once, must not wrap.  64 bits: n + a grid may not fit 32.
constexpr uint32_t kTraceBlock = 128;
constexpr uint32_t kTraceWalkSpheres = 65536, kTraceWalkRays = 1u << 18, kTraceWalkMost = 1u << 31;
struct TracePlan {
    uint32_t per_warp, grid;
    bool walk;
};
inline TracePlan trace_plan(uint32_t spheres, uint32_t n, bool both_outputs, uint32_t sms) {
    TracePlan p;
    p.walk = both_outputs && spheres >= kTraceWalkSpheres && n >= kTraceWalkRays && n <= kTraceWalkMost;
    const uint32_t warps = kTraceBlock / 32u;
    const uint64_t fill = (uint64_t)sms * 4u * warps;
    const uint64_t share = ((uint64_t)n + fill - 1u) / fill;
    p.per_warp = p.walk || share > 32u ? 32u : (uint32_t)share;
    p.grid = (uint32_t)(((uint64_t)n + warps * p.per_warp - 1u) / (warps * p.per_warp));
    return p;
}

// Device memory handed out in stream order and kept for reuse up to `keep`
// bytes (the default pool gives everything back at each synchronisation, and
// mapping it again costs 100 us and more); destroyed with its owner.  What it
// keeps is at most what was freed since the last trim.
struct DevPool {
    cudaMemPool_t pool = nullptr;
    uint64_t keep = 0, freed = 0;
    cudaError_t create(uint64_t keep_bytes) {
        keep = keep_bytes;
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        cudaError_t e = cudaGetDevice(&props.location.id);
        if (e == cudaSuccess) e = cudaMemPoolCreate(&pool, &props);
        if (e == cudaSuccess) e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        return e;
    }
    template <typename T>
    cudaError_t alloc(T** p, size_t bytes, cudaStream_t st) {
        return cudaMallocFromPoolAsync(reinterpret_cast<void**>(p), bytes, pool, st);
    }
    cudaError_t free(void* p, uint64_t bytes, cudaStream_t st) {
        freed += bytes;
        return cudaFreeAsync(p, st);
    }
    uint64_t kept_bound() const { return freed < keep ? freed : keep; }
    uint64_t kept() const {  // the bound, or the unused part of the pool where that is less
        uint64_t reserved = 0, used = 0;
        if (cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
            cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess || used > reserved)
            return kept_bound();
        return reserved - used < kept_bound() ? reserved - used : kept_bound();
    }
    // Gives the unused memory back; the frees must have completed.
    cudaError_t trim() {
        freed = 0;
        return cudaMemPoolTrimTo(pool, 0);
    }
    void destroy() {
        if (pool) cudaMemPoolDestroy(pool);
        pool = nullptr;
    }
};
}  // namespace venu

struct venu_scene {
    uint32_t n = 0;
    void* arena = nullptr;     // the one allocation that holds the buffers below (but the wide tree)
    float4* nodes = nullptr;   // 2 per internal node
    float4* trav = nullptr;    // 4 per internal node: both children (traversal layout)
    float4* sph = nullptr;     // slot order
    float4* mat = nullptr;
    uint32_t* meta = nullptr;  // original id | material << 30
    uint32_t* keys = nullptr;  // sorted Morton codes
    int32_t* parents = nullptr;  // [n-1] parent of each internal node, then [n] of each leaf (for refits)
    uint32_t* arrive = nullptr;  // [n-1] arrival counters of the build and of refits
    uint32_t* trace_err = nullptr;         // [kTraceWords] error word (0 unless one failed) and hand-out counter
                                           // of each venu_trace call
    mutable uint64_t trace_used = 0;       // the pairs in use (a bit each)
    mutable std::mutex trace_mu;
    // The 4-wide traversal tree (lbvh.cu), built on first use by a render
    // with traversal variant 4 or 5 (ensure_wide); a cache of the binary
    // tree, so it may be filled in through a const scene.
    mutable float4* wide = nullptr;      // kWideF4 float4 per wide node
    mutable int32_t* wide_src = nullptr; // kWideChildren per wide node: binary word of each child (for refits)
    mutable uint32_t nwide = 0;
    mutable float wide_ms = 0.0f;        // wall time of the wide tree's collapse
    mutable std::mutex wide_mu;          // serialises that first build
    // venu_scene_update's spheres on their way in: memory that no walk reads, so
    // that renders in flight on other streams never meet anything but records
    // in the traversal records.  Allocated by the first such update.
    venu_sphere* upload = nullptr;
    std::mutex update_mu;         // one upload at a time
    // Refits share the counters, so each waits on the device for the one before
    // it, on whatever stream that ran (refit_done, recorded by the first).  The first
    // build of the wide tree reads the records and waits for them as well.
    cudaEvent_t refit_done = nullptr;
    mutable std::mutex refit_mu;
    float bounds[6] = {0, 0, 0, 0, 0, 0};
    uint32_t nhoist = 0;          // huge spheres tested before traversal
    int32_t hoist[4] = {0, 0, 0, 0};
    float build_ms = 0.0f;
    mutable uint64_t bytes = 0;   // device bytes held (grows when the wide tree is built)
};

namespace venu {
// Builds the LBVH for `n` spheres in device or host memory into `s` (allocates
// its buffers).
venu_status build_scene(const venu_sphere* spheres, bool on_host, uint32_t n, cudaStream_t stream, venu_scene* s);
void free_scene(venu_scene* s);
// Moves the scene's spheres to `spheres` (same count, original order) and
// refits the boxes on `stream` (asynchronous).
venu_status update_scene(venu_scene* s, const venu_sphere* spheres, bool on_host, cudaStream_t stream);
// Builds the scene's 4-wide tree on `stream` unless it exists (blocking: the
// collapse reads each level's size on the host).  Thread-safe.
venu_status ensure_wide(const venu_scene* s, cudaStream_t stream);
DevPool* batch_pool(venu_batch* b);  // its job buffers
}  // namespace venu
