// Kernels of the compute rasteriser; the work itself is in raster_phases.cuh
// (shared with the persistent multi-view kernel).
#include "raster_phases.cuh"

#ifndef LH_RASTER_MIN_BLOCKS
#define LH_RASTER_MIN_BLOCKS 4  // resident blocks of k_raster per SM (registers: 65536 / 256 / this)
#endif
#ifndef LH_RASTER_BIG_MIN_BLOCKS
#define LH_RASTER_BIG_MIN_BLOCKS 4  // the same for the chunk kernel k_raster_big
#endif

namespace lh {
namespace {

// These kernels begin with pdl_wait, not pdl_enter: the next kernel's blocks do
// not become resident while they run.  Their blocks hold most of an SM's
// registers and shared memory and leave at different times, so early blocks of the
// next kernel came to stand unevenly, on SMs whose shared memory was still split for
// this one: by launches the 1080p frame of the benchmark took 359 or 391 us behind
// an L2 flush from one frame to the next, 346 so; back to back 345 -> 332, another
// 327 -> 312, foliage 411 -> 397, 32 probes 1736 -> 1688, none longer.
// The opaque class.  Four resident blocks per SM (64 registers), at three /
// four / five: main + 32 probes 1744 / 1677 / 1720 us, the 4K stress frame 10.12 /
// 9.78 / 10.01 ms; frames of few meshlets are a little better at three (1080p
// before walls 469 / 477 / 493 us, 512 x 512 training step 418 / 430 / 456).
template <int KIND>
__global__ void __launch_bounds__(kRasterWarps * 32, LH_RASTER_MIN_BLOCKS)
    k_raster(const __grid_constant__ FrameDev f, uint32_t view_begin, uint32_t n_views, RasterTune tune, uint32_t list) {
    __shared__ RasterSmemSmall sm;
    pdl_wait();
    phase_raster<KIND>(f, view_begin, n_views, tune, sm, list);
}

// The occluder pass: a few hundred meshlets, each large on screen.
__global__ void __launch_bounds__(kRasterWarps * 32, 3)
    k_raster_occluders(const __grid_constant__ FrameDev f, uint32_t view_begin, uint32_t n_views, RasterTune tune) {
    __shared__ RasterSmem sm;
    pdl_wait();
    phase_raster_general<0, false>(f, view_begin, n_views, tune, sm, nullptr, kListOccluders);
}

// The alpha-clip draw class (double sided, alpha tested).
template <int KIND>
__global__ void __launch_bounds__(kRasterWarps * 32, 3)
    k_raster_alpha(const __grid_constant__ FrameDev f, uint32_t view_begin, uint32_t n_views, RasterTune tune, uint32_t list) {
    __shared__ RasterSmemAlpha sm;
    pdl_wait();
    phase_raster_general<KIND, true>(f, view_begin, n_views, tune, sm, sm.alpha, list);
}

template <int KIND>
__global__ void __launch_bounds__(256, LH_RASTER_BIG_MIN_BLOCKS) k_raster_big(const __grid_constant__ FrameDev f) {
    __shared__ BigSmem sm;
    pdl_wait();
    phase_raster_big<KIND>(f, sm);
}

// Hierarchical depth of the visibility views after the occluder pass.
__global__ void __launch_bounds__(256) k_hiz(FrameDev f, uint32_t view_begin, uint32_t n_views) {
    pdl_wait();
    phase_hiz(f, view_begin, n_views);
}

// Depth test of the other visible meshlets' spheres; survivor lists.
__global__ void __launch_bounds__(256) k_occlusion_filter(FrameDev f, uint32_t view_begin, uint32_t n_views) {
    pdl_wait();
    phase_occlusion_filter(f, view_begin, n_views, (uint64_t)blockIdx.x * blockDim.x + threadIdx.x,
                           (uint64_t)gridDim.x * blockDim.x);
}

}  // namespace

cudaError_t launch_raster_kind(const FrameDev& f, uint32_t view_begin, uint32_t n_views, int kind, uint32_t small_px,
                               uint32_t medium_px, uint32_t raster_batch, cudaStream_t s, int sms) {
    if (n_views == 0) return cudaSuccess;
    if (n_views > kMaxViews) return cudaErrorInvalidValue;
    RasterTune tune{small_px, medium_px, raster_batch};
    // the raster words (clip count, claims, reduce counter, packed
    // big-triangle word) were zeroed by the meshlet cull launched before
    const dim3 rb(kRasterWarps * 32);
    cudaError_t e;
    if (kind == kViewVisibility) {
        auto opaque = [&](uint32_t list) {
            return launch_pdl(k_raster<0>, dim3(sms * LH_RASTER_MIN_BLOCKS), rb, s, f, view_begin, n_views, tune, list);
        };
        const dim3 big_grid(sms * LH_RASTER_BIG_MIN_BLOCKS);
        if (f.occlusion_px) {
            // occluders (and their chunks), hierarchical depth, the depth
            // test of every other meshlet, then the survivors
            e = launch_pdl(k_raster_occluders, dim3(sms * 3), rb, s, f, view_begin, n_views, tune);
            if (e == cudaSuccess) e = launch_pdl(k_raster_big<0>, big_grid, dim3(256), s, f);
            if (e == cudaSuccess) e = launch_pdl(k_hiz, dim3(sms * 4), dim3(256), s, f, view_begin, n_views);
            if (e == cudaSuccess)
                e = launch_pdl(k_occlusion_filter, dim3(sms * 8), dim3(256), s, f, view_begin, n_views);
            if (e == cudaSuccess) e = opaque(kListSurvivors);
            if (e == cudaSuccess && f.scene_alpha)
                e = launch_pdl(k_raster_alpha<0>, dim3(sms * 3), rb, s, f, view_begin, n_views, tune,
                               (uint32_t)kListSurvivors);
        } else {
            e = opaque(kListAll);
            if (e == cudaSuccess && f.scene_alpha)
                e = launch_pdl(k_raster_alpha<0>, dim3(sms * 3), rb, s, f, view_begin, n_views, tune,
                               (uint32_t)kListAll);
        }
        if (e == cudaSuccess) e = launch_pdl(k_raster_big<0>, big_grid, dim3(256), s, f);
    } else {
        e = launch_pdl(k_raster<1>, dim3(sms * LH_RASTER_MIN_BLOCKS), rb, s, f, view_begin, n_views, tune, (uint32_t)kListAll);
        if (e == cudaSuccess && f.scene_alpha)
            e = launch_pdl(k_raster_alpha<1>, dim3(sms * 3), rb, s, f, view_begin, n_views, tune, (uint32_t)kListAll);
        if (e == cudaSuccess) e = launch_pdl(k_raster_big<1>, dim3(sms * LH_RASTER_BIG_MIN_BLOCKS), dim3(256), s, f);
    }
    return e;
}

}  // namespace lh
