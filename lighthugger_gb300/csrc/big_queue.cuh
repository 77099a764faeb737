// Entries of the queue of big triangles (raster_phases.cuh), for host and
// device code.  A triangle's place comes from one 64-bit counter {triangles:
// hi 24, chunks: lo 40}: its index, and the number of its first chunk.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define LH_BQ_HD __host__ __device__ __forceinline__
#else
#define LH_BQ_HD inline
#endif

namespace lh {

constexpr uint32_t kBiasAlpha = 16u;  // TriSetup / BigTri bias: alpha-tested
constexpr uint32_t kBiasWhole = 32u;  // BigTri: taken whole by one warp, not by chunks

// An opaque triangle of at most this many chunks is queued whole (kBiasWhole)
// and adds no chunk.  KIND: the pass (0 visibility, 1 shadow).  One warp takes
// a whole triangle, at the launch's end: two visibility chunks (16 x 128 by
// default) are still one or two set-ups of rows, two shadow chunks (32 x 64) up
// to 4,096 pixels, which kept the cascades' launch waiting for a few warps.
// Shadow raster at limits 0 / 1 / 2 / 3, us: 1080p frame of the benchmark 75.7 /
// 75.8 / 81.9 / 84.0, before walls 210.9 / 186-188 / 192.5 / 211-213, 512 x 512
// training step 172-174 / 155.6 / 161.8 / 176.1; visibility raster at 1 / 2
// before walls: 163.5 / 149.2.  Whole frames at a shadow limit of 1 / 2: 327 / 333,
// 503 / 520, 341 / 351 (training step), 32 probes 1682 / 1690 and, the one that
// loses, 1943 / 1932.
#ifndef LH_WHOLE_CHUNKS
#define LH_WHOLE_CHUNKS 2
#endif
#ifndef LH_SHADOW_WHOLE_CHUNKS
#define LH_SHADOW_WHOLE_CHUNKS 1
#endif
template <int KIND> LH_BQ_HD bool taken_whole(uint64_t n, bool alpha) {
    return n <= (KIND == 0 ? LH_WHOLE_CHUNKS : LH_SHADOW_WHOLE_CHUNKS) && !alpha;
}
// What a triangle of n chunks adds to the counter.
template <int KIND> LH_BQ_HD uint64_t queue_word(uint64_t n, bool alpha) {
    return (1ull << 40) | (taken_whole<KIND>(n, alpha) ? 0ull : n);
}

// Write the entry of a triangle `t` of n chunks whose counter (before its own
// addition) is `old`; false when it does not fit and is dropped.  The chunk
// kernel walks every index the counter has handed out below the capacity, so
// an entry dropped for its chunk number (past 32 bits) is written all the same,
// as one that covers nothing: whole (no chunk is looked up in it), with an
// empty box, and a base above every chunk number so that the bases stay in
// order.  Left as it was, the slot would hold a triangle of an earlier pass.
template <int KIND, class Big, class Setup>
LH_BQ_HD bool store_queue_entry(Big* big, uint32_t* big_base, uint32_t cap, const Setup& t, uint32_t view, uint64_t old,
                                uint64_t n) {
    const uint64_t idx = old >> 40, base = old & ((1ull << 40) - 1);
    if (idx >= cap) return false;
    const bool fits = base + n <= 0xFFFFFFFFull;
    Big e;
    e.X0 = t.X0; e.Y0 = t.Y0; e.X1 = t.X1; e.Y1 = t.Y1; e.X2 = t.X2; e.Y2 = t.Y2;
    e.z0 = t.z0; e.s1 = t.s1; e.s2 = t.s2;
    e.id = t.id;
    e.view = view;
    e.bias = !fits ? kBiasWhole : t.bias | (taken_whole<KIND>(n, t.bias & kBiasAlpha) ? kBiasWhole : 0u);
    e.px0 = t.px0;
    e.px1 = t.px1;
    e.py0 = fits ? t.py0 : 1;
    e.py1 = fits ? t.py1 : 0;
    big[idx] = e;
    big_base[idx] = fits ? (uint32_t)base : 0xFFFFFFFFu;
    return fits;
}

}  // namespace lh
