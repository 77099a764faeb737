// Compute rasteriser for the visibility buffer and the cascade shadow maps.
//
// Replaces the reference's hardware draws: visbuffer_opaque_vertex/pixel
// (src/shaders/rasterization.glsl:12-58) with depth GREATER / clear 0 /
// back-face culling (src/pipelines.cpp:10-13,67-71,287-300), and
// shadowmap_opaque_vertex (rasterization.glsl:101-111) with depth LESS /
// clear 1 / front-face culling (pipelines.cpp:15-19,73-77,257-270), driven
// by drawIndirectCount over the draw lists (src/rendering.cpp:197-266,
// 325-438).  Alpha-clip draws (visbuffer_alpha_clip_vertex/pixel and
// shadowmap_alpha_clip*, rasterization.glsl:60-97,113-145) are double sided
// (pipelines.cpp:272-285,302-315) and alpha tested per fragment: the base
// texture's alpha, sampled bilinearly at the perspective-correct uv of the
// pixel centre, must not be below 0.5.
//
// Layout of the work:
//  k_raster       one warp per visible meshlet (claimed dynamically across
//                 all views of the launch): the meshlet's <= 64 vertices are
//                 transformed once, snapped to 1/256 px and kept in shared
//                 memory; then one lane per triangle tests whether its box
//                 holds a pixel centre, and the triangles whose box does are
//                 set up and rasterised, one per lane (raster_meshlet_small;
//                 raster_meshlet for clipped, very large or malformed
//                 meshlets).  Triangles covering <= `small` pixel centres are
//                 rasterised by their lane, up to `medium` by the whole warp,
//                 larger ones go to a queue of chunks (tiles of the bbox).
//                 A triangle that needs clipping is clipped by its lane
//                 (Sutherland-Hodgman in clip space against 0 <= z <= w and
//                 the guard band, fan triangulation) into the chunk queue.
//  k_raster_big   one warp per chunk: each row's run of covered pixels
//                 from the three edge functions, the runs walked row by
//                 row or compacted across the warp.
// The depth test is an atomicMax of (depth bits << 32 | packed ID) for the
// visibility buffer and an atomicMin of depth bits for shadow maps, so the
// result does not depend on the order of the work.
#pragma once

#include <type_traits>

#include "edge_run.cuh"
#include "exact_div.cuh"
#include "lh_device.cuh"
#include "lh_internal.cuh"

namespace lh {
namespace {

constexpr int kRasterWarps = 8;

// Most chunks of big triangles a warp claims per atomic, and the share of
// what is left that it claims (build knobs).
#ifndef LH_CHUNK_BATCH
#define LH_CHUNK_BATCH 32
#endif
#ifndef LH_CHUNK_SHIFT
#define LH_CHUNK_SHIFT 32
#endif
#ifndef LH_WHOLE_SHIFT
#define LH_WHOLE_SHIFT 32
#endif

// Upper bound of the warp bin in the shadow pass (0: the tuning's medium_px
// for both passes).  A shadow launch has about one unit per warp, so a warp
// that rasterises a run of 33-128-pixel triangles one after another sets the
// launch's time; sent to the chunk kernel instead, they spread over all
// warps: shadow raster stage 0.099 -> 0.087 ms at 32 (0.096 ms at 64) for the
// four 1024^2 cascades of the 4,096-instance frame.
#ifndef LH_SHADOW_MEDIUM_PX
#define LH_SHADOW_MEDIUM_PX 32
#endif

struct RasterTune {
    uint32_t small_px;   // lane path up to this many bbox pixels
    uint32_t medium_px;  // warp path up to this many; larger: chunk queue
    uint32_t batch;      // meshlets claimed per atomic (0: automatic)
};

// Upper bound of the warp bin in the pass.
template <int KIND>
__device__ __forceinline__ uint32_t medium_bin(RasterTune tune) {
    return KIND == 1 && LH_SHADOW_MEDIUM_PX ? min(tune.medium_px, (uint32_t)LH_SHADOW_MEDIUM_PX) : tune.medium_px;
}

__device__ __forceinline__ const lh_mat4& view_matrix(const FrameDev& f, const ViewDev* vw) {
    return vw->kind == kViewVisibility ? vw->uniforms->combined_perspective_view : f.misc->shadow_matrices[vw->cascade];
}

// Fields of a MeshInfo the raster needs.
struct MeshInfoRaster {
    uint64_t positions, indices, micro_indices, meshlets;
    uint32_t flags;
};
__device__ __forceinline__ MeshInfoRaster load_mesh_info_raster(const MeshInfo* mi) {
    const unsigned long long* w = reinterpret_cast<const unsigned long long*>(mi);
    MeshInfoRaster r;
    r.positions = __ldg(w + 0);
    r.indices = __ldg(w + 1);
    r.micro_indices = __ldg(w + 4);
    r.meshlets = __ldg(w + 5);
    r.flags = (uint32_t)((__ldg(w + 6) >> 16) & 0xFFu);
    return r;
}

// Asynchronous 16-byte copy global -> shared through L2 (cp.async.cg), and
// the wait for the issuing thread's copies.
__device__ __forceinline__ void cp_async16_cg(void* smem, const void* gmem) {
    const uint32_t sa = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ------------------------------------------------------------ alpha clip
// One vertex of an alpha-tested triangle: clip x, y, w and the uv the
// reference's vertex shader forms (uv * texture_scale + texture_offset).
struct AlphaVert {
    float x, y, w, u, v;
};

// Fields of a MeshInfo the alpha test needs.
struct MeshInfoAlpha {
    uint64_t uvs;
    float ts_x, ts_y, to_x, to_y;
    uint32_t tex;
};
__device__ __forceinline__ MeshInfoAlpha load_mesh_info_alpha(const MeshInfo* mi) {
    MeshInfoAlpha r;
    r.uvs = __ldg(&mi->uvs);
    r.ts_x = __ldg(&mi->texture_scale.x);
    r.ts_y = __ldg(&mi->texture_scale.y);
    r.to_x = __ldg(&mi->texture_offset.x);
    r.to_y = __ldg(&mi->texture_offset.y);
    r.tex = __ldg(&mi->base_color_texture_index);
    return r;
}
__device__ __forceinline__ AlphaVert alpha_vert(f4 c, const MeshInfoAlpha& ma, uint32_t flags, uint32_t index) {
    const f2 uv = load_uv_raw(ma.uvs, flags, index);
    return AlphaVert{c.x, c.y, c.w, uv.x * ma.ts_x + ma.to_x, uv.y * ma.ts_y + ma.to_y};
}

// 2D homogeneous edge functions of the unclipped triangle (Olano and Greer,
// "Triangle scan conversion using 2D homogeneous coordinates", 1997):
// E_k(nx, ny) = a_k nx + b_k ny + c_k with (a_k, b_k, c_k) = v_i x v_j for
// (i, j) = (1, 2), (2, 0), (0, 1) over v = (x, y, w); the perspective-correct
// barycentrics are E_k / (E_0 + E_1 + E_2), for clipped triangles too.
struct AlphaTri {
    float a[3], b[3], c[3];
    float u[3], v[3];
    uint32_t tex;
};
__device__ __forceinline__ void alpha_edge(const AlphaVert& p, const AlphaVert& q, float& a, float& b, float& c) {
    a = p.y * q.w - q.y * p.w;
    b = p.w * q.x - q.w * p.x;
    c = p.x * q.y - q.x * p.y;
}
__device__ __forceinline__ AlphaTri alpha_setup(const AlphaVert& v0, const AlphaVert& v1, const AlphaVert& v2,
                                                uint32_t tex) {
    AlphaTri t;
    alpha_edge(v1, v2, t.a[0], t.b[0], t.c[0]);
    alpha_edge(v2, v0, t.a[1], t.b[1], t.c[1]);
    alpha_edge(v0, v1, t.a[2], t.b[2], t.c[2]);
    t.u[0] = v0.u;
    t.u[1] = v1.u;
    t.u[2] = v2.u;
    t.v[0] = v0.v;
    t.v[1] = v1.v;
    t.v[2] = v2.v;
    t.tex = tex;
    return t;
}

// Alpha of the bilinear, repeat-addressed sample of texture `index` at uv.
__device__ __forceinline__ float sample_alpha(const FrameDev& f, uint32_t index, float uvx, float uvy) {
    if (index >= f.n_textures) return 0.0f;
    const lh_texture t = f.textures[index];
    const float4* tex = f.tex_linear[index];
    float u = uvx * (float)t.width - 0.5f, v = uvy * (float)t.height - 0.5f;
    if (!(fabsf(u) < 1e9f)) u = 0.0f;
    if (!(fabsf(v) < 1e9f)) v = 0.0f;
    const float fu = floorf(u), fv = floorf(v);
    const float a = u - fu, b = v - fv;
    const int32_t i0 = (int32_t)fu, j0 = (int32_t)fv, W = (int32_t)t.width, H = (int32_t)t.height;
    // i0 + 1 wraps to the texel after i0's (or 0 past the last)
    const int32_t ia = wrap_texel(i0, W), ib = ia + 1 == W ? 0 : ia + 1;
    const int32_t ja = wrap_texel(j0, H), jb = ja + 1 == H ? 0 : ja + 1;
    auto al = [&](int32_t i, int32_t j) { return __ldg(&tex[(size_t)j * W + i].w); };
    const float t00 = al(ia, ja), t10 = al(ib, ja), t01 = al(ia, jb), t11 = al(ib, jb);
    const float w00 = (1.0f - a) * (1.0f - b), w10 = a * (1.0f - b), w01 = (1.0f - a) * b, w11 = a * b;
    return ((t00 * w00 + t10 * w10) + t01 * w01) + t11 * w11;
}

// (p + 0.5) / n * 2 - 1 of a pixel column or row: the quotient is that of the
// integers 2 p + 1 and 2 n, whose reciprocal rcp_2n = 1 / (2 n) gives the same bits.
__device__ __forceinline__ float pixel_ndc(int32_t p, uint32_t n, float rcp_2n) {
    const float q = 2 * n <= (uint32_t)kExactDivMaxCount ? div_by_count((float)(2 * p + 1), (float)(2 * n), rcp_2n)
                                                         : ((float)p + 0.5f) / (float)n;
    return q * 2.0f - 1.0f;
}

// A target's size as the alpha test reads it.
struct AlphaSize {
    uint32_t W, H;
    float rcp_2w, rcp_2h;
};
__device__ __forceinline__ AlphaSize alpha_size(uint32_t W, uint32_t H) {
    return {W, H, 1.0f / (float)(2 * W), 1.0f / (float)(2 * H)};
}

// True when the fragment at pixel (px, py) survives.
__device__ __forceinline__ bool alpha_pass(const FrameDev& f, const AlphaTri& t, int32_t px, int32_t py, const AlphaSize& s) {
    const float nx = pixel_ndc(px, s.W, s.rcp_2w);
    const float ny = pixel_ndc(py, s.H, s.rcp_2h);
    const float e0 = (t.a[0] * nx + t.b[0] * ny) + t.c[0];
    const float e1 = (t.a[1] * nx + t.b[1] * ny) + t.c[1];
    const float e2 = (t.a[2] * nx + t.b[2] * ny) + t.c[2];
    const float sum = (e0 + e1) + e2;
    const float l0 = e0 / sum, l1 = e1 / sum, l2 = e2 / sum;
    const float u = (l0 * t.u[0] + l1 * t.u[1]) + l2 * t.u[2];
    const float v = (l0 * t.v[0] + l1 * t.v[1]) + l2 * t.v[2];
    return !(sample_alpha(f, t.tex, u, v) < 0.5f);
}

// The alpha set-up of triangle `id` (packed tri / draw slot) of view
// `view`, from the scene buffers (the chunk and clip paths).
__device__ AlphaTri alpha_tri_global(const FrameDev& f, uint32_t view, uint32_t id) {
    const ViewDev* vw = f.views + view;
    const uint32_t slot = id & ((1u << 24) - 1u), tri = id >> 24;
    const MeshletReference ref = vw->refs[slot];
    const Instance* inst = f.instances + ref.instance_index;
    lh_mat4 transform;
    const float4* src = reinterpret_cast<const float4*>(inst);
    float4* dst = reinterpret_cast<float4*>(&transform);
    for (int i = 0; i < 4; i++) dst[i] = __ldg(src + i);
    const MeshInfo* mip = mesh_info_of(inst);
    const MeshInfoRaster mi = load_mesh_info_raster(mip);
    const MeshInfoAlpha ma = load_mesh_info_alpha(mip);
    const Meshlet* ml = reinterpret_cast<const Meshlet*>(mi.meshlets) + ref.meshlet_index;
    const uint32_t tri_off = __ldg(&ml->triangle_offset), idx_off = __ldg(&ml->index_offset);
    const uint8_t* micro = reinterpret_cast<const uint8_t*>(mi.micro_indices) + tri_off + tri * 3;
    const lh_mat4& vp = view_matrix(f, vw);
    AlphaVert av[3];
    for (int k = 0; k < 3; k++) {
        const uint32_t idx = (mi.flags & MESH_INFO_FLAGS_32_BIT_INDICES)
                                 ? __ldg(reinterpret_cast<const uint32_t*>(mi.indices) + idx_off + __ldg(micro + k))
                                 : __ldg(reinterpret_cast<const uint16_t*>(mi.indices) + idx_off + __ldg(micro + k));
        const f3 w = world_pos(transform, load_position(mi.positions, mi.flags, idx));
        av[k] = alpha_vert(mul(vp, f4{w.x, w.y, w.z, 1.0f}), ma, mi.flags, idx);
    }
    return alpha_setup(av[0], av[1], av[2], ma.tex);
}
__device__ __forceinline__ uint32_t load_index_raw(uint64_t indices, uint32_t flags, uint32_t i) {
    if (flags & MESH_INFO_FLAGS_32_BIT_INDICES) return __ldg(reinterpret_cast<const uint32_t*>(indices) + i);
    return __ldg(reinterpret_cast<const uint16_t*>(indices) + i);
}

__device__ __forceinline__ void load_transform(const Instance* inst, lh_mat4& m) {
    const float4* s = reinterpret_cast<const float4*>(inst);
    float4* d = reinterpret_cast<float4*>(&m);
#pragma unroll
    for (int i = 0; i < 4; i++) d[i] = __ldg(s + i);
}

// Append big triangles with 64-bit atomics of {triangles:hi24, chunks:lo40}
// (the packed single-pass append of prefix_sum.glsl:17-30): the triangle's
// index and its first chunk come from the same word, so chunk bases ascend
// with the index and the chunk kernel finds a chunk's triangle by binary search.
// Opaque triangles of one or two chunks are queued whole (taken_whole,
// big_queue.cuh): the chunk kernel takes those by their index, without a
// search (alpha-tested pixels cost several times an opaque one: those stay in
// chunks).  (Entries without chunks keep the search exact: the last entry
// whose base is at most a chunk's number is the one that holds it.)
template <int KIND>
__device__ __forceinline__ unsigned long long box_chunks(const FrameDev& f, uint32_t w, uint32_t h) {  // extents - 1
    return (unsigned long long)((w >> f.chunk_shift[KIND][1]) + 1u) * ((h >> f.chunk_shift[KIND][0]) + 1u);
}
// Store the queue entry of a triangle of n chunks whose packed word (before
// its own addition) is `old`.
template <int KIND>
__device__ void store_big(const FrameDev& f, const TriSetup& t, uint32_t view, unsigned long long old,
                          unsigned long long n) {
    if (!store_queue_entry<KIND>(f.big, f.big_base, f.big_cap, t, view, old, n))
        atomicOr(&f.status[kStFlags], LH_FLAG_QUEUE_OVERFLOW);
}
// One thread's triangle.
template <int KIND>
__device__ void push_big(const FrameDev& f, const TriSetup& t, uint32_t view) {
    const unsigned long long n = box_chunks<KIND>(f, (uint32_t)(t.px1 - t.px0), (uint32_t)(t.py1 - t.py0));
    const unsigned long long old =
        atomicAdd(reinterpret_cast<unsigned long long*>(f.status + kStBigPacked), queue_word<KIND>(n, t.bias & kBiasAlpha));
    store_big<KIND>(f, t, view, old, n);
}
// Called by the whole warp: lanes with n != 0 append their triangle of n
// chunks with one atomic per warp (a warp scan of the lanes' words gives each
// lane the running total below it).  A sum reaching 2^32 chunks is flagged and
// dropped; the word's low 40 bits hold it up to half a million triangles
// that each fill a 16,384 x 16,384 view in the smallest chunks.
template <int KIND>
__device__ __forceinline__ unsigned long long reserve_big_warp(const FrameDev& f, unsigned long long n, bool alpha, uint32_t lane) {
    const unsigned long long mine = n ? queue_word<KIND>(n, alpha) : 0ull;
    unsigned long long incl = mine;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const unsigned long long v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += v;
    }
    unsigned long long old = 0;
    if (lane == 31) old = atomicAdd(reinterpret_cast<unsigned long long*>(f.status + kStBigPacked), incl);
    return __shfl_sync(0xFFFFFFFFu, old, 31) + (incl - mine);
}
template <int KIND>
__device__ void push_big_warp(const FrameDev& f, const TriSetup& t, uint32_t view, bool big, uint32_t lane) {
    const unsigned long long n = big ? box_chunks<KIND>(f, (uint32_t)(t.px1 - t.px0), (uint32_t)(t.py1 - t.py0)) : 0ull;
    const unsigned long long old = reserve_big_warp<KIND>(f, n, t.bias & kBiasAlpha, lane);
    if (big) store_big<KIND>(f, t, view, old, n);
}

// Sutherland-Hodgman against w-z, z, g*w-x, g*w+x, g*w-y, g*w+y >= 0.
__device__ int clip_polygon(f4* poly, int n) {
    f4 out[9];
    for (int plane = 0; plane < 6 && n >= 3; plane++) {
        int m = 0;
        for (int i = 0; i < n; i++) {
            f4 a = poly[i], b = poly[i + 1 < n ? i + 1 : 0];
            float ga = LH_GUARD_BAND * a.w, gb = LH_GUARD_BAND * b.w;
            float da, db;
            switch (plane) {
                case 0: da = a.w - a.z; db = b.w - b.z; break;
                case 1: da = a.z; db = b.z; break;
                case 2: da = ga - a.x; db = gb - b.x; break;
                case 3: da = ga + a.x; db = gb + b.x; break;
                case 4: da = ga - a.y; db = gb - b.y; break;
                default: da = ga + a.y; db = gb + b.y; break;
            }
            if (da >= 0.0f) out[m++] = a;
            if ((da >= 0.0f) != (db >= 0.0f)) {
                float tt = da / (da - db);
                out[m++] = f4{a.x + tt * (b.x - a.x), a.y + tt * (b.y - a.y), a.z + tt * (b.z - a.z), a.w + tt * (b.w - a.w)};
            }
        }
        n = m;
        for (int i = 0; i < n; i++) poly[i] = out[i];
    }
    return n;
}

// Triangle `tri` of the meshlet at draw slot `slot` of view `view`, one of
// whose vertices lies outside 0 <= z <= w, w > 0 or the guard band: clipped
// in clip space, fan-triangulated, the pieces appended to the chunk queue.
// Called by the lane that found it during the raster (rare, so the
// polygon's stack arrays stay out of the raster's register allocation).
template <int KIND>
__device__ __noinline__ void clip_triangle(const FrameDev& f, uint32_t view, uint32_t slot, uint32_t tri) {
    {
        const struct { uint32_t view, slot, tri; } it{view, slot, tri};
        const ViewDev* vw = f.views + it.view;
        const MeshletReference ref = vw->refs[it.slot];
        const Instance* inst = f.instances + ref.instance_index;
        lh_mat4 transform;
        load_transform(inst, transform);
        const MeshInfoRaster mi = load_mesh_info_raster(mesh_info_of(inst));
        MeshletBits mb;
        load_meshlet(reinterpret_cast<const Meshlet*>(mi.meshlets) + ref.meshlet_index, mb);
        const lh_mat4& vp = view_matrix(f, vw);
        const uint8_t* micro = reinterpret_cast<const uint8_t*>(mi.micro_indices) + mb.m.triangle_offset + it.tri * 3;
        const bool alpha = it.slot >= f.max_draws;  // alpha clip: double sided, alpha tested
        f4 poly[9];
        for (int k = 0; k < 3; k++) {
            uint32_t idx = load_index_raw(mi.indices, mi.flags, mb.m.index_offset + micro[k]);
            f3 w = world_pos(transform, load_position(mi.positions, mi.flags, idx));
            poly[k] = mul(vp, f4{w.x, w.y, w.z, 1.0f});
        }
        int np = clip_polygon(poly, 3);
        if (np < 3) return;
        bool projectable = true;  // false only for a triangle through the eye point
        for (int k = 0; k < np; k++) projectable = projectable && poly[k].w > 0.0f;
        if (!projectable) return;
        const uint32_t W = vw->width, H = vw->height;
        const float hw = (float)W * 0.5f, hh = (float)H * 0.5f;
        SnapV s[9];
        for (int k = 0; k < np; k++) s[k] = snap(poly[k], hw, hh);
        int64_t pc = 0;
        for (int k = 0; k < np; k++) {
            const SnapV &a = s[k], &b = s[k + 1 < np ? k + 1 : 0];
            pc += (int64_t)a.X * b.Y - (int64_t)b.X * a.Y;
        }
        if (pc == 0) return;
        if (!alpha && KIND == 0 && pc > 0) return;
        if (!alpha && KIND == 1 && pc < 0) return;
        const uint32_t id = LH_PACK_ID(it.tri, it.slot);
        for (int k = 1; k + 1 < np; k++) {
            SnapV a = s[0], b = s[k], c = s[k + 1];
            int64_t tc = cross3(a, b, c);
            if (tc == 0 || ((tc < 0) != (pc < 0))) continue;
            if (tc > 0) { SnapV tmp = b; b = c; c = tmp; }
            TriSetup st;
            if (make_setup(a, b, c, id, W, H, st)) {
                if (alpha) st.bias |= kBiasAlpha;
                push_big<KIND>(f, st, it.view);
            }
        }
    }
}

// A warp's covered pixels of alpha-tested triangles, waiting for the test.
// The test (three divisions and a bilinear sample, over 100 instructions) is
// taken by 32 covered pixels at a time, of whatever triangles: with the lanes
// testing their own triangles' pixels 14 of 32 were at work.
struct AlphaRing {
    uint32_t tri[64];    // vertices (6 bits each) and triangle of the meshlet
    uint32_t pixel[64];  // x | y << 16
    float depth[64];
};
// Where the warp's alpha-tested triangles find their vertices: its shared
// AlphaVert array (indexed by TriSetup::verts) and the meshlet's base texture.
struct AlphaSrc {
    const AlphaVert* av;
    uint32_t tex, slot;
    AlphaSize size;
};

// The bbox pixels of one triangle by one lane; `nfrag` counts the fragments
// written (depth-test reductions issued).
template <int KIND>
__device__ __forceinline__ void raster_lane(const TriSetup& t, void* target, uint32_t W, uint32_t& nfrag) {
    if (t.bias & 8u) {
        const EdgeSteps es = edge_steps(t);
        for (int32_t ry = 0; ry <= t.py1 - t.py0; ry++)
            for (int32_t rx = 0; rx <= t.px1 - t.px0; rx++) {
                float d;
                if (cover_step(t, es, rx, ry, d)) {
                    write_fragment<KIND>(target, W, t.px0 + rx, t.py0 + ry, d, t.id);
                    nfrag++;
                }
            }
        return;
    }
    for (int32_t py = t.py0; py <= t.py1; py++)
        for (int32_t px = t.px0; px <= t.px1; px++) {
            float d;
            if (cover(t, px, py, d)) {
                write_fragment<KIND>(target, W, px, py, d, t.id);
                nfrag++;
            }
        }
}

// All lanes of a warp cover the pixels of one triangle's bbox.
template <int KIND>
__device__ __forceinline__ void raster_warp(const TriSetup& t, void* target, uint32_t W, uint32_t lane,
                                            uint32_t& nfrag) {
    const uint32_t w = (uint32_t)(t.px1 - t.px0 + 1);
    const uint32_t npx = w * (uint32_t)(t.py1 - t.py0 + 1);
    const float inv_w = 1.0f / (float)w;
    for (uint32_t p = lane; p < npx; p += 32) {
        int32_t ry = (int32_t)(((float)p + 0.5f) * inv_w);
        int32_t rx = (int32_t)p - ry * (int32_t)w;
        if (rx < 0) { ry--; rx += (int32_t)w; }
        else if (rx >= (int32_t)w) { ry++; rx -= (int32_t)w; }
        int32_t px = t.px0 + rx, py = t.py0 + ry;
        float d;
        if (cover(t, px, py, d)) {
            write_fragment<KIND>(target, W, px, py, d, t.id);
            nfrag++;
        }
    }
}

// The ring's entries [first, first + n), n <= 32: tested and written; returns
// the lane's fragments.  Not inlined: the set-up and sampling state stays out
// of the register allocation of the meshlet's loop.
template <int KIND>
__device__ __noinline__ uint32_t alpha_fragments(const FrameDev& f, const AlphaRing& ring, uint32_t first, uint32_t n,
                                                 const AlphaSrc& as, void* target, uint32_t lane) {
    if (lane >= n) return 0u;
    const uint32_t i = (first + lane) & 63u, tri = ring.tri[i], pixel = ring.pixel[i];
    const int32_t px = (int32_t)(pixel & 0xFFFFu), py = (int32_t)(pixel >> 16);
    const AlphaTri at = alpha_setup(as.av[tri & 63u], as.av[(tri >> 6) & 63u], as.av[(tri >> 12) & 63u], as.tex);
    if (!alpha_pass(f, at, px, py, as.size)) return 0u;
    write_fragment<KIND>(target, as.size.W, px, py, ring.depth[i], LH_PACK_ID(tri >> 18, as.slot));
    return 1u;
}

__device__ __forceinline__ TriSetup shfl_setup(const TriSetup& s, int src) {
    TriSetup r;
    const uint32_t* a = reinterpret_cast<const uint32_t*>(&s);
    uint32_t* b = reinterpret_cast<uint32_t*>(&r);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(TriSetup) / 4); i++) b[i] = __shfl_sync(0xFFFFFFFFu, a[i], src);
    return r;
}

// Shared memory of the raster phase (declared by the calling kernel, so that
// the persistent kernel's phases reuse one copy).  The alpha-clip class adds
// AlphaVerts and a ring of pixels per warp (RasterSmemAlpha).
constexpr uint32_t kMicroWords = 4 * 32 * 3 / 4;  // four rounds of 32 triangles (MAX_MESHLET_TRIANGLES and a rest)
// A warp's vertices: absolute (the general path), or packed 16-bit offsets
// from the meshlet's corner (raster_meshlet_small), which needs no outcodes.
union MeshletVerts {
    SnapV v[MAX_MESHLET_UNIQUE_VERTICES];
    struct {
        uint32_t xy[MAX_MESHLET_UNIQUE_VERTICES];
        float z[MAX_MESHLET_UNIQUE_VERTICES];
        uint8_t list[MAX_MESHLET_TRIANGLES + 4];   // triangles whose box holds a pixel centre
        uint8_t large[MAX_MESHLET_TRIANGLES + 4];  // those above the lane bin
    } p;
};
// What the raster needs of a view besides its matrix.
struct ViewTarget {
    void* target;
    uint32_t W, H;
    const RasterDraw* rdraws;
    const uint32_t* list[2];   // by RasterLoop, the pass's slots (null: slots in order)
    uint64_t pad;
};
// The units of one of a launch's loops: the meshlets of its views (or a
// quarter of each), numbered one after another and claimed in batches.
struct RasterWork {
    uint32_t prefix[kMaxViews + 1];
    uint32_t n_units, batch, batch_shift, dyn_base, split_shift;
};
// A launch's two loops: the meshlets of the general path, then the ones
// expected to be small (raster_meshlet_small).
enum RasterLoop : uint32_t { kLoopSmall = 0, kLoopGeneral = 1 };
// A warp's claimed units: batches of at most kMaxBatch, the one in work and
// the next one, whose draw records are copied ahead.
constexpr uint32_t kMaxBatch = 8;
struct RasterUnit {
    uint32_t slot;  // draw slot
    uint32_t info;  // part << 8 | view of the launch
};
// Where the warp is in them, kept in shared memory while it leaves the loop
// over the small meshlets (raster_units).
struct RasterPlace {
    uint32_t i, n;       // next unit of the batch in work, its units
    uint32_t n_next;     // units of the next batch
    uint32_t end;        // one past the last unit claimed
    uint32_t buf;        // buffer of the batch in work
};
static_assert(sizeof(uint8_t[kRasterWarps][MAX_MESHLET_UNIQUE_VERTICES]) + sizeof(MeshletVerts) >= 256 * 4,
              "an 8-bit index from the last warp's vertices stays inside RasterSmem");
struct RasterSmem {
    RasterWork work[2];  // by RasterLoop
    __align__(16) lh_mat4 vp[kMaxViews];
    __align__(16) ViewTarget view[kMaxViews];
    MeshletVerts v[kRasterWarps];
    uint8_t oc[kRasterWarps][MAX_MESHLET_UNIQUE_VERTICES];
    uint32_t micro[kRasterWarps][kMicroWords];
};
struct AlphaSmem {
    AlphaVert av[MAX_MESHLET_UNIQUE_VERTICES];
    AlphaRing ring;
};
static_assert(MAX_MESHLET_UNIQUE_VERTICES <= 64 && MAX_MESHLET_TRIANGLES <= 1 << 14, "AlphaRing::tri");
struct RasterSmemAlpha : RasterSmem {
    AlphaSmem alpha[kRasterWarps];
};
struct RasterSmemSmall : RasterSmem {
    __align__(16) RasterDraw draw[kRasterWarps][2][kMaxBatch];
    RasterUnit unit[kRasterWarps][2][kMaxBatch];
    RasterPlace place[kRasterWarps];
    FrameDev f;  // for raster_meshlet_general (a kernel parameter's address would be read through memory)
};

// One claimed meshlet (or quarter of one) of a view, as the warp works on it.
struct MeshletWork {
    uint32_t view, slot, part, split, nv, nt, W, H;
    void* target;
    float hw, hh;
    const lh_mat4* vp;  // the view's matrix (shared memory)
    lh_mat4 transform;  // the instance's
    MeshInfoRaster mi;
    uint32_t index_offset, triangle_offset;
    const Instance* inst;
};

// The warp's pass over one meshlet: its vertices transformed and snapped into
// shared memory, then one lane per triangle (set-up, face culling, binning).
// ALPHA: the alpha-clip class (double sided, alpha tested per fragment).
template <int KIND, bool ALPHA>
__device__ __forceinline__ void raster_meshlet(const FrameDev& f, const MeshletWork w, RasterTune tune, SnapV* sv,
                                               uint8_t* so, uint32_t* micro_words, AlphaSmem* alpha, uint32_t lane,
                                               uint32_t& nfrag) {
    const uint32_t nv = w.nv, nt = w.nt, W = w.W, H = w.H;
    const MeshInfoRaster& mi = w.mi;
    AlphaSrc as{};
    MeshInfoAlpha ma{};
    if (ALPHA) {
        ma = load_mesh_info_alpha(mesh_info_of(w.inst));
        as = AlphaSrc{alpha->av, ma.tex, w.slot, alpha_size(W, H)};
    }
    // the ring's entries (the same in every lane); a covered pixel joins them,
    // and 32 of them are tested at once
    uint32_t ring_first = 0, ring_n = 0;
    auto join = [&](bool covered, uint32_t tri, int32_t px, int32_t py, float d) {
        const uint32_t mask = __ballot_sync(0xFFFFFFFFu, covered);
        if (covered) {
            const uint32_t i = (ring_first + ring_n + __popc(mask & ((1u << lane) - 1u))) & 63u;
            alpha->ring.tri[i] = tri;
            alpha->ring.pixel[i] = (uint32_t)px | (uint32_t)py << 16;
            alpha->ring.depth[i] = d;
        }
        ring_n += __popc(mask);
        if (ring_n < 32) return;
        __syncwarp();
        nfrag += alpha_fragments<KIND>(f, alpha->ring, ring_first, 32u, as, w.target, lane);
        ring_first = (ring_first + 32u) & 63u;
        ring_n -= 32u;
        __syncwarp();
    };
    // All of the meshlet's global loads are issued before any is used: the
    // micro-index words (at most 3 per lane; 4-byte aligned offsets, as the
    // meshletiser pads them), then both vertex indices of the lane, then both
    // positions -- two dependent round trips instead of seven.
    const uint64_t mbase = mi.micro_indices + w.triangle_offset;
    const uint32_t nbytes = nt * 3, nwords = (nbytes + 3) / 4;
    const bool micro_aligned = (mbase & 3) == 0;
    uint32_t mw[3] = {0u, 0u, 0u};
    if (micro_aligned) {
#pragma unroll
        for (uint32_t k = 0; k < 3; k++) {
            const uint32_t j = lane + 32u * k;
            if (j < nwords) mw[k] = __ldg(reinterpret_cast<const uint32_t*>(mbase) + j);
        }
    }
    const bool v0 = lane < nv, v1 = lane + 32u < nv;
    const uint32_t idx0 = v0 ? load_index_raw(mi.indices, mi.flags, w.index_offset + lane) : 0u;
    const uint32_t idx1 = v1 ? load_index_raw(mi.indices, mi.flags, w.index_offset + lane + 32u) : 0u;
    const f3 pos0 = v0 ? load_position(mi.positions, mi.flags, idx0) : f3{0.0f, 0.0f, 0.0f};
    const f3 pos1 = v1 ? load_position(mi.positions, mi.flags, idx1) : f3{0.0f, 0.0f, 0.0f};
    int32_t min_x = INT32_MAX, max_x = INT32_MIN, min_y = INT32_MAX, max_y = INT32_MIN;
    uint32_t any_oc = 0;
    auto vertex = [&](uint32_t j, uint32_t idx, f3 pos) {
        f3 wp = world_pos(w.transform, pos);
        f4 c = mul(*w.vp, f4{wp.x, wp.y, wp.z, 1.0f});
        uint32_t oc = outcode(c);
        SnapV s{0, 0, 0.0f};
        if (!oc) s = snap(c, w.hw, w.hh);
        sv[j] = s;
        so[j] = (uint8_t)oc;
        any_oc |= oc;
        min_x = min(min_x, s.X);
        max_x = max(max_x, s.X);
        min_y = min(min_y, s.Y);
        max_y = max(max_y, s.Y);
        if (ALPHA) alpha->av[j] = alpha_vert(c, ma, mi.flags, idx);
    };
    if (v0) vertex(lane, idx0, pos0);
    if (v1) vertex(lane + 32u, idx1, pos1);
    // A meshlet whose snapped vertices (all inside the guard band) span no
    // pixel centre produces no fragment: every triangle's bbox lies inside
    // the vertices' bbox.  Common for far meshlets in small views.
    if (nv > 0 && !__any_sync(0xFFFFFFFFu, any_oc != 0)) {
        min_x = __reduce_min_sync(0xFFFFFFFFu, min_x);
        max_x = __reduce_max_sync(0xFFFFFFFFu, max_x);
        min_y = __reduce_min_sync(0xFFFFFFFFu, min_y);
        max_y = __reduce_max_sync(0xFFFFFFFFu, max_y);
        if (max((min_x + 127) >> 8, 0) > min((max_x - 128) >> 8, (int32_t)W - 1) ||
            max((min_y + 127) >> 8, 0) > min((max_y - 128) >> 8, (int32_t)H - 1))
            return;
    }
    if (micro_aligned) {
#pragma unroll
        for (uint32_t k = 0; k < 3; k++) {
            const uint32_t j = lane + 32u * k;
            if (j < nwords) micro_words[j] = mw[k];
        }
    } else {
        uint8_t* d = reinterpret_cast<uint8_t*>(micro_words);
        for (uint32_t j = lane; j < nbytes; j += 32) d[j] = __ldg(reinterpret_cast<const uint8_t*>(mbase) + j);
    }
    __syncwarp();
    const uint8_t* mic = reinterpret_cast<const uint8_t*>(micro_words);
    for (uint32_t base = w.part * 32u; base < nt; base += 32u * w.split) {
        const uint32_t t = base + lane;
        bool small = false, medium = false, big = false;
        TriSetup st;
        if (t < nt) {
            const uint32_t m0 = mic[3 * t], m1 = mic[3 * t + 1], m2 = mic[3 * t + 2];
            if (m0 >= nv || m1 >= nv || m2 >= nv) {
                atomicOr(&f.status[kStFlags], LH_FLAG_BAD_MESHLET);
            } else {
                const uint32_t o0 = so[m0], o1 = so[m1], o2 = so[m2];
                if (((o0 | o1 | o2) & 64u) || (o0 & o1 & o2)) {
                    // non-finite / w <= 0, or entirely outside one plane
                } else if (o0 | o1 | o2) {
                    atomicAdd(&f.status[kStClipCount], 1u);  // statistics only
                    clip_triangle<KIND>(f, w.view, w.slot, t);
                } else {
                    SnapV a = sv[m0], b = sv[m1], c = sv[m2];
                    // most visible triangles hold no pixel centre: the 32-bit
                    // bbox test rejects them before the area.  The box and the
                    // area do not depend on the vertex order, so the set-up
                    // reuses both (make_setup's A is |cr| once oriented).
                    const TriBox box = tri_box(a, b, c, W, H);
                    int64_t cr = box_empty(box) ? 0 : cross_rel(a, b, c);
                    // alpha clip is double sided
                    bool keep = ALPHA ? cr != 0 : (KIND == 0 ? cr < 0 : cr > 0);
                    if (keep) {
                        if (cr > 0) { SnapV tmp = b; b = c; c = tmp; }
                        finish_setup(a, b, c, cr < 0 ? -cr : cr, box, LH_PACK_ID(t, w.slot), st);
                        if (ALPHA) {
                            st.bias |= kBiasAlpha;
                            st.verts = m0 | m1 << 6 | m2 << 12 | t << 18;
                        }
                        uint32_t npx = (uint32_t)(st.px1 - st.px0 + 1) * (uint32_t)(st.py1 - st.py0 + 1);
                        if (npx <= tune.small_px) {
                            if (ALPHA) small = true;  // below, the lanes' pixels together
                            else raster_lane<KIND>(st, w.target, W, nfrag);
                        } else if (npx <= medium_bin<KIND>(tune)) {
                            medium = true;
                        } else {
                            big = true;  // appended below, one atomic per warp
                        }
                    }
                }
            }
        }
        // one atomic per warp on the queue's counter word: shadow views and
        // the occluder pass hold few meshlets with many big triangles each,
        // whose appends would otherwise queue on that one word
        if (__any_sync(0xFFFFFFFFu, big)) push_big_warp<KIND>(f, st, w.view, big, lane);
        if (ALPHA && __any_sync(0xFFFFFFFFu, small)) {
            // each lane walks its triangle's box, all of them in step
            int32_t px = st.px0, py = st.py0;
            EdgeSteps es{};
            if (small && (st.bias & 8u)) es = edge_steps(st);
            do {
                float d = 0.0f;
                const int32_t x = px, y = py;
                bool covered = false;
                if (small) {
                    covered = (st.bias & 8u) ? cover_step(st, es, px - st.px0, py - st.py0, d) : cover(st, px, py, d);
                    if (px++ == st.px1) {
                        px = st.px0;
                        small = py++ != st.py1;
                    }
                }
                join(covered, st.verts, x, y, d);
            } while (__any_sync(0xFFFFFFFFu, small));
        }
        uint32_t mask = __ballot_sync(0xFFFFFFFFu, medium);
        while (mask) {
            int src = __ffs(mask) - 1;
            mask &= mask - 1;
            TriSetup b = shfl_setup(st, src);
            if (ALPHA) {
                const uint32_t bw = (uint32_t)(b.px1 - b.px0 + 1), npx = bw * (uint32_t)(b.py1 - b.py0 + 1);
                uint32_t rx = lane % bw, ry = lane / bw;
                const uint32_t step_x = 32u % bw, step_y = 32u / bw;
                for (uint32_t p = 0; p < npx; p += 32) {
                    float d = 0.0f;
                    const int32_t px = b.px0 + (int32_t)rx, py = b.py0 + (int32_t)ry;
                    join(p + lane < npx && cover(b, px, py, d), b.verts, px, py, d);
                    rx += step_x;
                    ry += step_y;
                    if (rx >= bw) rx -= bw, ry++;
                }
            } else {
                raster_warp<KIND>(b, w.target, W, lane, nfrag);
            }
        }
    }
    __syncwarp();
    if (ALPHA && ring_n) {
        nfrag += alpha_fragments<KIND>(f, alpha->ring, ring_first, ring_n, as, w.target, lane);
        __syncwarp();
    }
}

// A column-major matrix as row pairs: xy[c], zw[c] of column c.
struct Mat2 {
    f32x2 xy[4], zw[4];
};
template <bool GLOBAL>
__device__ __forceinline__ Mat2 load_mat2(const lh_mat4* m) {  // 16-byte aligned
    Mat2 r;
    const ulonglong2* p = reinterpret_cast<const ulonglong2*>(m);
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const ulonglong2 v = GLOBAL ? __ldg(p + c) : p[c];
        r.xy[c] = v.x;
        r.zw[c] = v.y;
    }
    return r;
}

// A meshlet's vertex through the instance and the view: world_pos(transform,
// p), then mul(vp, (world, 1)), in their operation order.
struct World2 {
    f32x2 xy;
    float z;
};
__device__ __forceinline__ World2 world_vertex(const Mat2& t, f3 p, f32x2 nz) {
    const f32x2 px = pack2(p.x, p.x), py = pack2(p.y, p.y), pz = pack2(p.z, p.z);
    World2 w;
    w.xy = add2(mul2(t.xy[0], px, nz), mul2(t.xy[1], py, nz));
    w.xy = add2(add2(w.xy, mul2(t.xy[2], pz, nz)), t.xy[3]);
    float t0, t1, t2, t3, unused;
    unpack2(t.zw[0], t0, unused);
    unpack2(t.zw[1], t1, unused);
    unpack2(t.zw[2], t2, unused);
    unpack2(t.zw[3], t3, unused);
    w.z = ((t0 * p.x + t1 * p.y) + t2 * p.z) + t3;
    return w;
}
struct Clip2 {
    f32x2 xy;
    float z, w;
};
__device__ __forceinline__ Clip2 clip_vertex(const Mat2& vp, const World2& v, f32x2 nz) {
    float wx, wy;
    unpack2(v.xy, wx, wy);
    const f32x2 bx = pack2(wx, wx), by = pack2(wy, wy), bz = pack2(v.z, v.z);
    Clip2 c;
    c.xy = add2(add2(add2(mul2(vp.xy[0], bx, nz), mul2(vp.xy[1], by, nz)), mul2(vp.xy[2], bz, nz)), vp.xy[3]);
    const f32x2 zw = add2(add2(add2(mul2(vp.zw[0], bx, nz), mul2(vp.zw[1], by, nz)), mul2(vp.zw[2], bz, nz)), vp.zw[3]);
    unpack2(zw, c.z, c.w);
    return c;
}
// outcode() == 0, for a w that 256 w cannot overflow (false sends the
// meshlet to the general path, which decides exactly).
__device__ __forceinline__ bool clip_inside(const Clip2& c) {
    float x, y;
    unpack2(c.xy, x, y);
    const float g = LH_GUARD_BAND * c.w;
    return c.w > 0.0f && c.w < 1e30f && c.z >= 0.0f && c.z <= c.w && fabsf(x) <= g && fabsf(y) <= g;
}
// snap() of a vertex inside the guard band.
__device__ __forceinline__ SnapV snap2(const Clip2& c, f32x2 half, f32x2 nz) {
    f32x2 nd = c.xy;
    SnapV s;
    s.z = c.z;
    if (c.w != 1.0f) {
        float x, y;
        unpack2(c.xy, x, y);
        nd = pack2(x / c.w, y / c.w);
        s.z = c.z / c.w;
    }
    float xf, yf;
    unpack2(mul2(add2(mul2(nd, half, nz), half), pack2(256.0f, 256.0f), nz), xf, yf);
    s.X = __float2int_rn(xf);
    s.Y = __float2int_rn(yf);
    return s;
}

enum SmallResult { kSmallGeneral, kSmallNothing, kSmallDone };

// A triangle of a meshlet in packed offsets, ready for coverage: orientation
// normalised, pixel box clamped to the view (pixels from (bx, by)), the
// doubled area, the vertices' depths, and -1 for each edge that is not
// top-left (0 for one that is).
struct SmallTri {
    int32_t ax, ay, bx, by, cx, cy;
    int32_t kx0, kx1, ky0, ky1;
    int32_t A, n12, n20, n01;
    float za, zb, zc;
};
// False when the triangle faces away or its clamped box is empty.
template <int KIND>
__device__ __forceinline__ bool small_tri(const MeshletVerts& mv, const uint8_t* mic, uint32_t t, int32_t bx, int32_t by,
                                          const ViewTarget& vt, SmallTri& s) {
    const uint32_t m0 = mic[3 * t];
    uint32_t m1 = mic[3 * t + 1], m2 = mic[3 * t + 2];
    if (KIND == 1) {  // kept with a positive area: orientation normalised
        const uint32_t x = m1;
        m1 = m2;
        m2 = x;
    }
    const uint32_t a = mv.p.xy[m0], b = mv.p.xy[m1], c = mv.p.xy[m2];
    s.ax = (int32_t)(a & 0xFFFFu), s.ay = (int32_t)(a >> 16);
    s.bx = (int32_t)(b & 0xFFFFu), s.by = (int32_t)(b >> 16);
    s.cx = (int32_t)(c & 0xFFFFu), s.cy = (int32_t)(c >> 16);
    // doubled area: differences below 2^15, so 32 bits hold it
    s.A = (s.cx - s.ax) * (s.by - s.ay) - (s.bx - s.ax) * (s.cy - s.ay);
    const uint32_t lo = __vimin3_u16x2(a, b, c) + 0x00FF00FFu, hi = __vimax3_u16x2(a, b, c);
    s.kx0 = max((int32_t)((lo >> 8) & 0xFFu), -bx), s.kx1 = min((int32_t)((hi >> 8) & 0xFFu), (int32_t)vt.W - 1 - bx);
    s.ky0 = max((int32_t)(lo >> 24), -by), s.ky1 = min((int32_t)(hi >> 24), (int32_t)vt.H - 1 - by);
    if (s.A <= 0 || s.kx0 > s.kx1 || s.ky0 > s.ky1) return false;
    s.za = mv.p.z[m0], s.zb = mv.p.z[m1], s.zc = mv.p.z[m2];
    // top-left (dy > 0, or dy == 0 and dx < 0) is 65536 dy - dx > 0 for
    // differences below 2^15; the words' difference is 65536 dy + dx
    s.n12 = ((int32_t)(c - b) - 2 * (s.cx - s.bx) - 1) >> 31;
    s.n20 = ((int32_t)(a - c) - 2 * (s.ax - s.cx) - 1) >> 31;
    s.n01 = ((int32_t)(b - a) - 2 * (s.bx - s.ax) - 1) >> 31;
    return true;
}

// The triangles of a small meshlet above the lane bin (mv.p.large): the warp
// bin, or the chunk queue.  Set-ups are formed from shared memory where they
// are used -- at the queue entry, or by every lane of the warp bin -- so
// none is held across the warp's scan and atomic.
template <int KIND>
__device__ __forceinline__ void setup_of(const SmallTri& s, uint32_t t, uint32_t slot, int32_t bx, int32_t by, TriSetup& st) {
    const int32_t ox = bx * 256 + 128, oy = by * 256 + 128;
    st.X0 = s.ax + ox; st.Y0 = s.ay + oy;
    st.X1 = s.bx + ox; st.Y1 = s.by + oy;
    st.X2 = s.cx + ox; st.Y2 = s.cy + oy;
    st.z0 = s.za;
    const float fA = __int2float_rn(s.A);
    st.s1 = (s.zb - s.za) / fA;
    st.s2 = (s.zc - s.za) / fA;
    st.id = LH_PACK_ID(t, slot);
    st.px0 = s.kx0 + bx; st.px1 = s.kx1 + bx;
    st.py0 = s.ky0 + by; st.py1 = s.ky1 + by;
    st.bias = (uint32_t)((s.n12 & 1) | (s.n20 & 2) | (s.n01 & 4)) | 8u;  // products fit 32 bits
    st.verts = 0;
}
template <int KIND>
__device__ __forceinline__ uint32_t raster_large(const FrameDev& f, const MeshletVerts& mv, const uint8_t* mic, uint32_t n,
                                                 int32_t bx, int32_t by, const ViewTarget& vt, uint32_t view,
                                                 uint32_t slot, uint32_t medium_px, uint32_t lane) {
    uint32_t nfrag = 0;
    for (uint32_t base = 0; base < n; base += 32u) {
        bool medium = false;
        unsigned long long chunks = 0;
        if (base + lane < n) {
            SmallTri s;
            small_tri<KIND>(mv, mic, mv.p.large[base + lane], bx, by, vt, s);
            const uint32_t w = (uint32_t)(s.kx1 - s.kx0), h = (uint32_t)(s.ky1 - s.ky0);
            medium = (w + 1u) * (h + 1u) <= medium_px;
            if (!medium) chunks = box_chunks<KIND>(f, w, h);
        }
        if (__any_sync(0xFFFFFFFFu, chunks != 0)) {
            const unsigned long long old = reserve_big_warp<KIND>(f, chunks, false, lane);
            if (chunks) {
                const uint32_t t = mv.p.large[base + lane];
                SmallTri s;
                small_tri<KIND>(mv, mic, t, bx, by, vt, s);
                TriSetup st;
                setup_of<KIND>(s, t, slot, bx, by, st);
                store_big<KIND>(f, st, view, old, chunks);
            }
        }
        uint32_t mask = __ballot_sync(0xFFFFFFFFu, medium);
        while (mask) {
            const uint32_t t = mv.p.large[base + __ffs(mask) - 1];
            mask &= mask - 1;
            SmallTri s;
            small_tri<KIND>(mv, mic, t, bx, by, vt, s);
            TriSetup st;
            setup_of<KIND>(s, t, slot, bx, by, st);
            raster_warp<KIND>(st, vt.target, vt.W, lane, nfrag);
        }
    }
    __syncwarp();
    return nfrag;
}

// The opaque meshlets that make up nearly all of a view: every vertex inside
// the clip volume and the guard band, the snapped vertices within 127 pixels
// of each other, micro indices 4-byte aligned and in range.  Returns false,
// with nothing written, for any other (raster_meshlet takes those).
//
// What bounds the general path on such a meshlet is instruction issue spent
// on triangles that hold no pixel centre (4 to 15 fragments per 124
// triangles in views from the air, in probes and in cascades): 32-bit
// gathers of three vertices per triangle, a box in 32-bit lanes, and set-up
// and pixel loop run once per 32 triangles for the two or three lanes left.
// Here a vertex is one 32-bit word -- 16-bit offsets from a pixel centre at
// the meshlet's corner -- so a triangle's box test is three shared loads and
// a handful of two-lane integer instructions, the triangles whose box holds
// a centre are listed, and set-up and pixels run once over the list.  All
// edge arithmetic is translation invariant and fits 32 bits (extents below
// 2^15: products below 2^30), so coverage and depth are those of the general
// path bit for bit.  Warp instructions a meshlet 1,349 -> 876 in a main view
// from the air (198,000 meshlets, 15 fragments each: 336 -> 195 us), 962 ->
// 592 in its cascades (440,000, 4 fragments each: 508 -> 282 us); now bound by
// issue (75 %), about a third of it set-up and pixels.
// `ahead` is called once, by the whole warp, when the vertices' loads are
// done with, `copy` before the pixels (unless the return comes first): the
// warp's next unit starts its way to the draw record behind this one's work.
template <int KIND, class Ahead, class Copy>
__device__ __forceinline__ SmallResult raster_meshlet_small(const FrameDev& f, const RasterDraw& rd, uint32_t view,
                                                            uint32_t slot, uint32_t part, uint32_t split,
                                                            const ViewTarget& vt, const lh_mat4* vp, RasterTune tune,
                                                            MeshletVerts& mv, uint32_t* micro_words, uint32_t lane,
                                                            uint32_t& nfrag, Ahead ahead, Copy copy) {
    const uint32_t nv = rd.bits & 0xFFu, nt = (rd.bits >> 8) & 0xFFu, flags = rd.bits >> 16;
    // every load of the meshlet issued before any is used (the formats'
    // branches below end what the compiler can move up)
    const Mat2 t = load_mat2<true>(&f.instances[rd.instance].transform);
    const uint32_t nwords = (nt * 3 + 3) / 4;
    uint32_t mw[3] = {0u, 0u, 0u};
#pragma unroll
    for (uint32_t k = 0; k < 3; k++) {
        const uint32_t j = lane + 32u * k;
        if (j < nwords) mw[k] = __ldg(reinterpret_cast<const uint32_t*>(rd.micro) + j);
    }
    // lanes past the last vertex repeat it
    const uint32_t j0 = min(lane, nv - 1u), j1 = min(lane + 32u, nv - 1u);
    uint32_t idx0, idx1;
    if (flags & MESH_INFO_FLAGS_32_BIT_INDICES) {
        idx0 = __ldg(reinterpret_cast<const uint32_t*>(rd.indices) + j0);
        idx1 = __ldg(reinterpret_cast<const uint32_t*>(rd.indices) + j1);
    } else {
        idx0 = __ldg(reinterpret_cast<const uint16_t*>(rd.indices) + j0);
        idx1 = __ldg(reinterpret_cast<const uint16_t*>(rd.indices) + j1);
    }
    f3 pos0, pos1;
    if (flags & MESH_INFO_FLAGS_FP32_VERTICES) {
        pos0 = load_position(rd.positions, MESH_INFO_FLAGS_FP32_VERTICES, idx0);
        pos1 = load_position(rd.positions, MESH_INFO_FLAGS_FP32_VERTICES, idx1);
    } else {
        pos0 = load_position(rd.positions, 0u, idx0);
        pos1 = load_position(rd.positions, 0u, idx1);
    }
    int32_t X0, Y0, X1, Y1;
    float z0, z1;
    {
        const World2 w0 = world_vertex(t, pos0, f.neg_zero2), w1 = world_vertex(t, pos1, f.neg_zero2);
        const Mat2 m = load_mat2<false>(vp);
        const Clip2 c0 = clip_vertex(m, w0, f.neg_zero2), c1 = clip_vertex(m, w1, f.neg_zero2);
        // a micro index of nv or more (nv <= 64: the byte sums do not carry)
        const uint32_t lim = (128u - nv) * 0x01010101u;
        uint32_t bad = 0;
#pragma unroll
        for (uint32_t k = 0; k < 3; k++) bad |= ((mw[k] & 0x7F7F7F7Fu) + lim) | mw[k];
        ahead();
        if (!__all_sync(0xFFFFFFFFu, clip_inside(c0) && clip_inside(c1) && !(bad & 0x80808080u))) return kSmallGeneral;
        const f32x2 half = pack2((float)vt.W * 0.5f, (float)vt.H * 0.5f);
        const SnapV s0 = snap2(c0, half, f.neg_zero2), s1 = snap2(c1, half, f.neg_zero2);
        X0 = s0.X, Y0 = s0.Y, z0 = s0.z;
        X1 = s1.X, Y1 = s1.Y, z1 = s1.z;
    }
    const int32_t min_x = __reduce_min_sync(0xFFFFFFFFu, min(X0, X1)), max_x = __reduce_max_sync(0xFFFFFFFFu, max(X0, X1));
    const int32_t min_y = __reduce_min_sync(0xFFFFFFFFu, min(Y0, Y1)), max_y = __reduce_max_sync(0xFFFFFFFFu, max(Y0, Y1));
    // no pixel centre in the vertices' box: no fragment
    if (max((min_x + 127) >> 8, 0) > min((max_x - 128) >> 8, (int32_t)vt.W - 1) ||
        max((min_y + 127) >> 8, 0) > min((max_y - 128) >> 8, (int32_t)vt.H - 1))
        return kSmallNothing;
    // offsets from the centre of pixel (bx, by), at or before the corner
    const int32_t bx = (min_x - 128) >> 8, by = (min_y - 128) >> 8;
    const int32_t ox = bx * 256 + 128, oy = by * 256 + 128;
    if (max_x - ox > 0x7FFF || max_y - oy > 0x7FFF) return kSmallGeneral;
    mv.p.xy[lane] = (uint32_t)(X0 - ox) | ((uint32_t)(Y0 - oy) << 16);
    mv.p.xy[lane + 32u] = (uint32_t)(X1 - ox) | ((uint32_t)(Y1 - oy) << 16);
    mv.p.z[lane] = z0;
    mv.p.z[lane + 32u] = z1;
#pragma unroll
    for (uint32_t k = 0; k < 3; k++) {
        const uint32_t j = lane + 32u * k;
        if (j < nwords) micro_words[j] = mw[k];
    }
    __syncwarp();
    const uint8_t* mic = reinterpret_cast<const uint8_t*>(micro_words);
    const uint32_t lanes_below = (1u << lane) - 1u;
    // the triangles whose box holds a pixel centre: offsets of centres are
    // multiples of 256, so the first column is ceil(min / 256), the last
    // floor(max / 256), both axes at once in the two halves of a word
    uint32_t n = 0;
    const uint8_t* tri = mic + 3u * (part * 32u + lane);
    for (uint32_t base = part * 32u; base < nt; base += 32u * split, tri += 96u * split) {
        const uint32_t t = base + lane;
        // (lanes past the last triangle gather at whatever bytes an earlier
        // meshlet left, inside the block's arrays, and drop the outcome)
        const uint32_t a = mv.p.xy[tri[0]], b = mv.p.xy[tri[1]], c = mv.p.xy[tri[2]];
        const uint32_t first = __byte_perm(__vimin3_u16x2(a, b, c) + 0x00FF00FFu, 0u, 0x4341);
        const uint32_t last = __byte_perm(__vimax3_u16x2(a, b, c), 1u, 0x4341);  // 256 + last
        const bool hit = t < nt && (~(last - first) & 0x01000100u) == 0u;
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, hit);
        if (hit) mv.p.list[n + __popc(m & lanes_below)] = (uint8_t)t;
        n += __popc(m);
    }
    __syncwarp();
    copy();
    uint32_t n_large = 0;
    for (uint32_t base = 0; base < n; base += 32u) {
        bool large = false;
        uint32_t t = 0;
        if (base + lane < n) {
            t = mv.p.list[base + lane];
            SmallTri s;
            if (small_tri<KIND>(mv, mic, t, bx, by, vt, s)) {
                const int32_t w = s.kx1 - s.kx0 + 1, npx = w * (s.ky1 - s.ky0 + 1);
                large = (uint32_t)npx > tune.small_px;
                if (!large) {
                    const float fA = __int2float_rn(s.A);
                    const float s1 = (s.zb - s.za) / fA, s2 = (s.zc - s.za) / fA;
                    const uint32_t id = LH_PACK_ID(t, slot);
                    // edge values less their bias at the box's first pixel,
                    // stepped along the rows (the three edge functions sum
                    // to the doubled area, their steps to zero)
                    const int32_t Px = s.kx0 * 256, Py = s.ky0 * 256;
                    int32_t e12 = (s.cy - s.by) * (Px - s.bx) - (s.cx - s.bx) * (Py - s.by);
                    int32_t e20 = (s.ay - s.cy) * (Px - s.cx) - (s.ax - s.cx) * (Py - s.cy);
                    // (unsigned: a sum on the way may wrap)
                    int32_t e01 = (int32_t)((uint32_t)s.A - (uint32_t)e12 - (uint32_t)e20 + (uint32_t)s.n01);
                    e12 += s.n12;
                    e20 += s.n20;
                    const int32_t x12 = (s.cy - s.by) * 256, x20 = (s.ay - s.cy) * 256;
                    const int32_t r12 = (s.bx - s.cx) * 256 - (w - 1) * x12, r20 = (s.cx - s.ax) * 256 - (w - 1) * x20;
                    uint32_t pix = (uint32_t)(s.ky0 + by) * vt.W + (uint32_t)(s.kx0 + bx);
                    const uint32_t row_step = vt.W - (uint32_t)w + 1u;
                    int32_t left = w;
                    for (int32_t k = npx; k > 0; k--) {
                        if ((e12 | e20 | e01) >= 0) {
                            const float d = (s.za + __int2float_rn(e20 - s.n20) * s1) + __int2float_rn(e01 - s.n01) * s2;
                            // clamped to [0, 1], NaN and -0 to +0
                            write_pixel<KIND>(vt.target, pix, fminf(fmaxf(d, 0.0f), 1.0f), id);
                            nfrag++;
                        }
                        const bool row = --left == 0;
                        left = row ? w : left;
                        pix += row ? row_step : 1u;
                        // (unsigned: the step past the last pixel may wrap)
                        const uint32_t d12 = (uint32_t)(row ? r12 : x12), d20 = (uint32_t)(row ? r20 : x20);
                        e12 = (int32_t)((uint32_t)e12 + d12);
                        e20 = (int32_t)((uint32_t)e20 + d20);
                        e01 = (int32_t)((uint32_t)e01 - d12 - d20);
                    }
                }
            }
        }
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, large);
        if (large) mv.p.large[n_large + __popc(m & lanes_below)] = (uint8_t)t;
        n_large += __popc(m);
    }
    __syncwarp();
    if (n_large) nfrag += raster_large<KIND>(f, mv, mic, n_large, bx, by, vt, view, slot, medium_bin<KIND>(tune), lane);
    return kSmallDone;
}

// A unit of the small loop that raster_meshlet_small leaves: not inlined, so
// its 64-bit state stays out of the small path's registers.  Returns the
// fragments the lane wrote.
template <int KIND>
__device__ __noinline__ uint32_t raster_meshlet_general(RasterSmemSmall& sm, uint32_t view_begin, uint32_t buf, uint32_t i,
                                                        RasterTune tune) {
    const FrameDev& f = sm.f;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const RasterDraw rd = sm.draw[warp][buf][i];
    const RasterUnit un = sm.unit[warp][buf][i];
    const uint32_t v = un.info & 0xFFu, part = un.info >> 8;
    const ViewTarget vt = sm.view[v];
    MeshletWork w;
    w.view = view_begin + v, w.slot = un.slot, w.part = part, w.split = 1u << sm.work[kLoopSmall].split_shift;
    w.nv = rd.bits & 0xFFu, w.nt = (rd.bits >> 8) & 0xFFu;
    if (w.nv > MAX_MESHLET_UNIQUE_VERTICES || w.nt > MAX_MESHLET_TRIANGLES) {
        // beyond the meshletiser limits: malformed, skipped and flagged
        if (lane == 0 && part == 0) atomicOr(&f.status[kStFlags], LH_FLAG_BAD_MESHLET);
        return 0u;
    }
    // a quarter without triangles, or no pixel centre in reach of the sphere
    if (part * 32u >= w.nt || (rd.bits & kDrawNoCentre)) return 0u;
    w.W = vt.W, w.H = vt.H;
    w.target = vt.target;
    w.hw = (float)vt.W * 0.5f, w.hh = (float)vt.H * 0.5f;
    w.vp = &sm.vp[v];
    w.inst = f.instances + rd.instance;
    load_transform(w.inst, w.transform);
    w.mi = MeshInfoRaster{rd.positions, rd.indices, rd.micro, 0, rd.bits >> 16};
    w.index_offset = w.triangle_offset = 0;
    uint32_t nfrag = 0;
    raster_meshlet<KIND, false>(f, w, tune, sm.v[warp].v, sm.oc[warp], sm.micro[warp], nullptr, lane, nfrag);
    return nfrag;
}

// Adds the warp's fragment count to the frame's statistics word of the
// pass (visibility or shadow views); called by every lane of the warp.
template <int KIND>
__device__ __forceinline__ void count_fragments(const FrameDev& f, uint32_t nfrag) {
    const uint32_t total = __reduce_add_sync(0xFFFFFFFFu, nfrag);
    if ((threadIdx.x & 31) == 0 && total) atomicAdd(&f.status[KIND == 0 ? kStFragVis : kStFragShadow], total);
}

// Meshlets of view `vw` one of a raster pass's loops covers: every visible
// one of the class (kListAll; the general loop the listed ones), or the
// entries of an occlusion list.  Occluders are on the general path: large on
// screen by definition.
__device__ __forceinline__ uint32_t raster_list_count(const FrameDev& f, const ViewDev* vw, bool alpha, uint32_t list,
                                                      RasterLoop loop) {
    if (loop == kLoopSmall && (alpha || list == kListOccluders)) return 0u;
    if (list == kListAll && (alpha || loop == kLoopSmall))
        return min(reinterpret_cast<const uint32_t*>(vw->draws)[alpha ? 1 : 0], f.max_draws);
    const uint32_t w = list == kListOccluders ? kClaimOccluders
                       : alpha ? kClaimSurvivorsAlpha : loop == kLoopGeneral ? kClaimGeneral : kClaimSurvivorsOpaque;
    return min(*reinterpret_cast<const volatile uint32_t*>(&vw->claim[w]), f.max_draws);
}
__device__ __forceinline__ const uint32_t* raster_list(const FrameDev& f, const ViewDev* vw, bool alpha, uint32_t list,
                                                       RasterLoop loop) {
    if (list == kListAll && (alpha || loop == kLoopSmall)) return nullptr;
    const uint32_t k = list == kListOccluders ? kSlotsOccluders
                       : alpha ? kSlotsAlpha : loop == kLoopGeneral ? kSlotsGeneral : kSlotsOpaque;
    return vw->lists + (size_t)k * f.max_draws;
}

// A warp's way through its units.
//
// A unit's way to its vertices is a chain of dependent loads (claim, list
// entry, draw record, indices, positions); the first three steps of the next
// batch run behind the last unit of the one in work: the claim is issued
// when that unit starts, the slots are read (a lane per unit) after its
// vertices, and the draw records are copied to shared memory (cp.async)
// before its pixels are written.
//
// Claims shrink as the units run out (guided self-scheduling): a warp claims
// 1 / 4 to 1 / 8 of an even share of what its last claim left, at most
// kMaxBatch units.  Every claim is an atomic on one word, which the L2 serves
// about 1.4 times a nanosecond: a unit per claim bounds a launch of 440,000
// meshlets at 300 us, whatever its work.
__device__ __forceinline__ uint32_t units_batch(uint32_t fixed, uint32_t left, uint32_t shift) {
    return min(fixed ? fixed : max(left >> shift, 1u), kMaxBatch);
}
// The claim of the batch after the one that ends at `end` (lane 0's value).
__device__ __forceinline__ uint32_t claim_batch(const RasterWork& k, uint32_t end, uint32_t* claim_word, uint32_t lane) {
    uint32_t got = 0;
    if (lane == 0 && k.dyn_base < k.n_units) got = atomicAdd(claim_word, units_batch(k.batch, k.n_units - end, k.batch_shift));
    return got;
}
// The lane's unit (first + lane): its view and slot.  A lane's units only
// increase, so the view search starts at its previous unit's view.
__device__ __forceinline__ RasterUnit unit_of(const RasterSmem& sm, RasterLoop loop, uint32_t first_slot, uint32_t unit, uint32_t& v) {
    const RasterWork& k = sm.work[loop];
    const uint32_t item = unit >> k.split_shift, part = unit & ((1u << k.split_shift) - 1u);
    while (item >= k.prefix[v + 1]) v++;
    const uint32_t local = item - k.prefix[v];
    const uint32_t* slots = sm.view[v].list[loop];
    return RasterUnit{slots ? __ldcg(slots + local) : first_slot + local, (part << 8) | v};
}
// The batch claimed as `claimed`: its units (0 when they have run out).
__device__ __forceinline__ uint32_t take_batch(const RasterSmem& sm, RasterLoop loop, uint32_t first_slot, uint32_t claimed,
                                               uint32_t& end, uint32_t lane, uint32_t& v, RasterUnit& mine) {
    const RasterWork& k = sm.work[loop];
    const uint32_t units = k.n_units, dyn_base = k.dyn_base;
    if (dyn_base >= units) return 0u;
    const uint32_t first = dyn_base + __shfl_sync(0xFFFFFFFFu, claimed, 0);
    if (first >= units) return 0u;
    const uint32_t n = min(units_batch(k.batch, units - end, k.batch_shift), units - first);  // as claim_batch
    end = first + n;
    if (lane < n) mine = unit_of(sm, loop, first_slot, first + lane, v);
    return n;
}
// The warp's static first window of a loop's units (warp g of the grid takes
// the g-th batch; the claim word hands out the rest from there on, so
// launches with fewer units than warps touch it not at all, and none start
// with every warp queueing on it).
__device__ __forceinline__ void first_window(const RasterWork& k, uint32_t gwarp, uint32_t& unit, uint32_t& end) {
    const uint32_t b = units_batch(k.batch, k.n_units, k.batch_shift);
    unit = min(gwarp * b, k.n_units);
    end = min(gwarp * b + b, k.n_units);
}

// Meshlets on the general path: the alpha-clip class, the occluders, and
// what the cull and the occlusion filter listed as kDrawGeneral.
template <int KIND, bool ALPHA>
__device__ __forceinline__ void raster_general_units(const FrameDev& f, uint32_t view_begin, RasterTune tune, uint32_t* claim_word,
                                                     RasterSmem& sm, AlphaSmem* alpha, uint32_t gwarp, uint32_t warp, uint32_t lane,
                                                     uint32_t& nfrag) {
    const RasterWork& work = sm.work[kLoopGeneral];
    const uint32_t first_slot = ALPHA ? f.max_draws : 0u;
    uint32_t unit, end, v_lane = 0;
    first_window(work, gwarp, unit, end);
    RasterUnit mine{0u, 0u}, next{0u, 0u};
    uint32_t n = end - unit;
    if (lane < n) mine = unit_of(sm, kLoopGeneral, first_slot, unit + lane, v_lane);
    while (n) {
        const uint32_t claimed = claim_batch(work, end, claim_word, lane);
        for (uint32_t i = 0; i < n; i++) {
            const uint32_t slot = __shfl_sync(0xFFFFFFFFu, mine.slot, i), info = __shfl_sync(0xFFFFFFFFu, mine.info, i);
            const uint32_t v = info & 0xFFu, part = info >> 8;
            const RasterDraw rd = sm.view[v].rdraws[slot];
            const Instance* inst = f.instances + rd.instance;
            lh_mat4 transform;
            load_transform(inst, transform);
            const uint32_t nv = rd.bits & 0xFFu, nt = (rd.bits >> 8) & 0xFFu;
            if (nv > MAX_MESHLET_UNIQUE_VERTICES || nt > MAX_MESHLET_TRIANGLES) {
                // beyond the meshletiser limits: malformed, skipped and flagged
                if (lane == 0 && part == 0) atomicOr(&f.status[kStFlags], LH_FLAG_BAD_MESHLET);
                continue;
            }
            if (part * 32u >= nt || (rd.bits & kDrawNoCentre)) continue;
            const uint32_t W = sm.view[v].W, H = sm.view[v].H;
            const MeshInfoRaster mi{rd.positions, rd.indices, rd.micro, 0, rd.bits >> 16};
            const MeshletWork w{view_begin + v, slot, part, 1u << work.split_shift, nv, nt, W, H, sm.view[v].target, (float)W * 0.5f,
                                (float)H * 0.5f, &sm.vp[v], transform, mi, 0u, 0u, inst};
            raster_meshlet<KIND, ALPHA>(f, w, tune, sm.v[warp].v, sm.oc[warp], sm.micro[warp], alpha, lane, nfrag);
        }
        n = take_batch(sm, kLoopGeneral, first_slot, claimed, end, lane, v_lane, next);
        mine = next;
    }
}

// The opaque meshlets that are expected to be small.  The loop over them
// holds no call: one for the general path inside it costs every meshlet 12
// local loads and 17 stores for the registers kept across it.  A unit that
// turns out not to be small (clipped, a span past the packed offsets) leaves
// the loop instead, the warp's place kept in shared memory.
template <int KIND>
__device__ __forceinline__ void raster_small_units(const FrameDev& f, uint32_t view_begin, RasterTune tune, uint32_t* claim_word,
                                                   RasterSmemSmall& sm, uint32_t gwarp, uint32_t warp, uint32_t lane,
                                                   uint32_t& nfrag) {
    const RasterWork& work = sm.work[kLoopSmall];
    auto copy_to = [&](uint32_t buf, const RasterUnit& mine) {  // the lane's unit of the next batch
        sm.unit[warp][buf][lane] = mine;
        const char* src = reinterpret_cast<const char*>(sm.view[mine.info & 0xFFu].rdraws + mine.slot);
        char* dst = reinterpret_cast<char*>(&sm.draw[warp][buf][lane]);
#pragma unroll
        for (uint32_t k = 0; k < sizeof(RasterDraw); k += 16) cp_async16_cg(dst + k, src + k);
    };
    {
        uint32_t unit, end, v = 0;
        first_window(work, gwarp, unit, end);
        if (lane < end - unit) copy_to(0u, unit_of(sm, kLoopSmall, 0u, unit + lane, v));
        if (lane == 0) sm.place[warp] = RasterPlace{0u, 0u, end - unit, end, 1u};  // the first batch is the next one
        __syncwarp();
    }
    for (;;) {
        uint32_t general = 0xFFFFFFFFu;  // a unit for the general path: its place in the batch
        RasterPlace at = sm.place[warp];
        uint32_t v_lane = 0, claimed = 0;
        RasterUnit mine{0u, 0u};
        for (;;) {
            if (at.i == at.n) {
                if (at.n_next == 0) break;
                at.i = 0;
                at.n = at.n_next;
                at.buf ^= 1u;
                cp_async_wait_all();
                __syncwarp();
            }
            const RasterDraw& rd = sm.draw[warp][at.buf][at.i];
            const RasterUnit un = sm.unit[warp][at.buf][at.i];
            at.i++;
            const bool last = at.i == at.n;
            if (last) claimed = claim_batch(work, at.end, claim_word, lane);
            auto ahead = [&]() {
                if (last) at.n_next = take_batch(sm, kLoopSmall, 0u, claimed, at.end, lane, v_lane, mine);
            };
            auto copy = [&]() {
                if (last && lane < at.n_next) copy_to(at.buf ^ 1u, mine);
            };
            const uint32_t bits = rd.bits;
            SmallResult res = kSmallNothing;
            if ((bits & (kDrawNoCentre | kDrawGeneral)) || (un.info >> 8) * 32u >= ((bits >> 8) & 0xFFu)) {
                // no pixel centre in reach of the sphere, a meshlet of the
                // general loop, or a quarter without triangles
                ahead();
            } else {
                const uint32_t v = un.info & 0xFFu;
                res = raster_meshlet_small<KIND>(f, rd, view_begin + v, un.slot, un.info >> 8, 1u << work.split_shift, sm.view[v],
                                                 &sm.vp[v], tune, sm.v[warp], sm.micro[warp], lane, nfrag, ahead, copy);
            }
            if (res != kSmallDone) copy();
            if (res == kSmallGeneral) {
                general = at.i - 1u;
                break;
            }
        }
        if (general == 0xFFFFFFFFu) break;
        __syncwarp();
        if (lane == 0) sm.place[warp] = at;
        __syncwarp();
        nfrag += raster_meshlet_general<KIND>(sm, view_begin, at.buf, general, tune);
    }
    cp_async_wait_all();  // no copy outlives the phase
}

// What a launch over views [view_begin, view_begin + n_views) reads of them,
// and its units, into shared memory.
template <bool ALPHA>
__device__ __forceinline__ void raster_setup(const FrameDev& f, uint32_t view_begin, uint32_t n_views, RasterTune tune,
                                             RasterSmem& sm, uint32_t list) {
    __syncthreads();  // `sm` may still be in use by a previous phase of the block
    if (threadIdx.x < 64 && (threadIdx.x & 31) == 0) {  // a warp per loop
        const RasterLoop loop = threadIdx.x == 0 ? kLoopSmall : kLoopGeneral;
        RasterWork& k = sm.work[loop];
        uint32_t run = 0;
        for (uint32_t v = 0; v < n_views; v++) {
            k.prefix[v] = run;
            run += raster_list_count(f, f.views + view_begin + v, ALPHA, list, loop);
        }
        k.prefix[n_views] = run;
        // Work units: a meshlet, or a quarter of its triangles when the views
        // hold fewer meshlets than the grid has warps.  Every quarter
        // transforms the meshlet's vertices again: with quarters up to two
        // meshlets per warp a 720p frame of 64 small spheres (7,600 meshlets
        // a view, 4,864 warps) takes 134 us, with this line 100.
        const uint32_t warps_total = gridDim.x * (blockDim.x >> 5);
        // Meshlets of the general path have more work in their triangles:
        // quarters up to two per warp (1080p before walls 476.5 against 477.5
        // us, the rest the same either way).
        k.split_shift = run < (loop == kLoopGeneral ? 2u * warps_total : warps_total) ? 2u : 0u;
        k.n_units = run << k.split_shift;
        k.batch = tune.batch;
        k.batch_shift = 34u - __clz(warps_total);  // 4 to 8 times the warps
        k.dyn_base = warps_total * units_batch(tune.batch, k.n_units, k.batch_shift);
    }
    for (uint32_t v = threadIdx.x; v < n_views; v += blockDim.x) {
        const ViewDev* vw = f.views + view_begin + v;
        ViewTarget& t = sm.view[v];
        t.target = vw->target;
        t.W = vw->width;
        t.H = vw->height;
        t.rdraws = vw->rdraws;
        t.list[kLoopSmall] = raster_list(f, vw, ALPHA, list, kLoopSmall);
        t.list[kLoopGeneral] = raster_list(f, vw, ALPHA, list, kLoopGeneral);
    }
    for (uint32_t i = threadIdx.x; i < n_views * 16; i += blockDim.x) {
        const lh_mat4& m = view_matrix(f, f.views + view_begin + i / 16);
        reinterpret_cast<float*>(&sm.vp[i / 16])[i % 16] = reinterpret_cast<const float*>(&m)[i % 16];
    }
    __syncthreads();
}

// One warp per meshlet of a pass over the views (`list`: a RasterList),
// claimed dynamically over all of them.  Persistent: returns when the claims
// run out.  The alpha-clip class and the occluders, all on the general path:
template <int KIND, bool ALPHA>
__device__ void phase_raster_general(const FrameDev& f, uint32_t view_begin, uint32_t n_views, RasterTune tune, RasterSmem& sm,
                                     AlphaSmem* s_alpha, uint32_t list) {
    raster_setup<ALPHA>(f, view_begin, n_views, tune, sm, list);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t nfrag = 0;  // fragments this lane wrote
    raster_general_units<KIND, ALPHA>(f, view_begin, tune, &f.status[ALPHA ? kStRasterClaimAlpha : kStRasterClaimGeneral], sm,
                                      ALPHA ? s_alpha + warp : nullptr, blockIdx.x * (blockDim.x >> 5) + warp, warp, lane, nfrag);
    count_fragments<KIND>(f, nfrag);
}

// and the opaque class, in two loops (each skipped when it holds nothing: a
// launch of a few hundred units is bound by fetching the instructions it
// runs through).  As two launches, the second beside the first, the 1080p
// frame took 3 to 6 % longer.
template <int KIND>
__device__ void phase_raster(const FrameDev& f, uint32_t view_begin, uint32_t n_views, RasterTune tune, RasterSmemSmall& sm,
                             uint32_t list) {
    static_assert(sizeof(FrameDev) % 8 == 0 && sizeof(FrameDev) / 8 <= 256, "copied by one pass of the block");
    __syncthreads();
    if (threadIdx.x < sizeof(FrameDev) / 8)
        reinterpret_cast<unsigned long long*>(&sm.f)[threadIdx.x] = reinterpret_cast<const unsigned long long*>(&f)[threadIdx.x];
    raster_setup<false>(f, view_begin, n_views, tune, sm, list);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t warps_total = gridDim.x * (blockDim.x >> 5), gwarp = blockIdx.x * (blockDim.x >> 5) + warp;
    uint32_t nfrag = 0;  // fragments this lane wrote
    // (first windows from opposite ends of the grid)
    if (sm.work[kLoopGeneral].n_units)
        raster_general_units<KIND, false>(f, view_begin, tune, &f.status[kStRasterClaimGeneral], sm, nullptr,
                                          warps_total - 1u - gwarp, warp, lane, nfrag);
    if (sm.work[kLoopSmall].n_units)
        raster_small_units<KIND>(f, view_begin, tune, &f.status[kStRasterClaim], sm, gwarp, warp, lane, nfrag);
    count_fragments<KIND>(f, nfrag);
}

// Edge function of edge a->b at pixel centre (px, py).
__device__ __forceinline__ int64_t edge_at(int32_t ax, int32_t ay, int32_t bx, int32_t by, int32_t px, int32_t py) {
    return (int64_t)(by - ay) * ((int64_t)px * 256 + 128 - ax) - (int64_t)(bx - ax) * ((int64_t)py * 256 + 128 - ay);
}

// True when the edge's test fails at all four corners of the pixel
// rectangle (the edge function is affine, so it fails everywhere inside).
__device__ __forceinline__ bool edge_rejects(int32_t ax, int32_t ay, int32_t bx, int32_t by, int32_t x0, int32_t x1,
                                             int32_t y0, int32_t y1, int64_t bias) {
    return edge_at(ax, ay, bx, by, x0, y0) < bias && edge_at(ax, ay, bx, by, x1, y0) < bias &&
           edge_at(ax, ay, bx, by, x0, y1) < bias && edge_at(ax, ay, bx, by, x1, y1) < bias;
}

// Arithmetic of a chunk's edge values.  No covered pixel's value exceeds the
// triangle's doubled area 2A (= e12 + e20 + e01 at every point).  kEdge32:
// every edge product inside the triangle's box fits 32 bits (TriSetup's bias
// bit 3), so the whole chunk runs in 32 bits; kEdge46: 64-bit values, 2A
// below 2^46, converted with FP32 adds; kEdge64: the 64-bit conversion
// instruction.
enum EdgeMode { kEdge32 = 0, kEdge46 = 1, kEdge64 = 2 };
template <int MODE>
struct EdgeVal {
    using T = typename std::conditional<MODE == kEdge32, int32_t, int64_t>::type;
};
template <int MODE>
__device__ __forceinline__ typename EdgeVal<MODE>::T shfl_edge(typename EdgeVal<MODE>::T v, uint32_t src) {
    if (MODE == kEdge32) return (int32_t)__shfl_sync(0xFFFFFFFFu, (int32_t)v, src);
    return (int64_t)__shfl_sync(0xFFFFFFFFu, (unsigned long long)v, src);
}

// The triangle's depth plane and ID, held in registers during a walk.
struct ChunkDepth {
    float z0;
    f32x2 s;  // s1, s2
    uint32_t id;
    f32x2 nz;  // FrameDev::neg_zero2
};

// A covered pixel: depth from its two edge values (the per-pixel test's
// arithmetic; both values converted and scaled in one register pair), then
// the depth test at linear pixel index `pix`.
template <int KIND, int MODE>
__device__ __forceinline__ void chunk_fragment(const ChunkDepth& t, void* target, uint32_t pix,
                                               typename EdgeVal<MODE>::T a20, typename EdgeVal<MODE>::T a01) {
    f32x2 e;
    if (MODE == kEdge32) {
        e = pack2(__int2float_rn((int32_t)a20), __int2float_rn((int32_t)a01));
    } else if (MODE == kEdge46) {  // u46_to_f32_rn of both
        const f32x2 hi = pack2(__uint_as_float(0x56800000u | (uint32_t)((uint64_t)a20 >> 23)),
                               __uint_as_float(0x56800000u | (uint32_t)((uint64_t)a01 >> 23)));
        const f32x2 lo = pack2(__uint_as_float(0x4B000000u | ((uint32_t)a20 & 0x7FFFFFu)),
                               __uint_as_float(0x4B000000u | ((uint32_t)a01 & 0x7FFFFFu)));
        e = add2(add2(hi, pack2(-70368744177664.0f, -70368744177664.0f)), add2(lo, pack2(-8388608.0f, -8388608.0f)));
    } else {
        e = pack2(__ll2float_rn((int64_t)a20), __ll2float_rn((int64_t)a01));
    }
    float d20, d01;
    unpack2(mul2(e, t.s, t.nz), d20, d01);
    const float d = (t.z0 + d20) + d01;
    // clamped to [0, 1], NaN and -0 to +0
    write_pixel<KIND>(target, pix, fminf(fmaxf(d, 0.0f), 1.0f), t.id);
}

// Row by row: the warp's lanes along each run (long runs).  Lane r holds
// row r's run: its length, the linear index of its first pixel and the two
// edge values there.
template <int KIND, int MODE>
__device__ __forceinline__ void chunk_rows(const ChunkDepth& t, void* target, uint32_t rows, uint32_t lane, int32_t len,
                                           uint32_t pix_first, typename EdgeVal<MODE>::T f20, typename EdgeVal<MODE>::T f01,
                                           typename EdgeVal<MODE>::T dx20, typename EdgeVal<MODE>::T dx01) {
    using T = typename EdgeVal<MODE>::T;
    using U = typename std::make_unsigned<T>::type;  // (the step past a run's end may wrap)
    const U step20 = (U)32 * (U)dx20, step01 = (U)32 * (U)dx01;
    const U lane20 = (U)lane * (U)dx20, lane01 = (U)lane * (U)dx01;
    for (uint32_t r = 0; r < rows; r++) {
        const int32_t l = __shfl_sync(0xFFFFFFFFu, len, r);
        if (l == 0) continue;
        uint32_t pix = __shfl_sync(0xFFFFFFFFu, pix_first, r) + lane;
        U a20 = (U)shfl_edge<MODE>(f20, r) + lane20, a01 = (U)shfl_edge<MODE>(f01, r) + lane01;
        for (int32_t k = (int32_t)lane; k < l; k += 32, pix += 32, a20 += step20, a01 += step01)
            chunk_fragment<KIND, MODE>(t, target, pix, (T)a20, (T)a01);
    }
}

// Compacted: the covered pixels of all rows numbered one after another,
// 32 consecutive per step, one per lane (short runs: slivers, corners).
// The non-empty rows are ranked in row order and lane k holds the k-th
// one's run: its first number, and the linear index and edge values
// extrapolated to number 0.  A step over numbers [base, base + 32) marks
// the runs that start inside it in one word (a warp OR of one bit per
// run), so a lane's run is the last one started at or before its number:
// the runs started before the step plus those marked up to its own bit.
template <int KIND, int MODE>
__device__ __forceinline__ void chunk_compact(const ChunkDepth& t, void* target, uint32_t lane, int32_t total, int32_t first,
                                              uint32_t pix_zero, typename EdgeVal<MODE>::T z20, typename EdgeVal<MODE>::T z01,
                                              typename EdgeVal<MODE>::T dx20, typename EdgeVal<MODE>::T dx01,
                                              uint32_t nonempty) {
    using T = typename EdgeVal<MODE>::T;
    using U = typename std::make_unsigned<T>::type;  // (exact modulo the word for the covered pixels)
    const uint32_t upto_me = 0xFFFFFFFFu >> (31u - lane);  // bits 0 .. lane
    int32_t before = 0;  // runs started before the step
    for (int32_t base = 0; base < total; base += 32) {
        const uint32_t off = (uint32_t)(first - base);
        const uint32_t starts = __reduce_or_sync(0xFFFFFFFFu, lane < nonempty && off < 32u ? 1u << off : 0u);
        const int32_t k = before + __popc(starts & upto_me) - 1;  // the lane's run
        before += __popc(starts);
        const int32_t p = base + (int32_t)lane;
        const uint32_t src = (uint32_t)k & 31u;
        const uint32_t pix = (uint32_t)p + __shfl_sync(0xFFFFFFFFu, pix_zero, src);
        const U a20 = (U)shfl_edge<MODE>(z20, src) + (U)p * (U)dx20, a01 = (U)shfl_edge<MODE>(z01, src) + (U)p * (U)dx01;
        if (p < total) chunk_fragment<KIND, MODE>(t, target, pix, (T)a20, (T)a01);
    }
}

// Per-row run state of a chunk, then the cheaper of the two walks.
template <int KIND, int MODE>
__device__ __forceinline__ void chunk_walk(const FrameDev& f, const BigTri& b, void* target, uint32_t W, int32_t x0, int32_t y0,
                                           uint32_t rows, uint32_t lane, int32_t lo, int32_t len, int32_t pre, int32_t total,
                                           typename EdgeVal<MODE>::T e20, typename EdgeVal<MODE>::T e01,
                                           typename EdgeVal<MODE>::T dx20, typename EdgeVal<MODE>::T dx01) {
    using T = typename EdgeVal<MODE>::T;
    using U = typename std::make_unsigned<T>::type;
    const ChunkDepth t{b.z0, pack2(b.s1, b.s2), b.id, f.neg_zero2};
    // steps of the row walk (plus a row's own cost) against the compacted
    // walk's, whose steps cost about twice as much
    const uint32_t row_steps = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)(len + 31) >> 5);
    const uint32_t ne_mask = __ballot_sync(0xFFFFFFFFu, len > 0);
    const uint32_t nonempty = __popc(ne_mask);
    const uint32_t pix_row = (uint32_t)(y0 + (int32_t)lane) * W + (uint32_t)x0;
    if (row_steps + nonempty / 4u <= 2u * (uint32_t)((total + 31) >> 5)) {
        chunk_rows<KIND, MODE>(t, target, rows, lane, len, pix_row + (uint32_t)lo, (T)((U)e20 + (U)lo * (U)dx20),
                               (T)((U)e01 + (U)lo * (U)dx01), dx20, dx01);
        return;
    }
    // rank the non-empty rows: lane k takes the k-th one's values
    const uint32_t src = __fns(ne_mask, 0, (int32_t)lane + 1);  // 0xFFFFFFFF past the last
    const uint32_t s = src < 32u ? src : 0u;
    const int32_t first = __shfl_sync(0xFFFFFFFFu, pre, s);
    const uint32_t pix_zero = __shfl_sync(0xFFFFFFFFu, pix_row + (uint32_t)(lo - pre), s);
    const T z20 = shfl_edge<MODE>((T)((U)e20 + (U)(T)(lo - pre) * (U)dx20), s);
    const T z01 = shfl_edge<MODE>((T)((U)e01 + (U)(T)(lo - pre) * (U)dx01), s);
    chunk_compact<KIND, MODE>(t, target, lane, total, first, pix_zero, z20, z01, dx20, dx01, nonempty);
}

// The pixels [x0, x1] x [y0, y1] (at most 32 rows of at most 256) of an
// opaque big triangle, by the whole warp.  Lane r finds the run of covered
// pixels of row y0 + r (the three edges' runs intersected, clip_run); the
// runs are walked row by row when they are long, else compacted (every lane
// of a step on a covered pixel).  Either walk forms, at every pixel, the
// very integers the per-pixel test forms, so coverage and depth are the
// same; a step's pixels lie in one or two rows, so its reductions stay
// coalesced.  Returns the fragments written.
struct ChunkSteps {  // reciprocals of a triangle's edge steps along x
    float inv12, inv20, inv01;
};
__device__ __forceinline__ ChunkSteps chunk_steps(const BigTri& b) {
    return ChunkSteps{run_inv_step(b.Y2 - b.Y1), run_inv_step(b.Y0 - b.Y2), run_inv_step(b.Y1 - b.Y0)};
}

// Edge function of edge a->b at pixel centre (px, py), in the mode's width.
template <int MODE>
__device__ __forceinline__ typename EdgeVal<MODE>::T edge_as(int32_t ax, int32_t ay, int32_t bx, int32_t by, int32_t px,
                                                             int32_t py) {
    if (MODE == kEdge32) return (by - ay) * (px * 256 + 128 - ax) - (bx - ax) * (py * 256 + 128 - ay);
    return (typename EdgeVal<MODE>::T)edge_at(ax, ay, bx, by, px, py);
}

// The runs of the chunk's rows in 32 bits (SMALL: TriSetup's bias bit 3) or
// 64, then the walk.  Most chunks by number are whole triangles of tens to
// thousands of pixels, whose set-up costs more than their walk.
template <int KIND, bool SMALL>
__device__ __forceinline__ uint32_t raster_chunk_as(const FrameDev& f, const BigTri& b, const ChunkSteps& k, int32_t x0,
                                                    int32_t x1, int32_t y0, int32_t y1, uint32_t lane, void* target,
                                                    uint32_t W) {
    constexpr int kMode = SMALL ? kEdge32 : kEdge46;
    using T = typename EdgeVal<kMode>::T;
    const int32_t n = x1 - x0 + 1;
    const uint32_t rows = (uint32_t)(y1 - y0 + 1);
    const T dx20 = (T)(b.Y0 - b.Y2) * 256, dx01 = (T)(b.Y1 - b.Y0) * 256;
    int32_t lo = 0, hi = -1;
    T e12 = 0, e20 = 0, e01 = 0;
    if (lane < rows) {
        const int32_t y = y0 + (int32_t)lane;
        e12 = edge_as<kMode>(b.X1, b.Y1, b.X2, b.Y2, x0, y);
        e20 = edge_as<kMode>(b.X2, b.Y2, b.X0, b.Y0, x0, y);
        e01 = edge_as<kMode>(b.X0, b.Y0, b.X1, b.Y1, x0, y);
        hi = n - 1;
        clip_run_as<T>(e12, (T)(b.Y2 - b.Y1) * 256, (T)(b.bias & 1u), n, k.inv12, lo, hi);
        clip_run_as<T>(e20, dx20, (T)((b.bias >> 1) & 1u), n, k.inv20, lo, hi);
        clip_run_as<T>(e01, dx01, (T)((b.bias >> 2) & 1u), n, k.inv01, lo, hi);
    }
    const int32_t len = hi >= lo ? hi - lo + 1 : 0;
    int32_t incl = len;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const int32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += v;
    }
    const int32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    if (total == 0) return 0;
    const int32_t pre = incl - len;
    if (!SMALL) {
        // 2A: the sum of the three edge functions, the same at every point
        const uint64_t area2 = (uint64_t)__shfl_sync(0xFFFFFFFFu, (unsigned long long)(e12 + e20 + e01), 0);
        if (area2 >= (1ull << 46)) {
            chunk_walk<KIND, kEdge64>(f, b, target, W, x0, y0, rows, lane, lo, len, pre, total, e20, e01, dx20, dx01);
            return (uint32_t)total;
        }
    }
    chunk_walk<KIND, kMode>(f, b, target, W, x0, y0, rows, lane, lo, len, pre, total, e20, e01, dx20, dx01);
    return (uint32_t)total;
}
template <int KIND>
__device__ __forceinline__ uint32_t raster_chunk_runs(const FrameDev& f, const BigTri& b, const ChunkSteps& k, int32_t x0,
                                                      int32_t x1, int32_t y0, int32_t y1, uint32_t lane, void* target,
                                                      uint32_t W) {
    return (b.bias & 8u) ? raster_chunk_as<KIND, true>(f, b, k, x0, x1, y0, y1, lane, target, W)
                         : raster_chunk_as<KIND, false>(f, b, k, x0, x1, y0, y1, lane, target, W);
}

// Number of entries of the ascending array `base` that are <= c (the upper
// bound), known to lie in [lo, hi], found by the whole warp: 32 probes per round narrow the
// range 32-fold, so a queue of 16k triangles takes 3 dependent loads instead
// of 14.
__device__ __forceinline__ uint32_t upper_bound_warp(const uint32_t* base, uint32_t lo, uint32_t hi, uint32_t c,
                                                     uint32_t lane) {  // the answer lies in [lo, hi]
    for (;;) {
        const uint32_t span = hi - lo;
        const uint32_t step = span <= 32u ? 1u : (span + 31u) / 32u;
        const uint32_t p = lo + lane * step;
        const bool le = p < hi && __ldcg(base + p) <= c;
        const uint32_t k = __popc(__ballot_sync(0xFFFFFFFFu, le));  // true lanes form a prefix
        if (step == 1u) return lo + k;
        const uint32_t nlo = k ? lo + (k - 1u) * step + 1u : lo;
        const uint32_t nhi = (k < 32u && lo + k * step < hi) ? lo + k * step : hi;
        lo = nlo;
        hi = nhi;
    }
}

// The pixels [x0, x1] x [y0, y1] of an alpha-tested big triangle by the whole
// warp: covered ones, found 32 of a row at a time, wait in `wait` (64 x {pixel,
// depth}) until 32 of them are tested at once.  Not inlined, as the other
// alpha paths; the triangle is read from the queue, not handed over in
// registers.
template <int KIND>
__device__ __noinline__ uint32_t raster_chunk_alpha(const FrameDev& f, const BigTri* entry, int32_t x0, int32_t x1,
                                                    int32_t y0, int32_t y1, uint32_t lane, uint2* wait) {
    const BigTri b = *entry;
    const ViewDev* vw = f.views + b.view;
    void* target = vw->target;
    const AlphaSize size = alpha_size(vw->width, vw->height);
    const AlphaTri at = alpha_tri_global(f, b.view, b.id);
    TriSetup t;
    t.X0 = b.X0; t.Y0 = b.Y0; t.X1 = b.X1; t.Y1 = b.Y1; t.X2 = b.X2; t.Y2 = b.Y2;
    t.z0 = b.z0; t.s1 = b.s1; t.s2 = b.s2;
    t.id = b.id;
    t.bias = b.bias;
    uint32_t n = 0, first = 0, waiting = 0;
    int32_t py = y0, px = x0;
    for (;;) {
        while (waiting < 32 && py <= y1) {
            float d = 0.0f;
            const int32_t x = px + (int32_t)lane;
            const bool covered = x <= x1 && cover(t, x, py, d);
            const uint32_t mask = __ballot_sync(0xFFFFFFFFu, covered);
            if (covered)
                wait[(first + waiting + __popc(mask & ((1u << lane) - 1u))) & 63u] =
                    make_uint2((uint32_t)x | (uint32_t)py << 16, f2u(d));
            waiting += __popc(mask);
            px += 32;
            if (px > x1) px = x0, py++;
        }
        if (!waiting) return n;
        const uint32_t now = min(waiting, 32u);
        __syncwarp();
        if (lane < now) {
            const uint2 w = wait[(first + lane) & 63u];
            const int32_t wx = (int32_t)(w.x & 0xFFFFu), wy = (int32_t)(w.x >> 16);
            if (alpha_pass(f, at, wx, wy, size)) {
                write_fragment<KIND>(target, size.W, wx, wy, u2f(w.y), t.id);
                n++;
            }
        }
        __syncwarp();
        first = (first + now) & 63u;
        waiting -= now;
    }
}

// The opaque or alpha-tested pixels [x0, x1] x [y0, y1] (at most 32 x 256) of
// the big triangle `b` (queue entry `entry`), by the whole warp: opaque ones by
// runs of covered pixels (raster_chunk_runs), alpha-tested ones pixel by pixel
// unless the rectangle lies outside one edge.  Returns the fragments this lane
// counts.
template <int KIND>
__device__ __forceinline__ uint32_t raster_chunk(const FrameDev& f, const BigTri& b, const BigTri* entry, const ChunkSteps& ks,
                                                 int32_t x0, int32_t x1, int32_t y0, int32_t y1, uint32_t lane, void* target,
                                                 uint32_t W, uint2* wait) {
    if (b.bias & kBiasAlpha) {
        if (edge_rejects(b.X1, b.Y1, b.X2, b.Y2, x0, x1, y0, y1, b.bias & 1u) ||
            edge_rejects(b.X2, b.Y2, b.X0, b.Y0, x0, x1, y0, y1, (b.bias >> 1) & 1u) ||
            edge_rejects(b.X0, b.Y0, b.X1, b.Y1, x0, x1, y0, y1, (b.bias >> 2) & 1u))
            return 0u;
        return raster_chunk_alpha<KIND>(f, entry, x0, x1, y0, y1, lane, wait);
    }
    const uint32_t written = raster_chunk_runs<KIND>(f, b, ks, x0, x1, y0, y1, lane, target, W);
    return lane == 0 ? written : 0u;
}

// Shared memory of the chunk kernel.
constexpr uint32_t kWholeBatch = 8;  // whole triangles claimed per atomic, at most (their entries: 16 bytes a lane)
struct BigSmem {
    // the views' targets and widths, read once per block
    unsigned long long target[kMaxViews];
    uint32_t width[kMaxViews];
    // each warp's entries: the current and the next triangle of the chunks
    // (copied ahead with cp.async while the current one's chunks are walked),
    // then two batches of whole triangles; kept here, not in registers
    __align__(16) BigTri tri[kRasterWarps][2 * kWholeBatch];
    ChunkSteps steps[kRasterWarps];
    uint2 wait[kRasterWarps][64];  // covered pixels of alpha-tested triangles
};

// The chunks of the triangles too large to be taken whole, claimed in order.
template <int KIND>
__device__ __forceinline__ void raster_big_chunks(const FrameDev& f, BigSmem& sm, uint32_t ntri, uint32_t total32, uint32_t w,
                                                  uint32_t lane, uint32_t& nfrag) {
    // static first batch per warp, then claims that shrink as the chunks run
    // out (the claim costs an atomic's and a search's round trips)
    const uint32_t warps_total = gridDim.x * (blockDim.x >> 5);
    // (a chunk of an alpha-tested triangle costs several times an opaque one's:
    // claims a quarter as large, 2258 x 406 close to foliage 1305 -> 1184 us)
    const uint32_t shift = LH_CHUNK_SHIFT - __clz(warps_total) + (f.scene_alpha ? 2u : 0u);
    // (never fewer than the chunks beside one another that one set-up of runs
    // serves, below: 1920 x 1080 before large walls 337 -> 317 us a frame;
    // alpha-tested chunks go one by one and cost more: 423 -> 437 with foliage)
    const uint32_t fewest = f.scene_alpha ? 1u : max(256u >> f.chunk_shift[KIND][1], 1u);
    auto batch_of = [&](uint32_t left) { return min(max(left >> shift, fewest), (uint32_t)LH_CHUNK_BATCH); };
    const uint32_t first_batch = batch_of(total32);
    const uint32_t gwarp = blockIdx.x * (blockDim.x >> 5) + w;
    const uint64_t dyn_base = (uint64_t)warps_total * first_batch;
    const uint32_t rs = f.chunk_shift[KIND][0], cs = f.chunk_shift[KIND][1];
    uint32_t c = (uint32_t)min((uint64_t)gwarp * first_batch, (uint64_t)total32);
    uint32_t c_end = (uint32_t)min((uint64_t)gwarp * first_batch + first_batch, (uint64_t)total32);
    // the current triangle, kept while consecutive chunks belong to it:
    // its index, chunk range [t_base, t_end), chunk columns, shared-memory
    // slot, and the chunk coordinates after the last one taken (c_next - 1);
    // the copied-ahead next entry (index pre_idx)
    uint32_t t_idx = 0, t_base = 1, t_end = 0, nbx = 1, c_next = 0xFFFFFFFFu, slot = 0;
    uint32_t pre_idx = 0xFFFFFFFFu;
    int32_t cx = 0, cy = 0;
    const ChunkSteps& ks = sm.steps[w];
    BigTri* s_tri = sm.tri[w];
    for (;;) {
        if (c >= c_end) {
            if (dyn_base >= total32) break;
            uint32_t claimed = 0;
            const uint32_t batch = batch_of(total32 - c_end);
            if (lane == 0) claimed = atomicAdd(&f.status[kStBigClaim], batch);
            const uint64_t first = dyn_base + __shfl_sync(0xFFFFFFFFu, claimed, 0);
            if (first >= total32) break;
            c = (uint32_t)first;
            c_end = (uint32_t)min(first + batch, (uint64_t)total32);
        }
        if (c >= t_base && c < t_end) {
            // the same triangle: the next chunk in row order, or any other
            if (c == c_next) {
                if (cx == (int32_t)nbx) {
                    cx = 0;
                    cy++;
                }
            } else {
                cx = (int32_t)((c - t_base) % nbx);
                cy = (int32_t)((c - t_base) / nbx);
            }
        } else {
            // another triangle, by a 32-ary search of the bases; often the
            // copied-ahead next entry
            __syncwarp();  // every lane is done with the current slot
            uint32_t i = pre_idx, base = t_end;
            bool next = false;
            if (c == t_end && pre_idx != 0xFFFFFFFFu) {
                // bases ascend without gaps: the chunk after a triangle's last is
                // the next entry's first, unless that one is taken whole
                cp_async_wait_all();
                __syncwarp();
                next = !(s_tri[slot ^ 1u].bias & kBiasWhole);
            }
            if (!next) {
                const uint32_t first = upper_bound_warp(f.big_base, t_end ? t_idx : 0u, ntri, c, lane);
                if (first == 0) {
                    c++;
                    continue;
                }
                i = first - 1;
                base = f.big_base[i];
            }
            if (i == pre_idx) {
                cp_async_wait_all();
                __syncwarp();
                slot ^= 1u;
            } else {
                const BigTri nb = f.big[i];
                if (lane == 0) s_tri[slot] = nb;
                __syncwarp();
            }
            const BigTri& nb = s_tri[slot];
            const uint32_t nx = ((uint32_t)(nb.px1 - nb.px0) >> cs) + 1;
            const uint32_t ny = ((uint32_t)(nb.py1 - nb.py0) >> rs) + 1;
            if ((nb.bias & kBiasWhole) || (unsigned long long)(c - base) >= (unsigned long long)nx * ny) {
                t_base = 1;  // chunk of a dropped triangle: the slot no longer holds the current one
                t_end = 0;
                pre_idx = 0xFFFFFFFFu;
                c++;
                continue;
            }
            if (lane == 0) sm.steps[w] = chunk_steps(nb);
            t_idx = i;
            t_base = base;
            t_end = base + nx * ny;
            nbx = nx;
            cx = (int32_t)((c - base) % nx);
            cy = (int32_t)((c - base) / nx);
            // copy the queue's next entry into the other slot meanwhile
            pre_idx = 0xFFFFFFFFu;
            if (i + 1u < ntri) {
                if (lane < 4) {
                    cp_async_wait_all();  // a copy still in flight to that slot
                    cp_async16_cg(reinterpret_cast<char*>(&s_tri[slot ^ 1u]) + 16 * lane,
                                  reinterpret_cast<const char*>(f.big + i + 1u) + 16 * lane);
                    cp_async_commit();
                }
                pre_idx = i + 1u;
            }
            __syncwarp();
        }
        // the batch's chunks beside this one in the same chunk row go with it,
        // up to 256 columns: one set-up of the rows' runs for all of them
        const BigTri& b = s_tri[slot];
        const uint32_t along = (b.bias & kBiasAlpha) ? 1u : min(min(nbx - (uint32_t)cx, c_end - c), 256u >> cs);
        const int32_t x0 = b.px0 + (cx << cs), x1 = min(b.px1, x0 + (int32_t)(along << cs) - 1);
        const int32_t y0 = b.py0 + (cy << rs), y1 = min(b.py1, y0 + (1 << rs) - 1);
        c += along;
        c_next = c;
        cx += (int32_t)along;
        nfrag += raster_chunk<KIND>(f, b, f.big + t_idx, ks, x0, x1, y0, y1, lane, reinterpret_cast<void*>(sm.target[b.view]),
                                    sm.width[b.view], sm.wait[w]);
    }
    cp_async_wait_all();
    __syncwarp();
}

// The triangles taken whole, claimed by their index in the queue; the next
// batch's claim and entries travel behind the current batch.
template <int KIND>
__device__ __forceinline__ void raster_big_whole(const FrameDev& f, BigSmem& sm, uint32_t ntri, uint32_t w, uint32_t lane,
                                                 uint32_t& nfrag) {
    const uint32_t warps_total = gridDim.x * (blockDim.x >> 5);
    const uint32_t shift = LH_WHOLE_SHIFT - __clz(warps_total);
    auto batch_of = [&](uint32_t left) { return min(max(left >> shift, 1u), kWholeBatch); };
    const uint32_t first_batch = batch_of(ntri), dyn_base = warps_total * first_batch;
    // (first windows from the end of the grid: the chunks' from its start)
    const uint32_t gwarp = warps_total - 1u - (blockIdx.x * (blockDim.x >> 5) + w);
    uint32_t i0 = min(gwarp * first_batch, ntri), end = min(gwarp * first_batch + first_batch, ntri), buf = 0;
    auto copy = [&](uint32_t first, uint32_t n, uint32_t to) {
        if (lane < 4 * n)
            cp_async16_cg(reinterpret_cast<char*>(&sm.tri[w][to * kWholeBatch]) + 16 * lane,
                          reinterpret_cast<const char*>(f.big + first) + 16 * lane);
    };
    copy(i0, end - i0, 0u);
    while (i0 < end) {
        const uint32_t n = end - i0, batch = batch_of(ntri - end);
        uint32_t claimed = 0, next = 0, next_end = 0;
        if (lane == 0 && dyn_base < ntri) claimed = atomicAdd(&f.status[kStWholeClaim], batch);
        cp_async_wait_all();
        __syncwarp();
        for (uint32_t k = 0; k < n; k++) {
            const BigTri& b = sm.tri[w][buf * kWholeBatch + k];
            if (k == n - 1u && dyn_base < ntri) {
                next = min(dyn_base + __shfl_sync(0xFFFFFFFFu, claimed, 0), ntri);
                next_end = min(next + batch, ntri);
                copy(next, next_end - next, buf ^ 1u);
            }
            if (!(b.bias & kBiasWhole)) continue;
            const ChunkSteps ks = chunk_steps(b);
            for (int32_t y0 = b.py0; y0 <= b.py1; y0 += 32)
                for (int32_t x0 = b.px0; x0 <= b.px1; x0 += 256)
                    nfrag += raster_chunk<KIND>(f, b, f.big + i0 + k, ks, x0, min(b.px1, x0 + 255), y0, min(b.py1, y0 + 31), lane,
                                                reinterpret_cast<void*>(sm.target[b.view]), sm.width[b.view], sm.wait[w]);
        }
        __syncwarp();
        i0 = next;
        end = next_end;
        buf ^= 1u;
    }
    cp_async_wait_all();  // no copy outlives the phase
}

// The chunk queue: the large triangles' chunks first, then the whole
// triangles, which fill the launch's end.  A claim of a chunk is a chain of an
// atomic, a three-step search and an entry's load behind the warp's own
// reductions; most triangles are one or two chunks, so claims take several, the
// chunks of a claim are merged along their row, and small triangles go whole,
// by their index.  Limit of a whole triangle in the visibility pass, 0 / 1 / 2 / 3
// chunks: the 4K stress frame 10.23 / 10.06 / 9.78 / 9.62 ms, 1080p before walls
// 490 / 490 / 477 / 477 us, another 305 / 296 / 290 / 293.  Most chunks a claim
// takes, 8 / 16 / 32 / 64: stress 9.95 / 9.83 / 9.78 / 9.79 ms, the rest the same.
// Share of what is left that a claim takes (LH_CHUNK_SHIFT 31 / 32 / 33): 32 probes
// 1719 / 1677 / 1681 us, before walls 472 / 477 / 477; the same of whole triangles
// (LH_WHOLE_SHIFT): 1080p 320 / 310 / 311, another 281 / 290 / 290, before walls
// 485 / 477 / 492, training step 428 / 430 / 437.
template <int KIND>
__device__ void phase_raster_big(const FrameDev& f, BigSmem& sm) {
    __syncthreads();  // `sm` may still be in use by a previous phase of the block
    for (uint32_t v = threadIdx.x; v < f.n_views; v += blockDim.x) {
        sm.target[v] = reinterpret_cast<unsigned long long>(f.views[v].target);
        sm.width[v] = f.views[v].width;
    }
    __syncthreads();
    const unsigned long long packed = *reinterpret_cast<volatile unsigned long long*>(f.status + kStBigPacked);
    const uint32_t ntri = (uint32_t)min((unsigned long long)f.big_cap, packed >> 40);
    const unsigned long long total = packed & ((1ull << 40) - 1);
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (ntri == 0) return;
    uint32_t nfrag = 0;
    // (chunk numbers fit 32 bits: store_big drops triangles beyond)
    if (total) raster_big_chunks<KIND>(f, sm, ntri, (uint32_t)min(total, 0xFFFFFFFFull), w, lane, nfrag);
    raster_big_whole<KIND>(f, sm, ntri, w, lane, nfrag);
    count_fragments<KIND>(f, nfrag);
}

// ------------------------------------------------------------ occlusion
// Hierarchical depth of the visibility views [view_begin, view_begin +
// n_views) that cull by occlusion, after the occluder pass: one block of 256
// threads per 64 x 64-pixel region (regions of all these views numbered one
// after another), claimed round robin by the grid.  Warp w takes pixel rows
// 8w .. 8w + 7 of the region in two 32-pixel halves, keeps the minimum depth
// bits of each lane's column, then of each 8 x 8 tile (lanes in groups of
// 8); the block takes the region's minimum over its 64 tiles.  Pixels
// outside the view do not count; a pixel without a fragment is depth 0.
__device__ void phase_hiz(const FrameDev& f, uint32_t view_begin, uint32_t n_views) {
    __shared__ uint32_t s_region_min[8];
    __shared__ uint32_t s_first[kMaxViews + 1];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();  // shared memory may still be in use by a previous phase of the block
    if (threadIdx.x == 0) {
        uint32_t run = 0;
        for (uint32_t v = 0; v < n_views; v++) {
            const ViewDev* vw = f.views + view_begin + v;
            s_first[v] = run;
            if (vw->kind == kViewVisibility && vw->hiz) run += vw->hiz_rx * vw->hiz_ry;
        }
        s_first[n_views] = run;
    }
    __syncthreads();
    const uint32_t total = s_first[n_views];
    uint32_t v = 0;
    for (uint32_t region = blockIdx.x; region < total; region += gridDim.x) {
        while (region >= s_first[v + 1]) v++;
        const ViewDev* vw = f.views + view_begin + v;
        const uint32_t r = region - s_first[v], rx = r % vw->hiz_rx, ry = r / vw->hiz_rx;
        const uint32_t W = vw->width, H = vw->height;
        const uint64_t* vis = reinterpret_cast<const uint64_t*>(vw->target);
        uint32_t* level0 = vw->hiz;
        const uint32_t pitch0 = vw->hiz_rx * 8u;
        uint32_t wmin = 0xFFFFFFFFu;
#pragma unroll
        for (uint32_t half = 0; half < 2; half++) {
            const uint32_t x = rx * kHizRegion + half * 32u + lane;
            uint32_t m = 0xFFFFFFFFu;
#pragma unroll
            for (uint32_t k = 0; k < 8; k++) {
                const uint32_t y = ry * kHizRegion + warp * 8u + k;
                if (x < W && y < H) m = min(m, (uint32_t)(__ldcg(vis + (size_t)y * W + x) >> 32));
            }
            m = min(m, __shfl_xor_sync(0xFFFFFFFFu, m, 1));
            m = min(m, __shfl_xor_sync(0xFFFFFFFFu, m, 2));
            m = min(m, __shfl_xor_sync(0xFFFFFFFFu, m, 4));
            if ((lane & 7u) == 0) level0[(size_t)(ry * 8u + warp) * pitch0 + rx * 8u + half * 4u + (lane >> 3)] = m;
            wmin = min(wmin, m);
        }
        wmin = __reduce_min_sync(0xFFFFFFFFu, wmin);
        if (lane == 0) s_region_min[warp] = wmin;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t m = s_region_min[0];
            for (uint32_t k = 1; k < 8; k++) m = min(m, s_region_min[k]);
            level0[(size_t)pitch0 * vw->hiz_ry * 8u + r] = m;  // level 1
        }
        __syncthreads();
    }
}

// True when no fragment of a meshlet inside the world sphere `sp` can pass
// the depth test against what the view holds already: every 8 x 8 tile (or
// 64 x 64 region) its screen box touches has a minimum depth above the
// largest depth the sphere can reach.  The box and that depth come from the
// 8 corners of the sphere's axis-aligned box through the view's matrix,
// widened by 2 pixels and by 1/128 of the depth (the kernels' float
// rounding of the vertices is far below both); a corner at or behind the
// camera plane culls nothing.  Exact: a culled meshlet's every fragment
// would have lost the atomicMax (its depth strictly below the pixel's).
__device__ __forceinline__ bool hiz_occluded(const ViewDev* vw, const lh_mat4& pv, const float (&sp)[4]) {
    const f4 cc = mul(pv, f4{sp[0], sp[1], sp[2], 1.0f});
    const float r = sp[3];
    const f4 a{pv.cols[0].x * r, pv.cols[0].y * r, pv.cols[0].z * r, pv.cols[0].w * r};
    const f4 b{pv.cols[1].x * r, pv.cols[1].y * r, pv.cols[1].z * r, pv.cols[1].w * r};
    const f4 d{pv.cols[2].x * r, pv.cols[2].y * r, pv.cols[2].z * r, pv.cols[2].w * r};
    const float hw = (float)vw->width * 0.5f, hh = (float)vw->height * 0.5f;
    float x0 = 3.0e38f, x1 = -3.0e38f, y0 = 3.0e38f, y1 = -3.0e38f, zmax = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const float sa = (k & 1) ? 1.0f : -1.0f, sb = (k & 2) ? 1.0f : -1.0f, sd = (k & 4) ? 1.0f : -1.0f;
        const float cw = cc.w + sa * a.w + sb * b.w + sd * d.w;
        // (approximate reciprocals: their 2^-22 is far inside the margins below)
        if (!(cw > 1e-6f && cw < 1e30f)) return false;
        const float rw = __fdividef(1.0f, cw);
        const float cx = cc.x + sa * a.x + sb * b.x + sd * d.x;
        const float cy = cc.y + sa * a.y + sb * b.y + sd * d.y;
        const float cz = cc.z + sa * a.z + sb * b.z + sd * d.z;
        const float px = (cx * rw) * hw + hw, py = (cy * rw) * hh + hh, pz = cz * rw;
        x0 = fminf(x0, px);
        x1 = fmaxf(x1, px);
        y0 = fminf(y0, py);
        y1 = fmaxf(y1, py);
        zmax = fmaxf(zmax, pz);
    }
    if (!(zmax >= 0.0f) || !(x1 >= x0) || !(y1 >= y0)) return false;  // NaN
    const float zt = zmax + zmax * (1.0f / 128.0f);
    if (!(zt < 1.0f)) return false;
    const uint32_t zbits = __float_as_uint(zt);
    const int32_t W = (int32_t)vw->width, H = (int32_t)vw->height;
    // the box, widened and clamped to [-1, W] x [-1, H] before conversion
    auto px_lo = [](float v, float lim) { return fminf(fmaxf(floorf(v) - 2.0f, -1.0f), lim); };
    auto px_hi = [](float v, float lim) { return fminf(fmaxf(ceilf(v) + 2.0f, -1.0f), lim); };
    const int32_t ix0 = max((int32_t)px_lo(x0, (float)W), 0), ix1 = min((int32_t)px_hi(x1, (float)W), W - 1);
    const int32_t iy0 = max((int32_t)px_lo(y0, (float)H), 0), iy1 = min((int32_t)px_hi(y1, (float)H), H - 1);
    if (ix0 > ix1 || iy0 > iy1) return true;  // no pixel centre of the view in reach
    const uint32_t pitch0 = vw->hiz_rx * 8u;
    const uint32_t* level0 = vw->hiz;
    // the ≤ 16 tiles (or regions) under the box, loaded all at once (no
    // load waits on the previous one's compare), then their minimum
    auto box_min = [](const uint32_t* level, uint32_t pitch, int32_t tx0, int32_t tx1, int32_t ty0, int32_t ty1) {
        const int32_t n = (tx1 - tx0 + 1) * (ty1 - ty0 + 1);
        uint32_t m = 0xFFFFFFFFu;
        int32_t tx = tx0, ty = ty0;
#pragma unroll
        for (int32_t k = 0; k < 16; k++) {
            if (k < n) {
                m = min(m, __ldcg(level + (size_t)ty * pitch + tx));
                if (++tx > tx1) {
                    tx = tx0;
                    ty++;
                }
            }
        }
        return m;
    };
    int32_t tx0 = ix0 >> 3, tx1 = ix1 >> 3, ty0 = iy0 >> 3, ty1 = iy1 >> 3;
    if ((tx1 - tx0 + 1) * (ty1 - ty0 + 1) <= 16) return box_min(level0, pitch0, tx0, tx1, ty0, ty1) > zbits;
    const uint32_t* level1 = level0 + (size_t)pitch0 * vw->hiz_ry * 8u;
    tx0 = ix0 >> 6, tx1 = ix1 >> 6, ty0 = iy0 >> 6, ty1 = iy1 >> 6;
    if ((tx1 - tx0 + 1) * (ty1 - ty0 + 1) > 16) return false;
    return box_min(level1, vw->hiz_rx, tx0, tx1, ty0, ty1) > zbits;
}

// After the hierarchical depth: every visible meshlet of the visibility
// views that is not an occluder (opaque, then alpha clip) is tested against
// it, and the survivors go to the view's survivor lists for the second
// raster pass (warp-aggregated appends, any order).  Threads stride over
// the (view, meshlet) pairs.  Also resets the raster's claim and big-triangle
// words for that pass (nothing of the occluder pass runs any more).
__device__ void phase_occlusion_filter(const FrameDev& f, uint32_t view_begin, uint32_t n_views, uint64_t gtid,
                                       uint64_t gstride) {
    const uint32_t md = f.max_draws, lane = threadIdx.x & 31;
    if (gtid == 0) {
        f.status[kStRasterClaim] = 0u;
        f.status[kStRasterClaimGeneral] = 0u;
        f.status[kStBigClaim] = 0u;
        f.status[kStWholeClaim] = 0u;
        *reinterpret_cast<unsigned long long*>(f.status + kStBigPacked) = 0ull;
    }
    for (uint32_t v = 0; v < n_views; v++) {
        const ViewDev* vw = f.views + view_begin + v;
        if (vw->kind != kViewVisibility || !vw->lists) continue;
        const uint32_t* cnt = reinterpret_cast<const uint32_t*>(vw->draws);
        const uint32_t nop = min(cnt[0], md), nal = min(cnt[1], md);
        const lh_mat4& pv = vw->uniforms->combined_perspective_view;
        const uint64_t n = (uint64_t)nop + nal;
        // whole warps iterate together (the appends are warp collectives)
        for (uint64_t base = gtid - lane; base < n; base += gstride) {
            const uint64_t i = base + lane;
            uint32_t cl = kSlotsOccluders, slot = 0;  // the list it joins; none: an occluder, or culled
            if (i < n) {
                const bool alpha = i >= nop;
                slot = alpha ? md + (uint32_t)(i - nop) : (uint32_t)i;
                const RasterDraw* rd = vw->rdraws + slot;
                // both loads issued together (one round trip)
                const uint32_t bits = __ldcg(&rd->bits);
                const float4 sp4 = __ldcg(reinterpret_cast<const float4*>(rd->sphere));
                if (!(bits & (kDrawOccluder | kDrawNoCentre))) {
                    const float sp[4] = {sp4.x, sp4.y, sp4.z, sp4.w};
                    if (!vw->hiz || !hiz_occluded(vw, pv, sp)) cl = alpha ? kSlotsAlpha : (bits & kDrawGeneral) ? kSlotsGeneral : kSlotsOpaque;
                }
            }
#pragma unroll
            for (uint32_t k = 0; k < kViewLists; k++) {
                if (k == kSlotsOccluders) continue;
                const uint32_t m = __ballot_sync(0xFFFFFFFFu, cl == k);
                if (!m) continue;
                const uint32_t leader = __ffs(m) - 1;
                uint32_t first = 0;
                if (lane == leader)
                    first = atomicAdd(&vw->claim[k == kSlotsOpaque  ? kClaimSurvivorsOpaque
                                                 : k == kSlotsAlpha ? kClaimSurvivorsAlpha
                                                                    : kClaimGeneral],
                                      __popc(m));
                first = __shfl_sync(0xFFFFFFFFu, first, leader);
                const uint32_t pos = first + __popc(m & ((1u << lane) - 1u));
                if (cl == k && pos < md) vw->lists[(size_t)k * md + pos] = slot;
            }
        }
    }
}

}  // namespace
}  // namespace lh
