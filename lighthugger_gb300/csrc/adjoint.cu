// Backward of the lighting resolve (render_geometry.comp:70-266) with the
// visibility held fixed: one thread per pixel recomputes the forward inputs
// from the visibility buffer (triangle, vertices, cascade, compare results)
// and runs the hand-written reverse pass of shade.cuh, then adds the
// gradients into the caller's buffers.  Targets every lane of a warp shares
// (light direction / colour, a material's base-colour factor) are summed
// across the warp first, so they take one atomic per warp.
//
// Bound by instruction issue and the latency of its gathers at 16 warps an
// SM (128 registers; 24 warps at 80 spill and take 760 us).  Every pixel by
// itself: triangles are small where it matters (15 distinct ones in a row of
// 32 pixels in the 1080p scene seen from above; records shared by a warp's
// pixels, 8 to 16 triangles at a time, took 4 times as long).  The gradients
// of slivers are ill-conditioned, so a pixel's arithmetic keeps its order
// and rounding.  That scene: 505 us with the triangle's terms formed three
// times a pixel and four looks at the runs per texture sample, 405 now.
#include <algorithm>

#include "exact_div.cuh"
#include "frame_phases.cuh"
#include "shade.cuh"
#include "tma.cuh"

namespace lh {
namespace {

using shade::Bilinear;
using shade::PixelGrad;
using shade::PixelParams;
using shade::v2;
using shade::v3;

struct DeviceSampler {
    const FrameDev* f;
    __device__ Bilinear<float> sample(uint32_t index, v2<float> uv) const {
        Bilinear<float> s;
        s.index = index;
        if (index >= f->n_textures) {
            for (int c = 0; c < 4; c++) s.t00[c] = s.t10[c] = s.t01[c] = s.t11[c] = 0.0f;
            s.a = s.b = 0.0f;
            s.size_u = s.size_v = 0.0f;
            s.i0 = s.i1 = s.j0 = s.j1 = 0;
            return s;
        }
        const lh_texture t = f->textures[index];
        const float4* tex = f->tex_linear[index];
        float u = uv.x * (float)t.width - 0.5f, v = uv.y * (float)t.height - 0.5f;
        if (!(fabsf(u) < 1e9f)) u = 0.0f;
        if (!(fabsf(v) < 1e9f)) v = 0.0f;
        float fu = floorf(u), fv = floorf(v);
        s.a = u - fu;
        s.b = v - fv;
        const int32_t i0 = (int32_t)fu, j0 = (int32_t)fv;
        const int32_t W = (int32_t)t.width, H = (int32_t)t.height;
        s.size_u = (float)t.width;
        s.size_v = (float)t.height;
        // i0 + 1 wraps to the texel after i0's (or 0 past the last)
        s.i0 = wrap_texel(i0, W);
        s.i1 = s.i0 + 1 == W ? 0 : s.i0 + 1;
        s.j0 = wrap_texel(j0, H);
        s.j1 = s.j0 + 1 == H ? 0 : s.j0 + 1;
        auto texel = [&](int32_t i, int32_t j, float* o) {
            const float4 p = __ldg(tex + ((size_t)j * W + i));
            o[0] = p.x;
            o[1] = p.y;
            o[2] = p.z;
            o[3] = p.w;
        };
        texel(s.i0, s.j0, s.t00);
        texel(s.i1, s.j0, s.t10);
        texel(s.i0, s.j1, s.t01);
        texel(s.i1, s.j1, s.t11);
        return s;
    }
    __device__ float shadow_cmp(uint32_t layer, int32_t i, int32_t j, float ref) const {
        const int32_t S = (int32_t)f->shadow_size;
        i = i < 0 ? 0 : (i > S - 1 ? S - 1 : i);
        j = j < 0 ? 0 : (j > S - 1 ? S - 1 : j);
        return ref < __ldg(f->shadow_maps + ((size_t)layer * S + j) * S + i) ? 1.0f : 0.0f;
    }
};

// The 4 x 4 window inside the map: no clamping (compare_window of shade.cuh).
__device__ uint32_t compare_window(const DeviceSampler& smp, uint32_t layer, int32_t i, int32_t j, float ref) {
    const int32_t S = (int32_t)smp.f->shadow_size;
    uint32_t win = 0;
    if (i >= 0 && j >= 0 && i <= S - 4 && j <= S - 4) {
        const float* row = smp.f->shadow_maps + ((size_t)layer * S + j) * S + i;
#pragma unroll
        for (int r = 0; r < 4; r++, row += S)
#pragma unroll
            for (int c = 0; c < 4; c++) win |= (ref < __ldg(row + c) ? 1u : 0u) << (4 * r + c);
        return win;
    }
#pragma unroll 1
    for (int k = 0; k < 16; k++) win |= (smp.shadow_cmp(layer, i + (k & 3), j + (k >> 2), ref) != 0.0f ? 1u : 0u) << k;
    return win;
}

constexpr uint32_t kFull = 0xFFFFFFFFu;
// Launch shape: tiles of 32 x ROWS pixels (ROWS = 4, 8 or 16, chosen at run
// time through lh_tuning.backward_rows), one warp per row, and the threads
// per SM the register budget is cut for (LH_BWD_MIN_BLOCKS blocks of 8 rows:
// 512 threads, 128 registers a thread, at every ROWS).
#ifndef LH_BWD_MIN_BLOCKS
#define LH_BWD_MIN_BLOCKS 2
#endif
constexpr uint32_t kCacheSlots = 256;     // shared-memory accumulators of hot gradient addresses
constexpr uint32_t kSmallTexture = 64;    // textures of at most this many texels go through them

// Shared-memory reads that the compiler neither merges nor moves: a value is
// read where it is used instead of held in a register through the pixel.
__device__ __forceinline__ float lds_f32(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}

// The terms of a pixel's triangle (shade.cuh's TriTerms and the instance's
// normal transform) in the thread's own column of shared memory, word j of
// the warp's 32 threads side by side.  They serve the forward and both parts
// of the reverse, each computed once: in registers they would not last
// through the BRDF, and recomputed where they are used they were a fifth of
// the kernel's instructions.
enum : uint32_t {
    kTermW = 0,        // 9: camera-relative positions
    kTermN = 9,        // 9: normalised normals
    kTermRn = 18,      // 3: 1 / length of the raw normals
    kTermC = 21,       // 6: clip x, y
    kTermIw = 27,      // 3: 1 / clip w
    kTermProj = 30,    // 6: projected x, y
    kTermSlope = 36,   // 6: slopes of lambda / w
    kTermSum = 42,     // 2: their sums
    kTermInvDet = 44,  // 1
    kTermUv = 45,      // 6: uvs times the texture scale
    kTermTs = 51,      // 2: texture scale
    kTermToff = 53,    // 2: texture offset
    kTermNt = 55,      // 9: normal transform
    kTerms = 64
};
struct ThreadTri {
    uint32_t at;  // shared-memory address of the thread's word 0
    __device__ float get(uint32_t j) const { return lds_f32(at + 128 * j); }
    __device__ void set(uint32_t j, float v) const { asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + 128 * j), "f"(v)); }
    __device__ v2<float> get2(uint32_t j) const { return {get(j), get(j + 1)}; }
    __device__ v3<float> get3(uint32_t j) const { return {get(j), get(j + 1), get(j + 2)}; }
    __device__ void set2(uint32_t j, v2<float> v) const { set(j, v.x), set(j + 1, v.y); }
    __device__ void set3(uint32_t j, v3<float> v) const { set(j, v.x), set(j + 1, v.y), set(j + 2, v.z); }
    __device__ v3<float> W(int k) const { return get3(kTermW + 3 * k); }
    __device__ v3<float> nk(int k) const { return get3(kTermN + 3 * k); }
    __device__ float rn(int k) const { return get(kTermRn + k); }
    __device__ v2<float> C(int k) const { return get2(kTermC + 2 * k); }
    __device__ float iw(int k) const { return get(kTermIw + k); }
    __device__ v2<float> n(int k) const { return get2(kTermProj + 2 * k); }
    __device__ v2<float> dd(int k) const { return get2(kTermSlope + 2 * k); }
    __device__ v2<float> s() const { return get2(kTermSum); }
    __device__ float inv_det() const { return get(kTermInvDet); }
    __device__ v2<float> uvs(int k) const { return get2(kTermUv + 2 * k); }
    __device__ v2<float> ts() const { return get2(kTermTs); }
    __device__ v2<float> toff() const { return get2(kTermToff); }
};

// Fixed inputs of a pixel for shade.cuh; its matrices are read from shared
// memory at each use: PV and the cascade's UVS, camera-relative, from the
// block's copies, the normal transform from the thread's terms.  `uvs3`
// points at the column 3 in use (absolute for the decisions).
struct DeviceFixed : shade::PixelScalars {
    uint32_t pv;         // 16 floats, column-major
    uint32_t uvs, uvs3;  // 16 floats of the pixel's cascade; 4 floats
    uint32_t nt;         // 9 words of the thread's
    __device__ float PV(int c, int r) const { return lds_f32(pv + 16 * c + 4 * r); }
    __device__ float UVS(int c, int r) const { return lds_f32((c == 3 ? uvs3 : uvs + 16 * c) + 4 * r); }
    __device__ float NT(int c, int r) const { return lds_f32(nt + 128 * (3 * c + r)); }
};
// The same with PV in registers, for the transforms of the three vertices.
struct VertexFixed : shade::PixelScalars {
    const float *pv, *pv3;  // shared
    __device__ float PV(int c, int r) const { return c == 3 ? pv3[r] : pv[4 * c + r]; }
};

// Block-shared copies of the frame's matrices for DeviceFixed.
struct FrameMats {
    float pv[16];        // combined_perspective_view
    float uvs[4][16];    // uv_space_shadow_matrices
    float rel[20];       // column 3 of PV T(cam) and of UVS_c T(cam) (rel_columns)
};

__device__ __forceinline__ float warp_sum(float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

// Per-block accumulators for addresses that many pixels of a block add to
// (a material's base-colour factor, the texels of 1 x 1 constant textures):
// open addressing over 256 slots keyed by the destination address, four
// probes, then a plain global atomic.  Slots are flushed once at block end.
struct HotCache {
    unsigned long long key[kCacheSlots];
    float sum[kCacheSlots];
};

__device__ __forceinline__ void cache_add(HotCache& c, float* addr, float v) {
    const unsigned long long k = (unsigned long long)addr;
    const uint32_t h = ((uint32_t)(k >> 2) * 2654435761u) >> 24;
    for (uint32_t probe = 0; probe < 4; probe++) {
        const uint32_t s = (h + probe) & (kCacheSlots - 1u);
        unsigned long long cur = *reinterpret_cast<volatile unsigned long long*>(&c.key[s]);
        if (cur == 0ull) cur = atomicCAS(&c.key[s], 0ull, k);
        if (cur == 0ull || cur == k) {
            atomicAdd(&c.sum[s], v);
            return;
        }
    }
    atomicAdd(addr, v);
}

// Runs of equal keys along the warp (a warp is one row of 32 pixels, so a
// triangle or a texel covers contiguous lanes): `end` is one past the last
// lane of this lane's run, `head` marks its first lane.
#ifndef LH_RUN_SPAN
#define LH_RUN_SPAN 1
#endif
struct Run {
    uint32_t end;   // first lane after this lane's run
    uint32_t span;  // longest run of the warp (warp uniform)
    bool head;
};

__device__ __forceinline__ Run run_of(unsigned long long key) {
    const uint32_t lane = threadIdx.x;
    const unsigned long long prev = __shfl_up_sync(kFull, key, 1);
    const bool head = lane == 0 || prev != key;
    const uint32_t heads = __ballot_sync(kFull, head);
    const uint32_t later = heads & ~((2u << lane) - 1u);
    const uint32_t end = later ? (uint32_t)__ffs(later) - 1u : 32u;
    return {end, __reduce_max_sync(kFull, end - lane), head};
}

// Sums of v[i] over the lanes [lane, end) of the run: the full run sums at
// its head.  Doubling steps stop at the warp's longest run: a step of
// o >= span adds nothing for any lane (end - lane <= span), so the sums are
// those of the full five steps; the N values share each step's shuffles.
template <int N>
__device__ __forceinline__ void run_sums(float (&v)[N], const Run& r) {
    const uint32_t lane = threadIdx.x;
#if LH_RUN_SPAN
    for (uint32_t o = 1; o < r.span; o <<= 1) {
#else
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
#endif
#pragma unroll
        for (int i = 0; i < N; i++) {
            const float w = __shfl_down_sync(kFull, v[i], o);
            if (lane + o < r.end) v[i] += w;
        }
    }
}

// What the scatter needs of a differentiated pixel besides its gradients.
struct PixelOut {
    bool ok;                // differentiated (covered, no normal map)
    uint32_t packed;        // visibility ID: triangle within the view
    const Instance* inst;
    const lh_mesh_grads* rec;  // may be null
    uint32_t idx[3];
};

// Recompute the forward of pixel (x, y) from the visibility buffer and run
// the surface half of the reverse pass of shade.cuh for the upstream
// gradient at that pixel; fx, tri and st carry what the geometry half needs.
// `M` holds the block's copies of the frame matrices.
__device__ __forceinline__ void pixel_backward(const FrameDev& f, const float4* grad, const lh_grad_targets& t,
                                               const FrameMats& M, uint32_t x, uint32_t y, float rcp_w,
                                               PixelGrad<float>& g, PixelOut& o, DeviceFixed& fx, const ThreadTri& tri,
                                               shade::SurfaceState<float>& st) {
    const Uniforms& u = *f.uniforms;
    const uint32_t W = u.window_size.x, H = u.window_size.y;
    o.ok = false;
    bool active = x < W && y < H;
    unsigned long long vis = 0;
    if (active) vis = __ldcs(reinterpret_cast<const unsigned long long*>(f.visibility) + (size_t)y * W + x);
    active = active && u2f((uint32_t)(vis >> 32)) != 0.0f;
    if (!active) return;
    const uint32_t packed = (uint32_t)vis;
    const uint32_t slot = packed & ((1u << 24) - 1u), tri_index = packed >> 24;
    // the slot's draw record (written by the meshlet cull): the instance and
    // the index / micro-index addresses already offset to the meshlet, so
    // the vertex loads do not wait on the reference, MeshInfo and Meshlet
    const RasterDraw rd = f.views[0].rdraws[slot];
    const Instance* inst = f.instances + rd.instance;
    const MeshInfoResolve mi = load_mesh_info_resolve(mesh_info_of(inst));
    if (mi.normal_tex != UNUSED_TEXTURE_INDEX) return;  // normal-mapped: not differentiated
    const float4 gp = __ldcs(grad + (size_t)y * W + x);
    const uint8_t* micro = reinterpret_cast<const uint8_t*>(rd.micro) + tri_index * 3;
    const uint32_t flags = mi.flags;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const uint32_t vi = __ldg(micro + k);
        o.idx[k] = (flags & MESH_INFO_FLAGS_32_BIT_INDICES) ? __ldg(reinterpret_cast<const uint32_t*>(rd.indices) + vi)
                                                            : __ldg(reinterpret_cast<const uint16_t*>(rd.indices) + vi);
    }
    PixelParams<float> p;
    const lh_mat4& T = inst->transform;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        f3 w = world_pos(T, load_position(rd.positions, flags, o.idx[k]));
        p.W[k] = {w.x, w.y, w.z};
        f3 nr = load_normal_raw(mi.normals, flags, o.idx[k]);
        p.N[k] = {nr.x, nr.y, nr.z};
        f2 uvr = load_uv_raw(mi.uvs, flags, o.idx[k]);
        p.UV[k] = {uvr.x, uvr.y};
    }
    p.bcf = {mi.base_color_factor.x, mi.base_color_factor.y, mi.base_color_factor.z};
    p.sun = {u.sun_dir.x, u.sun_dir.y, u.sun_dir.z};
    p.light = {u.sun_intensity.x, u.sun_intensity.y, u.sun_intensity.z};
    // x / W * 2 - 1 with the quotient from the reciprocal (the same bits)
    const float qx = W <= (uint32_t)kExactDivMaxCount ? div_by_count((float)x, (float)W, rcp_w) : (float)x / (float)W;
    VertexFixed vx;
    vx.pv = M.pv;
    vx.pv3 = M.pv + 12;
    vx.ndc[0] = fx.ndc[0] = qx * 2.0f - 1.0f;
    vx.ndc[1] = fx.ndc[1] = (float)y / (float)H * 2.0f - 1.0f;
    vx.ts[0] = mi.texture_scale.x;
    vx.ts[1] = mi.texture_scale.y;
    vx.toff[0] = mi.texture_offset.x;
    vx.toff[1] = mi.texture_offset.y;
    fx.thin = (flags & MESH_INFO_FLAGS_ALPHA_CLIP) ? 1u : 0u;
    fx.bias = fx.thin ? 0.000002f : 0.0f;
    fx.shadow_size = (float)f.shadow_size;
    fx.base_tex = mi.base_tex;
    fx.mr_tex = mi.mr_tex;
    fx.has_normal_map = 0u;
    DeviceSampler smp{&f};
    {
        // the world position the forward interpolated, in its absolute float
        // arithmetic, picks the cascade (render_geometry.comp:183-196) and
        // places the PCF taps
        const v3<float> world = shade::forward_world(vx, p);
        uint32_t ci;
        for (ci = 0; ci < 4; ci++) {
            const lh_mat4& m = *reinterpret_cast<const lh_mat4*>(M.uvs[ci]);
            f4 sc = mul(m, f4{world.x, world.y, world.z, 1.0f});
            float ox = sc.x - 0.5f, oy = sc.y - 0.5f;
            if (fabsf(ox) < 0.5f && fabsf(oy) < 0.5f) break;
        }
        fx.cascade = ci;
        fx.uvs = smem_u32(M.uvs[ci > 3 ? 3 : ci]);
        fx.uvs3 = fx.uvs + 48;
        // face flip, far-plane test and compare results exactly as the forward
        const f3 a{p.W[0].x, p.W[0].y, p.W[0].z}, b{p.W[1].x, p.W[1].y, p.W[1].z}, c{p.W[2].x, p.W[2].y, p.W[2].z};
        fx.flip = faces_away(cross(b - a, c - a), ld3(u.camera_pos) - f3{world.x, world.y, world.z}) ? -1.0f : 1.0f;
        shade::decide_shadow(fx, world, smp);
    }
    // the continuous part in camera-relative coordinates: W - cam is
    // (nearly) exact, and PV T(cam), UVS T(cam) were formed in double
    const uint32_t layer = fx.cascade > 3 ? 3u : fx.cascade;
    fx.uvs3 = smem_u32(M.rel + 4 + 4 * layer);
    fx.pv = smem_u32(M.pv);
    fx.nt = tri.at + 128 * kTermNt;
    fx.cam[0] = fx.cam[1] = fx.cam[2] = 0.0f;
    {
#pragma unroll
        for (int k = 0; k < 3; k++)
            p.W[k] = {p.W[k].x - u.camera_pos.x, p.W[k].y - u.camera_pos.y, p.W[k].z - u.camera_pos.z};
        vx.pv3 = M.rel;
        const shade::TriTerms<float> terms = shade::tri_terms(vx, p);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            tri.set3(kTermW + 3 * k, terms.w_[k]);
            tri.set3(kTermN + 3 * k, terms.nk_[k]);
            tri.set(kTermRn + k, terms.rn_[k]);
            tri.set2(kTermC + 2 * k, terms.c_[k]);
            tri.set(kTermIw + k, terms.iw_[k]);
            tri.set2(kTermProj + 2 * k, terms.n_[k]);
            tri.set2(kTermSlope + 2 * k, terms.dd_[k]);
            tri.set2(kTermUv + 2 * k, terms.uvs_[k]);
            const lh_vec3& nt = inst->normal_transform.cols[k];
            tri.set3(kTermNt + 3 * k, v3<float>{nt.x, nt.y, nt.z});
        }
        tri.set2(kTermSum, terms.s_);
        tri.set(kTermInvDet, terms.inv_det_);
        tri.set2(kTermTs, terms.ts_);
        tri.set2(kTermToff, terms.toff_);
    }
    v3<float> out;
    shade::shade_surface<float>(fx, p, tri, smp, &out, v3<float>{gp.x, gp.y, gp.z}, &g, &st);
    o.ok = true;
    o.packed = packed;
    o.inst = inst;
    o.rec = t.instance_grads ? reinterpret_cast<const lh_mesh_grads*>(
                                   reinterpret_cast<const uint64_t*>(t.instance_grads)[rd.instance])
                             : nullptr;
}

// The four texels of one bilinear sample (00, 10, 01, 11): summed over the
// run of pixels along the warp that sample the same four, and added to the
// texture's gradient image, channels [c0, c0 + NC).  Equal first texels of
// one texture (`index`; others may share its image) have equal others, so one
// look at the runs serves all four (each by itself: 120 us of the kernel's
// 470 at 1920 x 1080, 74 so).  In a texture one texel wide or high, taps on the
// same texel are merged.
template <int NC>
__device__ __forceinline__ void scatter_texels(HotCache& cache, float* dst, const lh_texture& t, uint32_t index, const int32_t ij[4],
                                               float v[4][NC], int c0) {
    const int32_t W = dst ? (int32_t)t.width : 0;
    float* const first = dst ? dst + 4 * ((size_t)ij[2] * W + ij[0]) : nullptr;
    if (!__any_sync(kFull, first != nullptr)) return;
    const Run r = run_of((unsigned long long)first ^ ((unsigned long long)index << 48));  // (addresses have 48 bits)
    if (r.span > 1) {
        float s[4 * NC];
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int c = 0; c < NC; c++) s[q * NC + c] = v[q][c];
        run_sums(s, r);
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int c = 0; c < NC; c++) v[q][c] = s[q * NC + c];
    }
    if (!r.head || !first) return;
    const bool one_wide = ij[0] == ij[1], one_high = ij[2] == ij[3];
    if (one_wide || one_high) {
#pragma unroll
        for (int c = 0; c < NC; c++) {
            if (one_wide) v[0][c] += v[1][c], v[2][c] += v[3][c];
            if (one_high) v[0][c] += v[2][c], v[1][c] += v[3][c];
        }
    }
    const bool small = t.width * t.height <= kSmallTexture;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        if (((q & 1) && one_wide) || ((q >> 1) && one_high)) continue;
        float* a = dst + 4 * ((size_t)ij[2 + (q >> 1)] * W + ij[q & 1]);
        if (!small && ((uintptr_t)a & 15u) == 0) {
            // one vector reduction per texel (the other channels add 0)
            float4 d = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            float* dc = &d.x;
#pragma unroll
            for (int c = 0; c < NC; c++) dc[c0 + c] = v[q][c];
            atomicAdd(reinterpret_cast<float4*>(a), d);
        } else {
#pragma unroll
            for (int c = 0; c < NC; c++) {
                if (small) cache_add(cache, a + c0 + c, v[q][c]);
                else atomicAdd(a + c0 + c, v[q][c]);
            }
        }
    }
}

// Three neighbouring floats: a pair and a single, the pair where it is
// aligned to 8 bytes.
__device__ __forceinline__ void add3(float* p, f3 v) {
    const bool even = ((uintptr_t)p & 7u) == 0;
    atomicAdd(reinterpret_cast<float2*>(even ? p : p + 1), even ? make_float2(v.x, v.y) : make_float2(v.y, v.z));
    atomicAdd(even ? p + 2 : p, even ? v.z : v.x);
}

// Column 3 of PV T(cam) and of UVS_c T(cam) for the 4 cascades, in double
// and rounded once: rel[r] for PV, rel[4 + 4c + r] for cascade c.  Threads
// 0..19 of the block each form one entry.
__device__ __forceinline__ void rel_columns(const FrameDev& f, uint32_t tid, float* rel) {
    if (tid >= 20) return;
    const Uniforms& u = *f.uniforms;
    const lh_mat4& m = tid < 4 ? u.combined_perspective_view : f.misc->uv_space_shadow_matrices[(tid - 4) / 4];
    const uint32_t r = tid & 3u;
    const float* c0 = &m.cols[0].x;
    const float* c1 = &m.cols[1].x;
    const float* c2 = &m.cols[2].x;
    const float* c3 = &m.cols[3].x;
    const double cx = u.camera_pos.x, cy = u.camera_pos.y, cz = u.camera_pos.z;
    rel[tid] = (float)((double)c3[r] + (((double)c0[r] * cx + (double)c1[r] * cy) + (double)c2[r] * cz));
}

// One thread per pixel over 32 x kBwdRows tiles; a grid of resident blocks strides
// over the tiles.  Gradients of the three vertices of a triangle are summed
// over the triangle's run of pixels in the warp's row before the atomics;
// the light gradients stay in registers until block end; base-colour
// factors and small textures accumulate in the block's HotCache.
template <int ROWS>
__global__ void __launch_bounds__(32 * ROWS, LH_BWD_MIN_BLOCKS * 8 / ROWS)
    k_resolve_backward(FrameDev f, const float4* grad, lh_grad_targets t, uint32_t tiles_x, uint32_t n_tiles) {
    __shared__ HotCache cache;
    __shared__ float s_light[ROWS][6];
    pdl_enter();
    __shared__ __align__(16) FrameMats s_mats;
    extern __shared__ __align__(16) float s_terms[];  // [ROWS][kTerms][32]
    const uint32_t tid = threadIdx.y * 32 + threadIdx.x;
    for (uint32_t s = tid; s < kCacheSlots; s += 32 * ROWS) {
        cache.key[s] = 0ull;
        cache.sum[s] = 0.0f;
    }
    if (tid < 16) s_mats.pv[tid] = (&f.uniforms->combined_perspective_view.cols[0].x)[tid];
    if (tid < 64) s_mats.uvs[tid / 16][tid % 16] = (&f.misc->uv_space_shadow_matrices[tid / 16].cols[0].x)[tid % 16];
    rel_columns(f, tid, s_mats.rel);
    __syncthreads();
    float acc[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    const uint64_t* tex_targets = reinterpret_cast<const uint64_t*>(t.texture_grads);
    const ThreadTri tri{smem_u32(s_terms + threadIdx.y * (kTerms * 32) + threadIdx.x)};
    const float rcp_w = 1.0f / (float)f.uniforms->window_size.x;
    for (uint32_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const uint32_t x = (tile % tiles_x) * 32 + threadIdx.x, y = (tile / tiles_x) * ROWS + threadIdx.y;
        PixelGrad<float> g;
        PixelOut o;
        DeviceFixed fx;
        shade::SurfaceState<float> st;
        pixel_backward(f, grad, t, s_mats, x, y, rcp_w, g, o, fx, tri, st);
        if (o.ok) {
            acc[0] += g.sun.x;
            acc[1] += g.sun.y;
            acc[2] += g.sun.z;
            acc[3] += g.light.x;
            acc[4] += g.light.y;
            acc[5] += g.light.z;
        }
        const lh_mesh_grads* mg = o.ok ? o.rec : nullptr;
        // base-colour factor of the pixel's MeshInfo record
        float* bcf_dst = mg ? reinterpret_cast<float*>(mg->base_color_factor) : nullptr;
        if (__any_sync(kFull, bcf_dst != nullptr)) {
            const Run r = run_of((unsigned long long)bcf_dst);
            float b[3] = {bcf_dst ? g.bcf.x : 0.0f, bcf_dst ? g.bcf.y : 0.0f, bcf_dst ? g.bcf.z : 0.0f};
            run_sums(b, r);
            if (r.head && bcf_dst) {
                cache_add(cache, bcf_dst, b[0]);
                cache_add(cache, bcf_dst + 1, b[1]);
                cache_add(cache, bcf_dst + 2, b[2]);
            }
        }
        if (tex_targets) {
            // base colour (rgb of the texel) and metallic-roughness (g, b)
            const uint32_t bi = o.ok && g.base_index < f.n_textures ? g.base_index : 0u;
            const uint32_t mi = o.ok && g.mr_index < f.n_textures ? g.mr_index : 0u;
            float* base = o.ok && g.base_index < f.n_textures ? reinterpret_cast<float*>(tex_targets[bi]) : nullptr;
            float* mr = o.ok && g.mr_index < f.n_textures ? reinterpret_cast<float*>(tex_targets[mi]) : nullptr;
            scatter_texels<3>(cache, base, f.textures[bi], bi, g.base_ij, g.base_texel, 0);
            scatter_texels<2>(cache, mr, f.textures[mi], mi, g.mr_ij, g.mr_texel, 1);  // roughness (g), metallic (b)
        }
        // the geometry half of the reverse, then the vertex attributes: one
        // run per triangle
        if (o.ok) shade::shade_geometry<float>(fx, tri, st, &g);
        if (__any_sync(kFull, mg != nullptr)) {
            const Run r = run_of(mg ? (unsigned long long)o.packed : ~0ull);
            float v[24];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                v[k * 8 + 0] = g.W[k].x;
                v[k * 8 + 1] = g.W[k].y;
                v[k * 8 + 2] = g.W[k].z;
                v[k * 8 + 3] = g.N[k].x;
                v[k * 8 + 4] = g.N[k].y;
                v[k * 8 + 5] = g.N[k].z;
                v[k * 8 + 6] = g.UV[k].x;
                v[k * 8 + 7] = g.UV[k].y;
            }
            run_sums(v, r);
            if (r.head && mg) {
                const lh_mesh_grads d = *mg;
                const lh_mat4& T = o.inst->transform;
                const f3 c0{T.cols[0].x, T.cols[0].y, T.cols[0].z}, c1{T.cols[1].x, T.cols[1].y, T.cols[1].z},
                    c2{T.cols[2].x, T.cols[2].y, T.cols[2].z};
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const float* vk = v + k * 8;
                    if (d.positions) {
                        // W = M3 P + t: dP = M3^T dW
                        const f3 gw{vk[0], vk[1], vk[2]};
                        add3(reinterpret_cast<float*>(d.positions) + (size_t)o.idx[k] * 3,
                             f3{dot(c0, gw), dot(c1, gw), dot(c2, gw)});
                    }
                    if (d.normals)
                        add3(reinterpret_cast<float*>(d.normals) + (size_t)o.idx[k] * 3, f3{vk[3], vk[4], vk[5]});
                    if (d.uvs) {
                        float* p = reinterpret_cast<float*>(d.uvs) + (size_t)o.idx[k] * 2;
                        if (((uintptr_t)p & 7u) == 0) {
                            atomicAdd(reinterpret_cast<float2*>(p), make_float2(vk[6], vk[7]));
                        } else {
                            atomicAdd(p, vk[6]);
                            atomicAdd(p + 1, vk[7]);
                        }
                    }
                }
            }
        }
    }
    // light direction / colour: one atomic per value per block
#pragma unroll
    for (int i = 0; i < 6; i++) {
        const float s = warp_sum(acc[i]);
        if (threadIdx.x == 0) s_light[threadIdx.y][i] = s;
    }
    __syncthreads();
    if (tid < 6) {
        float s = 0.0f;
        for (int w = 0; w < ROWS; w++) s += s_light[w][tid];
        float* dst = tid < 3 ? reinterpret_cast<float*>(t.light_dir) : reinterpret_cast<float*>(t.light_color);
        if (dst) atomicAdd(dst + (tid % 3), s);
    }
    for (uint32_t s = tid; s < kCacheSlots; s += 32 * ROWS)
        if (cache.key[s]) atomicAdd(reinterpret_cast<float*>(cache.key[s]), cache.sum[s]);
}

int g_backward_blocks_per_sm[3] = {-1, -1, -1};

template <int ROWS>
cudaError_t launch_backward_rows(const FrameDev& f, uint32_t width, uint32_t height, const float4* grad,
                                 const lh_grad_targets& t, cudaStream_t s, int& blocks_per_sm) {
    constexpr uint32_t kShared = ROWS * kTerms * 32 * (uint32_t)sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(k_resolve_backward<ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kShared);
    if (e != cudaSuccess) return e;
    if (blocks_per_sm < 0) {
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_resolve_backward<ROWS>, 32 * ROWS, kShared) != cudaSuccess)
            n = 1;
        blocks_per_sm = n > 0 ? n : 1;
    }
    int dev = 0, sms = 0;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    const uint32_t tiles_x = (width + 31) / 32, tiles_y = (height + ROWS - 1) / ROWS;
    const uint32_t n_tiles = tiles_x * tiles_y;
    if (n_tiles == 0) return cudaSuccess;
    const uint32_t grid = std::min<uint32_t>(n_tiles, (uint32_t)(sms * blocks_per_sm));
    return launch_pdl_shared(k_resolve_backward<ROWS>, dim3(grid), dim3(32, ROWS), kShared, s, f, grad, t, tiles_x, n_tiles);
}

}  // namespace

cudaError_t launch_resolve_backward(const FrameDev& f, uint32_t width, uint32_t height, const float4* grad,
                                    const lh_grad_targets& t, cudaStream_t s) {
    switch (f.backward_rows) {
        case 4: return launch_backward_rows<4>(f, width, height, grad, t, s, g_backward_blocks_per_sm[0]);
        case 16: return launch_backward_rows<16>(f, width, height, grad, t, s, g_backward_blocks_per_sm[2]);
        default: return launch_backward_rows<8>(f, width, height, grad, t, s, g_backward_blocks_per_sm[1]);
    }
}

}  // namespace lh
