// Display transform (src/shaders/display_transform.comp:5-81): the
// scene-referred HDR image through a 48^3 LUT tonemap (tony_mc_mapface's
// encoding: stimulus / (stimulus + 1), LUT sampled trilinearly with clamp to
// edge at texel centres), the optional cascade overlay of debug_shadowmaps,
// and the sRGB transfer function, written as RGBA8.  The reference's LUT
// (external/tony-mc-mapface) is an empty submodule here, so callers pass
// their LUT or get a stand-in identity LUT (display = stimulus / (1 +
// stimulus) per channel).
#include "frame_phases.cuh"

namespace lh {
namespace {

constexpr int kLutDims = 48;

__device__ __forceinline__ float log2f_approx(float x) {
    float r;
    asm("lg2.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float exp2f_approx(float x) {
    float r;
    asm("ex2.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Trilinear sample of a float4[48][48][48] LUT (x fastest) at normalised
// coordinates, clamp to edge.  Red and green are blended in one register pair
// (each product and sum rounded on its own; nz: two -0.0f the compiler cannot
// see, as in the rasteriser's packed transform).
__device__ __forceinline__ f3 lut_sample(const float4* lut, f3 uvw, f32x2 nz) {
    const float tx = uvw.x * (float)kLutDims - 0.5f, ty = uvw.y * (float)kLutDims - 0.5f,
                tz = uvw.z * (float)kLutDims - 0.5f;
    const float fx = floorf(tx), fy = floorf(ty), fz = floorf(tz);
    const float a = tx - fx, b = ty - fy, c = tz - fz;
    auto cl = [](int i) { return i < 0 ? 0 : (i > kLutDims - 1 ? kLutDims - 1 : i); };
    const int x0 = cl((int)fx), x1 = cl((int)fx + 1), y0 = cl((int)fy), y1 = cl((int)fy + 1), z0 = cl((int)fz),
              z1 = cl((int)fz + 1);
    struct Rgb {
        f32x2 rg;
        float b;
    };
    auto row = [&](int y, int z) { return lut + (z * kLutDims + y) * kLutDims; };
    auto blend = [&](const Rgb& p, const Rgb& q, float w) {
        const float v = 1.0f - w;
        return Rgb{add2(mul2(p.rg, pack2(v, v), nz), mul2(q.rg, pack2(w, w), nz)), p.b * v + q.b * w};
    };
    auto texel = [&](const float4* r, int x) {
        const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(r + x));
        float blue, alpha;
        unpack2(v.y, blue, alpha);
        return Rgb{v.x, blue};
    };
    const float4 *r00 = row(y0, z0), *r10 = row(y1, z0), *r01 = row(y0, z1), *r11 = row(y1, z1);
    const Rgb c00 = blend(texel(r00, x0), texel(r00, x1), a), c10 = blend(texel(r10, x0), texel(r10, x1), a);
    const Rgb c01 = blend(texel(r01, x0), texel(r01, x1), a), c11 = blend(texel(r11, x0), texel(r11, x1), a);
    const Rgb o = blend(blend(c00, c10, b), blend(c01, c11, b), c);
    f3 v;
    unpack2(o.rg, v.x, v.y);
    v.z = o.b;
    return v;
}

// Bilinear sample (clamp to edge) of shadow layer `layer` at uv.
__device__ __forceinline__ float shadow_texel_bilinear(const float* maps, uint32_t S, uint32_t layer, float u, float v) {
    const float* m = maps + (size_t)layer * S * S;
    const float tu = u * (float)S - 0.5f, tv = v * (float)S - 0.5f;
    const float fu = floorf(tu), fv = floorf(tv);
    const float a = tu - fu, b = tv - fv;
    auto cl = [&](int i) { return i < 0 ? 0 : (i > (int)S - 1 ? (int)S - 1 : i); };
    const int i0 = cl((int)fu), i1 = cl((int)fu + 1), j0 = cl((int)fv), j1 = cl((int)fv + 1);
    const float t00 = __ldg(m + (size_t)j0 * S + i0), t10 = __ldg(m + (size_t)j0 * S + i1),
                t01 = __ldg(m + (size_t)j1 * S + i0), t11 = __ldg(m + (size_t)j1 * S + i1);
    return ((t00 * ((1.0f - a) * (1.0f - b)) + t10 * (a * (1.0f - b))) + t01 * ((1.0f - a) * b)) + t11 * (a * b);
}

__device__ __forceinline__ float srgb_oetf(float v) {
    return v <= 0.003130f ? v * 12.92f : 1.055f * powf(v, 1.0f / 2.4f) - 0.055f;
}

__device__ __forceinline__ uint32_t unorm8(float v) {
    v = v > 0.0f ? v : 0.0f;
    v = v < 1.0f ? v : 1.0f;
    return (uint32_t)floorf(v * 255.0f + 0.5f);
}

// unorm8(srgb_oetf(v)).  powf is most of the kernel's instructions, and only
// decides where the result stands between two bytes: an estimate through the
// approximate log2 and exp2 (within 6.2e-5 of the code powf gives, over all
// floats in (0.00313, 1), measured) rounds to the same byte unless it lies
// within kByteGuard of a boundary, where powf decides (0.1 % of the values).
// 3840 x 2160: 112 us with powf throughout and scalar blends, 82 us now.
constexpr float kByteGuard = 1.0f / 2048.0f;
__device__ __forceinline__ uint32_t srgb_byte(float v) {
    if (!(v > 0.003130f)) return unorm8(srgb_oetf(v));
    if (v >= 1.0f) return 255u;
    const float x = (1.055f * exp2f_approx(log2f_approx(v) * (1.0f / 2.4f)) - 0.055f) * 255.0f + 0.5f;
    const float r = floorf(x), d = x - r;
    if (d < kByteGuard || d > 1.0f - kByteGuard) return unorm8(srgb_oetf(v));
    return (uint32_t)r;
}

// One thread per pixel (blocks of 32 x 8).
__global__ void __launch_bounds__(256) k_display_transform(FrameDev f, const float4* lut, uchar4* out) {
    pdl_enter();
    const Uniforms& u = *f.uniforms;
    const uint32_t W = u.window_size.x, H = u.window_size.y;
    const uint32_t x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y;
    if (x >= W || y >= H) return;
    const float4 hdr = load_hdr(f.hdr, f.hdr_half, (size_t)y * W + x);
    const f3 stimulus{hdr.x, hdr.y, hdr.z};
    // tony_mc_mapface (display_transform.comp:5-17)
    const f3 encoded{stimulus.x / (stimulus.x + 1.0f), stimulus.y / (stimulus.y + 1.0f),
                     stimulus.z / (stimulus.z + 1.0f)};
    const float scale = ((float)kLutDims - 1.0f) / (float)kLutDims, bias = 0.5f / (float)kLutDims;
    f3 v = lut_sample(lut, f3{encoded.x * scale + bias, encoded.y * scale + bias, encoded.z * scale + bias},
                      f.neg_zero2);
    if (u.debug_shadowmaps) {
        // display_transform.comp:51-75
        const float uvx = ((float)x + 0.5f) / (float)W, uvy = ((float)y + 0.5f) / (float)H;
        const float pct = 0.5f;
        if (uvx < pct && uvy < pct) {
            const float sx = uvx * 2.0f / pct, sy = uvy * 2.0f / pct;
            const uint32_t cascade = (sy > 1.0f ? 2u : 0u) + (sx > 1.0f ? 1u : 0u);
            const float d = shadow_texel_bilinear(f.shadow_maps, f.shadow_size, cascade, sx - floorf(sx), sy - floorf(sy));
            const float g = (d - 0.5f) * 100.0f + 0.5f;
            v = f3{g, g, g};
        }
    }
    out[(size_t)y * W + x] = make_uchar4((unsigned char)srgb_byte(v.x), (unsigned char)srgb_byte(v.y),
                                         (unsigned char)srgb_byte(v.z), 255);
}

}  // namespace

cudaError_t launch_display_transform(const FrameDev& f, uint32_t width, uint32_t height, const float4* lut, uchar4* out,
                                     cudaStream_t s) {
    dim3 grid((width + 31) / 32, (height + 7) / 8);
    return launch_pdl(k_display_transform, grid, dim3(32, 8), s, f, lut, out);
}

}  // namespace lh
