// Device check of two decisions taken through approximate instructions, against
// the plain forms they stand for: the display transform's byte (display.cu) for
// every float, and the normal-cone test (facing.cuh), whose reciprocal square
// root differs from the host's, near and away from the cutoff.
#include <cstdio>
#include <cstring>

#include "display.cu"

namespace lh {
namespace {

struct Counts {
    unsigned long long bytes, bytes_bad, cones, cones_bad, near;
    unsigned int worst;  // largest error of the byte's estimate, float bits
};

// Every float: a pattern per step, strided over the grid.
__global__ void k_bytes(Counts* c) {
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    unsigned long long n = 0, bad = 0;
    float worst = 0.0f;
    for (unsigned long long p = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; p < (1ull << 32); p += stride) {
        const float v = __uint_as_float((uint32_t)p);
        n++;
        bad += srgb_byte(v) != unorm8(srgb_oetf(v));
        if (v > 0.003130f && v < 1.0f) {
            const float estimate = (1.055f * exp2f_approx(log2f_approx(v) * (1.0f / 2.4f)) - 0.055f) * 255.0f + 0.5f;
            worst = fmaxf(worst, fabsf(estimate - (srgb_oetf(v) * 255.0f + 0.5f)));
        }
    }
    atomicAdd(&c->bytes, n);
    atomicAdd(&c->bytes_bad, bad);
    atomicMax(&c->worst, __float_as_uint(worst));
}

__device__ float unit(uint32_t& s) {  // [-1, 1)
    s = s * 1664525u + 1013904223u;
    uint32_t x = s;
    x = (x ^ (x >> 16)) * 0x7feb352du;
    x = (x ^ (x >> 15)) * 0x846ca68bu;
    x ^= x >> 16;
    return (float)(int32_t)x * (1.0f / 2147483648.0f);
}

// Cones: directions and axes of lengths 2^-20 .. 2^20 (and beyond the range the
// short form takes), cutoffs anywhere, or at the product in 64 bits up to a few
// rounding steps or 2^-17 of it.
__global__ void k_cones(Counts* c, uint32_t per_thread) {
    uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) * 2654435761u + 12345u;
    unsigned long long n = 0, bad = 0, near = 0;
    for (uint32_t i = 0; i < per_thread; i++) {
        const uint32_t kind = i & 3u;
        const float reach = kind == 3u ? 60.0f : 20.0f;
        const float sa = exp2f(unit(s) * reach), sd = i & 4u ? 1.0f : exp2f(unit(s) * reach);
        const float a[3] = {sa * unit(s), sa * unit(s), sa * unit(s)}, d[3] = {sd * unit(s), sd * unit(s), sd * unit(s)};
        const double la = sqrt((double)a[0] * a[0] + (double)a[1] * a[1] + (double)a[2] * a[2]);
        const double ld = sqrt((double)d[0] * d[0] + (double)d[1] * d[1] + (double)d[2] * d[2]);
        for (int times = 1; times <= 2; times++) {
            const bool is_unit = times == 1;
            float cutoff = unit(s);
            if (kind != 0u) {
                const double p = (double)a[0] * d[0] + (double)a[1] * d[1] + (double)a[2] * d[2];
                cutoff = (float)(p / (is_unit ? la : la * ld));
                const int steps = (int)(unit(s) * 40.0f);
                if (cutoff != 0.0f && isfinite(cutoff)) cutoff = __int_as_float(__float_as_int(cutoff) + steps);
                if (kind == 2u) cutoff += cutoff * unit(s) * (1.0f / 131072.0f);
                near++;
            }
            n++;
            bad += cone_behind(d, a, cutoff, is_unit, times) != cone_behind_ieee(d, a, cutoff, is_unit, times);
        }
    }
    atomicAdd(&c->cones, n);
    atomicAdd(&c->cones_bad, bad);
    atomicAdd(&c->near, near);
}

}  // namespace
}  // namespace lh

int main() {
    lh::Counts* c = nullptr;
    if (cudaMallocManaged(&c, sizeof(lh::Counts)) != cudaSuccess) return 2;
    *c = lh::Counts{};
    lh::k_bytes<<<1216, 256>>>(c);
    lh::k_cones<<<1216, 256>>>(c, 256u);
    if (cudaDeviceSynchronize() != cudaSuccess) return 3;
    float worst;
    memcpy(&worst, &c->worst, 4);
    std::printf("bytes %llu bad %llu worst estimate %.3g cones %llu near the cutoff %llu bad %llu\n", c->bytes, c->bytes_bad,
                worst, c->cones, c->near, c->cones_bad);
    return c->bytes_bad || c->cones_bad || !(worst < 1.0f / 4096.0f);
}
