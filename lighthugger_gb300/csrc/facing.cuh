// Signs of normalised dot products, decided without the normalisation.
//
// Whether a triangle with edge cross product n is seen from behind along v (the
// vector to the camera): the sign of dot(n, normalize(v)) as IEEE arithmetic
// gives it (dot = (x x' + y y') + z z'), mostly without the square root and the
// three divisions.  Their rounding moves the dot product by less than 2^-21
// of the sum of the terms' magnitudes, the undivided one's by less than 2^-22:
// only a sum of nearly cancelling terms, or of extreme ones, needs them.
#pragma once

#include <cmath>

#if defined(__CUDACC__)
#define LH_FACING_HD __host__ __device__ __forceinline__
#else
#define LH_FACING_HD inline
#endif

namespace lh {

LH_FACING_HD bool faces_away_ieee(float nx, float ny, float nz, float vx, float vy, float vz) {
    const float l = sqrtf((vx * vx + vy * vy) + vz * vz);
    return (nx * (vx / l) + ny * (vy / l)) + nz * (vz / l) < 0.0f;
}

LH_FACING_HD bool faces_away(float nx, float ny, float nz, float vx, float vy, float vz) {
    const float x = nx * vx, y = ny * vy, z = nz * vz, d2 = (vx * vx + vy * vy) + vz * vz;
    const float s = (x + y) + z, m = (fabsf(x) + fabsf(y)) + fabsf(z);
    if (fabsf(s) > m * (1.0f / 262144.0f) && fabsf(s) > 1e-30f && d2 > 1e-20f && d2 < 1e12f) return s < 0.0f;
    return faces_away_ieee(nx, ny, nz, vx, vy, vz);
}

// Whether a normal cone is seen from behind: dot(d', a') >= cutoff, where d' is
// d normalised (`unit`: d as it is) and a' is a normalised `times` times, in IEEE
// arithmetic.  Twelve divisions and roots lie behind that.  In units of 2^-24 of
// the sum of the terms' magnitudes their rounding moves the product by at most
// 13.5 (3.5 for each of three normalisations, 3 for the products and sums), that
// of the approximate reciprocal roots here by 16 (4 for each of two, 3 for the
// squared lengths, 2 for the scaling, 3 for the products and sums): less than
// 2^-19 together, so the plain form decides nearer than 2^-18 to the cutoff, or
// for extreme lengths.
LH_FACING_HD bool cone_behind_ieee(const float* d, const float* a, float cutoff, bool unit, int times) {
    float x = a[0], y = a[1], z = a[2], u = d[0], v = d[1], w = d[2];
    for (int i = 0; i < times; i++) {
        const float l = sqrtf((x * x + y * y) + z * z);
        x = x / l;
        y = y / l;
        z = z / l;
    }
    if (!unit) {
        const float l = sqrtf((u * u + v * v) + w * w);
        u = u / l;
        v = v / l;
        w = w / l;
    }
    return (u * x + v * y) + w * z >= cutoff;
}

LH_FACING_HD float rsqrt_near(float x) {
#if defined(__CUDA_ARCH__)
    return rsqrtf(x);
#else
    return 1.0f / sqrtf(x);
#endif
}

LH_FACING_HD bool cone_behind(const float* d, const float* a, float cutoff, bool unit, int times) {
    const float x = d[0] * a[0], y = d[1] * a[1], z = d[2] * a[2];
    const float dd = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2], aa = (a[0] * a[0] + a[1] * a[1]) + a[2] * a[2];
    const float q = unit ? rsqrt_near(aa) : rsqrt_near(aa) * rsqrt_near(dd);
    const float c = ((x + y) + z) * q, m = ((fabsf(x) + fabsf(y)) + fabsf(z)) * q;
    if (fabsf(c - cutoff) > m * (1.0f / 262144.0f) + 1e-20f && aa > 1e-16f && aa < 1e16f && dd > 1e-16f && dd < 1e16f)
        return c > cutoff;
    return cone_behind_ieee(d, a, cutoff, unit, times);
}

}  // namespace lh
