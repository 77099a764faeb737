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

}  // namespace lh
