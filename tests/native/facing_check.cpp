// CPU check of lighthugger_gb300/csrc/facing.cuh: faces_away against the plain
// IEEE evaluation, over random vectors, vectors nearly at right angles, extreme
// lengths and special values.
#include <cmath>
#include <cstdio>
#include <limits>
#include <random>

#include "facing.cuh"

int main() {
    std::mt19937 rng(7);
    std::uniform_real_distribution<float> U(-1.0f, 1.0f);
    long bad = 0, n = 0;
    auto check = [&](const float* a, const float* b) {
        n++;
        if (lh::faces_away(a[0], a[1], a[2], b[0], b[1], b[2]) != lh::faces_away_ieee(a[0], a[1], a[2], b[0], b[1], b[2])) bad++;
    };
    for (long i = 0; i < 4000000; i++) {
        const int kind = (int)(i % 4);
        const float sa = std::exp2(U(rng) * (kind == 3 ? 60.0f : 12.0f)), sb = std::exp2(U(rng) * (kind == 3 ? 60.0f : 12.0f));
        float a[3] = {sa * U(rng), sa * U(rng), sa * U(rng)}, b[3] = {sb * U(rng), sb * U(rng), sb * U(rng)};
        if (kind == 1 || kind == 2) {
            // b at right angles to a up to a few rounding steps of one component
            b[2] = (float)(-((double)a[0] * b[0] + (double)a[1] * b[1]) / a[2]);
            for (int k = (int)(rng() % 9) - 4; k != 0; k += k > 0 ? -1 : 1)
                b[2] = std::nextafter(b[2], k > 0 ? 1e30f : -1e30f);
            if (kind == 2) b[2] += b[2] * U(rng) * 1e-5f;
        }
        check(a, b);
    }
    const float inf = std::numeric_limits<float>::infinity(), nan = std::numeric_limits<float>::quiet_NaN();
    const float s[] = {0.0f, -0.0f, 1.0f, -1.0f, 1e-42f, -1e-42f, 3e38f, -3e38f, inf, -inf, nan};
    for (float p : s) for (float q : s) for (float r : s) for (float t : s) for (float u : s) {
        const float a[3] = {p, q, 1.0f}, b[3] = {r, t, u};
        check(a, b);
    }
    std::printf("checked %ld bad %ld\n", n, bad);
    return bad ? 1 : 0;
}
