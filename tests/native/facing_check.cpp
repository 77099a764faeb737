// CPU check of lighthugger_gb300/csrc/facing.cuh: faces_away and cone_behind
// against the plain IEEE evaluations, over random vectors, vectors nearly at
// right angles, cutoffs at and next to the product, extreme lengths and
// special values.
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
    auto cone = [&](const float* d, const float* a, float cutoff) {
        for (int times = 1; times <= 2; times++) {
            n++;
            if (lh::cone_behind(d, a, cutoff, times == 1, times) != lh::cone_behind_ieee(d, a, cutoff, times == 1, times)) bad++;
        }
    };
    for (long i = 0; i < 2000000; i++) {
        const int kind = (int)(i % 4);
        const float sa = std::exp2(U(rng) * (kind == 3 ? 60.0f : 6.0f)), sb = kind == 0 ? 1.0f : std::exp2(U(rng) * (kind == 3 ? 60.0f : 10.0f));
        const float a[3] = {sa * U(rng), sa * U(rng), sa * U(rng)}, d[3] = {sb * U(rng), sb * U(rng), sb * U(rng)};
        float cutoff = U(rng);
        if (kind != 0) {
            // the product itself (of either form), up to a few rounding steps
            const double l = std::sqrt((double)a[0] * a[0] + (double)a[1] * a[1] + (double)a[2] * a[2]) *
                             (i & 4 ? 1.0 : std::sqrt((double)d[0] * d[0] + (double)d[1] * d[1] + (double)d[2] * d[2]));
            cutoff = (float)(((double)a[0] * d[0] + (double)a[1] * d[1] + (double)a[2] * d[2]) / l);
            for (int k = (int)(rng() % 9) - 4; k != 0; k += k > 0 ? -1 : 1) cutoff = std::nextafter(cutoff, k > 0 ? 1e30f : -1e30f);
            if (kind == 2) cutoff += cutoff * U(rng) * 1e-5f;
        }
        cone(d, a, cutoff);
    }
    for (float p : s) for (float q : s) for (float r : s) for (float t : s) for (float u : s) {
        const float d[3] = {p, q, 1.0f}, a[3] = {r, t, 0.5f};
        cone(d, a, u);
    }
    std::printf("checked %ld bad %ld\n", n, bad);
    return bad ? 1 : 0;
}
