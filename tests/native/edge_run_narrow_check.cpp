// Host check of clip_run_as<int32_t> (edge_run.cuh): for triangles whose
// edge products inside their box fit 32 bits (the condition under which the
// chunk kernel takes it), every row of the box cut into windows of up to 256
// pixels gives the runs of the 64-bit form.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "edge_run.cuh"

int main() {
    std::mt19937_64 rng(23);
    long long rows = 0, bad = 0;
    for (int it = 0; it < 60000; it++) {
        // extents up to the limits: ext_x * ext_y < 2^30, both below 2^22
        const int sx = 1 + (int)(rng() % 22);
        int32_t ext_x = 1 + (int32_t)(rng() % (1u << sx)), ext_y = (int32_t)(((1ll << 30) - 1) / ext_x);
        if (ext_y > (1 << 22) - 1) ext_y = (1 << 22) - 1;
        if (it & 1) ext_y = 1 + (int32_t)(rng() % (uint32_t)ext_y);
        const int32_t ox = (int32_t)(rng() % (1u << 22)) - (1 << 21), oy = (int32_t)(rng() % (1u << 22)) - (1 << 21);
        int32_t X[3], Y[3];
        for (int k = 0; k < 3; k++) {
            X[k] = ox + (int32_t)(rng() % (uint32_t)(ext_x + 1));
            Y[k] = oy + (int32_t)(rng() % (uint32_t)(ext_y + 1));
        }
        if (it % 5 == 0) { X[0] = ox; X[1] = ox + ext_x; Y[1] = oy; Y[2] = oy + ext_y; }
        int32_t mx = X[0], Mx = X[0], my = Y[0], My = Y[0];
        for (int k = 1; k < 3; k++) {
            mx = X[k] < mx ? X[k] : mx, Mx = X[k] > Mx ? X[k] : Mx;
            my = Y[k] < my ? Y[k] : my, My = Y[k] > My ? Y[k] : My;
        }
        const int32_t px0 = (mx + 127) >> 8, px1 = (Mx - 128) >> 8, py0 = (my + 127) >> 8, py1 = (My - 128) >> 8;
        if (px0 > px1 || py0 > py1) continue;
        for (int r = 0; r < 4; r++) {
            const int32_t y = r == 0 ? py0 : r == 1 ? py1 : py0 + (int32_t)(rng() % (uint32_t)(py1 - py0 + 1));
            const int32_t x0 = r == 0 ? px0 : px0 + (int32_t)(rng() % (uint32_t)(px1 - px0 + 1));
            const int32_t n = px1 - x0 + 1 < 256 ? px1 - x0 + 1 : 256;
            for (int e = 0; e < 3; e++) {
                const int32_t ax = X[e], ay = Y[e], bx = X[(e + 1) % 3], by = Y[(e + 1) % 3];
                const int64_t e0 = (int64_t)(by - ay) * (x0 * 256 + 128 - ax) - (int64_t)(bx - ax) * (y * 256 + 128 - ay);
                const float inv = lh::run_inv_step(by - ay);
                for (int bias = 0; bias < 2; bias++) {
                    int32_t lo = 0, hi = n - 1, lo2 = 0, hi2 = n - 1;
                    lh::clip_run(e0, (int64_t)(by - ay) * 256, (int64_t)bias, n, inv, lo, hi);
                    lh::clip_run_as<int32_t>((int32_t)e0, (by - ay) * 256, bias, n, inv, lo2, hi2);
                    rows++;
                    const bool empty = lo > hi, empty2 = lo2 > hi2;
                    if (e0 != (int32_t)e0 || empty != empty2 || (!empty && (lo != lo2 || hi != hi2))) {
                        if (bad++ < 10) std::printf("it %d edge %d: [%d, %d] against [%d, %d]\n", it, e, lo2, hi2, lo, hi);
                    }
                }
            }
        }
    }
    std::printf("rows %lld bad %lld\n", rows, bad);
    return bad == 0 && rows > 100000 ? 0 : 1;
}
