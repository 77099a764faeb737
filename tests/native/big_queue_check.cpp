// Host check of the big-triangle queue's entries (big_queue.cuh) where the
// chunk numbers run past 32 bits: every index the counter hands out below the
// capacity is walked by the chunk kernel, so each has to hold what was pushed
// in this pass, or nothing that covers a pixel.  The slots hold triangles of an
// earlier pass beforehand (of a view that no longer exists).
#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>

#include "big_queue.cuh"

struct Setup {
    int32_t X0, Y0, X1, Y1, X2, Y2;
    float z0, s1, s2;
    uint32_t id;
    int32_t px0, py0, px1, py1;
    uint32_t bias, verts;
};
struct Big {
    int32_t X0, Y0, X1, Y1, X2, Y2;
    float z0, s1, s2;
    uint32_t id, view, bias;
    int32_t px0, px1, py0, py1;
};

long long entries = 0, dropped = 0, bad = 0;

// KIND: the pass.
template <int KIND> void run(uint64_t seed) {
    std::mt19937_64 rng(seed);
    for (int it = 0; it < 200; it++) {
        const uint32_t cap = 1 + (uint32_t)(rng() % 6000), pushes = 1 + (uint32_t)(rng() % 7000);
        // every other queue: the smallest chunks and boxes of nearly 16,384 pixels a side
        const bool past = it & 1;
        const uint32_t rs = past ? 2 : 2 + (uint32_t)(rng() % 4), cs = past ? 5 : 5 + (uint32_t)(rng() % 4);
        std::vector<Big> big(cap, Big{0, 0, 1, 0, 0, 1, 0.f, 0.f, 0.f, 7u, 99u, lh::kBiasWhole, 0, 900, 0, 900});
        std::vector<uint32_t> base(cap, (uint32_t)rng());
        std::vector<Setup> sent;
        uint64_t word = 0;
        std::vector<char> fits;
        for (uint32_t k = 0; k < pushes; k++) {
            Setup t{};
            // boxes up to 16,384 pixels a side (2 million chunks), small ones between
            const bool big_one = rng() % 2;
            auto extent = [&] { return (int32_t)(!big_one ? rng() % 40 : past ? 16000 + rng() % 284 : rng() % 16284); };
            t.px1 = (t.px0 = (int32_t)(rng() % 100)) + extent();
            t.py1 = (t.py0 = (int32_t)(rng() % 100)) + extent();
            t.id = k;
            t.bias = rng() % 4 == 0 ? lh::kBiasAlpha : 0u;
            const uint64_t n = (uint64_t)(((uint32_t)(t.px1 - t.px0) >> cs) + 1) * (((uint32_t)(t.py1 - t.py0) >> rs) + 1);
            const uint64_t old = word;
            word += lh::queue_word<KIND>(n, t.bias & lh::kBiasAlpha);
            const bool ok = lh::store_queue_entry<KIND>(big.data(), base.data(), cap, t, 3u, old, n);
            const bool want = k < cap && (old & ((1ull << 40) - 1)) + n <= 0xFFFFFFFFull;
            if (ok != want) bad++;
            sent.push_back(t);
            fits.push_back(ok);
        }
        // the walks of the chunk kernel
        const uint32_t ntri = (uint32_t)std::min<uint64_t>(cap, word >> 40);
        const uint32_t total = (uint32_t)std::min<uint64_t>(word & ((1ull << 40) - 1), 0xFFFFFFFFull);
        for (uint32_t i = 0; i < ntri; i++) {
            const Big& b = big[i];
            entries++;
            if (i && base[i] < base[i - 1]) bad++;                          // the search needs them in order
            if (b.view != 3u || b.id != i) bad++;                           // this pass's entry
            if (fits[i] != (b.py0 <= b.py1)) bad++;                         // pixels only of what fits
            if (!fits[i] && (!(b.bias & lh::kBiasWhole) || base[i] != 0xFFFFFFFFu)) bad++;
            if (fits[i] && !(b.bias & lh::kBiasWhole) && (b.px1 != sent[i].px1 || b.py1 != sent[i].py1)) bad++;
            dropped += !fits[i];
        }
        for (int s = 0; s < 200 && total; s++) {
            const uint32_t c = s < 4 ? total - 1 - std::min((uint32_t)s, total - 1) : (uint32_t)(rng() % total);
            const auto at = std::upper_bound(base.begin(), base.begin() + ntri, c) - base.begin();
            if (at == 0) continue;
            const Big& b = big[at - 1];
            const uint64_t n = (uint64_t)(((uint32_t)(b.px1 - b.px0) >> cs) + 1) * (((uint32_t)(b.py1 - b.py0) >> rs) + 1);
            const bool taken = !(b.bias & lh::kBiasWhole) && c - base[at - 1] < n;
            if (taken && !fits[at - 1]) bad++;
        }
    }
}

int main() {
    run<0>(5);
    run<1>(6);
    // whole up to two visibility chunks and one shadow chunk, alpha-tested never
    for (uint64_t n = 1; n < 5; n++)
        for (int alpha = 0; alpha < 2; alpha++) {
            if ((lh::queue_word<0>(n, alpha) & 0xFFFF) != (n <= 2 && !alpha ? 0 : n)) bad++;
            if ((lh::queue_word<1>(n, alpha) & 0xFFFF) != (n <= 1 && !alpha ? 0 : n)) bad++;
        }
    std::printf("entries %lld dropped %lld bad %lld\n", entries, dropped, bad);
    return bad != 0 || dropped == 0;
}
