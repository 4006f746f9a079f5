// Host-side unit test of the extraction's stream keys (kc_kernels.cuh),
// compiled by tests/test_stream_keys.py; runs on the CPU.
//
// For random tiles, every k and many window ends (tile edges, segment edges):
// key_of_window() and top_of_window() equal the canonical key built from the
// window itself; sequence_mask() and runs_at_least2() equal their definitions
// byte by byte.
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#include "../../kmertreecounter_b200/csrc/kc_kernels.cuh"

using namespace kc;

template <int NW>
static bool check(const std::vector<uint32_t>& sw, const std::vector<uint64_t>& seg, uint32_t e, uint32_t k) {
    const uint64_t* sc = seg.data() + HALO_SEGS + e / 32;
    uint64_t want[NW], got[NW];
    if constexpr (NW == 4) {
        uint64_t a, b, c, d;
        window_at4(sc[-4], sc[-3], sc[-2], sc[-1], sc[0], e % 32, a, b, c, d);
        const Key4 q = canonical4(a, b, c, d, k);
        want[0] = q.w0, want[1] = q.w1, want[2] = q.w2, want[3] = q.w3;
    } else {
        uint64_t lo, hi;
        window_at(sc[-2], sc[-1], sc[0], e % 32, lo, hi);
        if constexpr (NW == 1) {
            want[0] = canonical1(k >= 32 ? lo : lo & ((1ull << (2 * k)) - 1), k);
        } else {
            const Key2 q = canonical2(k >= 64 ? hi : hi & ((1ull << (2 * k - 64)) - 1), lo, k);
            want[0] = q.w0, want[1] = q.w1;
        }
    }
    const StreamPos p = stream_pos(e, k);
    key_of_window<NW>(sw.data(), p, k, got);
    for (int w = 0; w < NW; ++w)
        if (got[w] != want[w]) {
            std::printf("key mismatch NW=%d k=%u e=%u word %d\n", NW, k, e, w);
            return false;
        }
    if (top_of_window(sw.data(), p, key_mask(0, k)) != (uint32_t)(want[0] >> 32)) {
        std::printf("top mismatch NW=%d k=%u e=%u\n", NW, k, e);
        return false;
    }
    return true;
}

int main() {
    std::mt19937_64 rng(11);
    long checks = 0;
    for (int iter = 0; iter < 6; ++iter) {
        std::vector<uint64_t> seg(TILE_SEGS);
        // random codes, one base only (ties of every word), a period of two
        for (auto& s : seg) s = iter == 1 ? 0 : iter == 2 ? ~0ull : iter == 3 ? 0x3333333333333333ull : rng();
        if (iter == 4)  // palindromic neighbourhoods: orientations that agree far into the key
            for (int t = 1; t < TILE_SEGS; t += 2) seg[t] = ~rev_bases(seg[t - 1]);
        std::vector<uint32_t> sw(STREAM_WORDS, 0xDEADBEEFu);
        for (int t = 0; t < TILE_SEGS; ++t) stream_put(sw.data(), t, seg[t]);
        std::vector<uint32_t> ends = {0, 1, 15, 16, 31, 32, 63, 64, 127, EXT_TILE / 2, EXT_TILE - 33, EXT_TILE - 32,
                                      EXT_TILE - 17, EXT_TILE - 16, EXT_TILE - 2, EXT_TILE - 1};
        for (int i = 0; i < 60; ++i) ends.push_back((uint32_t)(rng() % EXT_TILE));
        for (uint32_t k = 1; k <= 128; ++k)
            for (uint32_t e : ends) {
                if (!(k <= 32 ? check<1>(sw, seg, e, k) : k <= 64 ? check<2>(sw, seg, e, k) : check<4>(sw, seg, e, k)))
                    return 1;
                ++checks;
            }
    }
    for (int i = 0; i < 20000; ++i) {
        const uint32_t line0 = (uint32_t)rng();
        uint32_t nls = (uint32_t)rng();
        for (int t = (int)(rng() % 5); t > 0; --t) nls &= (uint32_t)rng();
        uint32_t want = 0, line = line0;
        for (int j = 0; j < 32; ++j) {
            if ((line & 3) == 1) want |= 1u << j;
            if ((nls >> j) & 1) ++line;
        }
        if (sequence_mask(line0, nls) != want) {
            std::printf("sequence_mask mismatch\n");
            return 1;
        }
        const uint32_t prev = (uint32_t)(rng() | rng() | rng()), cur = (uint32_t)(rng() | rng() | rng() | rng());
        const uint32_t k = 1 + (uint32_t)(rng() % 32);
        want = 0;
        for (int j = 0; j < 32; ++j) {
            bool all = true;
            for (int b = j - (int)k + 1; b <= j; ++b) all &= b >= 0 ? (cur >> b) & 1 : (prev >> (32 + b)) & 1;
            if (all) want |= 1u << j;
        }
        if (runs_at_least2(prev, cur, k) != want) {
            std::printf("runs_at_least2 mismatch k=%u\n", k);
            return 1;
        }
        checks += 2;
    }
    std::printf("streams ok: %ld checks\n", checks);
    return 0;
}
