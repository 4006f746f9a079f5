// Host-side test of holds_unfenced() (kc_kernels.cuh), compiled and run by
// tests/test_slot_reads.py: a slot's key words, each read before or after it
// was written (EMPTY before), must never pass for another key.
#include <cstdio>

#include "../../kmertreecounter_b200/csrc/kc_kernels.cuh"

using namespace kc;

int main() {
    const uint64_t word[4] = {0, EMPTY, 0x123456789ABCDEF0ull, ~0ull << 2};
    auto key = [&](int i) { return Key4{word[i & 3], word[(i >> 2) & 3], word[(i >> 4) & 3], word[(i >> 6) & 3]}; };
    long wrong = 0, kept = 0;
    for (int p = 0; p < 256; ++p)      // the slot's key
        for (int q = 0; q < 256; ++q)  // the reader's
            for (int late = 0; late < 16; ++late) {
                Key4 have = key(p);
                if (!(late & 1)) have.w0 = EMPTY;
                if (!(late & 2)) have.w1 = EMPTY;
                if (!(late & 4)) have.w2 = EMPTY;
                if (!(late & 8)) have.w3 = EMPTY;
                const bool got = holds_unfenced(have, key(q));
                wrong += got && p != q;
                kept += got && p == q;
            }
    // keys without a word of all ones, read whole: one fetch settles them
    if (wrong || kept != 81) {
        std::printf("%ld wrong matches, %ld kept\n", wrong, kept);
        return 1;
    }
    std::printf("ok\n");
    return 0;
}
