// The memory rule by which a count takes a second key buffer (host only).
#include <cstdio>

#include "../../kmertreecounter_b200/csrc/kc_internal.h"

int main() {
    const double G = 1e9;
    int bad = 0;
    auto check = [&](bool got, bool want, const char* what) {
        if (got != want) {
            std::printf("%s: %d, want %d\n", what, got, want);
            ++bad;
        }
    };
    const KcNeed fresh[3] = {{8 * G, 0}, {8 * G, 0}, {4 * G, 0}};
    check(kc_needs_fit(fresh, 3, 22.6 * G), true, "an eighth and 64 MiB to spare");
    check(kc_needs_fit(fresh, 3, 22.5 * G), false, "the eighth alone");
    check(kc_needs_fit(fresh, 2, 18.1 * G), true, "without the last buffer");
    check(kc_needs_fit(fresh, 3, 18.1 * G), false, "room for all but the last buffer");
    const KcNeed held[3] = {{8 * G, 9 * G}, {8 * G, 8 * G}, {4 * G, 50 * G}};
    check(kc_needs_fit(held, 3, 0), true, "nothing to allocate");
    const KcNeed mixed[2] = {{8 * G, 7 * G}, {4 * G, 50 * G}};
    check(kc_needs_fit(mixed, 2, 2.1 * G), true, "a buffer is given back before it grows");
    check(kc_needs_fit(mixed, 2, 2 * G), false, "a buffer that stays gives nothing back");
    check(kc_windowed_keys(1e6, 512, false) == 1e6 + 64 * 512, true, "exact ranges");
    // the sub-routed keys' places against window_caps' sum over windows of
    // even, skewed and mostly empty contents
    for (int form = 0; form < 3; ++form)
        for (double keys = 1e5; keys < 1e10; keys *= 10)
            for (int windows : {256, 70'000, 250'000}) {
                double sum = 0, weight = 0;
                auto share = [&](int w) { return form == 0 ? 1.0 : form == 1 ? 1.0 / (1 + w) : (w % 50 == 0); };
                for (int w = 0; w < windows; ++w) weight += share(w);
                for (int w = 0; w < windows; ++w) {
                    const double est = keys * share(w) / weight;
                    sum += std::ceil((est * 1.1 + 4 * std::sqrt(est) + 64) / 64) * 64;
                }
                sum += std::max(65536.0, sum / 16);
                check(kc_windowed_keys(keys, windows, true) >= sum, true, "room for every window");
                if (keys > 1e6 * windows)
                    check(kc_windowed_keys(keys, windows, true) < 1.2 * keys, true, "no more than the windows' slack");
            }
    if (!bad) std::printf("ok\n");
    return bad != 0;
}
