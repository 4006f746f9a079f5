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
    if (!bad) std::printf("ok\n");
    return bad != 0;
}
