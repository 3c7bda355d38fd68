// Host-side check of fa::FastDiv (csrc/fast_div.h) against the language's division.  Prints "ok" and
// exits 0, or prints the first mismatch and exits 1.  Built and run by tests/test_fast_div_cpu.py.
#include <cstdio>
#include <initializer_list>

#include "fast_div.h"

static bool check(uint32_t d, uint32_t n) {
    if (n > 0x7FFFFFFFu) return true;
    if (fa::FastDiv(d).quot((int)n) == (int)(n / d)) return true;
    std::printf("FAILED %u / %u\n", n, d);
    return false;
}

int main() {
    const uint32_t top = 0x7FFFFFFFu;
    uint64_t seed = 1;
    auto next = [&] { seed = seed * 6364136223846793005ull + 1442695040888963407ull; return (uint32_t)(seed >> 33); };
    auto edges = [&](uint32_t d) {
        for (uint32_t q : {0u, 1u, 2u, 7u, top / d - 1u, top / d})
            for (int off : {-1, 0, 1})
                if (!check(d, q * d + off)) return false;
        return check(d, top) && check(d, 0);
    };
    for (uint32_t d = 1; d <= 5000; d++)
        if (!edges(d)) return 1;
    for (int s = 0; s < 31; s++)
        for (int off = -1; off <= 1; off++) {
            const uint32_t d = (1u << s) + off;
            if (d >= 1 && d <= top && !edges(d)) return 1;
        }
    for (int i = 0; i < 200000; i++) {
        const uint32_t d = next() >> (next() % 31);
        if (d == 0) continue;
        if (!edges(d) || !check(d, next())) return 1;
    }
    std::printf("ok\n");
    return 0;
}
