// Host-side check of fa::page_entry (csrc/page_entry.h) against the pages a tile's keys lie in.  Prints "ok"
// and exits 0, or prints what failed and exits 1.  Built and run by tests/test_page_entry_cpu.py.
#include <cstdio>
#include <initializer_list>

#include "page_entry.h"

int main() {
    for (int shift = 4; shift <= 30; shift++) {
        const long long page = 1ll << shift;
        const long long lens[] = {1, 15, 16, 17, 127, 128, 129, 1000, 4096, page - 1, page, page + 1, 3 * page + 5, 0x7fffff00ll};
        for (long long len : lens) {
            if (len < 1 || len > 0x7fffff00ll) continue;
            const long long tiles = (len + 127) / 128;
            for (long long t : {0ll, 1ll, page / 128, page / 128 + 1, tiles / 2, tiles - 1}) {
                if (t < 0 || t >= tiles) continue;
                const long long r0 = t * 128;
                const int n = page >= 128 ? 1 : (int)(128 / page);       // pages of the tile
                for (int lane = 0; lane < 32; lane++) {
                    const long long key = r0 + lane * page;              // first key of the tile in the lane's page
                    const long long want = lane < n && key < len ? key / page : -1;
                    const int got = fa::page_entry(lane, (int)r0, (int)len, shift);
                    if (got != want) {
                        std::printf("FAILED page 2^%d len %lld tile %lld lane %d: %d, not %lld\n", shift, len, t, lane, got, want);
                        return 1;
                    }
                }
            }
        }
    }
    std::printf("ok\n");
    return 0;
}
