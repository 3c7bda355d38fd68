// Which entry of a sequence's block table a lane looks up when a warp fetches one 128-key tile of a paged
// cache: lane i has the tile's i-th page.  Compiles for the host too, where a test compares it with the
// pages that the tile's keys lie in, for every page size the entry point takes.
//
// The reference has no paged cache.
#pragma once

#include "bounded_wait.h"       // FA_HOST_DEVICE

namespace fa {

// Entry for the tile that starts at key `r0` of a sequence of `kv_len` keys in pages of 2^page_shift keys, or
// -1: no such page.  A tile has max(1, 128 >> page_shift) pages; the lanes past them have none, whatever
// `lane << page_shift` would come to (it wraps for pages of 2^27 keys and more).
FA_HOST_DEVICE int page_entry(int lane, int r0, int kv_len, int page_shift) {
    if (lane != 0 && lane >= 128 >> page_shift) return -1;
    const int rr = r0 + (lane << page_shift);
    return rr < kv_len ? rr >> page_shift : -1;
}

}  // namespace fa
