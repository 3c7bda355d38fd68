// Division of a non-negative int by a launch constant: a multiply-high and a shift instead of the
// ~40 dependent instructions of a division by a variable (one of them on the MUFU pipe that the
// softmax needs).  Every role of a persistent CTA turns item indices into coordinates between two
// items, on its critical path: grouped-query attention of 512 new tokens on 1024 keys (B=8 Hq=32
// Hkv=8 D=128, 7 items a CTA) 90.5 -> 77 us.  Compiles for the host too, where a test compares it
// with the language's division.
//
// The reference divides by variables (kernels/flash_attention.cu:135-140, block index to head).
#pragma once

#include <cstdint>

#include "bounded_wait.h"       // FA_HOST_DEVICE

namespace fa {

// Exact for 0 <= n < 2^31 and 1 <= d < 2^31 (Granlund and Montgomery 1994, round-up method).
struct FastDiv {
    uint32_t mul = 1, shr = 0;
    FastDiv() = default;
    explicit FastDiv(uint32_t d) {
        while ((1ull << shr) < d) shr++;
        mul = static_cast<uint32_t>(((1ull << 32) * ((1ull << shr) - d)) / d + 1);
    }
    FA_HOST_DEVICE int quot(int n) const {
#if defined(__CUDA_ARCH__)
        const uint32_t hi = __umulhi(static_cast<uint32_t>(n), mul);
#else
        const uint32_t hi = static_cast<uint32_t>((static_cast<uint64_t>(static_cast<uint32_t>(n)) * mul) >> 32);
#endif
        return static_cast<int>((hi + static_cast<uint32_t>(n)) >> shr);
    }
};

}  // namespace fa
