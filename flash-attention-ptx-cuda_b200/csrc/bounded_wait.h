// The decision core of every device-side wait, kept free of device-only
// instructions so that the same code runs on the host: a unit test drives it
// with a poll that never succeeds and a fake clock, which is the only way the
// give-up branch is ever exercised (no test makes a GPU wait run out).
//
// The reference has no counterpart: its kernel synchronises with block-wide
// barriers only (kernels/flash_attention.cu:349,396,470) and its launcher
// reports errors by printing and exiting (include/flash_attention.h:35-43).
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define FA_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define FA_HOST_DEVICE inline
#endif

namespace fa {

// Error words written to the device status buffer: (code << 16) | detail.
enum : int {
    kErrNone        = 0,
    kErrWaitTimeout = 1,   // a bounded wait ran out of time; detail = barrier id
};

enum : int { kWaitDone = 0, kWaitAborted = 1, kWaitTimedOut = 2 };

// Polls until `poll()` returns true.  Every `check_every` polls (a power of two) it looks at
// `aborted()` - somebody else in the CTA already gave up - and at the clock `now_ns()`; the
// wait gives up once more than `limit_ns` have passed since its first look at the clock.
template <class Poll, class Aborted, class Clock>
FA_HOST_DEVICE int bounded_wait(Poll poll, Aborted aborted, Clock now_ns, unsigned long long limit_ns,
                                uint32_t check_every) {
    unsigned long long t0 = 0;
    bool have_t0 = false;
    uint32_t polls = 0;
    while (!poll()) {
        if ((++polls & (check_every - 1u)) == 0u) {
            if (aborted()) return kWaitAborted;
            const unsigned long long now = now_ns();
            if (!have_t0) {
                t0 = now;
                have_t0 = true;
            } else if (now - t0 > limit_ns) {
                return kWaitTimedOut;
            }
        }
    }
    return kWaitDone;
}

// Waits made by all lanes of a warp.  The lanes' answers can differ: one sees the phase complete while another
// runs out of time or sees the abort flag.  A warp that left its loop lane by lane on them would split, and
// those that stay would wait without limit, at the next full-mask instruction, for those that left.  So the
// warp votes; `all(x)` is true in every lane if x is true in all of them.
//
// The plain form votes on each wait: every lane gets the same answer.
template <class Wait, class All>
FA_HOST_DEVICE bool warp_wait(Wait wait, All all) {
    return all(wait());
}
// Several waits can share a vote: the lanes note what their waits said, and `all(ok)` decides for all of them.
// The warps that convert an e4m3 V tile vote once on both of its waits (B=32 Hkv=8 Skv=16384: 226 us with two
// votes, 219 with one, 218 without).  Where one elected lane issues MMAs, the vote comes after the issue, off its
// path; the elected lane issues if all of its own waits succeeded (what it issues is ready then).  A vote on
// each wait before the issue cost another 0.5 % at d_head 128 (bf16 B*H=32 S=8192 no mask: 975 us, 970 this
// way, 963 without any vote).  The backward's issuers vote once before an issue, which is shorter there (bf16
// D=128 B*H=32 S=4096 causal: 498 us, 502 with the vote after it, 492 without any).
struct LaneWaits {
    bool ok = true;
    template <class Wait>
    FA_HOST_DEVICE void wait(Wait w) {
        if (!w()) ok = false;
    }
};

// The status word a waiter records when it gives up on barrier `barrier_id`.
FA_HOST_DEVICE int wait_timeout_word(int barrier_id) { return (kErrWaitTimeout << 16) | (barrier_id & 0xFFFF); }

// Host side: what a status word read back from the device means for the caller.
// 0 -> 0 (FA_OK); a recorded wait timeout -> -6 (FA_ERR_DEVICE_TIMEOUT); any other
// non-zero word is reported the same way (a kernel recorded an error and stopped early).
FA_HOST_DEVICE int status_word_to_error(int word) { return word == 0 ? 0 : -6; }
FA_HOST_DEVICE int status_word_code(int word) { return (word >> 16) & 0xFFFF; }
FA_HOST_DEVICE int status_word_detail(int word) { return word & 0xFFFF; }

}  // namespace fa
