// Host-side driver of fa::bounded_wait (csrc/bounded_wait.h): the give-up branch of the device-side
// waits, exercised with polls that never succeed and a fake clock.  Prints "ok" and exits 0, or
// prints what failed and exits 1.  Built and run by tests/test_bounded_wait_cpu.py.
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>
#include <vector>

#include "bounded_wait.h"

#define CHECK(cond)                                                        \
    do {                                                                   \
        if (!(cond)) { std::printf("FAILED line %d: %s\n", __LINE__, #cond); return 1; } \
    } while (0)

// What the 32 lanes of a warp meet at (a full-mask vote): returns the AND of all lanes' values in every
// lane.  A lane that waits 10 s for lanes that have left sets `stuck` instead of waiting for good.
class Warp {
public:
    bool all(bool x) {
        std::unique_lock<std::mutex> lock(m_);
        const int phase = phase_;
        acc_ = acc_ && x;
        if (++arrived_ == 32) {
            result_ = acc_;
            acc_ = true;
            arrived_ = 0;
            phase_++;
            cv_.notify_all();
        } else if (!cv_.wait_for(lock, std::chrono::seconds(10), [&] { return phase_ != phase || stuck; })) {
            stuck = true;
            cv_.notify_all();
        }
        return result_;
    }
    bool stuck = false;

private:
    std::mutex m_;
    std::condition_variable cv_;
    bool acc_ = true, result_ = true;
    int arrived_ = 0, phase_ = 0;
};

// A role's loop of three waits, each followed by a full-mask instruction.  In the second wait lane i sees the
// phase complete if its bit of `done` is set and else runs out of time.  VOTE: the warp votes on each wait and
// lane 0 issues after it; else the lanes note the answer, lane 0 issues on its own one and the vote follows.
// Returns the number of steps issued, -1 if the lanes did not leave together or hung.
template <bool VOTE>
int walk(unsigned done) {
    Warp warp;
    std::vector<int> passed(32, 0);
    std::vector<std::thread> lanes;
    int issued = 0;
    for (int lane = 0; lane < 32; lane++)
        lanes.emplace_back([&, lane] {
            for (int step = 0; step < 3; step++) {
                unsigned long long clock = 1;
                const bool success = step != 1 || ((done >> lane) & 1u);
                auto own = [&] {
                    return fa::bounded_wait([&] { return success; }, [] { return false; },
                                            [&] { return clock += 1000000000ull; }, 2000000000ull, 16u) == fa::kWaitDone;
                };
                if (VOTE) {
                    if (!fa::warp_wait(own, [&](bool x) { return warp.all(x); })) break;
                    if (lane == 0) issued++;
                } else {
                    fa::LaneWaits lw;
                    lw.wait(own);
                    warp.all(true);                               // elect.sync
                    if (lane == 0 && lw.ok) issued++;
                    if (!warp.all(lw.ok)) break;
                }
                warp.all(true);
                passed[lane]++;
            }
        });
    for (auto& t : lanes) t.join();
    for (int n : passed)
        if (warp.stuck || n != passed[0]) return -1;
    return issued;
}

int main() {
    using namespace fa;
    const unsigned long long limit = 2000000000ull;        // 2 s, the device-side limit

    // 1. a poll that never succeeds: the wait must give up once the fake clock has moved past the limit
    {
        unsigned long long clock = 5, polls = 0, looks = 0;
        const int r = bounded_wait([&] { polls++; return false; }, [] { return false; },
                                   [&] { looks++; clock += 300000000ull; return clock; }, limit, 16u);
        CHECK(r == kWaitTimedOut);
        // first look starts the stopwatch; it then takes 7 more looks of 0.3 s to exceed 2 s
        CHECK(looks == 8);
        CHECK(polls == 8 * 16);                             // the clock is read every 16th poll only
    }
    // 2. a clock that starts at 0 must still start the stopwatch at its first look
    {
        unsigned long long clock = 0, looks = 0;
        const int r = bounded_wait([] { return false; }, [] { return false; },
                                   [&] { const unsigned long long now = clock; clock += limit + 1; looks++; return now; },
                                   limit, 4u);
        CHECK(r == kWaitTimedOut && looks == 2);
    }
    // 3. somebody else in the CTA gave up: leave at the next look, without reading the clock again
    {
        int polls = 0, looks = 0;
        bool abort_flag = false;
        const int r = bounded_wait([&] { if (++polls == 40) abort_flag = true; return false; },
                                   [&] { return abort_flag; }, [&] { looks++; return 1ull; }, limit, 16u);
        CHECK(r == kWaitAborted);
        CHECK(polls == 48 && looks == 2);                   // looks at polls 16 and 32; abort seen at poll 48
    }
    // 4. the awaited thing happens: no time-out however long it took in polls, as long as the clock is within the limit
    {
        int polls = 0;
        unsigned long long clock = 0;
        const int r = bounded_wait([&] { return ++polls == 1000; }, [] { return false; },
                                   [&] { clock += 1000; return clock; }, limit, 16u);
        CHECK(r == kWaitDone && polls == 1000);
    }
    // 5. success on the first poll never touches the clock or the abort flag
    {
        int looks = 0;
        const int r = bounded_wait([] { return true; }, [&] { looks++; return true; }, [&] { looks++; return 0ull; },
                                   limit, 16u);
        CHECK(r == kWaitDone && looks == 0);
    }
    // 6. a warp in which only some lanes run out of time stays together; nothing is issued after a failed wait
    for (unsigned done : {0x00000000u, 0xfffffffeu, 0x00000001u, 0x0f0f3355u}) {
        CHECK(walk<true>(done) == 1);
        CHECK(walk<false>(done) == ((done & 1u) ? 2 : 1));     // the issuing lane's own wait decides
    }
    CHECK(walk<true>(0xffffffffu) == 3);
    CHECK(walk<false>(0xffffffffu) == 3);
    // 7. the words a waiter records and what the host makes of them
    CHECK(wait_timeout_word(0x41) == ((1 << 16) | 0x41));
    CHECK(status_word_code(wait_timeout_word(7)) == kErrWaitTimeout && status_word_detail(wait_timeout_word(7)) == 7);
    CHECK(status_word_to_error(0) == 0);
    CHECK(status_word_to_error(wait_timeout_word(3)) == -6);
    std::printf("ok\n");
    return 0;
}
