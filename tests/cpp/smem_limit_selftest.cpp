// Threads that raise a kernel's shared-memory limit at the same time
// (lmb_smem.h), on a stand-in for the call that sets it: the limit is never
// set below an earlier size, every thread that was told its size is granted
// finds it so, and a refused size is asked for again.
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>

#include "lmb_smem.h"

int main()
{
    using namespace std::chrono_literals;
    int bad = 0;
    {
        // The smaller size's call is slow: set at once, the two would end on it.
        lmb::SmemLimit limit;
        std::atomic<size_t> set{0};
        std::atomic<bool> started{false};
        std::thread a([&] {
            limit.raise(0, 100, [&](size_t b) {
                started = true;
                std::this_thread::sleep_for(100ms);
                set = b;
                return 0;
            });
        });
        while (!started) std::this_thread::yield();
        limit.raise(0, 200, [&](size_t b) {
            set = b;
            return 0;
        });
        bad += set < 200;
        a.join();
        bad += set != 200;
    }
    {
        lmb::SmemLimit limit;
        std::atomic<size_t> set{0};
        std::atomic<int> lowered{0}, calls{0}, short_of{0};
        std::vector<std::thread> threads;
        for (size_t t = 0; t < 8; t++)
            threads.emplace_back([&, t] {
                for (size_t k = 0; k < 400; k++) {
                    const size_t want = (t * 37 + k * 101) % 1000 + 1;
                    const int rc = limit.raise(3, want, [&](size_t b) {
                        if (b < set) lowered++;
                        set = b;
                        calls++;
                        return 0;
                    });
                    if (rc != 0 || set < want) short_of++;
                }
            });
        for (std::thread &t : threads) t.join();
        bad += lowered != 0 || short_of != 0 || set != 1000 || calls > 1000;
    }
    {
        lmb::SmemLimit limit;
        int calls = 0;
        bad += limit.raise(1, 50, [&](size_t) { return calls++, 7; }) != 7;
        bad += limit.raise(1, 50, [&](size_t) { return calls++, 0; }) != 0;
        bad += limit.raise(1, 40, [&](size_t) { return calls++, 7; }) != 0;
        bad += limit.raise(2, 40, [&](size_t) { return calls++, 0; }) != 0;  // devices apart
        bad += calls != 3;
        bad += limit.raise(-1, 1, [](size_t) { return 0; }) != lmb::SmemLimit::BAD_DEVICE;
        bad += limit.raise(lmb::SmemLimit::DEVICES, 1, [](size_t) { return 0; }) != lmb::SmemLimit::BAD_DEVICE;
    }
    if (bad) std::printf("%d checks failed\n", bad);
    return bad ? 1 : 0;
}
