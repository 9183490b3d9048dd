// Recent (gmt_recent.h) under threads that keep and find values of more keys than it holds.  A value is 16 words
// of its key: prints how many were found, and how many of those were not whole.
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>

#include "../../glmmhdturb_b200/csrc/gmt_recent.h"

struct Value { long w[16]; };

int main() {
    gmt::Recent<long, Value, 4> recent;
    std::atomic<long> found{0}, torn{0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 4; ++t)
        threads.emplace_back([&, t] {
            for (long i = 0; i < 200000; ++i) {
                const long k = (i * 7 + t) % 6;
                Value v;
                if (recent.find(k, &v)) {
                    ++found;
                    for (long w : v.w)
                        if (w != k) { ++torn; break; }
                } else {
                    for (long& w : v.w) w = k;
                    recent.keep(k, v);
                }
            }
        });
    for (auto& t : threads) t.join();
    // one thread: the oldest of more keys than it holds is gone, the others are there
    gmt::Recent<long, Value, 4> last;
    Value v{};
    for (long k = 0; k < 5; ++k) last.keep(k, v);
    std::printf("%ld %ld %d %d%d%d%d\n", found.load(), torn.load(), last.find(0, &v), last.find(1, &v), last.find(2, &v),
                last.find(3, &v), last.find(4, &v));
    return 0;
}
