// ScratchTurn (gmt_turn.h) over stand-ins of the three runtime calls that it makes: each prints itself, and
// fails where the scenario says so.  Streams are numbers; the last line of a scenario is "end".
#include <chrono>
#include <cstdint>
#include <cstdio>
#include <thread>

#include "../../glmmhdturb_b200/csrc/gmt_turn.h"

static bool fail_wait, fail_record;
static int num(cudaStream_t s) { return (int)(intptr_t)s; }

extern "C" {
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t, unsigned) {
    std::printf("wait %d\n", num(s));
    return fail_wait ? cudaErrorInvalidValue : cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t s) {
    std::printf("record %d\n", num(s));
    return fail_record ? cudaErrorInvalidValue : cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    std::printf("synchronise %d\n", num(s));
    return cudaSuccess;
}
}

static std::mutex mu;

// a holder of stream s whose launches fail or not; left by return either way
static cudaError_t hold(int s, bool launches_fail) {
    gmt::ScratchTurn turn(mu, nullptr, (cudaStream_t)(intptr_t)s);
    if (turn.status() != cudaSuccess) return turn.status();
    std::printf("launch %d\n", s);
    if (launches_fail) return cudaErrorLaunchFailure;
    return turn.mark();
}

int main() {
    const struct { bool wait, record, launch; } cases[] = {{}, {false, false, true}, {true, false, false}, {false, true, false}};
    for (auto& c : cases) {
        fail_wait = c.wait;
        fail_record = c.record;
        std::printf("status %d\n", hold(1, c.launch) != cudaSuccess);
        fail_wait = fail_record = false;
        std::printf("free %d\n", mu.try_lock());
        mu.unlock();
        std::printf("end\n");
    }
    // another thread gets its turn only when the first has left, or marked the end of its work
    std::thread t;
    {
        gmt::ScratchTurn turn(mu, nullptr, (cudaStream_t)(intptr_t)1);
        t = std::thread([] { hold(2, false); });
        std::this_thread::sleep_for(std::chrono::milliseconds(50));
        std::printf("launch 1\n");
    }
    t.join();
    std::printf("end\n");
    {
        gmt::ScratchTurn turn(mu, nullptr, (cudaStream_t)(intptr_t)1);
        turn.mark();
        std::thread([] { hold(2, false); }).join();
    }
    std::printf("end\n");
    return 0;
}
