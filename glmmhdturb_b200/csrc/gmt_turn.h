// gmt_turn.h -- scratch that calls on several streams and threads use in turn (host code).
#pragma once
#include <cuda_runtime_api.h>

#include <mutex>

namespace gmt {

// One holder's turn: from construction the mutex is held and work put on the stream runs after the last
// holder's, which `ev` marks; however the holder leaves, `ev` then marks its own work, and the mutex is
// given back.  If the wait could not be put on the stream (status), nothing may be launched and `ev`
// keeps marking the last holder; if `ev` cannot be recorded, the work is waited for instead.
class ScratchTurn {
public:
    ScratchTurn(std::mutex& mu, cudaEvent_t ev, cudaStream_t s)
        : lock_(mu), ev_(ev), s_(s), status_(cudaStreamWaitEvent(s, ev, 0)), open_(status_ == cudaSuccess) {}
    ~ScratchTurn() { mark(); }
    ScratchTurn(const ScratchTurn&) = delete;
    ScratchTurn& operator=(const ScratchTurn&) = delete;
    cudaError_t status() const { return status_; }
    // all of the holder's work is on the stream: the next holder may come
    cudaError_t mark() {
        if (!open_) return cudaSuccess;
        open_ = false;
        const cudaError_t e = cudaEventRecord(ev_, s_);
        if (e != cudaSuccess) cudaStreamSynchronize(s_);
        lock_.unlock();
        return e;
    }

private:
    std::unique_lock<std::mutex> lock_;
    cudaEvent_t ev_;
    cudaStream_t s_;
    cudaError_t status_;
    bool open_;
};

}  // namespace gmt
