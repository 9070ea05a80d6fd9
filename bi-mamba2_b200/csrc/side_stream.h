// The backward's second stream: sets of (stream, events) per device, leased by a call for its duration.  Host code only.
#pragma once
#include <cuda_runtime_api.h>

#include <mutex>
#include <vector>

namespace bissd {

struct SideSet {
    cudaStream_t st = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    int dev = -1;
    bool busy = false;
};
inline std::mutex g_side_mu;
inline std::vector<SideSet *> g_side;

// May what `main` launches go to `side` now?  A stream that was forked into a capture belongs to it until the capture ends, long
// after its lease: only calls of the same capture may use it, anything else would break the capture.
inline bool side_usable(cudaStream_t side, cudaStream_t main) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone, st_main = st;
    unsigned long long id = 0, id_main = 0;
    if (cudaStreamGetCaptureInfo(side, &st, &id) != cudaSuccess) return false;
    if (st == cudaStreamCaptureStatusNone) return true;
    return st == cudaStreamCaptureStatusActive && cudaStreamGetCaptureInfo(main, &st_main, &id_main) == cudaSuccess && st_main == st && id_main == id;
}

// A free set of the current device, or null: the launch then stays in line.  Sets are created on first need - in practice
// by the first call on a device - but not while the caller's stream is being captured (creation belongs outside a capture).
inline SideSet *side_acquire(cudaStream_t s) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    std::lock_guard<std::mutex> lk(g_side_mu);
    for (SideSet *set : g_side)
        if (set->dev == dev && !set->busy && side_usable(set->st, s)) {
            set->busy = true;
            return set;
        }
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return nullptr;
    }
    SideSet made;
    if (cudaStreamCreateWithFlags(&made.st, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&made.fork, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&made.join, cudaEventDisableTiming) != cudaSuccess) {
        if (made.fork) cudaEventDestroy(made.fork);
        if (made.st) cudaStreamDestroy(made.st);
        cudaGetLastError();
        return nullptr;
    }
    made.dev = dev;
    made.busy = true;
    g_side.push_back(new SideSet(made));
    return g_side.back();
}

// One call's use of a second stream beside its own.  Between a fork and the next join the side stream may hold kernels that
// use the call's buffers, which the caller is free to give back in the order of its own stream once the call has
// returned: so the destructor joins, whichever way the call ends, and only then is the set free for another call.
class SideStream {
public:
    explicit SideStream(cudaStream_t main) : main_(main) {}
    SideStream(const SideStream &) = delete;
    SideStream &operator=(const SideStream &) = delete;
    ~SideStream() {
        if (!set_) return;
        if (join() != cudaSuccess) {
            cudaGetLastError();
            cudaStreamSynchronize(set_->st);                      // no event to wait for: wait here (refused under capture, which has failed anyway)
            cudaGetLastError();
        }
        std::lock_guard<std::mutex> lk(g_side_mu);
        set_->busy = false;
    }
    // What is launched on stream() from here on runs after what the caller's stream holds now.  Leases a set the first time;
    // without one, stream() stays the caller's.
    cudaError_t fork() {
        if (!set_ && !(set_ = side_acquire(main_))) return cudaSuccess;
        cudaError_t e = cudaEventRecord(set_->fork, main_);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(set_->st, set_->fork, 0);
        if (e == cudaSuccess) pending_ = true;
        return e;
    }
    // The caller's stream waits for what stream() holds.
    cudaError_t join() {
        if (!pending_) return cudaSuccess;
        cudaError_t e = cudaEventRecord(set_->join, set_->st);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(main_, set_->join, 0);
        if (e == cudaSuccess) pending_ = false;
        return e;
    }
    cudaStream_t stream() const { return pending_ ? set_->st : main_; }

private:
    cudaStream_t main_;
    SideSet *set_ = nullptr;
    bool pending_ = false;
};

}  // namespace bissd
