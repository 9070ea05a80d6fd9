// Drives csrc/side_stream.h against a CUDA runtime of a few fake functions that write down what is called.  Prints "ok".
#include <cstdio>
#include <cstdlib>
#include <map>
#include <string>

#include "../bi-mamba2_b200/csrc/side_stream.h"

static std::string calls;                                        // one letter per call: R record, W wait, S synchronize, C create
static std::string refuse;                                       // letters whose next call fails
static std::map<cudaStream_t, unsigned long long> capture;      // streams in a capture, and which
static long made = 100;
static cudaError_t note(char c) {
    const size_t at = refuse.find(c);
    calls += c;
    if (at == std::string::npos) return cudaSuccess;
    refuse.erase(at, 1);
    return cudaErrorUnknown;
}
extern "C" {
cudaError_t cudaGetDevice(int *dev) { *dev = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)++made; return note('C'); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    const cudaError_t r = note('E');
    if (r == cudaSuccess) *e = (cudaEvent_t)++made;
    return r;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return note('c'); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return note('e'); }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return note('R'); }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return note('W'); }
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t s, cudaStreamCaptureStatus *st, unsigned long long *id, cudaGraph_t *,
                                     const cudaGraphNode_t **, size_t *) {
    *st = capture.count(s) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    *id = capture.count(s) ? capture[s] : 0;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return note('S'); }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus *st) {
    *st = capture.count(s) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
}

static void expect(bool ok, const char *what) {
    if (ok) return;
    std::printf("%s (calls: %s)\n", what, calls.c_str());
    std::exit(1);
}
static std::string take() { std::string c; c.swap(calls); return c; }

int main() {
    using bissd::SideStream;
    const cudaStream_t s = (cudaStream_t)1, other = (cudaStream_t)2;
    {
        refuse = "E";
        SideStream side(s);
        expect(side.fork() == cudaSuccess && side.stream() == s, "no event, no second stream");
        expect(take() == "CEc", "the stream of a set that could not be made is destroyed");
    }
    cudaStream_t first;
    {                                                            // as a pass that succeeds: fork, join, fork, join
        SideStream side(s);
        expect(side.fork() == cudaSuccess && side.stream() != s, "forked");
        first = side.stream();
        expect(take() == "CEERW", "a set, then the fork");
        {
            SideStream beside(other);
            expect(beside.fork() == cudaSuccess && beside.stream() != first, "a leased set is not leased again");
        }
        expect(take() == "CEERWRW", "its fork and its join");
        expect(side.join() == cudaSuccess && side.stream() == s, "joined");
        expect(side.fork() == cudaSuccess && side.join() == cudaSuccess, "again");
        expect(take() == "RWRWRW", "join, fork, join");
    }
    expect(take().empty(), "nothing left to join");
    {                                                            // a launch fails after the fork: the call returns from here
        SideStream side(s);
        side.fork();
        expect(side.stream() == first && take() == "RW", "the freed set is used again");
    }
    expect(take() == "RW", "the destructor joins");
    {                                                            // and the join fails too
        SideStream side(s);
        side.fork();
        take();
        refuse = "R";
    }
    expect(take() == "RS", "without an event the host waits");
    {
        SideStream side(s);
        refuse = "W";
        expect(side.fork() != cudaSuccess && side.stream() == s, "a refused fork stays in line");
        take();
    }
    expect(take().empty(), "and has nothing to join");
    {                                                            // `first` was forked into capture 7 of s, which goes on after the call
        capture[s] = capture[first] = 7;
        SideStream beside(other);
        expect(beside.fork() == cudaSuccess && beside.stream() != first, "a stream in another's capture is left alone");
        SideStream same(s);
        expect(same.fork() == cudaSuccess && same.stream() == first, "the capture's own calls use it");
        capture[other] = 8;
        SideStream later(other);
        expect(later.fork() == cudaSuccess && later.stream() == other, "no set is made inside a capture");
    }
    std::printf("ok\n");
    return 0;
}
