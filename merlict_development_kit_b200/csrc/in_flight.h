// in_flight.h -- the work that calls on a scene have left on the GPU.
//
// A scene owns scratch memory (ray pools, photon lists, sort buffers) and the
// error word, and most calls return while their last kernels still use them.
// Calls on one stream follow one another there; a call on another stream
// first waits, on the device, for what the calls before it left: every entry
// point that writes the scene's scratch begins with wait() and ends with
// mark().  No host wait, and no wait at all for calls that only mark (a small
// batch uses no scratch, but its errors and inputs are in use).
//
// Work that is being captured into a graph is not followed: an event of a
// capture means nothing outside it, and the other way round.
#ifndef MLGPU_IN_FLIGHT_H_
#define MLGPU_IN_FLIGHT_H_

#include <cuda_runtime.h>

namespace mlgpu {

class InFlight {
 public:
    // Work queued on `s` from now on starts after what was marked so far (on
    // `s` itself it does anyway).
    cudaError_t wait(cudaStream_t s) {
        if (used_ == 0 && (!on_default_ || s == nullptr)) return cudaSuccess;
        unsigned long long id = 0;
        cudaError_t e = cudaStreamGetId(s, &id);
        if (e != cudaSuccess) return e;
        if (used_ == 1 && marks_[0].stream == id && !on_default_) return cudaSuccess;
        if (capturing(s)) return cudaSuccess;
        if (on_default_ && s != nullptr) {
            if (!default_) e = cudaEventCreateWithFlags(&default_, cudaEventDisableTiming);
            if (e == cudaSuccess) e = cudaEventRecord(default_, nullptr);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(s, default_, 0);
        }
        for (int k = 0; k < used_ && e == cudaSuccess; k++)
            if (marks_[k].stream != id) e = cudaStreamWaitEvent(s, marks_[k].event, 0);
        return e;
    }

    // The work queued on `s` so far is in flight.  A stream keeps its event
    // (by its id, as a handle can come to stand for another stream); with more
    // streams than events, what a reused event stood for comes to `s` first,
    // so nothing is forgotten.  The default stream is always there, so its
    // event can be left to the wait: an event per call is 1.4 us of the 94 us
    // that 300 photons take.
    cudaError_t mark(cudaStream_t s) {
        if (s == nullptr) {
            on_default_ = true;
            return cudaSuccess;
        }
        if (capturing(s)) return cudaSuccess;
        unsigned long long id = 0;
        cudaError_t e = cudaStreamGetId(s, &id);
        if (e != cudaSuccess) return e;
        int k = 0;
        while (k < used_ && marks_[k].stream != id) k++;
        if (k == used_ && used_ < kStreams) {
            e = cudaEventCreateWithFlags(&marks_[k].event, cudaEventDisableTiming);
            if (e == cudaSuccess) used_++;
        } else if (k == used_) {
            k = next_++ % kStreams;
            e = cudaStreamWaitEvent(s, marks_[k].event, 0);
        }
        if (e != cudaSuccess) return e;
        marks_[k].stream = id;
        return cudaEventRecord(marks_[k].event, s);
    }

    void release() {
        for (int k = 0; k < used_; k++) cudaEventDestroy(marks_[k].event);
        if (default_) cudaEventDestroy(default_);
        used_ = 0;
        default_ = nullptr;
        on_default_ = false;
    }

 private:
    static constexpr int kStreams = 8;
    struct Mark {
        unsigned long long stream;
        cudaEvent_t event;
    };
    Mark marks_[kStreams] = {};
    int used_ = 0;
    unsigned next_ = 0;
    bool on_default_ = false;        // something may be in flight on the default stream
    cudaEvent_t default_ = nullptr;

    static bool capturing(cudaStream_t s) {
        cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(s, &st) != cudaSuccess) {
            cudaGetLastError();   // the default stream during another one's capture
            return true;
        }
        return st != cudaStreamCaptureStatusNone;
    }
};

}  // namespace mlgpu

#endif  // MLGPU_IN_FLIGHT_H_
