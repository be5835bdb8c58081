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
    // Work queued on `s` from now on starts after what was marked so far.
    cudaError_t wait(cudaStream_t s) {
        if (used_ == 0 || capturing(s)) return cudaSuccess;
        for (int k = 0; k < used_; k++) {
            const cudaError_t e = cudaStreamWaitEvent(s, marks_[k].event, 0);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }

    // The work queued on `s` so far is in flight.  A stream keeps its event
    // (by its id, as a handle can come to stand for another stream); with more
    // streams than events, what a reused event stood for comes to `s` first,
    // so nothing is forgotten.
    cudaError_t mark(cudaStream_t s) {
        unsigned long long id = 0;
        if (capturing(s)) return cudaSuccess;
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
        used_ = 0;
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
