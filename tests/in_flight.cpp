// Host-side check of csrc/in_flight.h against a model of streams and events
// (built by tests/test_in_flight.py): a stream's work is a count, an event
// the work of every stream that is done before it, and waiting for an event
// adds what it stands for to the stream's past.
#include <cstdint>
#include <map>
#include <random>
#include <vector>

#include "in_flight.h"

namespace {

using Past = std::map<cudaStream_t, int64_t>;   // work of each stream that came before
std::map<cudaStream_t, Past> streams;
std::map<cudaEvent_t, Past> events;
std::map<cudaStream_t, bool> captures;
std::map<cudaStream_t, unsigned long long> ids;   // of the stream a handle stands for
unsigned long long next_id = 1;
int64_t waits = 0, live_events = 0, next_event = 1;

void merge(Past* to, const Past& from) {
    for (const auto& p : from) (*to)[p.first] = std::max((*to)[p.first], p.second);
}

// stream 0 is the default stream, which is never another
cudaStream_t handle(int k) { return reinterpret_cast<cudaStream_t>((intptr_t)(k ? 16 + k : 0)); }

void work(cudaStream_t s) { streams[s][s]++; }

bool after(cudaStream_t s, const Past& p) {
    for (const auto& q : p)
        if (streams[s][q.first] < q.second) return false;
    return true;
}

}  // namespace

extern "C" {

cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = reinterpret_cast<cudaEvent_t>((intptr_t)next_event++);
    live_events++;
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { events.erase(e); live_events--; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { events[e] = streams[s]; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    waits++;
    merge(&streams[s], events[e]);
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* st) {
    *st = captures[s] ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamGetId(cudaStream_t s, unsigned long long* id) {
    if (!ids[s]) ids[s] = next_id++;
    *id = ids[s];
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }

// `steps` calls on `num` streams in random order, some of which use the
// scratch (they wait) and some do not: violations of the order.
int64_t in_flight_violations(int num, int steps, uint32_t seed) {
    streams.clear(); events.clear(); captures.clear();
    mlgpu::InFlight f;
    std::mt19937 rng(seed);
    Past marked;
    int64_t bad = 0;
    for (int k = 0; k < steps; k++) {
        const cudaStream_t s = handle((int)(rng() % (unsigned)num));
        if (rng() % 3 != 0) {
            f.wait(s);
            if (!after(s, marked)) bad++;
        }
        if (s != nullptr && rng() % 16 == 0) {      // the handle of another stream now
            streams[s] = Past();
            ids[s] = next_id++;
            if (rng() % 2) { f.wait(s); if (!after(s, marked)) bad++; }
        }
        // work counts go on where the handle's earlier streams stopped
        streams[s][s] = marked[s];
        work(s);
        f.mark(s);
        merge(&marked, streams[s]);
    }
    f.release();
    return bad + live_events;
}

// Calls that only mark do not wait for one another on up to eight streams.
int64_t in_flight_order_among_small() {
    streams.clear(); events.clear(); captures.clear();
    mlgpu::InFlight f;
    int64_t bad = 0;
    for (int k = 0; k < 8; k++) { work(handle(k)); f.mark(handle(k)); }
    for (int k = 0; k < 8; k++)
        for (int j = 0; j < 8; j++)
            if (j != k && streams[handle(k)][handle(j)] != 0) bad++;
    f.release();
    return bad;
}

// A capturing stream neither waits for an event nor is followed.
int64_t in_flight_capture() {
    streams.clear(); events.clear(); captures.clear();
    mlgpu::InFlight f;
    work(handle(0));
    f.mark(handle(0));
    work(handle(2));
    f.mark(handle(2));
    captures[handle(1)] = true;
    const int64_t before = waits, had = live_events;
    f.wait(handle(1));
    work(handle(1));
    f.mark(handle(1));
    const int64_t bad = (waits - before) + (live_events - had);
    f.release();
    return bad;
}

}
