// signal_chain.cu -- the signal chain after binning for one event, on the
// device: photon pipelines (merlict_signal_processing/PipelinePhoton.cpp:
// 25-65), night-sky background (merlict_portal_plenoscope/
// night_sky_background/Injector.cpp:8-98), photo-electric conversion
// (merlict_signal_processing/PhotoElectricConverter.cpp:31-90) and
// single-pulse extraction (merlict_signal_processing/pulse_extraction.cpp:
// 9-35).
//
// Layout of the work:
//   1. pipelines: a counting sort by sensor (photons without one are left
//      out; its scan gives every pipeline's offset), then every sensor's
//      run by (arrival time, input index) -- ranks in shared memory for runs
//      of up to 4096 photons, a stable radix sort of each longer run by one
//      block (device_sort.cu) -- then per photon, in pipeline order and
//      contiguous per lixel: time, truth id, the quantum efficiency at its
//      wavelength and two of its lixel's conversion draws;
//   2. the exposure window: min/max of the Cherenkov arrival times (one
//      atomic per warp), their histogram on 2 + sqrt(n) linearly spaced
//      edges (block-private bins in shared memory), the first fullest bin;
//   3. one thread per lixel walks its pipeline merged with its background
//      photons (the Poisson stream first, to know their number, then their
//      wavelengths) and converts every photon to electric pulses -- twice:
//      a counting pass, a scan of the counts (the host reads the total and
//      sizes the pulse buffer), a writing pass with the same draws, which
//      writes a Cherenkov photon's pulses as its place in the pipelines;
//   4. extraction, one thread per pulse: pulse j of lixel i takes draws 2j
//      and 2j + 1 of its stream; the kept pulses are compacted (a scan of
//      the keep flags), which also gives each channel's offset.
//
// Draws: stage s (1 background, 2 conversion, 3 extraction) of lixel i
// draws uniforms k = 0, 1, ... of the Philox stream ((0xF0 | s) << 56) |
// (offset + i) in the order merlict's code asks for them; a normal deviate
// is mean + std sqrt(-2 ln(1 - u1)) cos(2 pi u2) of two uniforms.
// Compiled with --fmad=false: the arithmetic is merlict's, in merlict's
// order, so only log and cos (CUDA's, not the C library's) can differ in
// the last bit.
#include <cmath>
#include <cstdint>

#include "merlict_b200_philox.h"
#include "mlgpu_internal.h"
#include "fp64_geometry.cuh"

namespace mlgpu {
namespace {

constexpr int32_t kNightSkyBackground = -100;      // simulation_truth.h:15-17
constexpr int32_t kAccidental = -201;
constexpr int32_t kCrosstalk = -202;
constexpr double kNumberTimeSlices = 100.0;         // pulse_extraction.h:13
constexpr uint32_t kMaxDraws = 0xFFFFFF00u;         // counter space of one stream
constexpr int kSmemBins = 12288;                    // block-private histogram limit
constexpr int kHistThreads = 1024;                  // one block per SM: each adds its bins once

__device__ __forceinline__ uint64_t time_key(double t) {
    const uint64_t b = (uint64_t)__double_as_longlong(t);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

__device__ __forceinline__ double key_time(uint64_t k) {
    const uint64_t b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
    return __longlong_as_double((long long)b);
}

__device__ __forceinline__ uint64_t stage_stream(uint64_t stage, uint64_t offset, uint64_t lixel) {
    return ((0xF0ull | stage) << 56) | ((offset + lixel) & ((1ull << 56) - 1));
}

// Generator::expovariate (merlict/random/Generator.cpp:36-39)
__device__ __forceinline__ double expovariate(double u, double rate) {
    return -log(u)/rate;
}

__device__ __forceinline__ void raise_error(unsigned int* err, int code) {
    atomicCAS(err, 0u, (unsigned)code);
}

// ---- 1. pipelines ------------------------------------------------------------

// Photon i's rank among the photons of its sensor, in no particular order:
// the counting atomic already returns it, so placing a photon later needs no
// second one.  Photons with equal sensors within a warp are merged
// (__match_any_sync), one atomic per sensor and warp: a bright lixel's
// atomics would else line up at one address.  Photons without a sensor are
// neither counted nor placed; as one more key (half of an event's photons
// may miss) their atomics alone bounded the two passes: 27 + 30 us for 1e6
// photons, now 13 + 13.
constexpr int kRankRun = 4;        // photons of a thread whose atomics are in flight together

__global__ void __launch_bounds__(256)
sc_rank_kernel(const int32_t* __restrict__ sensor, uint64_t n, uint32_t num_sensors,
               uint32_t* __restrict__ count, uint32_t* __restrict__ rank,
               unsigned long long* __restrict__ minmax, unsigned int* __restrict__ err) {
    const int lane = threadIdx.x & 31;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        minmax[0] = 0xffefffffffffffffull;     // the time keys of DBL_MAX and DBL_MIN
        minmax[1] = 0x8010000000000000ull;
    }
    for (uint64_t b = kRankRun*((uint64_t)blockIdx.x*blockDim.x + (threadIdx.x & ~31u)); b < n;
         b += kRankRun*(uint64_t)gridDim.x*blockDim.x) {
        int32_t s[kRankRun];
        unsigned peers[kRankRun];
        uint32_t first[kRankRun];
#pragma unroll
        for (int k = 0; k < kRankRun; k++) {
            const uint64_t i = b + 32*k + lane;
            s[k] = i < n ? __ldg(sensor + i) : -1;
        }
#pragma unroll
        for (int k = 0; k < kRankRun; k++) {
            if (s[k] >= (int32_t)num_sensors) {
                raise_error(err, MLGPU_ERR_INVALID_ARGUMENT);
                s[k] = -1;
            }
            // photons without a sensor make one group, which nothing is done for
            peers[k] = __match_any_sync(0xffffffffu, s[k] < 0 ? -1 : s[k]);
            first[k] = 0;
            if (s[k] >= 0 && lane == __ffs(peers[k]) - 1)
                first[k] = atomicAdd(count + s[k], (unsigned)__popc(peers[k]));
        }
#pragma unroll
        for (int k = 0; k < kRankRun; k++) {
            first[k] = __shfl_sync(0xffffffffu, first[k], __ffs(peers[k]) - 1);
            if (s[k] >= 0)
                rank[b + 32*k + lane] = first[k] + __popc(peers[k] & ((1u << lane) - 1u));
        }
    }
}

// time key and input index of every photon with a sensor into its pipeline
__global__ void __launch_bounds__(256)
sc_place_kernel(const int32_t* __restrict__ sensor, const double* __restrict__ time, uint64_t n,
                uint32_t num_sensors, const uint32_t* __restrict__ rank,
                const uint64_t* __restrict__ pipe_off, uint64_t* __restrict__ key,
                uint32_t* __restrict__ idx) {
    for (uint64_t i = blockIdx.x*(uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x*blockDim.x) {
        const int32_t s = __ldg(sensor + i);
        if (s < 0 || s >= (int32_t)num_sensors) continue;
        const uint64_t j = __ldg(pipe_off + s) + __ldg(rank + i);
        key[j] = time_key(__ldg(time + i));
        idx[j] = (uint32_t)i;
    }
}

// Every sensor's run by (time key, input index), i.e. stable by time: runs
// of up to kWarpSegment photons by one warp in shared memory, up to
// kBlockSegment by one block (sc_segsort_block_kernel), longer ones by a
// radix sort of the run by (time key, index) by one block (sort_long_runs).
// Each element's place is its rank in the run, so the order the placing
// left within a sensor does not matter.
constexpr uint32_t kWarpSegment = 256;
constexpr uint32_t kBlockSegment = 4096;
constexpr int kSegWarps = 8;

__device__ __forceinline__ bool sorts_before(uint64_t ka, uint32_t va, uint64_t kb, uint32_t vb) {
    return ka < kb || (ka == kb && va < vb);
}

__global__ void __launch_bounds__(kSegWarps*32)
sc_segsort_warp_kernel(const uint64_t* __restrict__ key_in, const uint32_t* __restrict__ val_in,
                       const uint64_t* __restrict__ pipe_off, uint32_t num_sensors,
                       uint64_t* __restrict__ key_out, uint32_t* __restrict__ val_out,
                       uint32_t* __restrict__ medium, unsigned int* __restrict__ num_medium,
                       uint64_t* __restrict__ large_begin, uint64_t* __restrict__ large_end,
                       unsigned int* __restrict__ num_large) {
    __shared__ __align__(16) uint64_t sk[kSegWarps][kWarpSegment];
    __shared__ uint32_t sv[kSegWarps][kWarpSegment];
    __shared__ uint8_t sr[kSegWarps][kWarpSegment];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t l = blockIdx.x*kSegWarps + w;
    if (l >= num_sensors) return;
    const uint64_t b = pipe_off[l];
    const uint64_t m = pipe_off[l + 1] - b;
    if (m == 0) return;
    if (m > kWarpSegment) {
        if (lane == 0) {
            if (m <= kBlockSegment) {
                medium[atomicAdd(num_medium, 1u)] = l;
            } else {
                const unsigned int k = atomicAdd(num_large, 1u);
                large_begin[k] = b;
                large_end[k] = b + m;
            }
        }
        return;
    }
    const uint32_t mm = (uint32_t)m;
    for (uint32_t i = lane; i < mm; i += 32) {
        sk[w][i] = key_in[b + i];
        sv[w][i] = val_in[b + i];
    }
    // an odd run's last pair: no key is above this one, so it counts for none
    if ((mm & 1u) && lane == 0) sk[w][mm] = ~0ull;
    __syncwarp();
    // the rank by time alone, two keys a load; the ranks are a permutation,
    // with the sum 0 + 1 + ..., unless some times are equal (a tied element
    // ranks below its place)
    uint32_t sum = 0;
    for (uint32_t i = lane; i < mm; i += 32) {
        const uint64_t ki = sk[w][i];
        uint32_t r = 0;
        for (uint32_t j = 0; j < mm; j += 2) {
            const ulonglong2 kk = *reinterpret_cast<const ulonglong2*>(&sk[w][j]);
            r += kk.x < ki ? 1u : 0u;
            r += kk.y < ki ? 1u : 0u;
        }
        sr[w][i] = (uint8_t)r;
        sum += r;
    }
    const bool ties = __reduce_add_sync(0xffffffffu, sum) != mm*(mm - 1)/2;
    for (uint32_t i = lane; i < mm; i += 32) {
        const uint64_t ki = sk[w][i];
        const uint32_t vi = sv[w][i];
        uint32_t r = sr[w][i];
        if (ties)
            for (uint32_t j = 0; j < mm; j++) r += sk[w][j] == ki && sv[w][j] < vi ? 1u : 0u;
        key_out[b + r] = ki;
        val_out[b + r] = vi;
    }
}

__global__ void __launch_bounds__(512)
sc_segsort_block_kernel(const uint64_t* __restrict__ key_in, const uint32_t* __restrict__ val_in,
                        const uint64_t* __restrict__ pipe_off, const uint32_t* __restrict__ medium,
                        const unsigned int* __restrict__ num_medium, uint64_t* __restrict__ key_out,
                        uint32_t* __restrict__ val_out) {
    extern __shared__ uint64_t seg_smem[];
    uint64_t* sk = seg_smem;
    uint32_t* sv = reinterpret_cast<uint32_t*>(seg_smem + kBlockSegment);
    const unsigned int count = *num_medium;
    for (unsigned int t = blockIdx.x; t < count; t += gridDim.x) {
        const uint32_t l = medium[t];
        const uint64_t b = pipe_off[l];
        const uint32_t m = (uint32_t)(pipe_off[l + 1] - b);
        for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
            sk[i] = key_in[b + i];
            sv[i] = val_in[b + i];
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
            const uint64_t ki = sk[i];
            const uint32_t vi = sv[i];
            uint32_t r = 0;
            for (uint32_t j = 0; j < m; j++) r += sorts_before(sk[j], sv[j], ki, vi) ? 1u : 0u;
            key_out[b + r] = ki;
            val_out[b + r] = vi;
        }
        __syncthreads();
    }
}

// What the conversion needs of every photon, in pipeline order: its time
// (from its key, in place), its truth id, the quantum efficiency at its
// wavelength, and for the r-th photon of the pipeline uniforms 2r and
// 2r + 1 of its lixel's conversion stream, each with how many draws from it
// on give crosstalk (up to kLongRun).  The conversion of a lixel is one
// serial chain; whatever of it does not depend on the draws before it is
// computed here, one photon per thread.  A wavelength outside the table
// fails the call, as it does in the chain.
constexpr uint32_t kLongRun = 255;

__global__ void __launch_bounds__(256)
sc_gather_kernel(SignalChainParams P, uint64_t seed, uint64_t offset,
                 const uint32_t* __restrict__ idx, const int32_t* __restrict__ sensor,
                 const double* __restrict__ wavelength, const int32_t* __restrict__ truth,
                 const uint64_t* __restrict__ pipe_off, uint32_t num_sensors,
                 double* __restrict__ t, double* __restrict__ q_out, int32_t* __restrict__ r_out,
                 double2* __restrict__ u_out, uchar2* __restrict__ run_out,
                 unsigned int* __restrict__ err) {
    const uint64_t n = pipe_off[num_sensors];
    for (uint64_t j = blockIdx.x*(uint64_t)blockDim.x + threadIdx.x; j < n;
         j += (uint64_t)gridDim.x*blockDim.x) {
        const uint32_t i = __ldg(idx + j);
        const uint32_t l = (uint32_t)__ldg(sensor + i);
        t[j] = key_time((uint64_t)__double_as_longlong(t[j]));
        int e = 0;
        q_out[j] = fp64::func_eval_points(P.qe, P.num_qe, __ldg(wavelength + i), &e);
        if (e) raise_error(err, e);
        r_out[j] = __ldg(truth + i);
        const uint32_t k = 2u*(uint32_t)(j - __ldg(pipe_off + l));
        const uint64_t s_pec = stage_stream(2, offset, l);
        const double u0 = mlgpu_philox_uniform(seed, s_pec, k);
        const double u1 = mlgpu_philox_uniform(seed, s_pec, k + 1);
        u_out[j] = make_double2(u0, u1);
        uint32_t run = 0;
        if (P.second_puls >= u1)
            do run++;
            while (run < kLongRun &&
                   P.second_puls >= mlgpu_philox_uniform(seed, s_pec, k + 1 + run));
        const uint32_t run0 = P.second_puls >= u0 ? (run < kLongRun ? run + 1 : run) : 0u;
        run_out[j] = make_uchar2((unsigned char)run0, (unsigned char)run);
    }
}

// The earliest and latest Cherenkov arrival (Injector.cpp:21-41: min over
// the pipelines' fronts from DBL_MAX, max over their backs from DBL_MIN);
// one atomic per warp.
__global__ void __launch_bounds__(128)
sc_minmax_kernel(const double* __restrict__ t, const uint64_t* __restrict__ pipe_off,
                 uint32_t num_sensors, unsigned long long* __restrict__ minmax) {
    const uint32_t s = blockIdx.x*blockDim.x + threadIdx.x;
    unsigned long long lo = 0xffffffffffffffffull, hi = 0ull;
    if (s < num_sensors) {
        const uint64_t b = pipe_off[s], e = pipe_off[s + 1];
        if (e > b) {
            lo = time_key(t[b]);
            hi = time_key(t[e - 1]);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long a = __shfl_xor_sync(0xffffffffu, lo, o);
        const unsigned long long c = __shfl_xor_sync(0xffffffffu, hi, o);
        lo = a < lo ? a : lo;
        hi = c > hi ? c : hi;
    }
    if ((threadIdx.x & 31) == 0) {
        if (lo != 0xffffffffffffffffull) atomicMin(minmax + 0, lo);
        if (hi != 0ull) atomicMax(minmax + 1, hi);
    }
}

// ---- 2. the exposure window, Injector.cpp:43-59 -----------------------------------

struct Edges {
    double lo, step;
    uint32_t count;             // bin edges; count - 1 bins
    __device__ double at(uint32_t i) const { return lo + step*(double)i; }   // numeric::linspace
};

__device__ __forceinline__ Edges make_edges(const unsigned long long* minmax, uint64_t n) {
    Edges e;
    const double lo = key_time(minmax[0]), hi = key_time(minmax[1]);
    e.count = (uint32_t)(2.0 + sqrt((double)n));
    e.lo = lo;
    e.step = (hi - lo)/(double)(e.count - 1);
    return e;
}

// Histogram1::fill_in (Histogram1.cpp:29-44): std::upper_bound over the edges
__device__ __forceinline__ int64_t bin_of(const Edges& e, double t) {
    uint32_t first = 0, len = e.count;
    while (len > 0) {
        const uint32_t half = len >> 1, mid = first + half;
        if (t < e.at(mid)) { len = half; }
        else { first = mid + 1; len -= half + 1; }
    }
    if (first == 0 || first == e.count) return -1;     // under- or overflow
    return (int64_t)first - 1;
}

__global__ void __launch_bounds__(kHistThreads)
sc_histogram_kernel(const double* __restrict__ t, const uint64_t* __restrict__ pipe_off,
                    uint32_t num_sensors, const unsigned long long* __restrict__ minmax,
                    uint32_t* __restrict__ bins, int use_smem) {
    extern __shared__ uint32_t sbins[];
    const uint64_t n = pipe_off[num_sensors];
    if (n == 0) return;
    const Edges e = make_edges(minmax, n);
    const uint32_t nb = e.count - 1;
    if (use_smem) {
        for (uint32_t i = threadIdx.x; i < nb; i += blockDim.x) sbins[i] = 0;
        __syncthreads();
    }
    for (uint64_t j = blockIdx.x*(uint64_t)blockDim.x + threadIdx.x; j < n;
         j += (uint64_t)gridDim.x*blockDim.x) {
        const int64_t b = bin_of(e, t[j]);
        if (b >= 0) atomicAdd(use_smem ? sbins + b : bins + b, 1u);
    }
    if (use_smem) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < nb; i += blockDim.x)
            if (sbins[i]) atomicAdd(bins + i, sbins[i]);
    }
}

// Histogram1::mode / arg_max (Histogram1.cpp:46-60): the first fullest bin
__global__ void __launch_bounds__(1024)
sc_window_kernel(const uint64_t* __restrict__ pipe_off, uint32_t num_sensors,
                 const unsigned long long* __restrict__ minmax, const uint32_t* __restrict__ bins,
                 double exposure_time, double* __restrict__ start) {
    __shared__ uint64_t best[32];
    const uint64_t n = pipe_off[num_sensors];
    double mode = 0.0;
    if (n > 0) {
        const Edges e = make_edges(minmax, n);
        const uint32_t nb = e.count - 1;
        // (count << 32) | (~index): the max is the fullest, then the first
        uint64_t v = 0;
        for (uint32_t i = threadIdx.x; i < nb; i += blockDim.x) {
            const uint64_t c = ((uint64_t)bins[i] << 32) | (uint64_t)(0xffffffffu - i);
            if (bins[i] > 0 && c > v) v = c;
        }
        for (int o = 16; o > 0; o >>= 1) {
            const uint64_t w = __shfl_xor_sync(0xffffffffu, v, o);
            v = w > v ? w : v;
        }
        if ((threadIdx.x & 31) == 0) best[threadIdx.x >> 5] = v;
        __syncthreads();
        if (threadIdx.x < 32) {
            v = threadIdx.x < (blockDim.x >> 5) ? best[threadIdx.x] : 0;
            for (int o = 16; o > 0; o >>= 1) {
                const uint64_t w = __shfl_xor_sync(0xffffffffu, v, o);
                v = w > v ? w : v;
            }
        }
        const uint32_t arg = v ? 0xffffffffu - (uint32_t)v : 0u;
        mode = 0.5*(e.at(arg + 1) + e.at(arg));
    }
    if (threadIdx.x == 0) *start = mode - 0.5*exposure_time;
}

// ---- 3. background and conversion, one lixel per thread ----------------------------

// The electric pulses of lixel l: counted (kWrite false) or written at
// e_off[l].  A pulse of a Cherenkov photon is written as the photon's place
// in the pipelines (kFromPhoton in its lixel word; kOwnTruth in the place
// where the pulse has the photon's truth id, not the crosstalk's), and the
// extraction, one pulse per thread, looks its time and id up.
//
// Bound by latency: 13 warps per SM, each of some 2,500 instructions that
// follow one another, the longest chain as long as the brightest lixel's
// pipeline (80 photons of the measured event).  A step of the chain is
// therefore kept to what depends on the step before it: the efficiencies,
// the draws and the lengths of their crosstalk runs come from the gather,
// so that an accepted photon and its crosstalk are one step without a draw;
// a warp copies those of its 32 neighbouring pipelines -- one contiguous
// range -- into its part of the block's kPool photons of shared memory first
// (loaded by each lane for itself, some lane of the warp waits for L2 at
// nearly every step); the place of the next background photon is searched
// once instead of compared at every step.  What finds no room in the pool is
// read from global memory.  One block per SM, as its warps share the pool:
// with 32 lixels per block and fixed room for the brightest group, 4 warps
// per SM.  63,379 lixels, 6.2e5 photons, per pass (count, write): 115 + 118
// us with Philox, the table searches and the loads in the chain; 107 + 111
// without the first two; 49 + 67 with the copy and the runs; 39 + 54 with
// the shared pool.
constexpr int kLixelWarps = 16;
constexpr int kLixelThreads = 32*kLixelWarps;
constexpr int kNsbKeep = 2;
constexpr uint32_t kPool = 8192;
constexpr size_t kLixelSmem = kPool*(sizeof(double2) + sizeof(double) + sizeof(uchar2)) +
                              2*kNsbKeep*kLixelThreads*sizeof(double);
constexpr uint32_t kFromPhoton = 0x80000000u;
constexpr uint64_t kOwnTruth = 1ull << 63;

__device__ __forceinline__ void copy_async16(void* to, const void* from) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                 :: "r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from) : "memory");
}
__device__ __forceinline__ void copy_async8(void* to, const void* from) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;"
                 :: "r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from) : "memory");
}
__device__ __forceinline__ void copies_done() {
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// The first photon in [c, c_end) with t < time: the pipeline's photons before
// it come before a background photon at t (Injector.cpp:73-97).  The times
// ascend, except that what is not a number may end them; such a pipeline is
// looked through in order.  Eight probes are in flight at a time.
__device__ __forceinline__ uint64_t merge_place(const double* __restrict__ time, uint64_t c,
                                                uint64_t c_end, double t) {
    if (c == c_end) return c_end;
    const double last = __ldg(time + c_end - 1);
    if (last != last) {
        while (c < c_end && !(t < __ldg(time + c))) c++;
        return c;
    }
    if (!(t < last)) return c_end;
    // the answer is in [c, end]
    uint64_t end = c_end - 1;
    while (c < end) {
        const uint64_t part = (end - c + 8)/9;        // 8 probes, the last below end
        uint32_t below = 0;
        double probe[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint64_t j = c + (i + 1)*part - 1;
            probe[i] = j < end ? __ldg(time + j) : last;
        }
#pragma unroll
        for (int i = 0; i < 8; i++) below += !(t < probe[i]) ? 1u : 0u;
        const uint64_t above = c + (below + 1)*part - 1;
        c += below*part;
        end = below < 8 && above < end ? above : end;
    }
    return c;
}

template <bool kWrite>
__global__ void __launch_bounds__(kLixelThreads)
sc_lixel_kernel(SignalChainParams P, uint64_t seed, uint64_t offset,
                const uint64_t* __restrict__ pipe_off, const double* __restrict__ time,
                const double* __restrict__ efficacy, const double2* __restrict__ draws,
                const uchar2* __restrict__ runs, const float* __restrict__ efficiency,
                uint32_t num_sensors, const double* __restrict__ start,
                uint64_t* __restrict__ count, int32_t* __restrict__ nsb_count, const uint64_t* __restrict__ e_off,
                double* __restrict__ e_time, int32_t* __restrict__ e_truth,
                uint32_t* __restrict__ e_lixel, unsigned int* __restrict__ err) {
    extern __shared__ double2 pool_u[];
    double* const pool_q = reinterpret_cast<double*>(pool_u + kPool);
    double* const nsb_time = pool_q + kPool + threadIdx.x;            // one per thread and turn
    double* const nsb_q = nsb_time + kNsbKeep*kLixelThreads;
    uchar2* const pool_run =
        reinterpret_cast<uchar2*>(pool_q + kPool + 2*kNsbKeep*kLixelThreads);
    __shared__ uint32_t pool_used;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t groups = (num_sensors + 31)/32;
    const double S = *start;
    const double T = P.exposure_time;
    for (uint32_t round = 0; round*kLixelWarps*gridDim.x < groups; round++) {
        // neighbouring groups, bright or dark alike, go to different SMs
        const uint32_t g = (round*kLixelWarps + warp)*gridDim.x + blockIdx.x;
        __syncthreads();
        if (threadIdx.x == 0) pool_used = 0;
        __syncthreads();
        [&]() {
            if (g >= groups) return;
            const uint32_t l = 32*g + lane;
            const uint64_t base = pipe_off[32*g];
            uint32_t staged, at = 0;
            {
                const uint32_t next = 32*(g + 1);
            const uint64_t all = pipe_off[next < num_sensors ? next : num_sensors] - base;
                const uint32_t want = all < kPool ? (uint32_t)all : kPool;
                if (lane == 0) at = atomicAdd(&pool_used, want);
                at = __shfl_sync(0xffffffffu, at, 0);
                at = at < kPool ? at : kPool;
                staged = want < kPool - at ? want : kPool - at;
            }
            double2* const staged_u = pool_u + at;
            double* const staged_q = pool_q + at;
            uchar2* const staged_run = pool_run + at;
            for (uint32_t i = lane; i < staged; i += 32) {
                copy_async16(staged_u + i, draws + base + i);
                copy_async8(staged_q + i, efficacy + base + i);
                staged_run[i] = runs[base + i];
            }
            const bool live = l < num_sensors;
            const uint64_t s_nsb = stage_stream(1, offset, l);
            const uint64_t s_pec = stage_stream(2, offset, l);
            uint64_t c = live ? pipe_off[l] : 0;
            const uint64_t c_end = live ? pipe_off[l + 1] : 0;
            int e = 0;
            uint64_t out = kWrite && live ? e_off[l] : 0;
            uint32_t pulses = 0;
            auto pulse = [&](double t, int32_t id) {
                if (kWrite) {
                    e_time[out] = t;
                    e_truth[out] = id;
                    e_lixel[out] = l;
                    out++;
                }
                pulses++;
            };
            auto photon_pulse = [&](uint64_t place) {
                if (kWrite) {
                    e_time[out] = __longlong_as_double((long long)place);
                    e_truth[out] = kCrosstalk;
                    e_lixel[out] = l | kFromPhoton;
                    out++;
                }
                pulses++;
            };
            // draw k: staged, beyond the staged photons from the gather, beyond two
            // per photon of the pipeline from Philox
            const uint32_t num_drawn = 2u*(uint32_t)(c_end - c);
            const double* near = reinterpret_cast<const double*>(staged_u) + 2*(c - base);
            const unsigned char* near_run =
                reinterpret_cast<const unsigned char*>(staged_run) + 2*(c - base);
            const double* far = reinterpret_cast<const double*>(draws + c);
            const uint32_t num_near = c >= base + staged ? 0u
                                    : c_end <= base + staged ? num_drawn
                                                             : 2u*(uint32_t)(base + staged - c);
            auto draw = [&](uint32_t k) {
                return k < num_near ? near[k]
                     : k < num_drawn ? __ldg(far + k) : mlgpu_philox_uniform(seed, s_pec, k);
            };
            auto efficacy_of = [&](uint64_t j) {
                return j - base < staged ? staged_q[j - base] : __ldg(efficacy + j);
            };
            // background photons: the Poisson stream first (Injector.cpp:62-72)
            const double rate = live ? P.nsb_rate*(double)__ldg(efficiency + l)/P.num_lixel : 0.0;
            uint32_t nsb = 0;
            if (live) {
                double sum = expovariate(mlgpu_philox_uniform(seed, s_nsb, 0), rate);
                nsb_time[0] = sum;
                uint32_t kk = 1;
                while (sum < T) {
                    if (kk >= kMaxDraws) { e = MLGPU_ERR_RUNTIME; break; }
                    sum = sum + expovariate(mlgpu_philox_uniform(seed, s_nsb, kk), rate);
                    if (kk < kNsbKeep) nsb_time[kk*kLixelThreads] = sum;
                    kk++;
                    nsb++;
                }
            }
            if (!kWrite && live && nsb_count) nsb_count[l] = (int32_t)nsb;
            uint32_t kp = 0;           // conversion draws
            uint32_t m = 0, kept = 0;  // background photons: merged, with their efficiency kept
            // the efficiencies of the next background photons, and their times beyond
            // the first kNsbKeep (photon m is at S + nsb_time)
            auto keep_background = [&]() {
                const uint32_t first = kept;
                for (int i = 0; i < kNsbKeep && kept < nsb; i++, kept++) {
                    if (first) {
                        const int before = i ? i - 1 : kNsbKeep - 1;
                        nsb_time[i*kLixelThreads] =
                            nsb_time[before*kLixelThreads] +
                            expovariate(mlgpu_philox_uniform(seed, s_nsb, kept), rate);
                    }
                    const double u = mlgpu_philox_uniform(seed, s_nsb, nsb + 1 + kept);
                    // SamplesFromDistribution::draw
                    const double w =
                        fp64::func_eval_points(P.cdf, P.num_cdf, u*P.total_integral, &e);
                    nsb_q[i*kLixelThreads] = fp64::func_eval_points(P.qe, P.num_qe, w, &e);
                }
            };
            if (!e) keep_background();
            copies_done();
            __syncwarp();
            if (!live) return;
            // the pipeline merged with the background photons, in time order
            // (Injector.cpp:73-97, Cherenkov photons first on equal times), each
            // converted (PhotoElectricConverter.cpp:35-50)
            double tn = S + nsb_time[0], qn = nsb_q[0];
            int slot = 0;
            // the photon that the next background photon comes before
            uint64_t stop = m < nsb ? merge_place(time, c, c_end, tn) : c_end;
            while (!e && (c < c_end || m < nsb)) {
                // up to there: an accepted photon and its crosstalk in one step, by
                // the run from the draw after its own
                while (c < stop && kp + 2 <= num_near && c - base < staged) {
                    const uint32_t run = near_run[kp + 1];
                    if (run == kLongRun) break;
                    if (staged_q[c - base] >= near[kp]) {
                        if (kWrite) {
                            photon_pulse(c | kOwnTruth);
                            for (uint32_t i = 0; i < run; i++) photon_pulse(c);
                        } else {
                            pulses += 1 + run;
                        }
                        kp += 2 + run;
                    } else {
                        kp++;
                    }
                    c++;
                }
                if (c >= c_end && m >= nsb) break;
                const bool cherenkov = c < stop;
                const uint64_t place = c;
                const double t_rel = tn - S;
                double q = qn;
                if (cherenkov) {
                    q = efficacy_of(c);
                    c++;
                } else {
                    m++;
                    slot++;
                    if (m < nsb) {
                        if (m == kept) {
                            keep_background();
                            if (e) break;
                            slot = 0;
                        }
                        tn = S + nsb_time[slot*kLixelThreads];
                        qn = nsb_q[slot*kLixelThreads];
                        stop = merge_place(time, c, c_end, tn);
                    } else {
                        stop = c_end;
                    }
                }
                if (kp >= kMaxDraws) { e = MLGPU_ERR_RUNTIME; break; }
                if (q >= draw(kp++)) {
                    if (cherenkov) photon_pulse(place | kOwnTruth);
                    else pulse(t_rel, kNightSkyBackground);
                    // Converter::add_pulse: crosstalk while the draw allows it
                    while (kp < kMaxDraws && P.second_puls >= draw(kp++)) {
                        if (cherenkov) photon_pulse(place);
                        else pulse(t_rel, kCrosstalk);
                    }
                }
            }
            // dark pulses (PhotoElectricConverter.cpp:70-88)
            if (!e) {
                double sum = expovariate(draw(kp++), P.dark_rate);
                while (sum < T) {
                    if (kp >= kMaxDraws || pulses >= kMaxDraws/2) { e = MLGPU_ERR_RUNTIME; break; }
                    const double next = expovariate(draw(kp++), P.dark_rate);
                    pulse(sum, kAccidental);
                    while (kp < kMaxDraws && P.second_puls >= draw(kp++)) pulse(sum, kCrosstalk);
                    sum = sum + next;
                }
            }
            if (e) raise_error(err, e);
            if (!kWrite) {
                count[l] = e ? 0 : pulses;
                // one more, so that the scan gives the total
                if (l == 0) count[num_sensors] = 0;
            }
        }();
        __syncwarp();
    }
}

// ---- 4. extraction, one pulse per thread (pulse_extraction.cpp:17-30) ---------------

__global__ void __launch_bounds__(256)
sc_extract_kernel(SignalChainParams P, uint64_t seed, uint64_t offset,
                  const uint64_t* __restrict__ e_off, const double* __restrict__ e_time,
                  int32_t* __restrict__ e_truth, const uint32_t* __restrict__ e_lixel,
                  const double* __restrict__ time, const int32_t* __restrict__ truth,
                  const double* __restrict__ start, uint64_t num_pulses,
                  uint32_t num_sensors, uint8_t* __restrict__ slice,
                  uint32_t* __restrict__ keep) {
    const double S = *start;
    for (uint64_t p = blockIdx.x*(uint64_t)blockDim.x + threadIdx.x; p < num_pulses;
         p += (uint64_t)gridDim.x*blockDim.x) {
        const uint32_t word = e_lixel[p];
        const uint32_t l = word & ~kFromPhoton;
        if (l >= num_sensors) {            // not written: the writing pass stopped early
            slice[p] = 0;
            keep[p] = 0u;
            continue;
        }
        const uint32_t j = (uint32_t)(p - e_off[l]);
        const uint64_t st = stage_stream(3, offset, l);
        const double u1 = mlgpu_philox_uniform(seed, st, 2*j);
        const double u2 = mlgpu_philox_uniform(seed, st, 2*j + 1);
        const double z = 0.0 + P.arrival_time_std*(sqrt(-2.0*log(1.0 - u1))*cos(2.0*M_PI*u2));
        double t = e_time[p];
        if (word & kFromPhoton) {
            const uint64_t place = (uint64_t)__double_as_longlong(t);
            t = __ldg(time + (place & ~kOwnTruth)) - S;
            if (place & kOwnTruth) e_truth[p] = __ldg(truth + (place & ~kOwnTruth));
        }
        const double r = round((t + z)/P.time_slice_duration);
        const bool k = r >= 0.0 && r < kNumberTimeSlices;
        slice[p] = k ? (uint8_t)(int32_t)r : (uint8_t)0;
        keep[p] = k ? 1u : 0u;
    }
    // one more flag so that the scan also gives the total
    if (blockIdx.x == 0 && threadIdx.x == 0) keep[num_pulses] = 0u;
}

__global__ void __launch_bounds__(256)
sc_scatter_kernel(const uint8_t* __restrict__ slice, const int32_t* __restrict__ e_truth,
                  const uint32_t* __restrict__ keep, const uint64_t* __restrict__ pos,
                  uint64_t num_pulses, uint8_t* __restrict__ out_slice,
                  int32_t* __restrict__ out_truth) {
    for (uint64_t p = blockIdx.x*(uint64_t)blockDim.x + threadIdx.x; p < num_pulses;
         p += (uint64_t)gridDim.x*blockDim.x) {
        if (keep[p]) {
            const uint64_t q = pos[p];
            out_slice[q] = slice[p];
            out_truth[q] = e_truth[p];
        }
    }
}

// channel c's first kept pulse: the kept pulses before lixel c's first pulse
__global__ void __launch_bounds__(128)
sc_channel_offsets_kernel(const uint64_t* __restrict__ e_off, const uint64_t* __restrict__ pos,
                          uint32_t num_sensors, uint64_t* __restrict__ channel_offset) {
    const uint32_t s = blockIdx.x*blockDim.x + threadIdx.x;
    if (s <= num_sensors) channel_offset[s] = pos[e_off[s]];
}

// one block per SM; without 32 lixels for each, as many as there are
template <bool kWrite>
cudaError_t prepare_lixels(uint32_t num_sensors, int* blocks) {
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(sc_lixel_kernel<kWrite>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLixelSmem);
    const uint32_t groups = (num_sensors + 31)/32;
    *blocks = groups < (uint32_t)sms ? (int)groups : sms;
    return e;
}

// ---- scratch --------------------------------------------------------------------

inline uint64_t align256(uint64_t b) { return (b + 255) & ~uint64_t(255); }

struct PhotonScratch {
    uint32_t *rank, *idx_in, *idx_out;
    uint64_t* tkey_in;
    double *t, *q;                    // t holds the sorted time keys until the gather
    uchar2* run;
    double2* u;                       // over tkey_in, which the gather no longer needs
    int32_t* r;
    void* zeroed;                     // from runs to seg_counts
    size_t zeroed_bytes;
    uint32_t* runs;                   // photons per sensor
    uint64_t *pipe_off, *counts, *e_off;
    uint32_t* medium;                 // sensors with kWarpSegment < photons <= kBlockSegment
    uint64_t *large_begin, *large_end;
    uint64_t large_slots;             // at most n / (kBlockSegment + 1) longer runs
    uint32_t* bins;
    uint64_t nbins;
    unsigned long long* minmax;
    unsigned int* seg_counts;         // [0] medium, [1] large
    double* start;
    void* temp;
    size_t temp_bytes;
};

uint64_t large_slots_for(uint64_t n) { return n/(kBlockSegment + 1) + 1; }

PhotonScratch photon_layout(uint64_t n, uint32_t ns, void* scratch, size_t bytes) {
    PhotonScratch c;
    char* p = static_cast<char*>(scratch);
    const uint64_t a4 = align256(n*4), a8 = align256(n*8), as = align256((uint64_t)(ns + 2)*8);
    c.rank = reinterpret_cast<uint32_t*>(p);
    c.run = reinterpret_cast<uchar2*>(p); p += a4;      // the ranks are used up by then
    c.idx_in = reinterpret_cast<uint32_t*>(p); p += a4;
    c.idx_out = reinterpret_cast<uint32_t*>(p); p += a4;
    c.tkey_in = reinterpret_cast<uint64_t*>(p);
    c.u = reinterpret_cast<double2*>(p); p += 2*a8;
    c.t = reinterpret_cast<double*>(p); p += a8;
    c.q = reinterpret_cast<double*>(p); p += a8;
    c.r = reinterpret_cast<int32_t*>(p); p += a4;
    c.pipe_off = reinterpret_cast<uint64_t*>(p); p += as;
    c.counts = reinterpret_cast<uint64_t*>(p); p += as;
    c.e_off = reinterpret_cast<uint64_t*>(p); p += as;
    c.medium = reinterpret_cast<uint32_t*>(p); p += align256((uint64_t)(ns + 1)*4);
    c.zeroed = p;
    c.runs = reinterpret_cast<uint32_t*>(p); p += align256((uint64_t)(ns + 1)*4);
    c.large_slots = large_slots_for(n);
    c.large_begin = reinterpret_cast<uint64_t*>(p); p += align256(c.large_slots*8);
    c.large_end = reinterpret_cast<uint64_t*>(p); p += align256(c.large_slots*8);
    c.nbins = (uint64_t)(2.0 + sqrt((double)n)) + 1;
    c.bins = reinterpret_cast<uint32_t*>(p); p += align256(c.nbins*4);
    c.minmax = reinterpret_cast<unsigned long long*>(p);
    c.start = reinterpret_cast<double*>(p + 16);
    c.seg_counts = reinterpret_cast<unsigned int*>(p + 24);
    p += 256;
    c.zeroed_bytes = (size_t)(p - static_cast<char*>(c.zeroed));
    c.temp = p;
    c.temp_bytes = bytes - (size_t)(p - static_cast<char*>(scratch));
    return c;
}

struct PulseScratch {
    double* time;
    int32_t* truth;
    uint32_t *lixel, *keep;
    uint8_t* slice;
    uint64_t* pos;
    void* temp;
    size_t temp_bytes;
};

size_t pulse_temp_bytes(uint64_t np) { return exclusive_sum_temp_bytes(np + 1); }

PulseScratch pulse_layout(uint64_t np, void* scratch, size_t bytes) {
    PulseScratch c;
    char* p = static_cast<char*>(scratch);
    c.time = reinterpret_cast<double*>(p); p += align256(np*8);
    c.truth = reinterpret_cast<int32_t*>(p); p += align256(np*4);
    c.lixel = reinterpret_cast<uint32_t*>(p); p += align256(np*4);
    c.keep = reinterpret_cast<uint32_t*>(p); p += align256((np + 1)*4);
    c.slice = reinterpret_cast<uint8_t*>(p); p += align256(np);
    c.pos = reinterpret_cast<uint64_t*>(p); p += align256((np + 1)*8);
    c.temp = p;
    c.temp_bytes = bytes - (size_t)(p - static_cast<char*>(scratch));
    return c;
}

}  // namespace

size_t signal_chain_photon_scratch_bytes(uint64_t n, uint32_t ns) {
    const uint64_t a4 = align256(n*4), a8 = align256(n*8), as = align256((uint64_t)(ns + 2)*8);
    const uint64_t nbins = (uint64_t)(2.0 + sqrt((double)n)) + 1;
    return 4*a4 + 4*a8 + 3*as + 2*align256((uint64_t)(ns + 1)*4) +
           2*align256(large_slots_for(n)*8) + align256(nbins*4) + 256 +
           exclusive_sum_temp_bytes((uint64_t)ns + 1) + 256;
}

size_t signal_chain_pulse_scratch_bytes(uint64_t num_pulses) {
    const uint64_t np = num_pulses;
    return align256(np*8) + 2*align256(np*4) + align256((np + 1)*4) + align256(np) +
           align256((np + 1)*8) + pulse_temp_bytes(np) + 256;
}

// Steps 1-3a: pipelines, window, the conversion's counting pass and the scan
// of its counts.  *total_dev receives the electric pulses of the event,
// *start_dev the window start (both in the scratch).
cudaError_t launch_signal_chain_count(const SignalChainArgs& a, void* scratch, size_t bytes,
                                      int grid, cudaStream_t s, const uint64_t** total_dev,
                                      const double** start_dev) {
    const uint64_t n = a.num_photons;
    const uint32_t ns = a.num_sensors;
    if (n >= (1ull << 31) || ns >= (1u << 31)) return cudaErrorInvalidValue;
    const PhotonScratch c = photon_layout(n, ns, scratch, bytes);
    *total_dev = c.e_off + ns;
    *start_dev = c.start;
    cudaError_t e = cudaMemsetAsync(c.zeroed, 0, c.zeroed_bytes, s);
    if (e != cudaSuccess) return e;
    // 1. by sensor, then every sensor's run by (time, input index)
    if (n > 0)
        sc_rank_kernel<<<grid, 256, 0, s>>>(a.sensor, n, ns, c.runs, c.rank, c.minmax, a.err);
    e = exclusive_sum_u32(c.runs, c.pipe_off, (uint64_t)ns + 1, c.temp, s);
    if (e != cudaSuccess) return e;
    if (n > 0) {
        sc_place_kernel<<<grid, 256, 0, s>>>(a.sensor, a.time, n, ns, c.rank, c.pipe_off,
                                             c.tkey_in, c.idx_out);
        uint64_t* sorted = reinterpret_cast<uint64_t*>(c.t);
        if (ns > 0) {
            sc_segsort_warp_kernel<<<(ns + kSegWarps - 1)/kSegWarps, kSegWarps*32, 0, s>>>(
                c.tkey_in, c.idx_out, c.pipe_off, ns, sorted, c.idx_in, c.medium, c.seg_counts,
                c.large_begin, c.large_end, c.seg_counts + 1);
            if (n > kWarpSegment) {
                const uint64_t medium_max = n/(kWarpSegment + 1) + 1;
                const int blocks = (int)(medium_max < 296 ? medium_max : 296);
                sc_segsort_block_kernel<<<blocks, 512, kBlockSegment*12, s>>>(
                    c.tkey_in, c.idx_out, c.pipe_off, c.medium, c.seg_counts, sorted, c.idx_in);
            }
            if (n > kBlockSegment) {
                e = sort_long_runs(c.tkey_in, c.idx_out, sorted, c.idx_in, c.large_begin,
                                   c.large_end, (uint32_t)c.large_slots, s);
                if (e != cudaSuccess) return e;
            }
        }
        sc_gather_kernel<<<grid, 256, 0, s>>>(a.params, a.seed, a.offset, c.idx_in, a.sensor,
                                              a.wavelength, a.truth, c.pipe_off, ns, c.t, c.q,
                                              c.r, c.u, c.run, a.err);
    }
    // 2. the exposure window
    if (ns > 0)
        sc_minmax_kernel<<<(ns + 127)/128, 128, 0, s>>>(c.t, c.pipe_off, ns, c.minmax);
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int use_smem = c.nbins <= (uint64_t)kSmemBins;
    if (n > 0)
        sc_histogram_kernel<<<sms, kHistThreads, use_smem ? c.nbins*4 : 0, s>>>(c.t, c.pipe_off, ns,
                                                                        c.minmax, c.bins,
                                                                        use_smem);
    sc_window_kernel<<<1, 1024, 0, s>>>(c.pipe_off, ns, c.minmax, c.bins, a.params.exposure_time,
                                        c.start);
    // 3a. the counting pass and the scan of the counts
    if (ns == 0) {
        e = cudaMemsetAsync(c.counts, 0, 8, s);
        if (e != cudaSuccess) return e;
    } else {
        int blocks = 0;
        e = prepare_lixels<false>(ns, &blocks);
        if (e != cudaSuccess) return e;
        sc_lixel_kernel<false><<<blocks, kLixelThreads, kLixelSmem, s>>>(
            a.params, a.seed, a.offset, c.pipe_off, c.t, c.q, c.u, c.run, a.efficiency, ns, c.start,
            c.counts, a.nsb_count, nullptr, nullptr, nullptr, nullptr, a.err);
    }
    e = exclusive_sum_u64(c.counts, c.e_off, (uint64_t)ns + 1, c.temp, s);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

// Steps 3b-4 up to the scan of the keep flags: the electric pulses written,
// extracted, their kept positions and the channel offsets.  *kept_dev
// receives the number of kept pulses (in the pulse scratch).
cudaError_t launch_signal_chain_extract(const SignalChainArgs& a, void* scratch, size_t bytes,
                                        void* pulse_scratch, size_t pulse_bytes,
                                        uint64_t num_pulses, int grid, cudaStream_t s,
                                        const uint64_t** kept_dev) {
    const uint32_t ns = a.num_sensors;
    const PhotonScratch c = photon_layout(a.num_photons, ns, scratch, bytes);
    const PulseScratch q = pulse_layout(num_pulses, pulse_scratch, pulse_bytes);
    *kept_dev = q.pos + num_pulses;
    if (num_pulses > 0) {
        const cudaError_t e = cudaMemsetAsync(q.lixel, 0xff, num_pulses*4, s);
        if (e != cudaSuccess) return e;
    }
    if (ns > 0) {
        int blocks = 0;
        const cudaError_t e = prepare_lixels<true>(ns, &blocks);
        if (e != cudaSuccess) return e;
        sc_lixel_kernel<true><<<blocks, kLixelThreads, kLixelSmem, s>>>(
            a.params, a.seed, a.offset, c.pipe_off, c.t, c.q, c.u, c.run, a.efficiency, ns, c.start,
            nullptr, nullptr, c.e_off, q.time, q.truth, q.lixel, a.err);
    }
    sc_extract_kernel<<<grid, 256, 0, s>>>(a.params, a.seed, a.offset, c.e_off, q.time, q.truth,
                                           q.lixel, c.t, c.r, c.start, num_pulses, ns, q.slice, q.keep);
    cudaError_t e = exclusive_sum_u32(q.keep, q.pos, num_pulses + 1, q.temp, s);
    if (e != cudaSuccess) return e;
    sc_channel_offsets_kernel<<<(ns + 1 + 127)/128, 128, 0, s>>>(c.e_off, q.pos, ns,
                                                                 a.channel_offset);
    return cudaGetLastError();
}

// Step 4 end: the kept pulses into the caller's photon stream.
cudaError_t launch_signal_chain_scatter(const SignalChainArgs& a, void* pulse_scratch,
                                        size_t pulse_bytes, uint64_t num_pulses, int grid,
                                        cudaStream_t s) {
    const PulseScratch q = pulse_layout(num_pulses, pulse_scratch, pulse_bytes);
    if (num_pulses > 0)
        sc_scatter_kernel<<<grid, 256, 0, s>>>(q.slice, q.truth, q.keep, q.pos, num_pulses,
                                               a.slice, a.slice_truth);
    return cudaGetLastError();
}

}  // namespace mlgpu
