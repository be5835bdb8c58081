// corsika.cu -- CORSIKA photon bunches to photons on the device: merlict's
// EventIoPhotonFactory (merlict_corsika/PhotonFactory.cpp:8-136).
//
// A bunch is 8 floats: x, y on the observation level (cm), direction
// cosines u, v, relative arrival time (ns), production height (cm), weight
// (photons in the bunch, 0..16), wavelength (nm).  It becomes floor(weight)
// photons plus one more if a uniform draw is <= the weight's fraction
// (PhotonFactory.cpp:14-24), all with the same support and direction: the
// direction of motion (u, v, -sqrt(1 - u^2 - v^2)) (:113-118), the support
// the ground point moved up the ray by c t + 1 km (:31-62), the wavelength
// |lambda| 1e-9 (:128-130).  The arithmetic is merlict's, in the same
// order, compiled with --fmad=false, so the photons are bit-identical to
// the reference's given the same draws.
//
// Three passes: counts per bunch and their sums, a scan of the sums, the
// expansion (a block per 256 bunches, writing their photons as one
// contiguous run).
#include <cstdint>

#include "merlict_b200_philox.h"
#include "mlgpu_internal.h"

namespace mlgpu {
namespace {

constexpr int kScan = 1024;
constexpr int kTile = 256;                 // bunches of one expanding block
constexpr int kTilePhotons = kTile*17;     // at most 17 photons per bunch

struct Planes {
    double* p[7];
};

__device__ __forceinline__ void store4(double* to, double a, double b, double c, double d) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};"
                 :: "l"(to), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

__device__ __forceinline__ double bunch_uniform(const DevRng& r, uint64_t i) {
    if (r.mode == MLGPU_RNG_REPLAY) return __ldg(r.uniforms + i*(uint64_t)(r.stride ? r.stride : 1));
    return mlgpu_philox_uniform(r.seed, r.photon_offset + i, 0);
}

// One bunch per thread: its photons, those of the block's bunches, and
// where each tile of kTile bunches starts among them.  The expansion scans
// the counts of its own tile, so no offset per bunch is written or read:
// counting and scanning took 43 us of 316 for 2e6 bunches with one, 22
// without.
__global__ void __launch_bounds__(kScan)
corsika_count_kernel(const float* __restrict__ b, uint64_t n, DevRng rng,
                     uint8_t* __restrict__ count, uint32_t* __restrict__ tile_start,
                     uint64_t* __restrict__ sums, unsigned int* __restrict__ err) {
    __shared__ uint32_t warp_sum[kScan/32];
    const uint64_t i = blockIdx.x*(uint64_t)kScan + threadIdx.x;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t c = 0;
    if (i < n) {
        const double w = (double)__ldg(b + 8*i + 6);
        if (!(w >= 0.0 && w <= 16.0)) {
            // EventIoPhotonFactory::assert_bunch_weight throws
            atomicCAS(err, 0u, (unsigned)MLGPU_ERR_INVALID_ARGUMENT);
        } else {
            // fmod(w, 1): exact as a difference for weights from 0 to 16
            const double whole = floor(w);
            c = (uint32_t)whole;
            if (bunch_uniform(rng, i) <= w - whole) c += 1;
        }
        count[i] = (uint8_t)c;
    }
    const uint32_t sum = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) warp_sum[wid] = sum;
    __syncthreads();
    if (wid == 0) {
        const uint32_t v = warp_sum[lane];
        uint32_t x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane % (kTile/32) == 0)
            tile_start[blockIdx.x*(uint64_t)(kScan/kTile) + lane/(kTile/32)] = x - v;
        if (lane == 31) sums[blockIdx.x] = x;
    }
}

// Exclusive scan of up to kScan * kScan block sums in one block (serial
// over chunks of kScan).
__global__ void __launch_bounds__(kScan)
scan_sums_kernel(uint64_t* __restrict__ sums, uint64_t blocks, uint64_t* __restrict__ total) {
    __shared__ uint64_t warp_sum[kScan/32];
    __shared__ uint64_t carry;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (uint64_t base = 0; base < blocks; base += kScan) {
        const uint64_t i = base + threadIdx.x;
        const uint64_t v = i < blocks ? sums[i] : 0;
        uint64_t x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sum[wid] = x;
        __syncthreads();
        if (wid == 0) {
            uint64_t s = warp_sum[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const uint64_t y = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o) s += y;
            }
            warp_sum[lane] = s;
        }
        __syncthreads();
        const uint64_t before = (wid > 0 ? warp_sum[wid - 1] : 0) + carry;
        if (i < blocks) sums[i] = before + x - v;
        __syncthreads();
        if (threadIdx.x == kScan - 1) carry = before + x;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

// The expansion, a block per tile of kTile consecutive bunches: each thread
// computes its bunch's photon (merlict's arithmetic) into shared memory and
// marks the photons it owns in an owner list, then the block writes the
// tile's photons as one contiguous run per plane.  Bound by the writes, 60
// bytes a photon: a thread writes four photons of a plane at once, on a
// 32-byte boundary, so that all but the ends of a run are whole sectors.
// With 8 bytes per thread from wherever a run of 32 bunches began, every
// store of a warp split two sectors with its neighbours: 252 us for the
// 1.6e7 photons of 2e6 bunches, 163 now (6.3 TB/s with the bunches read; a
// fill of the same size reaches 7.5).  Planes that do not lie alike on 32 bytes (the ids on
// 16) are written photon by photon.
__global__ void __launch_bounds__(kTile)
corsika_expand_kernel(const float* __restrict__ b, uint64_t n, const uint8_t* __restrict__ count,
                      const uint32_t* __restrict__ tile_start, const uint64_t* __restrict__ sums,
                      const int32_t* __restrict__ ids, Planes out, int32_t* __restrict__ out_id) {
    __shared__ double s_val[7][kTile];
    __shared__ int32_t s_id[kTile];
    __shared__ uint8_t s_owner[kTilePhotons];
    __shared__ uint32_t warp_sum[kTile/32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t i = blockIdx.x*(uint64_t)kTile + threadIdx.x;
    const uint32_t c = i < n ? count[i] : 0u;
    uint32_t incl = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += y;
    }
    if (lane == 31) warp_sum[warp] = incl;
    // the tile's first photon
    const uint64_t o0 = sums[blockIdx.x/(kScan/kTile)] + tile_start[blockIdx.x];
    if (c != 0) {
        const float* r = b + 8*i;
        // direction_of_motion, PhotonFactory.cpp:113-118
        const double u = (double)__ldg(r + 2), v = (double)__ldg(r + 3);
        const double z = sqrt(1.0 - u*u - v*v);
        const double cx = u, cy = v, cz = -z;
        // Ray(ground point, -direction): direction normalised (Ray.cpp:16-20)
        const double ux = cx*-1.0, uy = cy*-1.0, uz = cz*-1.0;
        const double un = sqrt(ux*ux + uy*uy + uz*uz);
        const double nx = ux/un, ny = uy/un, nz = uz/un;
        // ray_parameter_for_production_point, PhotonFactory.cpp:58-62
        const double t = (double)__ldg(r + 4)*1e-9;
        const double par = t*299792458.0 + 1e3;
        const double gx = (double)__ldg(r + 0)*1e-2, gy = (double)__ldg(r + 1)*1e-2, gz = 0.0;
        s_val[0][threadIdx.x] = gx + nx*par;
        s_val[1][threadIdx.x] = gy + ny*par;
        s_val[2][threadIdx.x] = gz + nz*par;
        s_val[3][threadIdx.x] = cx;
        s_val[4][threadIdx.x] = cy;
        s_val[5][threadIdx.x] = cz;
        s_val[6][threadIdx.x] = fabs((double)__ldg(r + 7)*1e-9);
        s_id[threadIdx.x] = ids ? __ldg(ids + i) : (int32_t)i;
    }
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kTile/32; w++) {
        const uint32_t t = warp_sum[w];
        if (w < warp) before += t;
        total += t;
    }
    for (uint32_t k = before + incl - c; k < before + incl; k++)
        s_owner[k] = (uint8_t)threadIdx.x;
    __syncthreads();
    uint32_t phase = (uint32_t)(reinterpret_cast<uintptr_t>(out.p[0]) >> 3) & 3u;
    bool alike = true;
#pragma unroll
    for (int k = 1; k < 7; k++)
        alike = alike && ((uint32_t)(reinterpret_cast<uintptr_t>(out.p[k]) >> 3) & 3u) == phase;
    if (out_id)
        alike = alike && ((uint32_t)(reinterpret_cast<uintptr_t>(out_id) >> 2) & 3u) == phase;
    if (!alike) {
        for (uint32_t ph = threadIdx.x; ph < total; ph += kTile) {
            const uint32_t w = s_owner[ph];
#pragma unroll
            for (int k = 0; k < 7; k++) out.p[k][o0 + ph] = s_val[k][w];
            if (out_id) out_id[o0 + ph] = s_id[w];
        }
        return;
    }
    // photon `first` (of the tile; up to 3 before it) begins a 32-byte word
    const int64_t first = -(int64_t)((phase + (uint32_t)o0) & 3u);
    for (int64_t ph = first + 4*(int64_t)threadIdx.x; ph < (int64_t)total; ph += 4*kTile) {
        if (ph >= 0 && ph + 4 <= (int64_t)total) {
            uint32_t w[4];
#pragma unroll
            for (int j = 0; j < 4; j++) w[j] = s_owner[ph + j];
#pragma unroll
            for (int k = 0; k < 7; k++)
                store4(out.p[k] + o0 + ph, s_val[k][w[0]], s_val[k][w[1]], s_val[k][w[2]],
                       s_val[k][w[3]]);
            if (out_id)
                *reinterpret_cast<int4*>(out_id + o0 + ph) =
                    make_int4(s_id[w[0]], s_id[w[1]], s_id[w[2]], s_id[w[3]]);
        } else {
            for (int64_t q = ph < 0 ? 0 : ph; q < ph + 4 && q < (int64_t)total; q++) {
                const uint32_t w = s_owner[q];
#pragma unroll
                for (int k = 0; k < 7; k++) out.p[k][o0 + q] = s_val[k][w];
                if (out_id) out_id[o0 + q] = s_id[w];
            }
        }
    }
}

// the tiles' starts (32-bit), the blocks' sums, the bunches' counts (8-bit)
struct Scratch {
    uint32_t* tile_start;
    uint64_t* sums;
    uint8_t* count;
    uint64_t blocks;
    size_t bytes;
};

Scratch scratch_layout(uint64_t n, void* scratch) {
    Scratch l;
    l.blocks = (n + kScan - 1)/kScan;
    const uint64_t starts = (l.blocks*(kScan/kTile)*4 + 255) & ~uint64_t(255);
    const uint64_t sums = (l.blocks*8 + 255) & ~uint64_t(255);
    char* p = static_cast<char*>(scratch);
    l.tile_start = reinterpret_cast<uint32_t*>(p);
    l.sums = reinterpret_cast<uint64_t*>(p + starts);
    l.count = reinterpret_cast<uint8_t*>(p + starts + sums);
    l.bytes = starts + sums + ((n + 255) & ~uint64_t(255));
    return l;
}

}  // namespace

size_t corsika_scratch_bytes(uint64_t n) { return scratch_layout(n, nullptr).bytes; }

cudaError_t launch_corsika_count(const float* bunches, uint64_t n, const DevRng& rng, void* scratch,
                                 uint64_t* total_dev, unsigned int* err, cudaStream_t s) {
    const Scratch l = scratch_layout(n, scratch);
    if (l.blocks > (uint64_t)kScan*kScan*64) return cudaErrorInvalidValue;
    corsika_count_kernel<<<(unsigned)l.blocks, kScan, 0, s>>>(bunches, n, rng, l.count,
                                                              l.tile_start, l.sums, err);
    scan_sums_kernel<<<1, kScan, 0, s>>>(l.sums, l.blocks, total_dev);
    return cudaGetLastError();
}

cudaError_t launch_corsika_expand(const float* bunches, uint64_t n, const int32_t* ids,
                                  void* scratch, double* const* planes, int32_t* out_id,
                                  cudaStream_t s) {
    const Scratch l = scratch_layout(n, scratch);
    Planes out;
    for (int k = 0; k < 7; k++) out.p[k] = planes[k];
    corsika_expand_kernel<<<(unsigned)((n + kTile - 1)/kTile), kTile, 0, s>>>(
        bunches, n, l.count, l.tile_start, l.sums, ids, out, out_id);
    return cudaGetLastError();
}

}  // namespace mlgpu
