// wave_resolve.cuh -- the kernels of the wavefront tracers, shared by the
// FP64 and FP32 forms.  With the closest-hit walk (the default):
//   hit        new photons and the pool's rays: the closest hit of each by
//              the walk of closest_hit.cuh;
//   resolve    one thread per ray: the winner's point and normal (FP64: at
//              the distance the walk found; the single-precision forms solve
//              the winner again with its point refined), the interaction with
//              the surface (merlict/PhotonAndFrame.cpp:13-124), the history
//              entry and the time-of-flight term; survivors are compacted into
//              the next pool with a warp ballot and one atomic per warp,
//              finished photons write their results;
//   first      FP64: ends a large batch's photons that miss the scenery and
//              lists the others;
//   finish     FP64: photons from where they are to their ends in one launch.
// With the level kernels (wavefront_fp64.cu), which propose candidate leaves:
//   intersect  one thread per (ray, candidate leaf): the distance to the
//              leaf's hit; the smallest distance of each ray is kept with a
//              64-bit atomic minimum on its bits (positive doubles order like
//              their bit patterns);
//   ties       one thread per candidate: among the candidates at exactly that
//              distance the lowest leaf index wins, which is the leaf merlict
//              visits first (RayAndFrame.cpp:160-173);
//   overflow   rays whose walk overflowed a queue get merlict's own walk of
//              the frame tree;
//   resolve    as above.
//
// kIsect selects the intersection arithmetic: FP64 (merlict's, bit-identical
// when the translation unit is compiled with --fmad=false), or the FP32
// intersections of fp32_geometry.cuh (with or without the FP64 Newton step).
// The interaction, positions and time of flight are FP64 in every form.
#ifndef MLGPU_WAVE_RESOLVE_CUH_
#define MLGPU_WAVE_RESOLVE_CUH_

#include <climits>
#include <cstdint>

#include "closest_hit.cuh"
#include "merlict_b200_philox.h"

namespace mlgpu {
namespace {

using namespace fp64;

constexpr int kNoStep = -2;             // step state: the photon takes no step
constexpr int kStepNone = 0;            // it takes a step; nothing to queue (no candidates)
constexpr int kStepBvh = 1;             // it takes a step; the intake queues the BVH root
constexpr int kStepTree = 2;            // it takes a step; the intake walks its frame subtree

template <typename T>
__device__ __forceinline__ double load_in(const void* p, uint64_t i) {
    return (double)__ldg(static_cast<const T*>(p) + i);
}

__device__ __forceinline__ void store_hist(mlgpu_history_entry* h, v3 pos, v3 nrm, double dist,
                                           int32_t leaf, int kind, bool outside) {
    h->position[0] = pos.x; h->position[1] = pos.y; h->position[2] = pos.z;
    h->normal[0] = nrm.x; h->normal[1] = nrm.y; h->normal[2] = nrm.z;
    h->distance = dist;
    h->leaf = leaf;
    h->interaction = (uint8_t)kind;
    h->from_outside_to_inside = (uint8_t)outside;
    h->pad[0] = 0; h->pad[1] = 0;
}

// Reserves n consecutive entries of a queue for every lane of the (full,
// converged) warp with one atomic; returns this lane's first index.
__device__ __forceinline__ uint32_t warp_reserve(unsigned int* counter, uint32_t n) {
    const int lane = threadIdx.x & 31;
    uint32_t x = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    const uint32_t sum = __shfl_sync(kFull, x, 31);
    uint32_t base = 0;
    if (lane == 31 && sum) base = atomicAdd(counter, sum);
    base = __shfl_sync(kFull, base, 31);
    return base + x - n;
}

// Sends a slot to merlict's own walk (once per iteration).
__device__ __forceinline__ void mark_overflow(const WaveBuffers& w, const RayPool& cur,
                                              uint32_t slot) {
    uint32_t* flag = cur.overflow_flag;
    if (atomicExch(flag + slot, 1u) == 0u)
        w.overflow[atomicAdd(&w.counters->overflow_len, 1u)] = slot;
}

// The first index of this warp in a grid-stride loop whose trip count is
// the same for every lane of a warp (so that warp_reserve sees full warps).
__device__ __forceinline__ uint32_t warp_first() {
    return blockIdx.x*blockDim.x + (threadIdx.x & ~31u);
}

// The FP64 ray of a slot from its 48-byte record.
__device__ __forceinline__ void load_ray(const RayPool& p, uint32_t slot, v3* s, v3* d) {
    const double2 a = p.sd[3*slot], b = p.sd[3*slot + 1], c = p.sd[3*slot + 2];
    *s = mk(a.x, a.y, b.x);
    *d = mk(b.y, c.x, c.y);
}

__device__ __forceinline__ void store_ray(const RayPool& p, uint32_t slot, v3 s, v3 d) {
    p.sd[3*slot] = make_double2(s.x, s.y);
    p.sd[3*slot + 1] = make_double2(s.z, d.x);
    p.sd[3*slot + 2] = make_double2(d.y, d.z);
}

// The box inflation of a ray's FP32 slab tests: its rounding to FP32.
__device__ __forceinline__ float box_inflation(const DevScene& sc, float ox, float oy, float oz) {
    return sc.bvh_eps + 4e-7f*(fabsf(ox) + fabsf(oy) + fabsf(oz));
}

// How a ray about to take a step from s along d in the frame subtree `root`
// finds its hit: inside a lens (root != 0), or without a BVH, by merlict's
// own walk of the subtree (kStepTree); else merlict tests the root frame's
// sphere first (RayAndFrame.cpp:137-149) and the BVH walk follows if the ray
// passes it.
__device__ __forceinline__ int step_kind(const TraceArgs& a, const WaveBuffers& w, v3 s, v3 d,
                                         int32_t root) {
    const DevScene& sc = a.scene;
    if (root != 0 || (w.walk == MLGPU_WALK_LEVELS ? sc.bvh_nodes : sc.surf_levels) == 0 ||
        a.traversal == MLGPU_TRAVERSAL_FRAME_TREE)
        return kStepTree;
    const double2* np = reinterpret_cast<const double2*>(sc.node);
    const double2 n01 = __ldg(np), n23 = __ldg(np + 1);
    return sphere_cull(make_double4(n01.x, n01.y, n23.x, n23.y), s, d, dot(s, d)) ? kStepBvh
                                                                                 : kStepNone;
}

// The new photons of an iteration, which fill the pool's free slots; a fed
// propagation admits only those whose records have arrived.
__device__ __forceinline__ uint32_t new_photons(const TraceArgs& a, const WaveBuffers& w) {
    const unsigned long long limit = a.fed ? w.counters->avail_snap : a.num_photons;
    const unsigned long long remaining = limit - w.counters->next_input;
    const uint32_t room = w.pool - w.counters->active - w.counters->inside;
    return (uint32_t)(remaining < room ? remaining : room);
}

// What the level kernels keep of a ray in slot `slot`: its cleared closest
// hit and, for a BVH walk, its FP32 walk record.
__device__ __forceinline__ void prepare_levels(const DevScene& sc, const RayPool& p, uint32_t slot,
                                               v3 s, v3 d, int step) {
    p.best_key[slot] = kNoKey;
    p.best_leaf[slot] = kNoLeaf;
    p.overflow_flag[slot] = 0u;
    if (step != kStepBvh) return;
    const float ox = (float)s.x, oy = (float)s.y, oz = (float)s.z;
    float fdx = (float)d.x, fdy = (float)d.y, fdz = (float)d.z;
    if (fabsf(fdx) < kMinDirection) fdx = copysignf(kMinDirection, fdx);
    if (fabsf(fdy) < kMinDirection) fdy = copysignf(kMinDirection, fdy);
    if (fabsf(fdz) < kMinDirection) fdz = copysignf(kMinDirection, fdz);
    p.ray_o[slot] = make_float4(ox, oy, oz, box_inflation(sc, ox, oy, oz));
    p.ray_i[slot] = make_float4(1.0f/fdx, 1.0f/fdy, 1.0f/fdz, 0.0f);
}

// A photon between interactions (a merlict Photon: its ray, what its history
// adds up to, its random stream).
struct PhotonRay {
    v3 s, d;
    double lambda, tof;
    int32_t photon, root, n_int, k_draw;
    int32_t err;             // error | time-of-flight error << 8
};

__device__ __forceinline__ void load_photon(const RayPool& cur, uint32_t slot, PhotonRay* q) {
    load_ray(cur, slot, &q->s, &q->d);
    q->photon = cur.photon[slot];
    q->lambda = cur.lambda[slot];
    q->tof = cur.tof[slot];
    q->root = cur.root[slot];
    q->n_int = cur.n_int[slot];
    q->k_draw = cur.k_draw[slot];
    q->err = cur.err[slot];
}

// Photon q of the batch's tracing order as it sets out (merlict::Photon's
// constructor, Ray.cpp:16-20, RayForPropagation.cpp:52-64).  Returns its step.
template <typename In>
__device__ __forceinline__ int start_photon(const TraceArgs& a, const WaveBuffers& w, uint64_t q,
                                            PhotonRay* out) {
    const uint32_t max_int = a.max_interactions;
    uint64_t p;
    if (a.sorted) {
        // the photon's record in tracing order
        const double2* r = a.sorted + 4*q;
        const double2 r0 = __ldcg(r), r1 = __ldcg(r + 1), r2 = __ldcg(r + 2), r3 = __ldcg(r + 3);
        out->s = mk(r0.x, r0.y, r1.x);
        out->d = normalized_rn(mk(r1.y, r2.x, r2.y));
        out->lambda = r3.x;
        p = (uint64_t)__double_as_longlong(r3.y);
    } else {
        p = a.order ? (uint64_t)__ldg(a.order + q) : q;
        out->s = mk(load_in<In>(a.photons.sx, p), load_in<In>(a.photons.sy, p),
                    load_in<In>(a.photons.sz, p));
        out->d = normalized_rn(mk(load_in<In>(a.photons.dx, p), load_in<In>(a.photons.dy, p),
                                  load_in<In>(a.photons.dz, p)));
        out->lambda = load_in<In>(a.photons.wavelength, p);
    }
    out->photon = (int32_t)p;
    // Photon::assert_wavelength_is_positive (Photon.cpp:20-28): merlict
    // throws std::invalid_argument before propagating
    if (out->lambda <= 0.0) raise_error(a.scene.error_word, MLGPU_ERR_INVALID_ARGUMENT);
    out->tof = 0.0;
    out->root = a.start_node;
    out->n_int = 1;
    out->k_draw = 0;
    out->err = 0;
    if (a.results.history)
        store_hist(a.results.history + p*(max_int + 1), out->s, out->d, 0.0,
                   MLGPU_LEAF_PHOTON_SOURCE, MLGPU_PRODUCTION, dot(out->d, out->d) < 0.0);
    return 1u > max_int ? kNoStep : step_kind(a, w, out->s, out->d, out->root);
}

__device__ __forceinline__ void store_photon(const RayPool& p, uint32_t slot, const PhotonRay& q,
                                             int step) {
    p.photon[slot] = q.photon;
    store_ray(p, slot, q.s, q.d);
    p.lambda[slot] = q.lambda;
    p.tof[slot] = q.tof;
    p.root[slot] = q.root;
    p.n_int[slot] = q.n_int;
    p.k_draw[slot] = q.k_draw;
    p.err[slot] = q.err;
    p.step[slot] = step;
}

// The same into slot `slot` of the pool, prepared like the survivors the
// previous resolve step prepared.
template <typename In>
__device__ __forceinline__ int admit_photon(const TraceArgs& a, const WaveBuffers& w,
                                            const RayPool& cur, uint32_t slot, uint64_t q,
                                            v3* support, v3* direction) {
    PhotonRay ray;
    const int step = start_photon<In>(a, w, q, &ray);
    if (w.walk == MLGPU_WALK_LEVELS) prepare_levels(a.scene, cur, slot, ray.s, ray.d, step);
    store_photon(cur, slot, ray, step);
    *support = ray.s;
    *direction = ray.d;
    return step;
}

// Intake and closest hit in one kernel: new photons enter the free slots,
// and every ray that takes a step finds its closest hit (closest_hit.cuh)
// for the resolve step.  The grid's warps take the pool's slots in chunks of
// 32; a lane whose ray has been walked takes the next slot once kRefill
// lanes are free, so that a warp's lanes stay busy although rays visit
// different numbers of nodes.
constexpr int kRefill = 16;

template <typename In, int kIsect>
__global__ void __launch_bounds__(kWalkThreads, kWalkBlocks)
wave_hit_kernel(const TraceArgs a, const WaveBuffers w, const RayPool cur) {
    extern __shared__ double2 s_walk[];
    const DevScene& sc = a.scene;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kWarps = kWalkThreads/32;
    WalkWarp* sw = reinterpret_cast<WalkWarp*>(s_walk) + warp;
    uint32_t* stack = reinterpret_cast<uint32_t*>(reinterpret_cast<WalkWarp*>(s_walk) + kWarps) +
        threadIdx.x;
    const uint32_t active = w.counters->active;
    const unsigned long long next_input = w.counters->next_input;
    const uint32_t total = active + new_photons(a, w);
    const uint32_t chunks = (total + 31)/32;
    uint32_t chunk = blockIdx.x*kWarps + warp;   // then the next that no warp has
    int taken = 0;               // slots of this chunk given out
    WalkLane l;
    l.walking = false;
    l.eps = 0.0f;
    l.key = kNoKey;
    uint32_t slot = 0;
    bool have = false;           // the lane holds a ray whose hit is not written yet
    uint32_t listed = 0;         // lengths of the lists
    int groups = 0;
    while (true) {
        const unsigned idle = __ballot_sync(kFull, !l.walking);
        const int free_lanes = __popc(idle);
        const bool refill = free_lanes == 32 || (free_lanes >= kRefill && chunk < chunks);
        intersect_queued<kIsect>(sc, sw, lane, refill, &groups, &listed, &l);
        if (refill) {
            const bool is_free = (idle >> lane) & 1u;
            if (is_free && have) {
                cur.best_leaf[slot] = sw->leaf[lane];
                cur.best_key[slot] = sw->key[lane];
                have = false;
            }
            if (chunk >= chunks) break;   // all lanes are free and no slots are left
            const int rank = __popc(idle & ((1u << lane) - 1u));
            const int take = min(free_lanes, 32 - taken);
            const uint32_t next = chunk*32u + (uint32_t)(taken + rank);
            if (is_free && rank < take && next < total) {
                slot = next;
                v3 s, d;
                int step;
                if (slot >= active) {
                    step = admit_photon<In>(a, w, cur, slot, next_input + (slot - active), &s, &d);
                } else {
                    step = cur.step[slot];
                    load_ray(cur, slot, &s, &d);
                }
                if (step == kStepBvh) {
                    walk_begin(sc, s, d, sw, lane, &l);
                    have = true;
                } else {
                    cur.best_leaf[slot] = kNoLeaf;
                }
            }
            taken += take;
            if (taken == 32) {
                if (lane == 0) chunk = gridDim.x*kWarps + atomicAdd(&w.counters->chunks, 1u);
                chunk = __shfl_sync(kFull, chunk, 0);
                taken = 0;
            }
            __syncwarp();
        }
#pragma unroll 1
        for (int k = 0; k < kVisits; k++)
            groups = visit_nodes(sc, sw, stack, lane, groups, &l);
    }
}

template <int kIsect>
__global__ void __launch_bounds__(256)
wave_isect_kernel(const TraceArgs a, const WaveBuffers w, const RayPool cur) {
    const DevScene& sc = a.scene;
    const uint32_t n = w.counters->isect_len < w.isect_cap ? w.counters->isect_len : w.isect_cap;
    for (uint32_t e = blockIdx.x*blockDim.x + threadIdx.x; e < n; e += gridDim.x*blockDim.x) {
        const uint2 q = w.isect_q[e];
        const uint32_t slot = q.x;
        v3 s, d;
        load_ray(cur, slot, &s, &d);
        double dist = -1.0;
        if (kIsect == kIsectFp64) {
            double T[12], ti[3], pr[MLGPU_LEAF_PARAMS], r2;
            int32_t prim;
            load_leaf_slot(sc, q.y, T, ti, pr, &r2, &prim);
            // merlict's bounding-sphere test of the leaf (RayAndFrame.cpp:
            // 16-107; the sphere is centred on the frame's position,
            // Frame::position_in_world): the walk proposed the leaf with a
            // conservative single-precision version of it
            if (sphere_cull(make_double4(T[3], T[7], T[11], r2), s, d, dot(s, d))) {
                Isec h;
                intersect_leaf<-1>(sc, (int32_t)q.y, prim, pr, r2, position_inverse(T, ti, s),
                               orientation_inverse(T, d), &h);
                if (h.leaf >= 0) dist = h.dist;
            }
        } else {
            // by slot: the FP32 records in slot order, like the FP64 ones
            const fp32::Hit32 h = fp32::intersect32<false, true>(
                sc, (int32_t)q.y, fp32::dmk(s.x, s.y, s.z), fp32::dmk(d.x, d.y, d.z),
                kIsect == kIsectFp32Pure);
            if (h.leaf >= 0) dist = h.v;
        }
        w.isect_dist[e] = dist;
        if (dist >= 0.0) atomicMin(&cur.best_key[slot], (unsigned long long)__double_as_longlong(dist));
    }
}

__global__ void __launch_bounds__(256)
wave_tie_kernel(const WaveBuffers w, const RayPool cur) {
    const uint32_t n = w.counters->isect_len < w.isect_cap ? w.counters->isect_len : w.isect_cap;
    for (uint32_t e = blockIdx.x*blockDim.x + threadIdx.x; e < n; e += gridDim.x*blockDim.x) {
        const double dist = w.isect_dist[e];
        if (!(dist >= 0.0)) continue;
        const uint2 q = w.isect_q[e];
        if ((unsigned long long)__double_as_longlong(dist) == cur.best_key[q.x])
            atomicMin(&cur.best_leaf[q.x], __ldg(w.slot_leaf_of + q.y));
    }
}

// Rays whose walk overflowed a queue: merlict's own walk of the frame tree
// (FP64, in merlict's order) finds the closest hit.
__global__ void __launch_bounds__(128)
wave_overflow_kernel(const TraceArgs a, const WaveBuffers w, const RayPool cur) {
    const uint32_t n = w.counters->overflow_len;
    for (uint32_t e = blockIdx.x*blockDim.x + threadIdx.x; e < n; e += gridDim.x*blockDim.x) {
        const uint32_t slot = w.overflow[e];
        v3 s, d;
        load_ray(cur, slot, &s, &d);
        const Isec is = first_intersection_tree(a.scene, cur.root[slot], s, d);
        cur.best_leaf[slot] = is.leaf >= 0 ? is.leaf : kNoLeaf;
        cur.best_key[slot] = (unsigned long long)__double_as_longlong(is.dist);
    }
}

// The photon's step to the hit found for it, `best` (kNoLeaf: none) at
// best_dist: the intersection, the interaction with the surface
// (merlict/PhotonAndFrame.cpp:13-124), the history entry and the
// time-of-flight term.  Returns true if the photon goes on, then with its
// new ray; else its results are written.  `before` reads the ray before the
// step again where the results ask for it.
template <typename Out, int kIsect, typename Before>
__device__ __forceinline__ bool resolve_photon(const TraceArgs& a, const double* fn_pts,
                                               const int32_t* fn_off, int step, int32_t best,
                                               double best_dist, PhotonRay* q, Before before) {
    const DevScene& sc = a.scene;
    const uint32_t max_int = a.max_interactions;
    const uint32_t hist_len = max_int + 1;
    v3& s = q->s;
    v3& d = q->d;
    const double lambda = q->lambda;
    double& tof = q->tof;
    int32_t& root = q->root;
    int32_t& k_draw = q->k_draw;
    const int32_t photon = q->photon, n_int = q->n_int;
    int err = q->err & 0xff;
    int tof_error = (q->err >> 8) & 0xff;
    const uint64_t stream = a.rng.photon_offset + (uint64_t)photon;
    mlgpu_history_entry* hist =
        a.results.history ? a.results.history + (uint64_t)photon*hist_len : nullptr;

    Isec is;
    int kind = MLGPU_PRODUCTION;
    bool moved = false;      // then s and d are the photon's new ray
    double T[12];
    if (step == kNoStep) {
        is.leaf = MLGPU_LEAF_PHOTON_SOURCE;
        is.pos = s; is.normal = d; is.dist = 0.0; is.outside = dot(d, d) < 0.0;
#pragma unroll
        for (int k = 0; k < 12; k++) T[k] = IDENTITY[k];
    } else {
        // merlict's closest hit among the candidates: minimum distance,
        // ties to merlict's visiting order (RayAndFrame.cpp:160-173)
        {
            // the winner of the search at its distance; the FP32 forms
            // intersect it again with the hit point refined
            if (best == kNoLeaf) {
                set_void(&is, s, d);
            } else if (kIsect == kIsectFp64) {
                hit_at(sc, best, best_dist, s, d, T, &is);
            } else {
                const fp32::Hit32 h = fp32::intersect32<true>(sc, best, fp32::dmk(s.x, s.y, s.z),
                                                        fp32::dmk(d.x, d.y, d.z),
                                                        kIsect == kIsectFp32Pure);
                if (h.leaf < 0) {
                    set_void(&is, s, d);
                } else {
                    is.leaf = h.leaf;
                    is.pos = mk(h.p.x, h.p.y, h.p.z);
                    is.normal = mk(h.n.x, h.n.y, h.n.z);
                    is.dist = h.v;
                    is.outside = h.outside;
                }
            }
        }
        const bool hit = is.leaf >= 0;
        const LeafRec* L = hit ? sc.leaf + is.leaf : nullptr;
        // a property table of the surface, by the side the ray comes from.
        // FP64 reads an id where it needs it: the six ids held in registers
        // made 1e7 telescope photons 17.2 ms instead of 16.7.  The
        // single-precision forms, whose hit is solved again above, wait for
        // each id in turn, and have them read at once: 1e6 photons among all
        // primitives spend 379 us here instead of 558 (pure: 350, 522), 8e6 of
        // the large reflector take 4.85 ms instead of 4.94.
        constexpr bool kIdsAtOnce = kIsect != kIsectFp64;
        static_assert(offsetof(LeafRec, fn) % 16 == 0, "ids are read in 16- and 8-byte pieces");
        int32_t fn[6] = {0, 0, 0, 0, 0, 0};
        if (hit && kIsect != kIsectFp64) {
#pragma unroll
            for (int k = 0; k < 3; k++) load4(L->T + 4*k, T + 4*k);
            const int4 f03 = __ldg(reinterpret_cast<const int4*>(L->fn));
            const int2 f45 = __ldg(reinterpret_cast<const int2*>(L->fn + 4));
            fn[0] = f03.x; fn[1] = f03.y; fn[2] = f03.z; fn[3] = f03.w;
            fn[4] = f45.x; fn[5] = f45.y;
        } else if (!hit) {
#pragma unroll
            for (int k = 0; k < 12; k++) T[k] = IDENTITY[k];
        }
        auto table = [&](int outside, int inside) {
            return kIdsAtOnce ? fn[is.outside ? outside : inside]
                              : __ldg(L->fn + (is.outside ? outside : inside));
        };
        auto draw = [&]() -> double {
            const uint32_t k = (uint32_t)k_draw++;
            if (a.rng.mode == MLGPU_RNG_REPLAY) {
                if (k >= a.rng.stride) { if (!err) err = MLGPU_ERR_RUNTIME; return 0.5; }
                return __ldg(a.rng.uniforms + (uint64_t)photon*a.rng.stride + k);
            }
            return mlgpu_philox_uniform(a.rng.seed, stream, k);
        };
        bool absorbed = false;
        if (hit) {
            // absorbed_in_medium_before_reaching_surface, PhotonAndFrame.cpp:32-38
            const double depth = func_eval_tab(fn_pts, fn_off, table(MLGPU_SURF_OUTER_ABSORPTION, MLGPU_SURF_INNER_ABSORPTION), lambda, &err);
            if (depth != depth && a.rng.mode == MLGPU_RNG_PHILOX) {
                // merlict's default table evaluates to NaN, and no draw
                // is larger than that: only the draw is counted
                k_draw++;
            } else {
                const double survival = exp(-is.dist/depth);
                absorbed = draw() > survival;
            }
        }
        v3 out = d;              // the new direction in the leaf's frame, if it moves
        if (!hit || absorbed) {
            kind = MLGPU_ABSORPTION_IN_VOID;
        } else {
            const double refl = func_eval_tab(fn_pts, fn_off, table(MLGPU_SURF_OUTER_REFLECTION, MLGPU_SURF_INNER_REFLECTION), lambda, &err);
            if (refl >= draw()) {
                kind = MLGPU_REFLECTION_ON_SURFACE;
                out = mirror(is.normal, orientation_inverse(T, d));
                moved = true;
            } else if (!(__ldg(&L->flags) & MLGPU_FLAG_TRANSPARENT)) {
                kind = MLGPU_ABSORPTION_ON_SURFACE;
            } else {
                const v3 inc = orientation_inverse(T, d);
                const v3 nrm = is.outside ? is.normal : scale(is.normal, -1.0);
                const double n_from = func_eval_tab(fn_pts, fn_off, table(MLGPU_SURF_OUTER_REFRACTION, MLGPU_SURF_INNER_REFRACTION), lambda, &err);
                const double n_to = func_eval_tab(fn_pts, fn_off, table(MLGPU_SURF_INNER_REFRACTION, MLGPU_SURF_OUTER_REFRACTION), lambda, &err);
                const double cosI = dot(nrm, inc)*(-1.0);
                const double ratio = n_from/n_to;
                const double sinT2 = ratio*ratio*(1.0 - cosI*cosI);
                const double cosT = sqrt(1.0 - sinT2);
                double R;
                if (sinT2 > 1.0) {
                    R = 1.0;
                } else {
                    const double rOrth = (n_from*cosI - n_to*cosT) / (n_from*cosI + n_to*cosT);
                    const double rPar = (n_to*cosI - n_from*cosT) / (n_to*cosI + n_from*cosT);
                    R = (rOrth*rOrth + rPar*rPar) / 2.0;
                }
                if (R > draw()) {
                    kind = MLGPU_FRESNEL_REFLECTION_ON_SURFACE;
                    out = mirror(is.normal, inc);
                    moved = true;
                } else {
                    kind = is.outside ? MLGPU_REFRACTION_TO_INSIDE : MLGPU_REFRACTION_TO_OUTSIDE;
                    const int32_t flags = __ldg(&L->flags), allowed = __ldg(&L->allowed_node);
                    const bool to_default = is.outside
                        ? (flags & MLGPU_FLAG_INNER_REFRACTION_DEFAULT) != 0
                        : (flags & MLGPU_FLAG_OUTER_REFRACTION_DEFAULT) != 0;
                    root = (allowed >= 0 && !to_default) ? allowed : 0;
                    out = add(scale(inc, ratio), scale(nrm, ratio*cosI - cosT));
                    moved = true;
                }
            }
        }
        if (moved) {
            // the new ray, whichever way its direction came about
            s = position(T, is.pos);
            d = normalized(orientation(T, out));
        }
        if (hist) store_hist(&hist[n_int], is.pos, is.normal, is.dist, is.leaf, kind, is.outside);
        {
            // time-of-flight term, merlict/Photon.cpp:37-56
            const int32_t f = hit
                ? table(MLGPU_SURF_OUTER_REFRACTION, MLGPU_SURF_INNER_REFRACTION)
                : sc.default_refraction;
            int terr = 0;
            const double n = func_eval_tab(fn_pts, fn_off, f, lambda, &terr);
            if (terr && !tof_error) tof_error = terr;
            tof += n*is.dist/299792458.0;
        }
    }
    const int32_t n_next = n_int + (step == kNoStep ? 0 : 1);
    const bool survive = moved && (uint32_t)n_next <= max_int;
    q->n_int = n_next;
    if (survive) {
        q->err = err | (tof_error << 8);
    } else {
        // the photon ends: its results (Sensor.cpp:14-30)
        const int32_t sensor = is.leaf >= 0 ? __ldg(&sc.leaf[is.leaf].sensor) : -1;
        if (sensor >= 0 && tof_error && !err) err = tof_error;
        const DevResults& r = a.results;
        const uint64_t p = (uint64_t)photon;
        r.sensor[p] = sensor;
        if (r.x) static_cast<Out*>(r.x)[p] = (Out)is.pos.x;
        if (r.y) static_cast<Out*>(r.y)[p] = (Out)is.pos.y;
        if (r.time) r.time[p] = tof;
        if (r.final_leaf) r.final_leaf[p] = is.leaf;
        if (r.info)
            r.info[p] = (uint32_t)kind | ((uint32_t)n_next << 8) |
                ((k_draw > 255 ? 255u : (uint32_t)k_draw) << 16) | ((uint32_t)err << 24);
        if (r.theta_x || r.theta_y || r.final_position || r.final_direction) {
            // the last segment (RayForPropagation.cpp:114-136); the
            // transform and the ray before the step are read again, so
            // that the step itself need not keep them
            v3 s0, d0;
            before(&s0, &d0);
            if (is.leaf >= 0) {
#pragma unroll
                for (int k = 0; k < 3; k++) load4(sc.leaf[is.leaf].T + 4*k, T + 4*k);
            } else {
#pragma unroll
                for (int k = 0; k < 12; k++) T[k] = IDENTITY[k];
            }
            const v3 last_world = moved ? s : position(T, is.pos);
            const v3 second_last_world =
                step == kNoStep ? last_world : (n_int == 1 ? position(IDENTITY, s0) : s0);
            v3 inc = mk(0.0, 0.0, 0.0);
            if (n_next > 1) inc = orientation_inverse(T, normalized(sub(last_world, second_last_world)));
            if (r.theta_x) static_cast<Out*>(r.theta_x)[p] = (Out)(-1.0*inc.x);
            if (r.theta_y) static_cast<Out*>(r.theta_y)[p] = (Out)(-1.0*inc.y);
            if (r.final_position) {
                r.final_position[3*p] = last_world.x;
                r.final_position[3*p + 1] = last_world.y;
                r.final_position[3*p + 2] = last_world.z;
            }
            if (r.final_direction) {
                r.final_direction[3*p] = d.x;
                r.final_direction[3*p + 1] = d.y;
                r.final_direction[3*p + 2] = d.z;
            }
        }
        if (hist)
            for (uint32_t k = (uint32_t)n_next; k < hist_len; k++)
                store_hist(&hist[k], mk(0, 0, 0), mk(0, 0, 0), 0.0, MLGPU_LEAF_PHOTON_SOURCE, 0, false);
        if (err) raise_error(sc.error_word, (unsigned int)err);
    }
    return survive;
}

// The property tables, staged in shared memory when they fit.
__device__ __forceinline__ void stage_tables(const DevScene& sc, int bytes, double* s_fn,
                                             const double** pts, const int32_t** off) {
    *pts = sc.fn_points;
    *off = sc.fn_offset;
    if (!bytes) return;
    const int np = 3*sc.num_fn_points;
    int32_t* s_off = reinterpret_cast<int32_t*>(s_fn + np);
    for (int k = threadIdx.x; k < np; k += blockDim.x) s_fn[k] = __ldg(sc.fn_points + k);
    for (int k = threadIdx.x; k <= sc.num_functions; k += blockDim.x) s_off[k] = __ldg(sc.fn_offset + k);
    __syncthreads();
    *pts = s_fn;
    *off = s_off;
}

// The first look at a large batch: a photon that misses the root frame's
// sphere (most of an air shower's) ends here, its void result written where
// it is read, and the others' indices are listed in w.first for the tracer,
// so that only they pass through the pool.  Streams the planes once: 1.85e7
// photons of air showers, 2 % of which are listed, spend 0.42 ms here (3.7
// TB/s of planes and results) and 1.85 ms in all; through the pool in the
// coherent order they take 5.4 ms.
template <typename In, typename Out>
__global__ void __launch_bounds__(256, 4)
wave_first_kernel(const TraceArgs a, const WaveBuffers w) {
    extern __shared__ double s_fn[];
    const double* fn_pts;
    const int32_t* fn_off;
    stage_tables(a.scene, w.fn_smem_bytes, s_fn, &fn_pts, &fn_off);
    const int lane = threadIdx.x & 31;
    const uint64_t warps = (uint64_t)gridDim.x*8;
    // a warp looks at kRun x 32 consecutive photons per turn: one addition to
    // the list's length for all of them
    constexpr int kRun = 4;
    for (uint64_t first = ((uint64_t)blockIdx.x*8 + (threadIdx.x >> 5))*(32*kRun);
         first < a.num_photons; first += warps*(32*kRun)) {
        unsigned listed[kRun];
        uint32_t sum = 0;
#pragma unroll
        for (int r = 0; r < kRun; r++) {
            const uint64_t i = first + 32u*r + (uint64_t)lane;
            bool on = false;
            if (i < a.num_photons) {
                PhotonRay q;
                const int step = start_photon<In>(a, w, i, &q);
                on = step == kStepBvh || step == kStepTree;
                if (!on) {
                    const v3 s = q.s, d = q.d;
                    resolve_photon<Out, kIsectFp64>(a, fn_pts, fn_off, step, kNoLeaf, 0.0, &q,
                                                    [&](v3* s0, v3* d0) { *s0 = s; *d0 = d; });
                }
            }
            listed[r] = __ballot_sync(kFull, on);
            sum += (uint32_t)__popc(listed[r]);
        }
        if (sum == 0) continue;
        uint32_t at = 0;
        if (lane == 0) at = (uint32_t)atomicAdd(&w.counters->avail_snap, (unsigned long long)sum);
        at = __shfl_sync(kFull, at, 0);
#pragma unroll
        for (int r = 0; r < kRun; r++) {
            if ((listed[r] >> lane) & 1u)
                w.first[at + __popc(listed[r] & ((1u << lane) - 1u))] =
                    (uint32_t)(first + 32u*r) + (uint32_t)lane;
            at += (uint32_t)__popc(listed[r]);
        }
    }
}

// Photons from where they are to their ends, in one launch: the rays of the
// pool and, up to the batch's end, photons that have not set out.  Without a
// pool (kFinishBatchMode), the whole batch; with kFinishListMode, the photons
// that wave_first_kernel listed, unless there are more than kFinishRays.  A warp keeps its photons, one per
// lane, and alternates between searching their hits and resolving them; no
// host, no counters and no other kernel come between the interactions of a
// photon.  For few rays that is what counts: a wavefront iteration is two
// kernels, each with its ramp and its longest ray, however few rays it
// advances.  With fewer photons than the grid
// has lanes each warp takes fewer, since a warp lasts as long as its longest
// photon.
template <typename In, typename Out>
__global__ void __launch_bounds__(kWalkThreads, kFinishBlocks)
wave_finish_kernel(const TraceArgs a, const WaveBuffers w, const RayPool cur, int mode) {
    extern __shared__ double2 s_walk[];
    const DevScene& sc = a.scene;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kWarps = kWalkThreads/32;
    WalkWarp* sw = reinterpret_cast<WalkWarp*>(s_walk) + warp;
    uint32_t* stacks = reinterpret_cast<uint32_t*>(reinterpret_cast<WalkWarp*>(s_walk) + kWarps);
    uint32_t* stack = stacks + threadIdx.x;
    const double* fn_pts;
    const int32_t* fn_off;
    stage_tables(sc, w.fn_smem_bytes,
                 reinterpret_cast<double*>(stacks + kWalkThreads*sc.surf_levels), &fn_pts, &fn_off);
    const bool pool = mode == kFinishPoolMode;
    const uint32_t active = pool ? w.counters->active : 0u;
    const uint32_t inside = pool ? w.counters->inside : 0u;
    const unsigned long long next_input = pool ? w.counters->next_input : 0ull;
    const unsigned long long input = mode == kFinishListMode ? w.counters->avail_snap : a.num_photons;
    if (mode == kFinishListMode && input > kFinishRays) return;
    const uint32_t front = active + (uint32_t)(input - next_input);
    const uint32_t rays = front + inside;
    const uint32_t warps = gridDim.x*kWarps;
    const uint32_t share = (rays + warps - 1)/warps, per = share < 32u ? share : 32u;
    WalkLane l;
    l.eps = 0.0f;
    l.key = kNoKey;
    for (uint32_t first = (blockIdx.x*kWarps + warp)*per; first < rays; first += warps*per) {
        const uint32_t index = first + (uint32_t)lane;
        bool live = (uint32_t)lane < per && index < rays;
        PhotonRay q;
        int step = kNoStep;
        if (live) {
            const uint32_t slot = index < front ? index : w.pool - 1u - (index - front);
            if (index >= active && index < front) {
                step = start_photon<In>(a, w, next_input + (index - active), &q);
            } else {
                load_photon(cur, slot, &q);
                step = cur.step[slot];
            }
        }
        while (__any_sync(kFull, live)) {
            uint32_t listed = 0;
            int groups = 0;
            l.walking = false;
            if (live) {
                if (step == kStepBvh) {
                    walk_begin(sc, q.s, q.d, sw, lane, &l);
                } else {
                    sw->ray[0][lane] = make_double2(q.s.x, q.s.y);
                    sw->ray[1][lane] = make_double2(q.s.z, q.d.x);
                    sw->ray[2][lane] = make_double2(q.d.y, q.d.z);
                }
            }
            __syncwarp();
            while (true) {
                const bool walking = __any_sync(kFull, l.walking);
                intersect_queued<kIsectFp64>(sc, sw, lane, !walking, &groups, &listed, &l);
                if (!walking) break;
                groups = visit_nodes(sc, sw, stack, lane, groups, &l);
            }
            int32_t best = kNoLeaf;
            double dist = 0.0;
            if (live && step == kStepBvh) {
                best = sw->leaf[lane];
                dist = __longlong_as_double((long long)sw->key[lane]);
            }
            if (live && step == kStepTree)
                best = closest_hit_tree<kIsectFp64>(sc, q.root, q.s, q.d, &dist);
            if (live) {
                live = resolve_photon<Out, kIsectFp64>(
                    a, fn_pts, fn_off, step, best, dist, &q, [&](v3* s, v3* d) {
                        const double2 x = sw->ray[0][lane], y = sw->ray[1][lane],
                                      z = sw->ray[2][lane];
                        *s = mk(x.x, x.y, y.x);
                        *d = mk(y.y, z.x, z.y);
                    });
                if (live) step = step_kind(a, w, q.s, q.d, q.root);
            }
            __syncwarp();
        }
    }
}

// The value of avail the next iteration admits photons up to: read once
// per iteration, so that the intake and its counting agree on it.  avail is
// raised by kernels of another stream after the records they publish are
// written, so a fence orders the read before the intake's record reads.
__device__ __forceinline__ void snapshot_avail(WaveCounters* c) {
    c->avail_snap = atomicAdd(&c->avail, 0ull);
    __threadfence();
}

// One slot of the resolve step, all lanes of the warp: the photon's step,
// and the photon into the next pool if it goes on.
template <typename Out, int kIsect>
__device__ __forceinline__ void resolve_slot(const TraceArgs& a, const WaveBuffers& w,
                                             const RayPool& cur, const RayPool& nxt,
                                             const double* fn_pts, const int32_t* fn_off,
                                             bool valid, uint32_t slot, int lane) {
    const DevScene& sc = a.scene;
    bool survive = false;
    int32_t finished_chunk = -1;   // fed propagation: the chunk of a photon that ends here
    PhotonRay q;
    if (valid) {
        load_photon(cur, slot, &q);
        const int step = cur.step[slot];
        int32_t best = kNoLeaf;
        double dist = 0.0;
        if (kIsect != kIsectFp32Pure && step == kStepTree && w.walk != MLGPU_WALK_LEVELS) {
            // a ray inside a lens (or without a BVH); the pure form's rays
            // are always walked by the level kernels
            best = closest_hit_tree<kIsect>(sc, q.root, q.s, q.d, &dist);
        } else {
            best = cur.best_leaf[slot];
            if (kIsect == kIsectFp64) dist = __longlong_as_double((long long)cur.best_key[slot]);
        }
        survive = resolve_photon<Out, kIsect>(a, fn_pts, fn_off, step, best, dist, &q,
                                              [&](v3* s, v3* d) { load_ray(cur, slot, s, d); });
        if (!survive && a.fed) {
            int32_t c = 0;
            while (c + 1 < a.feed_chunks && (uint64_t)q.photon >= a.feed_start[c + 1]) c++;
            finished_chunk = c;
        }
    }
    // fed propagation: finished photons per chunk, one addition per chunk
    // and warp (a warp's photons mostly come from one chunk)
    if (a.fed) {
        const unsigned fin = __ballot_sync(kFull, finished_chunk >= 0);
        if (finished_chunk >= 0) {
            const unsigned same = __match_any_sync(fin, finished_chunk);
            if (lane == __ffs(same) - 1)
                atomicAdd(&w.counters->done[finished_chunk], (unsigned)__popc(same));
        }
    }
    // warp-ballot compaction of the surviving rays into the next pool; with
    // the closest-hit walk, the rays inside a lens from its end, so that the
    // warps of the next iteration hold rays of one kind
    int step = kNoStep;
    if (survive) step = step_kind(a, w, q.s, q.d, q.root);
    const bool inside = survive && step == kStepTree && w.walk != MLGPU_WALK_LEVELS;
    const unsigned m = __ballot_sync(kFull, survive && !inside);
    const unsigned mi = __ballot_sync(kFull, inside);
    if (m | mi) {
        uint32_t base = 0;
        if (lane == 0 && m) base = atomicAdd(&w.counters->next, (unsigned)__popc(m));
        if (lane == 1 && mi) base = atomicAdd(&w.counters->next_inside, (unsigned)__popc(mi));
        const uint32_t base_m = __shfl_sync(kFull, base, 0), base_i = __shfl_sync(kFull, base, 1);
        if (survive) {
            const unsigned below = (1u << lane) - 1u;
            const uint32_t o = inside ? w.pool - 1u - (base_i + __popc(mi & below))
                                      : base_m + __popc(m & below);
            // the ray as the next iteration takes it: merlict's state and
            // how it finds its hit
            store_photon(nxt, o, q, step);
            if (w.walk == MLGPU_WALK_LEVELS) prepare_levels(sc, nxt, o, q.s, q.d, step);
        }
    }
}

// A thread per ray; those inside a lens search their hit first, by merlict's
// walk of the lens.  96 registers and a few dozen bytes spilled, five blocks
// of 128 per SM: the step waits on its gathers and on chains of
// double-precision arithmetic.  1e7 photons of the light-field telescope take
// 16.8 ms so, and 16.7, 16.9, 17.1 and 17.3 ms with four, six, seven and eight
// blocks.  As three kernels (lens search, resolve, counters) of their own an
// iteration ended three times: 18.3 ms of an earlier build, 17.65 so.
constexpr int kResolveThreads = 128;
constexpr int kResolveBlocks = 5;

inline int resolve_blocks(uint32_t pool) {
    const uint32_t need = (pool + kResolveThreads - 1)/kResolveThreads;
    const uint32_t full = device_sms()*kResolveBlocks;
    return (int)(need < full ? need : full);
}

template <typename Out, int kIsect>
__global__ void __launch_bounds__(kResolveThreads, kResolveBlocks)
wave_resolve_kernel(const TraceArgs a, const WaveBuffers w, const RayPool cur, const RayPool nxt) {
    const DevScene& sc = a.scene;
    extern __shared__ double s_fn[];
    const double* fn_pts;
    const int32_t* fn_off;
    stage_tables(sc, w.fn_smem_bytes, s_fn, &fn_pts, &fn_off);
    const bool levels = w.walk == MLGPU_WALK_LEVELS;
    const uint32_t fresh = levels ? 0u : new_photons(a, w);
    const uint32_t front = levels ? w.counters->total : w.counters->active + fresh;
    const uint32_t rays = front + w.counters->inside;
    const int lane = threadIdx.x & 31;
    for (uint32_t first = warp_first(); first < rays; first += gridDim.x*blockDim.x) {
        const uint32_t index = first + (uint32_t)lane;
        resolve_slot<Out, kIsect>(a, w, cur, nxt, fn_pts, fn_off, index < rays,
                                  index < front ? index : w.pool - 1u - (index - front), lane);
    }
    if (levels) return;
    // the last block to end turns the counters over for the next iteration
    __shared__ bool s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&w.counters->blocks, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (s_last && threadIdx.x == 0) {
        WaveCounters* c = w.counters;
        __threadfence();
        c->next_input += fresh;
        c->active = *const_cast<volatile unsigned int*>(&c->next);
        c->inside = *const_cast<volatile unsigned int*>(&c->next_inside);
        c->next = 0;
        c->next_inside = 0;
        c->chunks = 0;
        c->blocks = 0;
        if (a.fed) snapshot_avail(c);
    }
}

}  // namespace
}  // namespace mlgpu

#endif  // MLGPU_WAVE_RESOLVE_CUH_
