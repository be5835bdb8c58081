// closest_hit.cuh -- merlict's first causal intersection of a ray
// (CausalIntersection, merlict/RayAndFrame.cpp:126-173): a warp walks the
// surface BVH for its rays, one ray per lane, nearest octant first, and
// intersects the leaves it reaches on the way, so that nodes beyond a ray's
// closest hit so far are left out.
//
// The walk tests boxes in single precision, widened by the ray's rounding;
// a leaf it reaches goes through merlict's own bounding-sphere test and
// merlict's own intersection, and equal distances go to the leaf merlict
// visits first (the lowest leaf index), so the hit is merlict's.
//
// A lane keeps its walk in a few registers and a column of shared memory
// (one stack word per tree level: first child << 8 | children left to visit,
// in visiting order).  The leaves that the lanes reach are queued per warp, a
// node's leaves as one group; 32 groups at a time are spread into three
// lists by the arithmetic of their intersection (caps, planes, other
// quadrics), and whenever a list holds 32 leaves the warp intersects 32, a
// lane each on whichever ray they belong to: the double-precision work runs
// on full warps of one kind instead of on the lanes that happen to have
// reached a leaf.
//
// What bounds it: instructions (53 % issue on the light-field telescope, no
// more warps: 116 registers, four blocks per SM; five blocks spill and measured
// 6 % slower).  Per photon of that scene, 2.5 rays of this kind visit 27.8
// nodes and intersect 13.0 leaves.  Propagating 1e7 photons, the searches
// took 22.5 ms as one kernel per BVH level over queued (ray, node) pairs plus
// intersection and tie kernels, and take 12.9 ms so, of which 1.6 ms are the
// walks inside lenses (of the build that brought the walk).  On the way: one thread per ray with its own leaf list
// 18.0 ms (15 of 32 lanes busy), refilled lanes and a shared leaf list 18.9,
// lists by kind 15.9, the same at 116 registers instead of 80 14.4, 32-byte
// loads instead of 16-byte ones 13.6, leaves queued in groups 12.9; now 11.3
// (10.1 in the coherent order), with the walks inside lenses in the
// interaction's kernel, 2^23 rays at a time and three-way integer minima for
// the slab test.
#ifndef MLGPU_CLOSEST_HIT_CUH_
#define MLGPU_CLOSEST_HIT_CUH_

#include <climits>
#include <cstdint>

#include "fp64_geometry.cuh"
#include "fp32_geometry.cuh"

namespace mlgpu {
namespace {

using namespace fp64;

constexpr unsigned kFull = 0xffffffffu;
constexpr int kIsectFp64 = 0;
constexpr int kIsectFp32 = 1;
constexpr int kIsectFp32Pure = 2;

constexpr int32_t kNoLeaf = INT32_MAX;  // no hit
constexpr unsigned long long kNoKey = ~0ull;

constexpr int kWalkThreads = 128;
constexpr int kWalkBlocks = 4;   // resident per SM
constexpr int kFinishBlocks = 3;
constexpr int kLists = 3;
constexpr int kLeafList = 96;                  // leaves a list holds
static_assert(kLeafList >= 32 + kBvhWidth, "a list of fewer than 32 takes any one group's leaves");
// nodes a lane visits between looks at the queue: with one, two and three, 1e6
// telescope photons take 2.30, 2.28 and 2.25 ms, 8e6 of the large reflector
// (whose walks are short) 4.55, 4.55 and 4.71 ms
constexpr int kVisits = 2;
constexpr int kGroups = 32 + 32*kVisits;       // groups: 31 and the visits of 32 lanes

// A warp's part of shared memory; the lanes' stacks follow all warps' parts.
struct WalkWarp {
    double2 ray[3][32];          // (sx, sy), (sz, dx), (dy, dz)
    unsigned long long key[32];  // smallest hit distance (bits of a positive double)
    int32_t leaf[32];            // its leaf
    uint2 group[kGroups];        // first leaf slot << 8 | leaves hit; kinds of the node's
                                 // slots: caps, planes, leaves (a byte each), lane of the ray
    uint32_t list[kLists][kLeafList];   // leaf slot << 5 | lane of the ray
};

inline size_t closest_hit_smem(int levels) {
    return (size_t)(kWalkThreads/32)*sizeof(WalkWarp) +
        (size_t)kWalkThreads*(size_t)levels*sizeof(uint32_t);
}

// Blocks of a walk over `rays` rays: as many as stay resident, each warp
// taking several chunks of 32.
inline int walk_blocks(uint32_t rays) {
    const uint32_t need = (rays + kWalkThreads - 1)/kWalkThreads, full = device_sms()*kWalkBlocks;
    return (int)(need < full ? need : full);
}

// Blocks of a launch that takes at most `rays` rays to their ends: a warp
// per ray up to a full GPU.
inline int finish_blocks(uint32_t rays) {
    const uint32_t need = (rays + kWalkThreads/32 - 1)/(kWalkThreads/32);
    const uint32_t full = device_sms()*kFinishBlocks;
    return (int)(need < full ? need : full);
}

// A lane's walk.
struct WalkLane {
    float ox, oy, oz;            // origin
    float ix, iy, iz;            // reciprocal direction
    float wx, wy, wz;            // box widening over |direction|
    float eps;                   // the widening
    float tbest;                 // no farther than this
    uint32_t octant;             // bit a: the direction is negative on axis a
    uint32_t node, group, base;  // node to visit next; its siblings left, first sibling
    int sp;
    bool walking;
    unsigned long long key;      // the lane's copy of WalkWarp::key
};

// Starts the lane's walk of the whole tree along (s, d); the caller has made
// merlict's test of the root frame's sphere.
__device__ __forceinline__ void walk_begin(const DevScene& sc, v3 s, v3 d, WalkWarp* w, int lane,
                                           WalkLane* l) {
    w->ray[0][lane] = make_double2(s.x, s.y);
    w->ray[1][lane] = make_double2(s.z, d.x);
    w->ray[2][lane] = make_double2(d.y, d.z);
    w->key[lane] = kNoKey;
    w->leaf[lane] = kNoLeaf;
    l->key = kNoKey;
    float fdx = (float)d.x, fdy = (float)d.y, fdz = (float)d.z;
    if (fabsf(fdx) < kMinDirection) fdx = copysignf(kMinDirection, fdx);
    if (fabsf(fdy) < kMinDirection) fdy = copysignf(kMinDirection, fdy);
    if (fabsf(fdz) < kMinDirection) fdz = copysignf(kMinDirection, fdz);
    l->ix = 1.0f/fdx; l->iy = 1.0f/fdy; l->iz = 1.0f/fdz;
    l->ox = (float)s.x; l->oy = (float)s.y; l->oz = (float)s.z;
    l->eps = sc.bvh_eps + 4e-7f*(fabsf(l->ox) + fabsf(l->oy) + fabsf(l->oz));
    l->wx = l->eps*fabsf(l->ix); l->wy = l->eps*fabsf(l->iy); l->wz = l->eps*fabsf(l->iz);
    l->octant = (fdx < 0.0f ? 1u : 0u) | (fdy < 0.0f ? 2u : 0u) | (fdz < 0.0f ? 4u : 0u);
    l->tbest = INFINITY;
    l->node = 0; l->group = 0; l->base = 0;
    l->sp = 0;
    // a ray that is not finite hits nothing: every intersection of merlict's
    // rejects it (support and hit differ by NaN)
    l->walking = (s.x - s.x) + (s.y - s.y) + (s.z - s.z) + (d.x - d.x) + (d.y - d.y) +
        (d.z - d.z) == 0.0;
}

// 32 bytes through the read-only path in one load: a gather costs the L1 a
// pass per lane and load, however wide the load is.
__device__ __forceinline__ void load32(const uint4* p, uint4* a, uint4* b) {
    asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(a->x), "=r"(a->y), "=r"(a->z), "=r"(a->w), "=r"(b->x), "=r"(b->y), "=r"(b->z),
          "=r"(b->w)
        : "l"(p));
}

// Visits the lane's next node and moves on; returns the group of its leaves
// that are hit (x's low byte is 0: none).
//
// The slab distance of a bound origin + q 2^e is q (2^e i) + (origin - o) i
// -+ w, one fused multiply-add per bound with the origin folded in: a byte q
// in bits 8-15 of a float with exponent 2^15 is 2^15 + q, and the 2^15 2^e i
// is taken off the constant; that rounds by 2^-9 of a step, which the
// builder has widened the boxes by.  Which bound of a pair is the near one
// is the octant's, so four bounds at a time are chosen instead of a minimum
// and a maximum per pair.
__device__ __forceinline__ uint2 walk_step(const DevScene& sc, WalkLane* l, uint32_t* stack) {
    uint4 h0, w1, b0, b1, b2, unused;
    const uint4* nu = reinterpret_cast<const uint4*>(sc.surf + l->node);
    load32(nu, &h0, &w1);
    load32(nu + 2, &b0, &b1);
    load32(nu + 4, &b2, &unused);
    const float4 w0 = make_float4(__uint_as_float(h0.x), __uint_as_float(h0.y),
                                  __uint_as_float(h0.z), __uint_as_float(h0.w));
    const uint32_t ex = __float_as_uint(w0.w);
    const float Sx = __uint_as_float((ex & 0xffu) << 23)*l->ix;
    const float Sy = __uint_as_float((ex & 0xff00u) << 15)*l->iy;
    const float Sz = __uint_as_float((ex & 0xff0000u) << 7)*l->iz;
    const float Lx = __fmaf_rn(-32768.0f, Sx, (w0.x - l->ox)*l->ix);
    const float Ly = __fmaf_rn(-32768.0f, Sy, (w0.y - l->oy)*l->iy);
    const float Lz = __fmaf_rn(-32768.0f, Sz, (w0.z - l->oz)*l->iz);
    const float nx = Lx - l->wx, ny = Ly - l->wy, nz = Lz - l->wz;
    const float fx = Lx + l->wx, fy = Ly + l->wy, fz = Lz + l->wz;
    const bool sx = (l->octant & 1u) != 0, sy = (l->octant & 2u) != 0, sz = (l->octant & 4u) != 0;
    const uint32_t nxw[2] = {sx ? b1.z : b0.x, sx ? b1.w : b0.y};
    const uint32_t fxw[2] = {sx ? b0.x : b1.z, sx ? b0.y : b1.w};
    const uint32_t nyw[2] = {sy ? b2.x : b0.z, sy ? b2.y : b0.w};
    const uint32_t fyw[2] = {sy ? b0.z : b2.x, sy ? b0.w : b2.y};
    const uint32_t nzw[2] = {sz ? b2.z : b1.x, sz ? b2.w : b1.y};
    const uint32_t fzw[2] = {sz ? b1.x : b2.z, sz ? b1.y : b2.w};
    uint32_t miss = 0;
#pragma unroll
    for (int k = kBvhWidth - 1; k >= 0; k--) {
        const int g = k >> 2;
        const uint32_t sel = 0x7404u | (uint32_t)(k & 3) << 4;
        auto dq = [sel](uint32_t word) {   // 2^15 + byte k & 3 of the word
            return __uint_as_float(__byte_perm(word, 0x47000000u, sel));
        };
        // largest of the near distances and 0, smallest of the far ones and
        // tbest, by their bits: floats that are not negative order like
        // integers, and a negative far distance misses whichever it is
        const float t0 = __int_as_float(__vimax3_s32_relu(
            __float_as_int(__fmaf_rn(dq(nxw[g]), Sx, nx)),
            __float_as_int(__fmaf_rn(dq(nyw[g]), Sy, ny)),
            __float_as_int(__fmaf_rn(dq(nzw[g]), Sz, nz))));
        const float t1 = __int_as_float(min(__vimin3_s32(
            __float_as_int(__fmaf_rn(dq(fxw[g]), Sx, fx)),
            __float_as_int(__fmaf_rn(dq(fyw[g]), Sy, fy)),
            __float_as_int(__fmaf_rn(dq(fzw[g]), Sz, fz))), __float_as_int(l->tbest)));
        miss = __funnelshift_l(__float_as_uint(t1 - t0), miss, 1);   // the sign: missed
    }
    uint32_t m = ~miss & (ex >> 24);
    if (m) {
        // into visiting order, bit (slot ^ octant)
        if (sx) m = ((m & 0x55u) << 1) | ((m >> 1) & 0x55u);
        if (sy) m = ((m & 0x33u) << 2) | ((m >> 2) & 0x33u);
        if (sz) m = ((m & 0x0fu) << 4) | (m >> 4);
        if (l->group) { stack[l->sp*kWalkThreads] = l->base << 8 | l->group; l->sp++; }
        l->group = m;
        l->base = w1.x;
    } else if (!l->group) {
        if (l->sp == 0) {
            l->walking = false;
        } else {
            l->sp--;
            const uint32_t e = stack[l->sp*kWalkThreads];
            l->group = e & 0xffu;
            l->base = e >> 8;
        }
    }
    if (l->group) {
        l->node = l->base + (((uint32_t)__ffs(l->group) - 1u) ^ l->octant);
        l->group &= l->group - 1u;
    }
    return make_uint2(w1.y & ~(miss & 0xffu), w1.z);
}

// The distance along (s, d) of merlict's intersection of leaf `leaf`, or a
// negative number.  kClass: the leaf's class, whose leaves the warp has
// listed (then merlict's test of the bounding sphere comes first), or -1 for
// any leaf of merlict's own walk (which has made that test).
template <int kIsect, int kClass>
__device__ __forceinline__ double leaf_distance(const DevScene& sc, int32_t leaf, v3 s, v3 d) {
    if (kIsect == kIsectFp64) {
        double T[12], ti[3], pr[MLGPU_LEAF_PARAMS], r2;
        int32_t prim;
        load_leaf(sc.leaf + leaf, T, ti, pr, &r2, &prim);
        if (kClass >= 0 && !sphere_cull(make_double4(T[3], T[7], T[11], r2), s, d, dot(s, d)))
            return -1.0;
        Isec h;   // only the distance is used; the rest is not computed
        const v3 ls = position_inverse(T, ti, s), ld = orientation_inverse(T, d);
        switch (kClass >= 0 ? kClass : leaf_class(prim)) {
        case kLeafCap: intersect_leaf<kLeafCap>(sc, leaf, prim, pr, r2, ls, ld, &h); break;
        case kLeafPlane: intersect_leaf<kLeafPlane>(sc, leaf, prim, pr, r2, ls, ld, &h); break;
        default: intersect_leaf<kLeafQuadric>(sc, leaf, prim, pr, r2, ls, ld, &h); break;
        }
        return h.leaf >= 0 ? h.dist : -1.0;
    }
    const fp32::Hit32 h = fp32::intersect32<false>(sc, leaf, fp32::dmk(s.x, s.y, s.z),
                                                   fp32::dmk(d.x, d.y, d.z), false);
    return h.leaf >= 0 ? h.v : -1.0;
}

// Spreads the last groups, up to 32 and a lane each, into the lists, lanes
// in order as far as their leaves fit (with every list below 32 leaves at
// least one group does); returns the number of groups left.  `listed` holds
// the three lists' lengths, ten bits each.
__device__ __forceinline__ int spread_groups(WalkWarp* w, int lane, int groups, uint32_t* listed) {
    const int first = max(groups - 32, 0), take = groups - first;
    uint2 g = make_uint2(0u, 0u);
    if (lane < take) g = w->group[groups - 1 - lane];
    uint32_t hit = g.x & 0xffu;
    const uint32_t caps = hit & g.y, planes = hit & (g.y >> 8);
    const uint32_t n = (uint32_t)__popc(caps) | (uint32_t)__popc(planes) << 10 |
        (uint32_t)__popc(hit & ~(caps | planes)) << 20;
    uint32_t end = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, end, o);
        if (lane >= o) end += y;
    }
    end += *listed;
    const bool fits = (end & 1023u) <= (uint32_t)kLeafList &&
        (end >> 10 & 1023u) <= (uint32_t)kLeafList && (end >> 20) <= (uint32_t)kLeafList;
    const unsigned no = __ballot_sync(kFull, !fits);
    const int cut = no ? __ffs(no) - 1 : 32;
    if (lane < cut) {
        const uint32_t owner = g.y >> 24, leaves = g.y >> 16 & 0xffu, base = g.x >> 8;
        uint32_t at = end - n;
        while (hit) {
            const uint32_t bit = hit & (0u - hit);
            hit ^= bit;
            const int c = caps & bit ? 0 : planes & bit ? 1 : 2;
            w->list[c][at >> (10*c) & 1023u] = (base + __popc(leaves & (bit - 1u))) << 5 | owner;
            at += 1u << (10*c);
        }
    }
    *listed = __shfl_sync(kFull, end, cut - 1);
    __syncwarp();
    return groups - min(cut, take);
}

// Intersects the last n <= 32 leaves of list kClass, of length `length`, and
// updates the lanes' closest hits.
template <int kIsect, int kClass>
__device__ __forceinline__ void intersect_listed(const DevScene& sc, WalkWarp* w, int lane,
                                                 int length, int n, WalkLane* l) {
    unsigned long long key = kNoKey;
    uint32_t owner = 0;
    int32_t leaf = 0;
    if (lane < n) {
        const uint32_t e = w->list[kClass][length - n + lane];
        owner = e & 31u;
        leaf = __ldg(sc.surf_leaf + (e >> 5));
        const double2 a = w->ray[0][owner], b = w->ray[1][owner], c = w->ray[2][owner];
        const double dist = leaf_distance<kIsect, kClass>(sc, leaf, mk(a.x, a.y, b.x),
                                                          mk(b.y, c.x, c.y));
        if (dist >= 0.0) {
            key = (unsigned long long)__double_as_longlong(dist);
            atomicMin(&w->key[owner], key);
        }
    }
    __syncwarp();
    const unsigned long long mine = w->key[lane];
    if (mine != l->key) {
        l->key = mine;
        l->tbest = (float)__longlong_as_double((long long)mine)*1.00001f + l->eps;
        w->leaf[lane] = kNoLeaf;
    }
    __syncwarp();
    if (key != kNoKey && key == w->key[owner]) atomicMin(&w->leaf[owner], leaf);
    __syncwarp();
}

// Works off the lists as long as one holds at least `least` leaves.
template <int kIsect>
__device__ __forceinline__ uint32_t work_off(const DevScene& sc, WalkWarp* w, int lane,
                                             uint32_t listed, int least, WalkLane* l) {
    int n = (int)(listed & 1023u);
    while (n >= least) {
        const int k = min(n, 32);
        intersect_listed<kIsect, kLeafCap>(sc, w, lane, n, k, l);
        n -= k;
    }
    int np = (int)(listed >> 10 & 1023u);
    while (np >= least) {
        const int k = min(np, 32);
        intersect_listed<kIsect, kLeafPlane>(sc, w, lane, np, k, l);
        np -= k;
    }
    int nq = (int)(listed >> 20);
    while (nq >= least) {
        const int k = min(nq, 32);
        intersect_listed<kIsect, kLeafQuadric>(sc, w, lane, nq, k, l);
        nq -= k;
    }
    return (uint32_t)n | (uint32_t)np << 10 | (uint32_t)nq << 20;
}

// One visit of every lane that walks; the groups of leaves reached join the
// queue.  Returns the groups queued.  All lanes of the warp call it, with
// fewer than 32 groups queued, up to kVisits times.
__device__ __forceinline__ int visit_nodes(const DevScene& sc, WalkWarp* w, uint32_t* stack,
                                           int lane, int groups, WalkLane* l) {
    uint2 group = make_uint2(0u, 0u);
    if (l->walking) group = walk_step(sc, l, stack);
    const unsigned reached = __ballot_sync(kFull, (group.x & 0xffu) != 0);
    if ((group.x & 0xffu) != 0)
        w->group[groups + __popc(reached & ((1u << lane) - 1u))] =
            make_uint2(group.x, group.y | (uint32_t)lane << 24);
    __syncwarp();
    return groups + __popc(reached);
}

// Intersects queued leaves while there are 32 groups, or 32 leaves of a
// kind; with `all`, every one.
template <int kIsect>
__device__ __forceinline__ void intersect_queued(const DevScene& sc, WalkWarp* w, int lane, bool all,
                                                 int* groups, uint32_t* listed, WalkLane* l) {
    while (*groups >= 32 || (all && (*groups | (int)*listed) != 0)) {
        *groups = spread_groups(w, lane, *groups, listed);
        *listed = work_off<kIsect>(sc, w, lane, *listed, all && *groups == 0 ? 1 : 32, l);
    }
}

// The closest hit in the frame subtree `root` by merlict's own walk of its
// bounding spheres (RayAndFrame.cpp:137-149), one thread by itself: inside a
// lens, or where there is no BVH.  The leaves it reaches are listed (in the
// caller's local array) and intersected together.
template <int kIsect>
__device__ __forceinline__ int32_t closest_hit_tree(const DevScene& sc, int32_t root, v3 s, v3 d,
                                                    double* distance) {
    constexpr int kList = 8;
    int32_t list[kList];
    int32_t best_leaf = kNoLeaf;
    double best = 0.0;
    const double sd = dot(s, d);
    int32_t i = root;
    const int32_t end = __ldg(&sc.node_meta[root].x);
    int n = 0;
    while (true) {
        while (i < end && n < kList) {
            const double2* np = reinterpret_cast<const double2*>(sc.node + i);
            const double2 n01 = __ldg(np), n23 = __ldg(np + 1);
            const int2 meta = __ldg(&sc.node_meta[i]);
            if (!sphere_cull(make_double4(n01.x, n01.y, n23.x, n23.y), s, d, sd)) {
                i = meta.x;
                continue;
            }
            if (meta.y >= 0) list[n++] = meta.y;
            i++;
        }
        for (int k = 0; k < n; k++) {
            const double dist = leaf_distance<kIsect, -1>(sc, list[k], s, d);
            if (dist >= 0.0 && (best_leaf == kNoLeaf || dist < best ||
                                (dist == best && list[k] < best_leaf))) {
                best = dist;
                best_leaf = list[k];
            }
        }
        n = 0;
        if (!(i < end)) break;
    }
    *distance = best;
    return best_leaf;
}

}  // namespace
}  // namespace mlgpu

#endif  // MLGPU_CLOSEST_HIT_CUH_
