// Host-side checks of the surface BVH the closest-hit walk uses
// (csrc/bvh_build.cu, csrc/closest_hit.cuh), built by
// tests/test_surface_bvh.py with the host compiler: every leaf with geometry
// is one leaf slot of one node, every index a walk follows is in range, the
// tree is no deeper than its stated levels; and the walk, with the kernel's
// single-precision arithmetic, reaches the leaf a ray is known to hit.
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "mlgpu_internal.h"

using mlgpu::SurfBvhHost;
using mlgpu::SurfNode;

namespace {

float bits(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }

// Leaf slots whose boxes the ray meets, as the kernel tests them.
void candidates(const SurfBvhHost& b, const double* s, const double* d, float eps,
                std::vector<uint32_t>* out) {
    float o[3], iv[3], w = eps;
    for (int a = 0; a < 3; a++) {
        o[a] = (float)s[a];
        float f = (float)d[a];
        if (std::fabs(f) < mlgpu::kMinDirection) f = std::copysign(mlgpu::kMinDirection, f);
        iv[a] = 1.0f/f;
    }
    w = eps + 4e-7f*(std::fabs(o[0]) + std::fabs(o[1]) + std::fabs(o[2]));
    std::vector<uint32_t> stack = {0};
    while (!stack.empty()) {
        const SurfNode& n = b.nodes[stack.back()];
        stack.pop_back();
        const uint32_t leaves = n.leaf_base_mask & 0xff, nodes = n.exps_nodes >> 24;
        uint32_t rank = 0;
        for (int k = 0; k < 8; k++) {
            float tmin = 0.0f, tmax = INFINITY;
            for (int a = 0; a < 3; a++) {
                const float S = bits(((n.exps_nodes >> (8*a)) & 0xff) << 23)*iv[a];
                const float L = std::fma(-32768.0f, S, (n.origin[a] - o[a])*iv[a]);
                const float W = w*std::fabs(iv[a]);
                const float ql = 32768.0f + (float)((n.qlo[a][k >> 2] >> (8*(k & 3))) & 0xff);
                const float qh = 32768.0f + (float)((n.qhi[a][k >> 2] >> (8*(k & 3))) & 0xff);
                const bool back = iv[a] < 0.0f;   // as the kernel: -0 is a negative direction
                const float x = std::fma(back ? qh : ql, S, L - W), y = std::fma(back ? ql : qh, S, L + W);
                tmin = std::fmax(tmin, x);
                tmax = std::fmin(tmax, y);
            }
            const bool hit = tmin <= tmax;
            if ((leaves >> k) & 1) {
                if (hit) out->push_back((n.leaf_base_mask >> 8) + rank);
                rank++;
            } else if (((nodes >> k) & 1) && hit) {
                stack.push_back(n.child_base + k);
            }
        }
    }
}

}  // namespace

// Violations; info = {nodes, leaves, levels}.
extern "C" int64_t surface_bvh_invariants(const mlgpu_flat_scene* f, int64_t* info) {
    SurfBvhHost b;
    mlgpu::build_surface_bvh(f, &b);
    info[0] = (int64_t)b.nodes.size();
    info[1] = (int64_t)b.leaf_ids.size();
    info[2] = b.levels;
    int64_t bad = 0;
    std::vector<int32_t> seen(b.leaf_ids.size() + 1, 0);
    struct Item { uint32_t node; int level; };
    std::vector<Item> todo;
    if (b.levels) todo.push_back({0, 1});
    while (!todo.empty()) {
        const Item it = todo.back();
        todo.pop_back();
        if (it.node >= b.nodes.size() || it.level > b.levels) { bad++; continue; }
        const SurfNode& n = b.nodes[it.node];
        const uint32_t leaves = n.leaf_base_mask & 0xff, nodes = n.exps_nodes >> 24;
        if (leaves & nodes) bad++;
        uint32_t slot = n.leaf_base_mask >> 8;
        for (int k = 0; k < 8; k++) {
            if ((leaves >> k) & 1) {
                if (slot >= b.leaf_ids.size()) { bad++; continue; }
                seen[slot++]++;
            }
            if ((nodes >> k) & 1) todo.push_back({n.child_base + (uint32_t)k, it.level + 1});
        }
    }
    std::vector<int32_t> of_leaf(f->num_leaves > 0 ? f->num_leaves : 1, 0);
    for (size_t j = 0; j < b.leaf_ids.size(); j++) {
        if (seen[j] != 1) bad++;
        if (b.leaf_ids[j] < 0 || b.leaf_ids[j] >= f->num_leaves) bad++;
        else of_leaf[b.leaf_ids[j]]++;
    }
    if (b.levels)
        for (int32_t l = 0; l < f->num_leaves; l++)
            if (of_leaf[l] != (f->leaf_primitive[l] != MLGPU_PRIM_NONE ? 1 : 0)) bad++;
    return bad;
}

// Of n rays (support, unit direction, the leaf each hits first or -1), those
// whose leaf the walk does not reach.  visits += leaves reached.
extern "C" int64_t surface_bvh_misses(const mlgpu_flat_scene* f, int64_t n, const double* s,
                                      const double* d, const int32_t* leaf, int64_t* visits) {
    SurfBvhHost b;
    mlgpu::build_surface_bvh(f, &b);
    const double* root = f->node_sphere;
    const double extent = std::fabs(root[0]) + std::fabs(root[1]) + std::fabs(root[2]) + 2.0*root[3];
    const float eps = (float)(1e-6 + 4e-7*extent);
    int64_t missed = 0;
    std::vector<uint32_t> c;
    for (int64_t i = 0; i < n; i++) {
        if (leaf[i] < 0) continue;
        c.clear();
        candidates(b, s + 3*i, d + 3*i, eps, &c);
        *visits += (int64_t)c.size();
        bool found = false;
        for (uint32_t j : c) found = found || b.leaf_ids[j] == leaf[i];
        if (!found) missed++;
    }
    return missed;
}
