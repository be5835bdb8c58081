// bvh_build.cu -- host-side construction of the 8-wide bounding-volume
// hierarchy the tracers use to find candidate leaves in the world tree.
//
// merlict finds candidates by walking its own frame tree, whose octant
// clustering (merlict/Frame.cpp:190-255) gives heavily overlapping bounding
// spheres: ~400 sphere tests per photon in the light-field telescope.  The
// tracers instead walk a BVH built here by binned surface-area-heuristic
// splits over the leaves' bounding spheres, collapsed to eight children per
// node.  The BVH only proposes candidates; every candidate is then put
// through merlict's own bounding-sphere test of that leaf and merlict's
// intersection, and ties are broken in merlict's visiting order, so the
// closest hit is merlict's.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <vector>

#include "mlgpu_internal.h"

namespace mlgpu {
namespace {

struct Box {
    double lo[3] = {DBL_MAX, DBL_MAX, DBL_MAX};
    double hi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
    void grow(const Box& b) {
        for (int k = 0; k < 3; k++) {
            lo[k] = std::min(lo[k], b.lo[k]);
            hi[k] = std::max(hi[k], b.hi[k]);
        }
    }
    void grow(const double* p) {
        for (int k = 0; k < 3; k++) {
            lo[k] = std::min(lo[k], p[k]);
            hi[k] = std::max(hi[k], p[k]);
        }
    }
    double area() const {
        if (hi[0] < lo[0]) return 0.0;
        const double dx = hi[0] - lo[0], dy = hi[1] - lo[1], dz = hi[2] - lo[2];
        return 2.0*(dx*dy + dy*dz + dz*dx);
    }
};

struct BNode {            // binary build node
    Box box;
    int32_t left = -1, right = -1;
    int32_t begin = 0, end = 0;   // leaf range when left < 0
};

constexpr int kLeafMax = 4;   // leaves of a leaf range (sphere BVH)
constexpr int kBins = 16;

class Builder {
 public:
    int leaf_max = kLeafMax;
    std::vector<Box> prim_box;
    std::vector<double> centroid;   // 3 per primitive
    std::vector<int32_t> order;     // permutation of primitive ids
    std::vector<BNode> nodes;

    int32_t build(int32_t begin, int32_t end, int depth) {
        const int32_t id = (int32_t)nodes.size();
        nodes.emplace_back();
        Box box, cbox;
        for (int32_t i = begin; i < end; i++) {
            box.grow(prim_box[order[i]]);
            cbox.grow(&centroid[3*(size_t)order[i]]);
        }
        nodes[id].box = box;
        const int32_t n = end - begin;
        if (n <= leaf_max) {
            nodes[id].begin = begin;
            nodes[id].end = end;
            return id;
        }
        int axis = 0;
        double ext = -1.0;
        for (int k = 0; k < 3; k++)
            if (cbox.hi[k] - cbox.lo[k] > ext) { ext = cbox.hi[k] - cbox.lo[k]; axis = k; }
        int32_t mid = begin + n/2;
        if (ext > 0.0 && depth <= 40) {
            Box bin_box[kBins];
            int32_t bin_count[kBins] = {0};
            const double scale = kBins/ext;
            auto bin_of = [&](int32_t p) {
                int b = (int)((centroid[3*(size_t)p + axis] - cbox.lo[axis])*scale);
                return std::min(std::max(b, 0), kBins - 1);
            };
            for (int32_t i = begin; i < end; i++) {
                const int b = bin_of(order[i]);
                bin_count[b]++;
                bin_box[b].grow(prim_box[order[i]]);
            }
            double best = DBL_MAX;
            int best_split = -1;
            for (int s = 1; s < kBins; s++) {
                Box l, r;
                int32_t nl = 0, nr = 0;
                for (int b = 0; b < s; b++) { if (bin_count[b]) { l.grow(bin_box[b]); nl += bin_count[b]; } }
                for (int b = s; b < kBins; b++) { if (bin_count[b]) { r.grow(bin_box[b]); nr += bin_count[b]; } }
                if (!nl || !nr) continue;
                const double cost = l.area()*nl + r.area()*nr;
                if (cost < best) { best = cost; best_split = s; }
            }
            if (best_split > 0) {
                int32_t* first = order.data() + begin;
                int32_t* last = order.data() + end;
                int32_t* m = std::partition(first, last, [&](int32_t p) { return bin_of(p) < best_split; });
                mid = (int32_t)(m - order.data());
                if (mid == begin || mid == end) mid = begin + n/2;
            } else {
                std::sort(order.begin() + begin, order.begin() + end, [&](int32_t a, int32_t b) {
                    return centroid[3*(size_t)a + axis] < centroid[3*(size_t)b + axis];
                });
            }
        }
        const int32_t l = build(begin, mid, depth + 1);
        const int32_t r = build(mid, end, depth + 1);
        nodes[id].left = l;
        nodes[id].right = r;
        return id;
    }
};

float round_down(double x) {
    float f = (float)x;
    if ((double)f > x) f = std::nextafter(f, -FLT_MAX);
    return f;
}
float round_up(double x) {
    float f = (float)x;
    if ((double)f < x) f = std::nextafter(f, FLT_MAX);
    return f;
}

}  // namespace

// Builds the BVH of all leaves with geometry.  `inflate` widens every leaf
// box (absolute, metres) so that single-precision slab tests stay
// conservative.
void build_bvh(const mlgpu_flat_scene* f, double inflate, BvhHost* out) {
    out->nodes.clear();
    out->leaf_ids.clear();
    out->levels = 0;
    Builder b;
    for (int32_t l = 0; l < f->num_leaves; l++) {
        if (f->leaf_primitive[l] == MLGPU_PRIM_NONE) continue;
        const double* c = f->node_sphere + 4*(size_t)f->leaf_node[l];
        Box box;
        const double r = c[3] + inflate;
        for (int k = 0; k < 3; k++) { box.lo[k] = c[k] - r; box.hi[k] = c[k] + r; }
        b.prim_box.push_back(box);
        b.centroid.push_back(c[0]);
        b.centroid.push_back(c[1]);
        b.centroid.push_back(c[2]);
        out->leaf_ids.push_back(l);
    }
    const int32_t n = (int32_t)out->leaf_ids.size();
    if (n == 0) return;
    b.order.resize(n);
    for (int32_t i = 0; i < n; i++) b.order[i] = i;
    b.nodes.reserve(2*(size_t)n);
    b.build(0, n, 0);
    // primitive order of the leaf ranges
    std::vector<int32_t> ids(n);
    for (int32_t i = 0; i < n; i++) ids[i] = out->leaf_ids[b.order[i]];
    out->leaf_ids.swap(ids);

    // collapse to kBvhWidth-wide nodes, breadth first from the root
    std::vector<int32_t> queue = {0};
    std::vector<int32_t> wide_of(b.nodes.size(), -1);
    std::vector<int32_t> level = {0};   // per wide node
    wide_of[0] = 0;
    out->nodes.emplace_back();
    out->levels = 1;
    for (size_t qi = 0; qi < queue.size(); qi++) {
        const int32_t bn = queue[qi];
        const int32_t w = wide_of[bn];
        std::vector<int32_t> kids;
        if (b.nodes[bn].left < 0) {
            kids.push_back(bn);   // a root that is a leaf
        } else {
            kids.push_back(b.nodes[bn].left);
            kids.push_back(b.nodes[bn].right);
            while (kids.size() < (size_t)kBvhWidth) {
                int best = -1;
                double area = -1.0;
                for (size_t k = 0; k < kids.size(); k++) {
                    const BNode& c = b.nodes[kids[k]];
                    if (c.left >= 0 && c.box.area() > area) { area = c.box.area(); best = (int)k; }
                }
                if (best < 0) break;
                const BNode c = b.nodes[kids[best]];
                kids[best] = c.left;
                kids.push_back(c.right);
            }
        }
        BvhNode node;
        std::memset(&node, 0, sizeof(node));
        for (int k = 0; k < kBvhWidth; k++) {
            node.lo[0][k] = 1.0f; node.hi[0][k] = -1.0f;   // empty slot never hits
            node.lo[1][k] = 1.0f; node.hi[1][k] = -1.0f;
            node.lo[2][k] = 1.0f; node.hi[2][k] = -1.0f;
            node.child[k] = kBvhEmpty;
        }
        for (size_t k = 0; k < kids.size(); k++) {
            const BNode& c = b.nodes[kids[k]];
            for (int a = 0; a < 3; a++) {
                node.lo[a][k] = round_down(c.box.lo[a]);
                node.hi[a][k] = round_up(c.box.hi[a]);
            }
            if (c.left < 0) {
                const int32_t count = c.end - c.begin;
                node.child[k] = kBvhLeafFlag | (c.begin << 3) | (count - 1);
            } else {
                const int32_t idx = (int32_t)out->nodes.size();
                out->nodes.emplace_back();
                level.push_back(level[w] + 1);
                out->levels = std::max(out->levels, level[w] + 2);
                wide_of[kids[k]] = idx;
                queue.push_back(kids[k]);
                node.child[k] = idx;
            }
        }
        out->nodes[w] = node;
    }
    // nodes were numbered in breadth-first order, so each level is a range
    out->level_start.assign((size_t)out->levels + 1, (int32_t)out->nodes.size());
    for (int32_t i = (int32_t)level.size() - 1; i >= 0; i--) out->level_start[level[i]] = i;
    out->level_start[0] = 0;
}

// Quantises a node's float boxes (already rounded outwards) to QNode: per
// axis the origin is the smallest low bound and the step the smallest power
// of two with 255 steps reaching the largest high bound; each bound is
// rounded outwards to whole steps.  origin + q * 2^e is evaluated in double,
// where it is exact for the magnitudes a scenery has, and each bound is
// checked against the float box it stands for.
void quantise_bvh_node(const BvhNode& n, QNode* q) {
    std::memset(q, 0, sizeof(*q));
    uint32_t exps = 0;
    for (int a = 0; a < 3; a++) {
        float lo = FLT_MAX, hi = -FLT_MAX;
        for (int k = 0; k < kBvhWidth; k++) {
            if (n.child[k] == kBvhEmpty) continue;
            lo = std::min(lo, n.lo[a][k]);
            hi = std::max(hi, n.hi[a][k]);
        }
        if (lo > hi) { lo = 0.0f; hi = 0.0f; }   // no children (not built)
        const double ext = (double)hi - (double)lo;
        int e = -126;                            // the smallest normal step
        while (e < 127 && std::ldexp(255.0, e) < ext) e++;
        const double step = std::ldexp(1.0, e);
        q->origin[a] = lo;
        exps |= (uint32_t)(e + 127) << (8*a);
        for (int k = 0; k < kBvhWidth; k++) {
            uint32_t ql = 0, qh = 0;
            if (n.child[k] != kBvhEmpty) {
                double l = std::floor(((double)n.lo[a][k] - (double)lo)/step);
                double h = std::ceil(((double)n.hi[a][k] - (double)lo)/step);
                l = std::min(std::max(l, 0.0), 255.0);
                h = std::min(std::max(h, 0.0), 255.0);
                while (l > 0.0 && (double)lo + l*step > (double)n.lo[a][k]) l -= 1.0;
                while (h < 255.0 && (double)lo + h*step < (double)n.hi[a][k]) h += 1.0;
                ql = (uint32_t)l;
                qh = (uint32_t)h;
            }
            q->qlo[a][k >> 2] |= ql << (8*(k & 3));
            q->qhi[a][k >> 2] |= qh << (8*(k & 3));
        }
    }
    q->exps = exps;
    for (int k = 0; k < kBvhWidth; k++) q->child[k] = n.child[k];
}

namespace {

// ---- the surface BVH ------------------------------------------------------

// World box of every point at which merlict's intersection of leaf l can
// report a hit (scenery/primitive/*.cpp): the bounds of the primitive in its
// own frame, turned into the world.  A spherical cap's hits lie on its
// sphere, inside its prism and inside the bounding sphere, |p|^2 = 2 R z <=
// r^2, so z is in [0, r^2 / (2 R)]; the plane family's hits lie in z = 0.
// Where that does not bound the hits -- a primitive without such bounds, a
// triangle so thin that its sign tests are rounding noise, values that are
// not finite -- the box of the bounding sphere stands in: merlict tests a
// leaf only for rays that pass it (RayAndFrame.cpp:137-149).  The box is
// widened by 1e-5 of the leaf's radius, a hundred times the rounding of the
// single-precision form's local coordinates.
bool corners_box(const double* T, const std::vector<double>& xy, double z0, double z1, Box* box) {
    for (size_t i = 0; i + 1 < xy.size(); i += 2)
        for (int e = 0; e < 2; e++) {
            const double x = xy[i], y = xy[i + 1], z = e ? z1 : z0;
            double w[3];
            for (int a = 0; a < 3; a++) {
                w[a] = T[4*a]*x + T[4*a + 1]*y + T[4*a + 2]*z + T[4*a + 3];
                if (!std::isfinite(w[a])) return false;
            }
            box->grow(w);
        }
    return !xy.empty();
}

void rectangle(double x0, double x1, double y0, double y1, std::vector<double>* xy) {
    *xy = {x0, y0, x1, y0, x0, y1, x1, y1};
}

// The corners of the hexagonal prism |u.p|, |v.p|, |w.p| < inner; none if
// the three directions do not bound a region of the plane.
void hexagon(const mlgpu_flat_scene* f, double inner, std::vector<double>* xy) {
    const double* u[3] = {f->hex_unit_u, f->hex_unit_v, f->hex_unit_w};
    for (int i = 0; i < 3; i++)
        if (!(std::fabs(u[i][2]) < 1e-9)) return;
    // two of the slabs bound a parallelogram; the third only cuts it, so its
    // corners count where they are inside (with a margin)
    for (int i = 0; i < 3; i++)
        for (int j = i + 1; j < 3; j++) {
            const double det = u[i][0]*u[j][1] - u[i][1]*u[j][0];
            if (!(std::fabs(det) > 0.1)) { xy->clear(); return; }
            for (int s = 0; s < 4; s++) {
                const double p = s & 1 ? inner : -inner, q = s & 2 ? inner : -inner;
                const double x = (p*u[j][1] - q*u[i][1])/det, y = (u[i][0]*q - u[j][0]*p)/det;
                const int k = 3 - i - j;
                if (std::fabs(u[k][0]*x + u[k][1]*y) <= inner*(1.0 + 1e-6)) {
                    xy->push_back(x);
                    xy->push_back(y);
                }
            }
        }
}

Box surface_box(const mlgpu_flat_scene* f, int32_t l) {
    const double* c = f->node_sphere + 4*(size_t)f->leaf_node[l];
    const double* T = f->leaf_frame2world + 12*(size_t)l;
    const double* p = f->leaf_params + MLGPU_LEAF_PARAMS*(size_t)l;
    const double r = c[3];
    double z0 = 0.0, z1 = 0.0;
    std::vector<double> xy;
    switch (f->leaf_primitive[l]) {
    case MLGPU_PRIM_SPHERE_CAP_HEX:
    case MLGPU_PRIM_SPHERE_CAP_CYL:
    case MLGPU_PRIM_SPHERE_CAP_RECT:
        if (!(p[0] > 0.0)) break;
        z1 = std::min(r, r*r/(2.0*p[0]));
        if (f->leaf_primitive[l] == MLGPU_PRIM_SPHERE_CAP_HEX) hexagon(f, p[1], &xy);
        else if (f->leaf_primitive[l] == MLGPU_PRIM_SPHERE_CAP_CYL)
            rectangle(-std::sqrt(p[1]), std::sqrt(p[1]), -std::sqrt(p[1]), std::sqrt(p[1]), &xy);
        else rectangle(-p[1], p[1], -p[2], p[2], &xy);
        break;
    case MLGPU_PRIM_DISC:
    case MLGPU_PRIM_ANNULUS: {
        const double o = std::sqrt(p[0]);
        rectangle(-o, o, -o, o, &xy);
        break;
    }
    case MLGPU_PRIM_HEX_PLANE: hexagon(f, p[0], &xy); break;
    case MLGPU_PRIM_PLANE: rectangle(-p[0], p[0], -p[1], p[1], &xy); break;
    case MLGPU_PRIM_PLANE_DUAL_SPHERE: {
        const double o = std::fabs(p[4]);
        rectangle(std::max(p[0], p[2]) - o, std::min(p[0], p[2]) + o,
                  std::max(p[1], p[3]) - o, std::min(p[1], p[3]) + o, &xy);
        break;
    }
    case MLGPU_PRIM_TRIANGLE: {
        const double ax = p[2] - p[0], ay = p[3] - p[1], bx = p[4] - p[0], by = p[5] - p[1];
        const double cx = bx - ax, cy = by - ay;
        const double longest = std::max(ax*ax + ay*ay, std::max(bx*bx + by*by, cx*cx + cy*cy));
        if (std::fabs(ax*by - ay*bx) > 1e-5*longest) xy = {p[0], p[1], p[2], p[3], p[4], p[5]};
        break;
    }
    case MLGPU_PRIM_CYLINDER:
        rectangle(-std::fabs(p[0]), std::fabs(p[0]), -std::fabs(p[0]), std::fabs(p[0]), &xy);
        z0 = -0.5*std::fabs(p[1]);
        z1 = 0.5*std::fabs(p[1]);
        break;
    default: break;
    }
    Box box;
    if (!corners_box(T, xy, z0, z1, &box)) {
        box = Box();
        for (int k = 0; k < 3; k++) { box.lo[k] = c[k] - r; box.hi[k] = c[k] + r; }
    }
    for (int k = 0; k < 3; k++) { box.lo[k] -= 1e-5*r; box.hi[k] += 1e-5*r; }
    return box;
}

// The binary tree's subtrees gathered into nodes of eight so that the sum
// of the nodes' surface areas -- the expected node visits of a random ray --
// is least (the dynamic program of Ylitie, Karras and Laine, HPG 2017, with
// leaves free): forest[n][i] = least cost of node n as at most i subtrees.
struct Collapse {
    const std::vector<BNode>& b;
    std::vector<double> cost;        // [node][9]
    std::vector<int8_t> left;        // [node][9]: subtrees the left child takes; 0: itself

    explicit Collapse(const std::vector<BNode>& nodes)
        : b(nodes), cost(9*nodes.size(), 0.0), left(9*nodes.size(), 0) {
        for (size_t n = b.size(); n-- > 0;) {      // children have higher indices
            if (b[n].left < 0) continue;
            const double* l = &cost[9*(size_t)b[n].left];
            const double* r = &cost[9*(size_t)b[n].right];
            double* c = &cost[9*n];
            int8_t* s = &left[9*n];
            double split[9];
            int8_t at[9];
            for (int i = 2; i <= 8; i++) {
                split[i] = DBL_MAX;
                at[i] = 1;
                for (int j = 1; j < i; j++)
                    if (l[j] + r[i - j] < split[i]) { split[i] = l[j] + r[i - j]; at[i] = (int8_t)j; }
            }
            c[1] = split[8] + b[n].box.area();
            s[0] = at[8];                          // of the node's own eight
            for (int i = 2; i <= 8; i++) {
                const bool open = split[i] < c[i - 1];
                c[i] = open ? split[i] : c[i - 1];
                s[i] = open ? at[i] : -1;          // -1: as with i - 1
            }
        }
    }
    void subtrees(int32_t n, int i, std::vector<int32_t>* out) const {
        while (i > 1 && b[n].left >= 0 && left[9*(size_t)n + i] < 0) i--;
        if (i == 1 || b[n].left < 0) { out->push_back(n); return; }
        const int j = left[9*(size_t)n + i];
        subtrees(b[n].left, j, out);
        subtrees(b[n].right, i - j, out);
    }
    void children(int32_t n, std::vector<int32_t>* out) const {
        if (b[n].left < 0) { out->push_back(n); return; }   // a root that is a leaf
        const int j = left[9*(size_t)n];
        subtrees(b[n].left, j, out);
        subtrees(b[n].right, 8 - j, out);
    }
};

// Slots for a node's children: the pair of child and slot that agree best,
// the offset of the child's centre along the slot's diagonal, first.
void octant_slots(const std::vector<BNode>& b, const std::vector<int32_t>& kids,
                  int32_t slot_of[kBvhWidth]) {
    Box all;
    for (int32_t k : kids) all.grow(b[k].box);
    bool taken[kBvhWidth] = {}, placed[kBvhWidth] = {};
    for (size_t round = 0; round < kids.size(); round++) {
        double best = -DBL_MAX;
        int bk = -1, bs = -1;
        for (size_t k = 0; k < kids.size(); k++) {
            if (placed[k]) continue;
            for (int s = 0; s < kBvhWidth; s++) {
                if (taken[s]) continue;
                double v = 0.0;
                for (int a = 0; a < 3; a++) {
                    const Box& c = b[kids[k]].box;
                    const double off = 0.5*(c.lo[a] + c.hi[a]) - 0.5*(all.lo[a] + all.hi[a]);
                    v += (s >> a) & 1 ? off : -off;
                }
                if (v > best || bk < 0) { best = v; bk = (int)k; bs = s; }
            }
        }
        slot_of[bk] = bs;
        placed[bk] = true;
        taken[bs] = true;
    }
}

}  // namespace

void build_surface_bvh(const mlgpu_flat_scene* f, SurfBvhHost* out) {
    *out = SurfBvhHost();
    Builder b;
    b.leaf_max = 1;
    std::vector<int32_t> ids;
    for (int32_t l = 0; l < f->num_leaves; l++) {
        if (f->leaf_primitive[l] == MLGPU_PRIM_NONE) continue;
        const Box box = surface_box(f, l);
        for (int k = 0; k < 3; k++) {
            if (!(std::isfinite(box.lo[k]) && std::isfinite(box.hi[k]))) return;
            b.centroid.push_back(0.5*(box.lo[k] + box.hi[k]));
        }
        b.prim_box.push_back(box);
        ids.push_back(l);
    }
    const int32_t n = (int32_t)ids.size();
    if (n == 0) return;
    b.order.resize(n);
    for (int32_t i = 0; i < n; i++) b.order[i] = i;
    b.nodes.reserve(2*(size_t)n);
    b.build(0, n, 0);
    for (int k = 0; k < 3; k++)
        if (b.nodes[0].box.hi[k] - b.nodes[0].box.lo[k] > kMaxSurfExtent) return;
    const Collapse collapse(b.nodes);
    struct Item { int32_t binary; size_t wide; int level; };
    std::vector<Item> queue = {{0, 0, 1}};
    out->nodes.emplace_back();
    for (size_t qi = 0; qi < queue.size(); qi++) {
        const Item it = queue[qi];
        out->levels = std::max(out->levels, it.level);
        std::vector<int32_t> kids;
        collapse.children(it.binary, &kids);
        int32_t slot_of[kBvhWidth];
        octant_slots(b.nodes, kids, slot_of);
        int32_t kid_in[kBvhWidth];
        for (int s = 0; s < kBvhWidth; s++) kid_in[s] = -1;
        for (size_t k = 0; k < kids.size(); k++) kid_in[slot_of[k]] = kids[k];
        BvhNode box;
        std::memset(&box, 0, sizeof(box));
        uint32_t nodes = 0, leaves = 0, caps = 0, planes = 0;
        const size_t leaf_base = out->leaf_ids.size();
        for (int s = 0; s < kBvhWidth; s++) {
            box.child[s] = kid_in[s] < 0 ? kBvhEmpty : 0;
            if (kid_in[s] < 0) continue;
            const BNode& c = b.nodes[kid_in[s]];
            for (int a = 0; a < 3; a++) {
                box.lo[a][s] = round_down(c.box.lo[a]);
                box.hi[a][s] = round_up(c.box.hi[a]);
            }
            if (c.left < 0) {
                leaves |= 1u << s;
                const int32_t l = ids[b.order[c.begin]];
                const int cls = leaf_class(f->leaf_primitive[l]);
                if (cls == kLeafCap) caps |= 1u << s;
                if (cls == kLeafPlane) planes |= 1u << s;
                out->leaf_ids.push_back(l);
            } else {
                nodes |= 1u << s;
            }
        }
        // the walk's arithmetic rounds by 2^-9 of a quantisation step, which is
        // at most 2/255 of the node's extent: widen by four times that
        for (int a = 0; a < 3; a++) {
            double lo = DBL_MAX, hi = -DBL_MAX;
            for (int s = 0; s < kBvhWidth; s++) {
                if (kid_in[s] < 0) continue;
                lo = std::min(lo, (double)box.lo[a][s]);
                hi = std::max(hi, (double)box.hi[a][s]);
            }
            const double m = 6.2e-5*(hi - lo);
            for (int s = 0; s < kBvhWidth; s++) {
                if (kid_in[s] < 0) continue;
                box.lo[a][s] = round_down((double)box.lo[a][s] - m);
                box.hi[a][s] = round_up((double)box.hi[a][s] + m);
            }
        }
        const size_t child_base = out->nodes.size();
        if (nodes) {
            // up to the last slot that is a node
            int last = kBvhWidth - 1;
            while (!((nodes >> last) & 1u)) last--;
            out->nodes.resize(child_base + last + 1, SurfNode{});
            for (int s = 0; s <= last; s++)
                if ((nodes >> s) & 1u) queue.push_back({kid_in[s], child_base + s, it.level + 1});
        }
        QNode q;
        quantise_bvh_node(box, &q);
        SurfNode w = {};
        for (int a = 0; a < 3; a++) {
            w.origin[a] = q.origin[a];
            for (int g = 0; g < 2; g++) { w.qlo[a][g] = q.qlo[a][g]; w.qhi[a][g] = q.qhi[a][g]; }
        }
        w.exps_nodes = q.exps | (nodes << 24);
        w.child_base = (uint32_t)child_base;
        w.leaf_base_mask = (uint32_t)leaf_base << 8 | leaves;
        w.leaf_kinds = caps | planes << 8 | leaves << 16;
        out->nodes[it.wide] = w;
    }
    // 24-bit node and leaf indices, a stack entry per level
    if (out->nodes.size() >= (1u << 24) || out->leaf_ids.size() >= (1u << 24) ||
        out->levels > kMaxSurfLevels)
        *out = SurfBvhHost();
}

}  // namespace mlgpu
