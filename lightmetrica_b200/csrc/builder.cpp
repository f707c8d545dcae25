// Host scene builder. Compiled by g++ with -ffp-contract=off so that every
// float operation rounds separately, as in the reference's float SSE build.
//
// Reference algorithms restated here (own code, same steps):
//   vertex transform    Mat4f * Vec4f, math.matrix.inl:692-702
//   TriAccel::Load      triaccel.h:57-98
//   BVHScene::Build     scene.bvh.cpp:202-388 (12-bucket binned SAH, cost
//                       0.125 + (n1 A1 + n2 A2) / A, leaf if cost >= n and
//                       n <= 255, 1-triangle and degenerate-centroid leaves)
// The tree is built in parallel over subtrees; its shape does not depend on
// the threading (every node's split is a function of its triangle set only).
#include "builder.h"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cfloat>
#include <cstring>
#include <exception>
#include <functional>
#include <limits>
#include <mutex>
#include <system_error>
#include <thread>

namespace lmgpu {
namespace {

// _mm_min_ps / _mm_max_ps semantics (second operand unless strictly smaller).
inline float min_sse(float a, float b) { return a < b ? a : b; }
inline float max_sse(float a, float b) { return a > b ? a : b; }

inline HostAabb aabb_empty()
{
    HostAabb b;
    for (int i = 0; i < 3; i++) { b.mn[i] = FLT_MAX; b.mx[i] = -FLT_MAX; }
    return b;
}
inline void aabb_grow(HostAabb& a, const HostAabb& b)
{
    for (int i = 0; i < 3; i++) { a.mn[i] = min_sse(a.mn[i], b.mn[i]); a.mx[i] = max_sse(a.mx[i], b.mx[i]); }
}
inline void aabb_grow_p(HostAabb& a, const float* p)
{
    for (int i = 0; i < 3; i++) { a.mn[i] = min_sse(a.mn[i], p[i]); a.mx[i] = max_sse(a.mx[i], p[i]); }
}
inline float aabb_area(const HostAabb& b)
{
    float dx = b.mx[0] - b.mn[0], dy = b.mx[1] - b.mn[1], dz = b.mx[2] - b.mn[2];
    float s = dx * dy;
    s = s + dy * dz;
    s = s + dz * dx;
    return 2.0f * s;
}
inline int aabb_longest(const HostAabb& b)
{
    float dx = b.mx[0] - b.mn[0], dy = b.mx[1] - b.mn[1], dz = b.mx[2] - b.mn[2];
    return (dx > dy && dx > dz) ? 0 : (dy > dz ? 1 : 2);
}

// Column-major 4x4 times (x, y, z, 1) in the SSE order (c0 x + c1 y) + (c2 z + c3).
inline void xform_point(const float* m, const float* p, float* out)
{
    for (int r = 0; r < 3; r++) {
        float a = m[0 + r] * p[0];
        float b = m[4 + r] * p[1];
        float c = m[8 + r] * p[2];
        float d = m[12 + r] * 1.0f;
        float ab = a + b;
        float cd = c + d;
        out[r] = ab + cd;
    }
}

// TriAccel constants in the reference's evaluation order.
void load_triaccel(TriRecord& t, const float* A, const float* B, const float* C)
{
    static const int wald_modulo[4] = { 1, 2, 0, 1 };
    float b[3], c[3], N[3];
    for (int i = 0; i < 3; i++) { b[i] = C[i] - A[i]; c[i] = B[i] - A[i]; }
    N[0] = c[1] * b[2] - c[2] * b[1];
    N[1] = c[2] * b[0] - c[0] * b[2];
    N[2] = c[0] * b[1] - c[1] * b[0];
    uint32_t k = 0;
    for (int j = 0; j < 3; j++)
        if (std::fabs(N[j]) > std::fabs(N[k])) k = static_cast<uint32_t>(j);
    const int u = wald_modulo[k], v = wald_modulo[k + 1];
    const float n_k = N[k];
    const float denom = b[u] * c[v] - b[v] * c[u];
    std::memset(&t, 0, sizeof(t));
    if (denom == 0.0f) { t.k_flags = 3; return; }
    t.k_flags = k;
    t.n_u = N[u] / n_k;
    t.n_v = N[v] / n_k;
    float dot = A[0] * N[0] + A[1] * N[1];
    dot = dot + A[2] * N[2];
    t.n_d = dot / n_k;
    t.b_nu = b[u] / denom;
    t.b_nv = -b[v] / denom;
    t.a_u = A[u];
    t.a_v = A[v];
    t.c_nu = c[v] / denom;
    t.c_nv = -c[u] / denom;
}

struct Builder {
    BuiltScene& s;
    std::vector<HostAabb> tri_bounds;
    std::vector<float> centroids;
    std::vector<BuildNode> pool;
    std::atomic<int32_t> pool_next{0};
    std::atomic<int64_t> leaves{0};
    std::atomic<int32_t> depth{0};
    int spawn_depth = 0;

    explicit Builder(BuiltScene& out) : s(out) {}

    int32_t alloc_node() { return pool_next.fetch_add(1); }

    inline int bucket_of(int32_t tri, int axis, const HostAabb& cb) const
    {
        float c = centroids[3 * (size_t)tri + axis];
        float num = c - cb.mn[axis];
        float den = cb.mx[axis] - cb.mn[axis];
        float x = 12.0f * (num / den);
        int b = static_cast<int>(x);
        return b < 11 ? b : 11;
    }

    int32_t make_leaf(int begin, int end, const HostAabb& bound)
    {
        int32_t id = alloc_node();
        BuildNode& n = pool[id];
        n.leaf = true; n.begin = begin; n.end = end; n.bound = bound;
        leaves.fetch_add(1);
        return id;
    }

    int32_t build(int begin, int end, int d)
    {
        int32_t cur = depth.load();
        while (d > cur && !depth.compare_exchange_weak(cur, d)) {}
        int32_t* order = s.tri_order.data();
        HostAabb bound = aabb_empty();
        for (int i = begin; i < end; i++) aabb_grow(bound, tri_bounds[order[i]]);
        const int n = end - begin;
        if (n == 1) return make_leaf(begin, end, bound);

        HostAabb cb = aabb_empty();
        for (int i = begin; i < end; i++) aabb_grow_p(cb, &centroids[3 * (size_t)order[i]]);
        const int axis = aabb_longest(cb);
        if (cb.mn[axis] == cb.mx[axis]) return make_leaf(begin, end, bound);

        HostAabb bb[12];
        int bc[12];
        for (int i = 0; i < 12; i++) { bb[i] = aabb_empty(); bc[i] = 0; }
        for (int i = begin; i < end; i++) {
            const int32_t t = order[i];
            const int b = bucket_of(t, axis, cb);
            bc[b]++;
            aabb_grow(bb[b], tri_bounds[t]);
        }
        // Prefix/suffix sweeps give the same unions as the reference's
        // per-split loops: min/max are exact and order-independent.
        HostAabb left[11], right[11];
        int lc[11], rc[11];
        {
            HostAabb acc = aabb_empty(); int c = 0;
            for (int i = 0; i < 11; i++) { aabb_grow(acc, bb[i]); c += bc[i]; left[i] = acc; lc[i] = c; }
            acc = aabb_empty(); c = 0;
            for (int i = 11; i >= 1; i--) { aabb_grow(acc, bb[i]); c += bc[i]; right[i - 1] = acc; rc[i - 1] = c; }
        }
        const float area = aabb_area(bound);
        float costs[11];
        for (int i = 0; i < 11; i++) {
            float num = static_cast<float>(lc[i]) * aabb_area(left[i]) + static_cast<float>(rc[i]) * aabb_area(right[i]);
            costs[i] = 0.125f + num / area;
        }
        int min_idx = 0;
        double min_cost = costs[0];
        for (int i = 1; i < 11; i++)
            if (min_cost > costs[i]) { min_cost = costs[i]; min_idx = i; }

        if (min_cost < static_cast<float>(n) || n > 255) {
            // Two-pointer (Hoare) partition, the algorithm of std::partition
            // on bidirectional iterators: same leaf order as the reference.
            int first = begin, last = end;
            for (;;) {
                while (first != last && bucket_of(order[first], axis, cb) <= min_idx) ++first;
                if (first == last) break;
                --last;
                while (first != last && !(bucket_of(order[last], axis, cb) <= min_idx)) --last;
                if (first == last) break;
                std::swap(order[first], order[last]);
                ++first;
            }
            const int mid = first;
            int32_t l, r;
            if (d < spawn_depth && n > 4096) {
                int32_t lres = -1;
                std::thread th([&] { lres = build(begin, mid, d + 1); });
                r = build(mid, end, d + 1);
                th.join();
                l = lres;
            } else {
                l = build(begin, mid, d + 1);
                r = build(mid, end, d + 1);
            }
            int32_t id = alloc_node();
            BuildNode& nd = pool[id];
            nd.leaf = false; nd.axis = axis; nd.left = l; nd.right = r;
            nd.bound = pool[l].bound;
            aabb_grow(nd.bound, pool[r].bound);
            return id;
        }
        return make_leaf(begin, end, bound);
    }
};

// DFS pre-order flatten into Bvh2Node (internal nodes only).
int32_t flatten_bvh2(const std::vector<BuildNode>& nodes, int32_t ni, std::vector<Bvh2Node>& out)
{
    const BuildNode& n = nodes[ni];
    if (n.leaf) return ~n.begin;
    const int32_t id = static_cast<int32_t>(out.size());
    out.emplace_back();
    const BuildNode& L = nodes[n.left];
    const BuildNode& R = nodes[n.right];
    {
        Bvh2Node& o = out[id];
        o.bx[0] = L.bound.mn[0]; o.bx[1] = L.bound.mx[0]; o.bx[2] = R.bound.mn[0]; o.bx[3] = R.bound.mx[0];
        o.by[0] = L.bound.mn[1]; o.by[1] = L.bound.mx[1]; o.by[2] = R.bound.mn[1]; o.by[3] = R.bound.mx[1];
        o.bz[0] = L.bound.mn[2]; o.bz[1] = L.bound.mx[2]; o.bz[2] = R.bound.mn[2]; o.bz[3] = R.bound.mx[2];
        o.axis = n.axis;
        o.split = 0;
    }
    const int32_t l = flatten_bvh2(nodes, n.left, out);
    const int32_t r = flatten_bvh2(nodes, n.right, out);
    out[id].left = l;
    out[id].right = r;
    return id;
}

// ------------------------------------------------------------ render tree

// Render tree: binned SAH over all three axes (the reference bins only the
// longest axis of the centroid bounds, into 12 buckets), cost
// RTREE_NODE_COST + (nL AL + nR AR) / A in units of one triangle test
// against a leaf's n, leaves of at most RTREE_MAX_LEAF triangles (unless
// their centroids coincide).
#ifndef LMGPU_RTREE_BINS
#define LMGPU_RTREE_BINS 32
#endif
#ifndef LMGPU_RTREE_NODE_COST
#define LMGPU_RTREE_NODE_COST 0.5f    // a node visit costs about half a triangle test (measured)
#endif
#ifndef LMGPU_RTREE_MAX_LEAF
#define LMGPU_RTREE_MAX_LEAF 8
#endif

struct RenderBuilder {
    static constexpr int NB = LMGPU_RTREE_BINS;
    const std::vector<HostAabb>& tri_bounds;
    const std::vector<float>& centroids;
    std::vector<int32_t> order;
    std::vector<BuildNode> pool;
    std::atomic<int32_t> pool_next{0};
    std::atomic<int64_t> leaves{0};
    std::atomic<int32_t> depth{0};
    int spawn_depth = 0;

    RenderBuilder(const std::vector<HostAabb>& tb, const std::vector<float>& c) : tri_bounds(tb), centroids(c) {}

    int32_t alloc_node() { return pool_next.fetch_add(1); }

    int32_t make_leaf(int begin, int end, const HostAabb& bound)
    {
        int32_t id = alloc_node();
        BuildNode& n = pool[id];
        n.leaf = true; n.begin = begin; n.end = end; n.bound = bound;
        leaves.fetch_add(1);
        return id;
    }

    static int bin_of(float c, float lo, float scale)
    {
        const int b = static_cast<int>((c - lo) * scale);
        return b < 0 ? 0 : (b >= NB ? NB - 1 : b);
    }

    int32_t build(int begin, int end, int d)
    {
        int32_t cur = depth.load();
        while (d > cur && !depth.compare_exchange_weak(cur, d)) {}
        HostAabb bound = aabb_empty(), cb = aabb_empty();
        for (int i = begin; i < end; i++) {
            aabb_grow(bound, tri_bounds[order[i]]);
            aabb_grow_p(cb, &centroids[3 * (size_t)order[i]]);
        }
        const int n = end - begin;
        if (n == 1) return make_leaf(begin, end, bound);
        const float area = aabb_area(bound);
        float best = FLT_MAX;
        int best_axis = -1, best_bin = 0;
        for (int axis = 0; axis < 3; axis++) {
            const float lo = cb.mn[axis], ext = cb.mx[axis] - cb.mn[axis];
            if (!(ext > 0.0f)) continue;
            const float scale = float(NB) / ext;
            HostAabb bb[NB];
            int bc[NB];
            for (int i = 0; i < NB; i++) { bb[i] = aabb_empty(); bc[i] = 0; }
            for (int i = begin; i < end; i++) {
                const int32_t t = order[i];
                const int b = bin_of(centroids[3 * (size_t)t + axis], lo, scale);
                bc[b]++;
                aabb_grow(bb[b], tri_bounds[t]);
            }
            float right_area[NB];
            int right_count[NB];
            HostAabb acc = aabb_empty();
            int c = 0;
            for (int i = NB - 1; i >= 1; i--) {
                aabb_grow(acc, bb[i]);
                c += bc[i];
                right_area[i] = aabb_area(acc);
                right_count[i] = c;
            }
            acc = aabb_empty();
            c = 0;
            for (int i = 0; i < NB - 1; i++) {         // split after bin i
                aabb_grow(acc, bb[i]);
                c += bc[i];
                if (c == 0 || right_count[i + 1] == 0) continue;
                const float cost = LMGPU_RTREE_NODE_COST +
                                   (float(c) * aabb_area(acc) + float(right_count[i + 1]) * right_area[i + 1]) / area;
                if (cost < best) { best = cost; best_axis = axis; best_bin = i; }
            }
        }
        if (best_axis < 0 || (n <= LMGPU_RTREE_MAX_LEAF && float(n) <= best)) return make_leaf(begin, end, bound);
        const float lo = cb.mn[best_axis], scale = float(NB) / (cb.mx[best_axis] - cb.mn[best_axis]);
        int32_t* o = order.data();
        const int32_t* mid_ptr = std::partition(o + begin, o + end, [&](int32_t t) {
            return bin_of(centroids[3 * (size_t)t + best_axis], lo, scale) <= best_bin;
        });
        const int mid = static_cast<int>(mid_ptr - o);
        int32_t l, r;
        if (d < spawn_depth && n > 4096) {
            int32_t lres = -1;
            std::thread th([&] { lres = build(begin, mid, d + 1); });
            r = build(mid, end, d + 1);
            th.join();
            l = lres;
        } else {
            l = build(begin, mid, d + 1);
            r = build(mid, end, d + 1);
        }
        int32_t id = alloc_node();
        BuildNode& nd = pool[id];
        nd.leaf = false; nd.axis = best_axis; nd.left = l; nd.right = r;
        nd.bound = pool[l].bound;
        aabb_grow(nd.bound, pool[r].bound);
        return id;
    }
};

}  // namespace

// ------------------------------------------------------- 8-wide collapse

namespace {

// Cost model of the collapse: a wide node's visit costs 1, a triangle test
// BVH8_TRI_COST, weighted by surface area. A triangle test runs with few lanes
// active (about 6 of 32, against 22 in a node visit), which makes it as dear as a
// visit: 0.3, 0.6 and 1.0 gave 1.82, 1.65 and 1.60 ms for 2^23 random rays through a
// 1,048,576-triangle soup, 1.51, 1.48 and 1.47 ms for 5.3 M shadow rays of a
// 3.4 M-triangle terrain. Leaves of more than BVH8_MAX_LEAF triangles are not formed
// by merging (6: slower on both).
constexpr float BVH8_TRI_COST = 1.0f;
constexpr int BVH8_MAX_LEAF = 3;

struct Box {
    float lo[3], hi[3];
};
inline float half_area(const Box& b)
{
    const float dx = b.hi[0] - b.lo[0], dy = b.hi[1] - b.lo[1], dz = b.hi[2] - b.lo[2];
    return dx * dy + dy * dz + dz * dx;
}
inline void box_join(Box& a, const Box& b)
{
    for (int k = 0; k < 3; k++) { a.lo[k] = std::min(a.lo[k], b.lo[k]); a.hi[k] = std::max(a.hi[k], b.hi[k]); }
}
inline Box box_empty()
{
    return Box{ { FLT_MAX, FLT_MAX, FLT_MAX }, { -FLT_MAX, -FLT_MAX, -FLT_MAX } };
}

// fn(0) .. fn(n - 1) on up to `threads` threads; the first exception is
// rethrown once all have ended.
template <class Fn>
void parallel_for(int threads, size_t n, Fn fn)
{
    threads = static_cast<int>(std::min<size_t>((size_t)threads, n));
    std::atomic<size_t> next{0};
    std::exception_ptr failed;
    std::mutex mu;
    auto work = [&] {
        try {
            for (size_t i; (i = next.fetch_add(1)) < n;) fn(i);
        } catch (...) {
            std::lock_guard<std::mutex> lock(mu);
            if (!failed) failed = std::current_exception();
            next.store(n);
        }
    };
    std::vector<std::thread> pool;
    pool.reserve((size_t)std::max(threads, 1));
    try {
        for (int t = 1; t < threads; t++) pool.emplace_back(work);
    } catch (const std::system_error&) {
        // fewer threads than asked for
    }
    work();
    for (auto& t : pool) t.join();
    if (failed) std::rethrow_exception(failed);
}

// How far outside its triangle's bounding box a point that TriAccel::Intersect
// reports as hit can lie, for ray origins and triangles whose coordinates are at
// most B and M. With eps = 2^-24 and Wald's projection: the projected point
// (hu, hv) is off by e0 = 4 eps (B + 4M); the barycentrics by e0 times the row
// norms of the inverse edge matrix plus the relative error K of its float
// determinant (large for slivers); each of the three edge tests then lets the
// point out by that times the longest edge L, and the plane equation adds its own
// rounding and tilt.
double triaccel_slack(const float* A, const float* B_, const float* C, double B, double M)
{
    const double eps = std::ldexp(1.0, -24);
    double b[3], c[3], L = 0.0;
    for (int k = 0; k < 3; k++) {
        b[k] = (double)C[k] - A[k];
        c[k] = (double)B_[k] - A[k];
        L = std::max(L, std::max(std::fabs(b[k]), std::fabs(c[k])));
    }
    const double N[3] = { c[1] * b[2] - c[2] * b[1], c[2] * b[0] - c[0] * b[2], c[0] * b[1] - c[1] * b[0] };
    const double Nk = std::max(std::fabs(N[0]), std::max(std::fabs(N[1]), std::fabs(N[2])));
    const double base = 32.0 * eps * (B + 4.0 * M);
    if (!(Nk > 0.0)) return base + 2.0 * M;
    const double K = 16.0 * eps * L * L / Nk;
    const double delta = 4.0 * eps * (B + 4.0 * M) * (4.0 * L / Nk) + 4.0 * K + 16.0 * eps;
    return std::min(base + 9.0 * delta * L + 4.0 * K * L, 4.0 * M + base);
}

// The dynamic programme of the collapse (Ylitie et al. 2017, section 4.1) over a binary
// tree in DFS pre-order: cost[n][i - 1] is the least cost of node n's subtree
// as at most i children of some wide node, i = 1 .. 7.
struct Collapse {
    static constexpr int W = 8;
    const BuiltScene& s;
    const std::vector<Bvh2Node>& nodes;
    const std::vector<TriRecord>& tris;
    double magnitude = 0.0;
    bool exact = false;
    std::vector<int32_t> run;            // triangles of the leaf starting at a record
    std::vector<Box> record_box;         // per record (inflated when exact)
    std::vector<Box> box;                // per binary node (inflated when exact)
    std::vector<int32_t> count;          // triangles below
    std::vector<float> cost;             // W - 1 per node
    std::vector<uint8_t> split;          // W + 1 per node: slots of the left child when node takes j (0: takes j - 1)
    std::vector<uint8_t> leaf;           // the node's subtree becomes one leaf

    struct Item {
        int32_t ref;
        Box b;
    };

    Collapse(const BuiltScene& s_, const std::vector<Bvh2Node>& n, const std::vector<TriRecord>& t)
        : s(s_), nodes(n), tris(t) {}

    Box tri_box(const TriRecord& t) const
    {
        const float* p[3];
        for (int c = 0; c < 3; c++) p[c] = &s.positions[3 * (size_t)s.tri_vidx[3 * (size_t)t.tri_id + c]];
        Box b;
        const float e = exact ? (float)(triaccel_slack(p[0], p[1], p[2], magnitude, scene_max) * 1.001) : 0.0f;
        for (int k = 0; k < 3; k++) {
            b.lo[k] = std::min(p[0][k], std::min(p[1][k], p[2][k])) - e;
            b.hi[k] = std::max(p[0][k], std::max(p[1][k], p[2][k])) + e;
        }
        return b;
    }
    Item item(int32_t ref) const
    {
        if (ref >= 0) return Item{ ref, box[(size_t)ref] };
        Item it{ ref, box_empty() };
        for (size_t i = (size_t)~ref;; i++) {
            box_join(it.b, record_box[i]);
            if (tris[i].k_flags & TRI_LAST_IN_LEAF) break;
        }
        return it;
    }
    // Costs of a child as at most 1 .. 7 children.
    void costs_of(const Item& it, float* c) const
    {
        if (it.ref < 0) std::fill(c, c + (W - 1), half_area(it.b) * (float)run[(size_t)~it.ref] * BVH8_TRI_COST);
        else std::memcpy(c, &cost[(size_t)it.ref * (W - 1)], (W - 1) * sizeof(float));
    }
    void solve(size_t n)
    {
        const Item l = item(nodes[n].left), r = item(nodes[n].right);
        Box u = l.b;
        box_join(u, r.b);
        box[n] = u;
        count[n] = (l.ref < 0 ? run[(size_t)~l.ref] : count[(size_t)l.ref]) + (r.ref < 0 ? run[(size_t)~r.ref] : count[(size_t)r.ref]);
        const float area = half_area(u);
        float cl[W - 1], cr[W - 1], dist[W + 1];
        costs_of(l, cl);
        costs_of(r, cr);
        for (int j = 2; j <= W; j++) {
            float best = cl[0] + cr[j - 2];
            int at = 1;
            for (int k = 2; k < j; k++) {
                const float c = cl[k - 1] + cr[j - k - 1];
                if (c < best) { best = c; at = k; }
            }
            dist[j] = best;
            split[n * (W + 1) + (size_t)j] = (uint8_t)at;
        }
        const float inner = area + dist[W];
        const float as_leaf = count[n] <= BVH8_MAX_LEAF ? area * (float)count[n] * BVH8_TRI_COST : FLT_MAX;
        leaf[n] = as_leaf <= inner;
        float* c = &cost[n * (W - 1)];
        c[0] = std::min(as_leaf, inner);
        for (int j = 2; j < W; j++) {
            if (dist[j] < c[j - 2]) c[j - 1] = dist[j];
            else { c[j - 1] = c[j - 2]; split[n * (W + 1) + (size_t)j] = 0; }
        }
    }
    // Children of a wide node that give binary subtree `it` j slots.
    void gather(const Item& it, int j, Item* out, int& n) const
    {
        if (it.ref < 0) { out[n++] = it; return; }
        const uint8_t* sp = &split[(size_t)it.ref * (W + 1)];
        j = std::min(j, W - 1);
        while (j > 1 && sp[j] == 0) j--;
        if (j == 1) { out[n++] = it; return; }
        gather(item(nodes[(size_t)it.ref].left), sp[j], out, n);
        gather(item(nodes[(size_t)it.ref].right), j - sp[j], out, n);
    }
    bool is_leaf(const Item& it) const { return it.ref < 0 || leaf[(size_t)it.ref]; }
    void emit_tris(int32_t ref, std::vector<TriRecord>& out) const
    {
        if (ref >= 0) { emit_tris(nodes[(size_t)ref].left, out); emit_tris(nodes[(size_t)ref].right, out); return; }
        for (size_t i = (size_t)~ref;; i++) {
            out.push_back(tris[i]);
            out.back().k_flags &= ~TRI_LAST_IN_LEAF;
            if (tris[i].k_flags & TRI_LAST_IN_LEAF) return;
        }
    }
    double scene_max = 0.0;

    // Writes the wide node of binary subtree `ref` to `node`, its leaves to `out_tris`, and
    // returns its internal children in slot order. Indices are relative to
    // the lists' present sizes.
    struct Made {
        int32_t ref[W];
        int n = 0;
    };
    Made make(const Item* in, int n, Bvh8Node& node, std::vector<TriRecord>& out_tris, uint32_t child_base) const
    {
        Box u = box_empty();
        for (int i = 0; i < n; i++) box_join(u, in[i].b);
        // Greedy assignment of children to octant slots: the best remaining
        // (child, slot) pair by projection of the child's centre on the slot's diagonal.
        int slot_of[W], child_in[W];
        for (int i = 0; i < W; i++) { slot_of[i] = -1; child_in[i] = -1; }
        float toward[W][W];
        for (int i = 0; i < n; i++) {
            float cen[3];
            for (int k = 0; k < 3; k++) cen[k] = (in[i].b.lo[k] + in[i].b.hi[k]) - (u.lo[k] + u.hi[k]);
            for (int sl = 0; sl < W; sl++)
                toward[i][sl] = (sl & 1 ? cen[0] : -cen[0]) + (sl & 2 ? cen[1] : -cen[1]) + (sl & 4 ? cen[2] : -cen[2]);
        }
        for (int r = 0; r < n; r++) {
            float best = -FLT_MAX;
            int bi = -1, bs = -1;
            for (int i = 0; i < n; i++) {
                if (slot_of[i] >= 0) continue;
                for (int sl = 0; sl < W; sl++) {
                    if (child_in[sl] >= 0) continue;
                    if (bi < 0 || toward[i][sl] > best) { best = toward[i][sl]; bi = i; bs = sl; }
                }
            }
            slot_of[bi] = bs;
            child_in[bs] = bi;
        }
        std::memset(&node, 0, sizeof(node));
        // Grid: steps are powers of two, at least 16 ulps of the largest
        // magnitude, so that a visit's rounding stays inside the planes' margin.
        const double top = std::max(magnitude, scene_max);
        const double ulp = top > 0.0 ? std::ldexp(1.0, std::ilogb(top) - 23) : std::ldexp(1.0, -126);
        uint8_t q[6][W];
        uint32_t exps = 0;
        for (int k = 0; k < 3; k++) {
            const double extra = 4.0 * ulp;
            const double need = std::max(16.0 * ulp, ((double)u.hi[k] - u.lo[k] + 2.0 * extra) / 253.0);
            int E = std::ilogb(need);
            if (std::ldexp(1.0, E) < need) E++;
            E = std::min(std::max(E, -126), 127);
            const double step = std::ldexp(1.0, E), inv_step = std::ldexp(1.0, -E);
            const double m = extra + step / 64.0;
            const double od = (double)u.lo[k] - m - step / 64.0;
            float of = (float)od;
            if ((double)of > od) of = std::nextafter(of, -std::numeric_limits<float>::infinity());
            node.origin[k] = of;
            for (int sl = 0; sl < W; sl++) {
                q[k][sl] = 255;          // an unused slot: lo > hi
                q[3 + k][sl] = 0;
                if (child_in[sl] < 0) continue;
                const Box& b = in[child_in[sl]].b;
                // (both quotients are in [0, 255]: truncation is the floor)
                q[k][sl] = (uint8_t)std::min(255.0, std::max(0.0, ((double)b.lo[k] - m - of) * inv_step));
                const double hi = std::min(255.0, std::max(0.0, ((double)b.hi[k] + m - of) * inv_step));
                q[3 + k][sl] = (uint8_t)((double)(int)hi < hi ? (int)hi + 1 : (int)hi);
            }
            exps |= (uint32_t)(E + 127) << (8 * k);
        }
        Made made;
        uint32_t inner = 0;
        for (int sl = 0; sl < W; sl++) {
            if (child_in[sl] < 0) continue;
            const Item& it = in[child_in[sl]];
            node.valid |= 1u << sl;
            if (!is_leaf(it)) {
                inner |= 1u << sl;
                made.ref[made.n++] = it.ref;
            } else {
                node.start[sl] = (uint32_t)out_tris.size();
                emit_tris(it.ref, out_tris);
                out_tris.back().k_flags |= TRI_LAST_IN_LEAF;
            }
        }
        node.exps = exps | inner << 24;
        node.child_base = child_base;
        std::memcpy(node.lox, q[0], W); std::memcpy(node.loy, q[1], W); std::memcpy(node.loz, q[2], W);
        std::memcpy(node.hix, q[3], W); std::memcpy(node.hiy, q[4], W); std::memcpy(node.hiz, q[5], W);
        return made;
    }
    Made make_from(int32_t ref, Bvh8Node& node, std::vector<TriRecord>& out_tris, uint32_t child_base) const
    {
        Item in[W];
        int n = 0;
        const int k = split[(size_t)ref * (W + 1) + W];
        gather(item(nodes[(size_t)ref].left), k, in, n);
        gather(item(nodes[(size_t)ref].right), W - k, in, n);
        return make(in, n, node, out_tris, child_base);
    }
    // Depth-first emission below the wide node already made at out.nodes[0].
    struct Todo {
        size_t at;
        int32_t ref;
        int depth;
    };
    void emit(std::vector<Todo> stack, Bvh8Tree& out) const
    {
        while (!stack.empty()) {
            const Todo t = stack.back();
            stack.pop_back();
            out.depth = std::max(out.depth, t.depth);
            Bvh8Node node;
            const size_t base = out.nodes.size();
            const Made m = make_from(t.ref, node, out.tris, (uint32_t)base);
            out.nodes[t.at] = node;
            out.nodes.resize(base + (size_t)m.n);
            for (int i = m.n - 1; i >= 0; i--) stack.push_back(Todo{ base + (size_t)i, m.ref[i], t.depth + 1 });
        }
    }
};

}  // namespace

void set_splits(std::vector<Bvh2Node>& nodes)
{
    std::vector<int32_t> first(nodes.size());         // pre-order: children follow their parent
    for (size_t i = nodes.size(); i-- > 0;) {
        auto begin = [&](int32_t ref) { return ref < 0 ? ~ref : first[(size_t)ref]; };
        first[i] = begin(nodes[i].left);
        nodes[i].split = begin(nodes[i].right);
    }
}

void collapse_bvh8(const BuiltScene& s, const std::vector<Bvh2Node>& nodes, const std::vector<TriRecord>& tris,
                   int32_t root, const float* root_box, double magnitude, bool exact, int threads,
                   Bvh8Tree& out)
{
    out = Bvh8Tree{};
    if (tris.empty()) return;
    if (threads <= 0) threads = static_cast<int>(std::max(1u, std::thread::hardware_concurrency()));
    Collapse C(s, nodes, tris);
    C.exact = exact;
    C.magnitude = magnitude;
    for (int k = 0; k < 3; k++)
        C.scene_max = std::max(C.scene_max, std::max((double)std::fabs(s.bounds.mn[k]), (double)std::fabs(s.bounds.mx[k])));
    if (tris.size() < 8192) threads = 1;
    C.record_box.resize(tris.size());
    const size_t chunk = 16384;
    parallel_for(threads, (tris.size() + chunk - 1) / chunk, [&](size_t t) {
        for (size_t i = t * chunk; i < std::min(tris.size(), (t + 1) * chunk); i++) C.record_box[i] = C.tri_box(tris[i]);
    });
    C.run.assign(tris.size(), 0);
    for (size_t i = 0, first = 0; i < tris.size(); i++)
        if (tris[i].k_flags & TRI_LAST_IN_LEAF) { C.run[first] = (int32_t)(i + 1 - first); first = i + 1; }
    if (root < 0) {                                   // one leaf
        out.nodes.resize(1);
        const Collapse::Item it = C.item(root);
        C.make(&it, 1, out.nodes[0], out.tris, 1);
        out.depth = 1;
    } else {
        const size_t n = nodes.size();
        C.box.resize(n);
        C.count.resize(n);
        C.cost.resize(n * (Collapse::W - 1));
        C.split.assign(n * (Collapse::W + 1), 0);
        C.leaf.resize(n);
        // Pre-order: a subtree is the index range [ref, end). Subtrees of at most
        // n / 64 nodes are solved in parallel, the nodes above them afterwards.
        struct Range { size_t at, end; };
        std::vector<Range> tasks;
        std::vector<size_t> above;
        std::vector<Range> open{ Range{ (size_t)root, n } };
        while (!open.empty()) {
            const Range r = open.back();
            open.pop_back();
            if (r.end - r.at <= std::max<size_t>(n / 64, 1024)) { tasks.push_back(r); continue; }
            above.push_back(r.at);
            const int32_t l = nodes[r.at].left, rt = nodes[r.at].right;
            if (l >= 0) open.push_back(Range{ (size_t)l, rt >= 0 ? (size_t)rt : r.end });
            if (rt >= 0) open.push_back(Range{ (size_t)rt, r.end });
        }
        parallel_for(threads, tasks.size(), [&](size_t t) {
            for (size_t i = tasks[t].end; i-- > tasks[t].at;) C.solve(i);
        });
        std::sort(above.begin(), above.end());
        for (size_t i = above.size(); i-- > 0;) C.solve(above[i]);
        // The top of the wide tree breadth first until there are enough subtrees
        // to share among the threads; each subtree's nodes and triangles then
        // follow in one block.
        std::vector<Collapse::Todo> front{ Collapse::Todo{ 0, root, 1 } };
        out.nodes.resize(1);
        const size_t want = threads > 1 ? 4 * (size_t)threads : 0;
        for (size_t head = 0; head < front.size() && front.size() - head < want;) {
            const Collapse::Todo t = front[head++];
            Bvh8Node node;
            const size_t base = out.nodes.size();
            const Collapse::Made m = C.make_from(t.ref, node, out.tris, (uint32_t)base);
            out.nodes[t.at] = node;
            out.nodes.resize(base + (size_t)m.n);
            out.depth = std::max(out.depth, t.depth);
            for (int i = 0; i < m.n; i++) front.push_back(Collapse::Todo{ base + (size_t)i, m.ref[i], t.depth + 1 });
            if (head == front.size() || front.size() - head >= want) {
                front.erase(front.begin(), front.begin() + (ptrdiff_t)head);
                break;
            }
        }
        std::vector<Bvh8Tree> part(front.size());
        parallel_for(threads, front.size(), [&](size_t t) {
            part[t].nodes.resize(1);
            C.emit({ Collapse::Todo{ 0, front[t].ref, front[t].depth } }, part[t]);
        });
        for (size_t t = 0; t < part.size(); t++) {
            // Local node 0 is the front node itself; node i > 0 lands at base + i - 1.
            const uint32_t node_base = (uint32_t)out.nodes.size() - 1, tri_base = (uint32_t)out.tris.size();
            for (Bvh8Node& x : part[t].nodes) {
                x.child_base += node_base;
                for (int sl = 0; sl < Collapse::W; sl++)
                    if ((x.valid & ~(x.exps >> 24)) >> sl & 1u) x.start[sl] += tri_base;
            }
            out.nodes[front[t].at] = part[t].nodes[0];
            out.nodes.insert(out.nodes.end(), part[t].nodes.begin() + 1, part[t].nodes.end());
            out.tris.insert(out.tris.end(), part[t].tris.begin(), part[t].tris.end());
            out.depth = std::max(out.depth, part[t].depth);
            part[t] = Bvh8Tree{};
        }
    }
    std::vector<LeafBox> by_id(tris.size());
    auto put = [&](int32_t ref, const float* x, const float* y, const float* z) {
        LeafBox b{ { x[0], y[0], z[0] }, { x[1], y[1], z[1] }, { 0.0f, 0.0f } };
        for (size_t i = (size_t)~ref;; i++) {
            by_id[tris[i].tri_id] = b;
            if (tris[i].k_flags & TRI_LAST_IN_LEAF) break;
        }
    };
    if (root < 0) {
        const float x[2] = { root_box[0], root_box[3] }, y[2] = { root_box[1], root_box[4] }, z[2] = { root_box[2], root_box[5] };
        put(root, x, y, z);
    }
    for (const Bvh2Node& n : nodes) {
        if (n.left < 0) put(n.left, n.bx, n.by, n.bz);
        if (n.right < 0) put(n.right, n.bx + 2, n.by + 2, n.bz + 2);
    }
    out.boxes.resize(tris.size());
    parallel_for(threads, (tris.size() + chunk - 1) / chunk, [&](size_t t) {
        for (size_t i = t * chunk; i < std::min(tris.size(), (t + 1) * chunk); i++) out.boxes[i] = by_id[out.tris[i].tri_id];
    });
}

void build_render_tree(BuiltScene& s, int threads)
{
    auto t0 = std::chrono::steady_clock::now();
    const int64_t ntris = s.num_tris;
    if (ntris <= 0) return;
    std::vector<HostAabb> tb((size_t)ntris);
    std::vector<float> cen(3 * (size_t)ntris);
    for (int64_t t = 0; t < ntris; t++) {
        const float* p1 = &s.positions[3 * (size_t)s.tri_vidx[3 * t]];
        const float* p2 = &s.positions[3 * (size_t)s.tri_vidx[3 * t + 1]];
        const float* p3 = &s.positions[3 * (size_t)s.tri_vidx[3 * t + 2]];
        HostAabb b;
        for (int c = 0; c < 3; c++) { b.mn[c] = min_sse(p1[c], p2[c]); b.mx[c] = max_sse(p1[c], p2[c]); }
        aabb_grow_p(b, p3);
        tb[(size_t)t] = b;
        for (int c = 0; c < 3; c++) cen[3 * (size_t)t + c] = (b.mn[c] + b.mx[c]) * 0.5f;
    }
    RenderBuilder B(tb, cen);
    B.order.resize((size_t)ntris);
    for (int64_t t = 0; t < ntris; t++) B.order[(size_t)t] = static_cast<int32_t>(t);
    if (threads <= 0) threads = static_cast<int>(std::max(1u, std::thread::hardware_concurrency()));
    while ((1 << B.spawn_depth) < threads) B.spawn_depth++;
    B.spawn_depth += 1;
    B.pool.resize(2 * (size_t)ntris);
    const int32_t root = B.build(0, static_cast<int32_t>(ntris), 0);
    B.pool.resize((size_t)B.pool_next.load());
    // Records in the render tree's leaf order: the same TriAccel constants.
    std::vector<TriRecord> by_id((size_t)ntris);
    for (int64_t i = 0; i < ntris; i++) by_id[s.tris[(size_t)i].tri_id] = s.tris[(size_t)i];
    s.rtris.resize((size_t)ntris);
    for (int64_t i = 0; i < ntris; i++) {
        s.rtris[(size_t)i] = by_id[(size_t)B.order[(size_t)i]];
        s.rtris[(size_t)i].k_flags &= ~TRI_LAST_IN_LEAF;
    }
    for (auto& n : B.pool)
        if (n.leaf) s.rtris[(size_t)(n.end - 1)].k_flags |= TRI_LAST_IN_LEAF;
    s.rbvh2.clear();
    s.rbvh2.reserve((size_t)std::max<int64_t>(1, ntris));
    s.rbvh2_root = flatten_bvh2(B.pool, root, s.rbvh2);
    const HostAabb& rb = B.pool[root].bound;
    for (int c = 0; c < 3; c++) { s.rroot_box[c] = rb.mn[c]; s.rroot_box[3 + c] = rb.mx[c]; }
    s.rnum_nodes = (int64_t)B.pool.size();
    s.rnum_leaves = B.leaves.load();
    s.rmax_depth = B.depth.load();
    s.has_render_tree = true;
    s.rbuild_seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
}

std::string build_scene(const std::vector<PrimitiveInput>& prims, int threads, bool want_bvh, BuiltScene& s)
{
    auto t0 = std::chrono::steady_clock::now();
    static const float identity[16] = { 1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1 };

    // ---- world-space geometry and TriAccel records (primitive-major order)
    int64_t ntris = 0, nverts = 0;
    for (auto& p : prims) {
        if (p.num_faces < 0 || p.num_vertices < 0) return "negative primitive size";
        if (p.num_faces > 0 && (!p.positions || !p.faces)) return "primitive without positions or faces";
        ntris += p.num_faces;
        nverts += p.num_vertices;
    }
    if (ntris >= (int64_t(1) << 31) - 1) return "too many triangles";
    s.num_tris = ntris;
    s.positions.resize(3 * (size_t)nverts);
    s.normals.resize(3 * (size_t)nverts);
    s.texcoords.assign(2 * (size_t)nverts, 0.0f);
    s.tri_vidx.resize(3 * (size_t)ntris);
    s.tri_prim.resize((size_t)ntris);
    s.has_uv.resize(prims.size());
    std::vector<TriRecord> ta((size_t)ntris);
    s.bounds = aabb_empty();

    int64_t vbase = 0, tbase = 0;
    for (size_t pi = 0; pi < prims.size(); pi++) {
        const PrimitiveInput& p = prims[pi];
        const float* m = p.transform ? p.transform : identity;
        s.has_uv[pi] = p.texcoords != nullptr;
        // Normal transform: transpose(inverse(M)) upper 3x3 (primitive.h:42-44).
        double inv[9];
        {
            const double a = m[0], b = m[4], c = m[8], d = m[1], e = m[5], f = m[9], g = m[2], h = m[6], i = m[10];
            const double det = a * (e * i - f * h) - b * (d * i - f * g) + c * (d * h - e * g);
            const double id = det != 0.0 ? 1.0 / det : 0.0;
            // inverse (row-major r,c) then transposed => normal matrix N[r][c] = inv[c][r]
            const double I[3][3] = {
                { (e * i - f * h) * id, (c * h - b * i) * id, (b * f - c * e) * id },
                { (f * g - d * i) * id, (a * i - c * g) * id, (c * d - a * f) * id },
                { (d * h - e * g) * id, (b * g - a * h) * id, (a * e - b * d) * id } };
            for (int r = 0; r < 3; r++)
                for (int c2 = 0; c2 < 3; c2++) inv[3 * r + c2] = I[c2][r];
        }
        for (int v = 0; v < p.num_vertices; v++) {
            float w[3];
            xform_point(m, p.positions + 3 * (size_t)v, w);
            std::memcpy(&s.positions[3 * (size_t)(vbase + v)], w, sizeof(w));
            float nn[3] = { 0, 0, 0 };
            if (p.normals) {
                const float* n0 = p.normals + 3 * (size_t)v;
                for (int r = 0; r < 3; r++)
                    nn[r] = static_cast<float>(inv[3 * r] * n0[0] + inv[3 * r + 1] * n0[1] + inv[3 * r + 2] * n0[2]);
            }
            std::memcpy(&s.normals[3 * (size_t)(vbase + v)], nn, sizeof(nn));
            if (p.texcoords) {
                s.texcoords[2 * (size_t)(vbase + v)] = p.texcoords[2 * (size_t)v];
                s.texcoords[2 * (size_t)(vbase + v) + 1] = p.texcoords[2 * (size_t)v + 1];
            }
        }
        for (int f = 0; f < p.num_faces; f++) {
            const int64_t t = tbase + f;
            uint32_t vi[3];
            for (int c = 0; c < 3; c++) {
                vi[c] = p.faces[3 * (size_t)f + c];
                if ((int64_t)vi[c] >= p.num_vertices) return "face index out of range";
                s.tri_vidx[3 * (size_t)t + c] = static_cast<uint32_t>(vbase + vi[c]);
            }
            s.tri_prim[(size_t)t] = static_cast<int32_t>(pi);
            const float* A = &s.positions[3 * (size_t)(vbase + vi[0])];
            const float* B = &s.positions[3 * (size_t)(vbase + vi[1])];
            const float* C = &s.positions[3 * (size_t)(vbase + vi[2])];
            load_triaccel(ta[(size_t)t], A, B, C);
            ta[(size_t)t].tri_id = static_cast<uint32_t>(t);
            ta[(size_t)t].prim = static_cast<uint32_t>(pi);
            // Geometric normal stands in for missing vertex normals.
            if (!p.normals) {
                float e1[3], e2[3], g[3];
                for (int c = 0; c < 3; c++) { e1[c] = B[c] - A[c]; e2[c] = C[c] - A[c]; }
                g[0] = e1[1] * e2[2] - e1[2] * e2[1];
                g[1] = e1[2] * e2[0] - e1[0] * e2[2];
                g[2] = e1[0] * e2[1] - e1[1] * e2[0];
                for (int c = 0; c < 3; c++)
                    for (int k = 0; k < 3; k++) s.normals[3 * (size_t)(vbase + vi[c]) + k] = g[k];
            }
        }
        vbase += p.num_vertices;
        tbase += p.num_faces;
    }

    // ---- bounds, centroids, BVH
    Builder B(s);
    B.tri_bounds.resize((size_t)ntris);
    B.centroids.resize(3 * (size_t)ntris);
    s.tri_order.resize((size_t)ntris);
    for (int64_t t = 0; t < ntris; t++) {
        const float* p1 = &s.positions[3 * (size_t)s.tri_vidx[3 * t]];
        const float* p2 = &s.positions[3 * (size_t)s.tri_vidx[3 * t + 1]];
        const float* p3 = &s.positions[3 * (size_t)s.tri_vidx[3 * t + 2]];
        HostAabb tb;
        for (int c = 0; c < 3; c++) { tb.mn[c] = min_sse(p1[c], p2[c]); tb.mx[c] = max_sse(p1[c], p2[c]); }
        aabb_grow_p(tb, p3);
        aabb_grow(s.bounds, tb);
        B.tri_bounds[(size_t)t] = tb;
        for (int c = 0; c < 3; c++) B.centroids[3 * (size_t)t + c] = (tb.mn[c] + tb.mx[c]) * 0.5f;
        s.tri_order[(size_t)t] = static_cast<int32_t>(t);
    }

    if (threads <= 0) threads = static_cast<int>(std::max(1u, std::thread::hardware_concurrency()));
    while ((1 << B.spawn_depth) < threads) B.spawn_depth++;
    B.spawn_depth += 1;

    if (want_bvh && ntris > 0) {
        B.pool.resize(2 * (size_t)ntris);
        const int32_t root = B.build(0, static_cast<int32_t>(ntris), 0);
        B.pool.resize((size_t)B.pool_next.load());
        s.nodes.swap(B.pool);
        s.root = root;
        s.num_leaves = B.leaves.load();
        s.max_depth = B.depth.load();
    }

    // ---- device layouts
    s.tris.resize((size_t)ntris);
    for (int64_t i = 0; i < ntris; i++) s.tris[(size_t)i] = ta[(size_t)s.tri_order[(size_t)i]];
    if (want_bvh && ntris > 0) {
        for (auto& n : s.nodes)
            if (n.leaf) s.tris[(size_t)(n.end - 1)].k_flags |= TRI_LAST_IN_LEAF;
        s.bvh2.reserve((size_t)std::max<int64_t>(1, ntris));
        s.bvh2_root = flatten_bvh2(s.nodes, s.root, s.bvh2);
        const HostAabb& rb = s.nodes[s.root].bound;
        for (int c = 0; c < 3; c++) { s.root_box[c] = rb.mn[c]; s.root_box[3 + c] = rb.mx[c]; }
        s.max_stack = s.max_depth + 2;
    } else if (ntris > 0) {
        s.tris[(size_t)(ntris - 1)].k_flags |= TRI_LAST_IN_LEAF;
    }
    s.build_seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    return std::string();
}

}  // namespace lmgpu
