// Traversal of the 8-wide compressed tree (Bvh8Node): the box test of a
// node's eight children, the renders' candidate rule and the exact walk's certificate.
//
// A visit is about 250 instructions a warp, half of them on the ALU pipe (48 byte
// permutes turn plane bytes into floats, 32 three-input min/max). On the first three
// bounces of a 1080p frame 24, 19 and 18 of 32 lanes are active; the walk issues on 82, 75
// and 70 % of cycles, its ALU pipe is busy on 73, 61 and 56 % and L1's data pipe on 55, 78
// and 82 %; DRAM on 3 to 4 %. It replaces the binary tree's visits (64-byte nodes as four
// 16-byte loads, L1 at 83 % of its wavefront peak on the bounce rays of a 3.4 M-triangle
// terrain): 38 visits of a bounce ray became 14.6, each of three 32-byte loads. Measured,
// binary -> 8-wide (one B200, render arithmetic): 2^23 random rays through a 1,048,576-triangle soup
// 2.97 -> 1.60 ms (exact, with the certificate below: 3.17 -> 2.32 ms);
// on the terrain 8.3 M camera rays 1.52 -> 1.44 ms, 5.3 M bounce rays
// 1.98 -> 1.51 ms, 5.3 M shadow rays 2.30 -> 1.47 ms. Float planes (224-byte nodes)
// took 2.5 / 2.2 ms on the soup / bounce rays, a 4-wide node of 8-bit planes
// 2.0 / 1.54 ms.
#pragma once
#include <type_traits>
#include "scene.cuh"
#include "trace.cuh"

namespace lmgpu {

// 32 bytes of read-only data by one load (sm_100).
struct Words8 { uint32_t w[8]; };
__device__ __forceinline__ Words8 load32(const void* p)
{
    Words8 v;
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]), "=r"(v.w[4]), "=r"(v.w[5]), "=r"(v.w[6]), "=r"(v.w[7])
        : "l"(p));
    return v;
}

// Byte B of `word` as the float 2^15 + byte: one byte permute puts it into the
// second mantissa byte under the exponent of 2^15. The 2^15 * step / d this adds is
// taken off the axis' bias, which rounds that at 2^-9 of a grid step, inside the
// margin of step / 64 that collapse_bvh8 leaves.
template <int B>
__device__ __forceinline__ float plane_byte(uint32_t word)
{
    return __uint_as_float(__byte_perm(word, 0x47000000u, 0x7404 | (B << 4)));
}

// One lane's walk: the group of deferred children it is in (bits 0-7 of mask: hit
// internal children still to visit, nearest first at bit 0; bits 8-15: which slots
// are internal) and the leaves found (bit s of leaves: slot s of leaf_node).
struct Walk8 {
    uint32_t base, mask;
    uint32_t leaf_node, leaves;
    int sp;
};

__device__ __forceinline__ void walk8_begin(Walk8& w, uint32_t oct)
{
    // The root as slot 0 of a group of one: child index popc(0) = 0.
    w.base = 0;
    w.mask = (1u << oct) | (1u << 8);
    w.leaves = 0;
    w.sp = 0;
}

// Visit order is slot ^ oct: exchanges the bits of an 8-bit slot mask so.
__device__ __forceinline__ uint32_t order_mask(uint32_t m, uint32_t oct)
{
    if (oct & 1u) m = ((m & 0x55u) << 1) | ((m >> 1) & 0x55u);
    if (oct & 2u) m = ((m & 0x33u) << 2) | ((m >> 2) & 0x33u);
    if (oct & 4u) m = ((m & 0x0fu) << 4) | ((m >> 4) & 0x0fu);
    return m;
}

// Takes the nearest child of the current group (which has one) and returns its node.
__device__ __forceinline__ uint32_t walk8_next(Walk8& w, uint32_t oct)
{
    const uint32_t slot = (uint32_t)(__ffs(w.mask) - 1) ^ oct;
    w.mask &= w.mask - 1;
    return w.base + __popc((w.mask >> 8) & ((1u << slot) - 1u));
}

// Tests the eight child boxes of `node` against the ray's [tmin, tmax]: sets the
// group of hit internal children and the hit leaves (`w.leaves` must be empty).
// A ray made by setup_ray<true>; oct = the signs of its direction.
__device__ __forceinline__ void walk8_visit(Walk8& w, const Bvh8Node* __restrict__ nodes, uint32_t node,
                                            const TraversalRay& r, uint32_t oct)
{
    const char* p = reinterpret_cast<const char*>(nodes + node);
    const Words8 h = load32(p), a = load32(p + 32), b = load32(p + 64);
    const float sx = __uint_as_float((h.w[3] << 23) & 0x7f800000u) * r.inv_min[0];
    const float sy = __uint_as_float((h.w[3] << 15) & 0x7f800000u) * r.inv_min[1];
    const float sz = __uint_as_float((h.w[3] << 7) & 0x7f800000u) * r.inv_min[2];
    const float bx = fmaf(-32768.0f, sx, fmaf(__uint_as_float(h.w[0]), r.inv_min[0], r.inv_max[0]));
    const float by = fmaf(-32768.0f, sy, fmaf(__uint_as_float(h.w[1]), r.inv_min[1], r.inv_max[1]));
    const float bz = fmaf(-32768.0f, sz, fmaf(__uint_as_float(h.w[2]), r.inv_min[2], r.inv_max[2]));
    const bool nx = oct & 1u, ny = oct & 2u, nz = oct & 4u;
    uint32_t miss = 0;
#pragma unroll
    for (int q = 1; q >= 0; q--) {
        const uint32_t lx = a.w[q], ly = a.w[2 + q], lz = a.w[4 + q], ux = a.w[6 + q], uy = b.w[q], uz = b.w[2 + q];
        const uint32_t near_x = nx ? ux : lx, far_x = nx ? lx : ux;
        const uint32_t near_y = ny ? uy : ly, far_y = ny ? ly : uy;
        const uint32_t near_z = nz ? uz : lz, far_z = nz ? lz : uz;
        auto child = [&](auto B) {
            constexpr int I = decltype(B)::value;
            float x0, x1, y0, y1, z0, z1;
            fma_pair(plane_byte<I>(near_x), plane_byte<I>(far_x), sx, bx, x0, x1);
            fma_pair(plane_byte<I>(near_y), plane_byte<I>(far_y), sy, by, y0, y1);
            fma_pair(plane_byte<I>(near_z), plane_byte<I>(far_z), sz, bz, z0, z1);
            const float tn = fmaxf(fmaxf(x0, y0), fmaxf(z0, r.tmin));
            const float tf = fminf(fminf(x1, y1), fminf(z1, r.tmax));
            miss = __funnelshift_l(__float_as_uint(tf - tn), miss, 1);   // shifts in the sign: 1 = entry after exit
        };
        child(std::integral_constant<int, 3>{});
        child(std::integral_constant<int, 2>{});
        child(std::integral_constant<int, 1>{});
        child(std::integral_constant<int, 0>{});
    }
    const uint32_t hit = ~miss & h.w[5], inner = h.w[3] >> 24;
    w.base = h.w[4];
    w.mask = order_mask(hit & inner, oct) | (inner << 8);
    w.leaf_node = node;
    w.leaves = hit & ~inner;
}

// First record of the next hit leaf.
__device__ __forceinline__ const float4* walk8_leaf(const Bvh8Node* __restrict__ nodes, const TriRecord* __restrict__ tris,
                                                    uint32_t node, uint32_t& leaves)
{
    const uint32_t slot = (uint32_t)(__ffs(leaves) - 1);
    leaves &= leaves - 1;
    return reinterpret_cast<const float4*>(tris + __ldg(&nodes[node].start[slot]));
}

// ------------------------------------------------------- candidate hits ----

// A render ray's hit is the one that a near-first walk of the binary tree through its
// float boxes finds. That walk enters a leaf only before the closest hit so far, so its answer
// depends on its order where a box is entered no sooner than its triangle's t: flat boxes
// are, by rounding, and rays within rounding of a shared edge hit both its triangles. So a
// hit has a window, from its t to the entry of its leaf's box if that is later (looked at near
// an edge only). The hit whose window ends first wins; of windows that end together, the
// binary walk's order decides (order_takes). This is a total order of a ray's hits: the answer
// depends on neither the nodes' width and rounding nor the warp's other rays. (With the wide
// walk's own order in its place, waves and one-thread passes, which walk the binary tree, gave
// albedo gradients of a 36,864-triangle Cornell box 1.4e-4 apart, now 4e-6. The frame takes
// 0.3 % longer, the six-scene batch 0.8 %.)
// Without the box test, the triangle test's rounding reports hits just outside a triangle that
// 8-bit boxes let through and float boxes do not (far from the origin, many). A hit well
// inside its triangle is well inside the box, so that only hits near an edge are tested
// (DeviceScene::box_margin). On every
// hit the test takes the 1080p frame from 13.15 to 13.70 ms; near edges only it costs 2 %
// (frame, six-scene batch and terrain alike).

// Entry distance of a box, in the arithmetic of render rays (multiply-adds).
__device__ __forceinline__ float box_entry(float lox, float hix, float loy, float hiy, float loz, float hiz, const TraversalRay& r)
{
    float x0, x1, y0, y1, z0, z1;
    fma_pair(lox, hix, r.inv_min[0], r.inv_max[0], x0, x1);
    fma_pair(loy, hiy, r.inv_min[1], r.inv_max[1], y0, y1);
    fma_pair(loz, hiz, r.inv_min[2], r.inv_max[2], z0, z1);
    return fmaxf(fmaxf(fminf(x0, x1), fminf(y0, y1)), fminf(z0, z1));
}

// The slab test of the record's binary leaf box in the same arithmetic.
__device__ __forceinline__ bool leaf_box_render(const LeafBox* __restrict__ boxes, int64_t at, const TraversalRay& r, float& te)
{
    const float4 a = __ldg(reinterpret_cast<const float4*>(boxes + at));
    const float4 b = __ldg(reinterpret_cast<const float4*>(boxes + at) + 1);
    return slab_render(r, a.x, a.w, a.y, b.x, a.z, b.y, te);
}

// Of two hits whose windows end at the same distance `end`, whether triangle b's (at tb) is the
// binary walk's answer rather than a's (at ta): the one visited later, if its leaf is entered
// before that, else the one visited first; in one leaf the nearer, of equal t the later record.
// Where the two paths part, the child entered later comes later, the right one if both are
// entered at once.
__device__ __forceinline__ bool order_takes(const Bvh2Node* __restrict__ nodes, const int32_t* __restrict__ pos, int32_t root,
                                            int32_t a, int32_t b, float ta, float tb, float end, const TraversalRay& r)
{
    const int32_t pa = __ldg(pos + a), pb = __ldg(pos + b);
    int32_t lo = min(pa, pb), hi = max(pa, pb);
    bool parted = false, b_later = pb > pa;
    float te = -FLT_MAX;                       // of the later one's leaf box
    for (int32_t ref = root; ref >= 0;) {
        const float4* n = reinterpret_cast<const float4*>(nodes + ref);
        const float4 x = __ldg(n), y = __ldg(n + 1), z = __ldg(n + 2);
        const int4 meta = __ldg(reinterpret_cast<const int4*>(n + 3));   // left, right, axis, split
        const float tl = box_entry(x.x, x.y, y.x, y.y, z.x, z.y, r), tr = box_entry(x.z, x.w, y.z, y.w, z.z, z.w, r);
        if (!parted && lo < meta.w && hi >= meta.w) {
            if (tr < tl) { b_later = pb < pa; hi = lo; }   // right child first: the left one comes later
            lo = hi;
            parted = true;
        }
        const bool right = lo >= meta.w;
        te = right ? tr : tl;
        ref = right ? meta.y : meta.x;
    }
    if (!parted) return tb < ta || (tb == ta && b_later);
    return (te < end) == b_later;
}

// Whether a candidate (record `at`, triangle id, t <= r.tmax) replaces the hit h (h.tri -1: none),
// whose window ends at r.tmax; `window`: the end of the candidate's own.
template <bool ANY>
__device__ __forceinline__ bool render_candidate(const DeviceScene& s, int64_t at, int32_t id, float t, float u, float v,
                                                 const TraversalRay& r, const Hit& h, bool any, float& window)
{
    window = t;
    if (fminf(fminf(u, v), 1.0f - u - v) < s.box_margin) {
        float te;
        if (!leaf_box_render(s.boxes8, at, r, te)) return false;
        if (ANY || any) return te < r.tmax;
        window = fmaxf(t, te);
    }
    if (ANY || any || window < r.tmax || h.tri < 0) return true;
    return window == r.tmax && order_takes(s.bvh2, s.tie_pos, s.root_ref, h.tri, id, h.t, t, window, r);
}

// Exact walk. The reference's answer for a ray is a fold over the triangles whose
// leaf box passes its slab test with t_enter < maxT (the ancestors' boxes then
// pass too: the test is monotone under containment) and whose TriAccel test
// passes. Call S the candidates at the ray's own maxT. If A in S has the least t
// and every other member has t > max(t_A, t_enter_A), the reference finds A
// whatever the order: its leaf is entered before any maxT that another hit can
// have set, and nothing is accepted after it. The wide walk therefore culls at
// max(t_A, t_enter_A), tests each candidate's leaf box with the reference's
// arithmetic, and hands the ray back (HIT_TIED) when two candidates lie within that
// window of one another; such rays, and rays for which the inflated boxes prove
// nothing (exact_wide_ok), take the reference's own walk.
constexpr int32_t HIT_TIED = -2;

__device__ __forceinline__ bool leaf_box_exact(const LeafBox* __restrict__ boxes, int64_t at, const TraversalRay& r,
                                               float& te)
{
    const float4 a = __ldg(reinterpret_cast<const float4*>(boxes + at));
    const float4 b = __ldg(reinterpret_cast<const float4*>(boxes + at) + 1);
    TraversalRay e;
    RayIn in;
#pragma unroll
    for (int c = 0; c < 3; c++) { in.o[c] = r.o[c]; in.d[c] = r.d[c]; }
    in.tmin = r.tmin;
    in.tmax = r.tmax;
    setup_ray(e, in);
    return slab_intrinsic(e, a.x, a.w, a.y, b.x, a.z, b.y, te);
}

// A candidate hit (t, u, v) of record `at` within the current window; tmax0 is
// the ray's own maxT.
__device__ __forceinline__ void exact_candidate(const LeafBox* __restrict__ boxes, int64_t at, int32_t tri, float t,
                                                float u, float v, float tmax0, TraversalRay& r, Hit& h)
{
    float te;
    if (!leaf_box_exact(boxes, at, r, te) || !(te < tmax0) || h.tri == HIT_TIED) return;
    const float window = fmaxf(t, te);
    if (h.tri >= 0 && (t >= h.t || h.t <= window)) { h.tri = HIT_TIED; return; }
    h.tri = tri; h.t = t; h.u = u; h.v = v;
    r.tmax = window;
}

// Whether the inflated boxes cover this ray, for scenes of largest coordinate M and
// origins within limit = 8 M:
//   * every non-zero direction component has an inverse below the clamp of setup_ray (1e18);
//   * a zero axis, on which the walk's box ends at 1e18 times its distance, must not end
//     the ray before its hit. Boxes that hold a hit reach at least 2^-21 * 8 M / 2 beyond
//     the origin on such an axis (collapse_bvh8's margin of 4 ulps), that is 1.9e12 M,
//     and a hit lies within 9.1 M of the origin on the direction's largest axis: any
//     largest component above 5e-12 will do, and 2^-30 leaves a factor of 190;
//   * inverses times grid steps (2^-83 and more) stay normal: at most 2^30.
// NaN fails every comparison.
__device__ __forceinline__ bool exact_wide_ok(const RayIn& in, float limit)
{
    bool ok = true;
    float longest = 0.0f;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const float a = fabsf(in.d[c]);
        ok = ok && fabsf(in.o[c]) <= limit && (a == 0.0f || a >= 0x1p-59f);
        longest = fmaxf(longest, a);
    }
    return ok && longest >= 0x1p-30f && longest <= 0x1p30f;
}

}  // namespace lmgpu
