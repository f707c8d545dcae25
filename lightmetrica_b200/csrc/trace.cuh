// Rays, triangle tests and one-thread walks of the binary trees (sm_100a). The
// batched traversals walk the 8-wide tree (trace8.cuh). The reference's own walk
// (trace_bvh2) answers the rays that one hands back, the work counts and the full hit
// records; render rays of one thread walk the binary render tree (trace_bvh2_render).
//
// Exactness contract: the closest hit (triangle id, t, u, v) is bit-identical
// to the reference BVHScene::Intersect
// (scene.bvh.cpp:405-473, TriAccel::Intersect triaccel.h:100-160):
//   * same tree (host builder) and the same near-first depth-first order
//     (the right child first iff the ray direction is negative along the
//     node's split axis);
//   * the slab test's maxT-independent part is evaluated when a node is
//     first seen; its `tmin < maxT` part is re-evaluated when the far child is
//     popped, i.e. with the same maxT the recursive reference sees there;
//   * every float operation uses an explicit round-to-nearest intrinsic
//     (__fadd_rn, __fmul_rn, __fdiv_rn, ...), so nvcc cannot fuse them into
//     FMAs and each rounds once, like the reference's float SSE build.
#pragma once
#include <cfloat>
#include <cstdint>
#include "layout.h"

namespace lmgpu {

struct RayIn {
    float o[3], d[3];
    float tmin, tmax;
};

struct TraversalRay {
    float o[3];
    float d[3];
    float inv_min[3];   // 1/d, or 0 where d == 0      (scene.bvh.cpp:124-127)
    float inv_max[3];   // 1/d, or FLT_MAX where d == 0 (scene.bvh.cpp:129-132)
    uint32_t neg;       // bit c set iff d[c] < 0        (scene.bvh.cpp:134-137);
                        // bit 3: finite origin, every d[c] != 0 with a finite 1/d
                        // (RAY_FINITE_INV)
    float tmin, tmax;
};

constexpr uint32_t RAY_FINITE_INV = 8u;

// Render rays and rays of the 8-wide walk (FMA) keep inv_min = 1/d, clamped to +-1e18 so that
// it stays finite, and inv_max = -o/d: a plane distance is then one
// multiply-add, (lo - o)/d = fma(lo, 1/d, -o/d). inv_min's sign is `neg`'s: both
// zeros give +1e18, since the walk picks near and far planes by `neg`.
template <bool FMA = false>
__device__ __forceinline__ void setup_ray(TraversalRay& r, const RayIn& in)
{
    if (FMA) {
        r.neg = RAY_FINITE_INV;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            r.o[c] = in.o[c];
            r.d[c] = in.d[c];
            float inv = __frcp_rn(in.d[c]);
            if (!(fabsf(inv) <= 1e18f)) inv = in.d[c] < 0.0f ? -1e18f : 1e18f;
            r.inv_min[c] = inv;
            r.inv_max[c] = -(in.o[c] * inv);
            r.neg |= (in.d[c] < 0.0f ? 1u : 0u) << c;
        }
        r.tmin = in.tmin;
        r.tmax = in.tmax;
        return;
    }
    r.neg = RAY_FINITE_INV;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        r.o[c] = in.o[c];
        r.d[c] = in.d[c];
        const bool z = in.d[c] == 0.0f;
        const float inv = __frcp_rn(in.d[c]);  // correctly rounded 1/d == 1.0f/d
        r.inv_min[c] = z ? 0.0f : inv;
        r.inv_max[c] = z ? FLT_MAX : inv;
        r.neg |= (in.d[c] < 0.0f ? 1u : 0u) << c;
        const float inf = __int_as_float(0x7f800000);
        if (z || !(fabsf(inv) < inf) || !(fabsf(in.o[c]) < inf)) r.neg &= ~RAY_FINITE_INV;
    }
    r.tmin = in.tmin;
    r.tmax = in.tmax;
}

// Slab test of one box, split into the maxT-independent verdict (`pass`)
// and the entry distance `t_enter`; the box is hit iff pass && t_enter < maxT.
// lo/hi are the box's per-axis bounds.
__device__ __forceinline__ bool slab_intrinsic(const TraversalRay& r,
                                               float lox, float hix, float loy, float hiy,
                                               float loz, float hiz, float& t_enter)
{
    const float nx = (r.neg & 1u) ? hix : lox, fx = (r.neg & 1u) ? lox : hix;
    const float ny = (r.neg & 2u) ? hiy : loy, fy = (r.neg & 2u) ? loy : hiy;
    const float nz = (r.neg & 4u) ? hiz : loz, fz = (r.neg & 4u) ? loz : hiz;
    float tmin = __fmul_rn(__fsub_rn(nx, r.o[0]), r.inv_min[0]);
    float tmax = __fmul_rn(__fsub_rn(fx, r.o[0]), r.inv_max[0]);
    const float tymin = __fmul_rn(__fsub_rn(ny, r.o[1]), r.inv_min[1]);
    const float tymax = __fmul_rn(__fsub_rn(fy, r.o[1]), r.inv_max[1]);
    if ((tmin > tymax) || (tymin > tmax)) return false;
    if (tymin > tmin) tmin = tymin;
    if (tymax < tmax) tmax = tymax;
    const float tzmin = __fmul_rn(__fsub_rn(nz, r.o[2]), r.inv_min[2]);
    const float tzmax = __fmul_rn(__fsub_rn(fz, r.o[2]), r.inv_max[2]);
    if ((tmin > tzmax) || (tzmin > tmax)) return false;
    if (tzmin > tmin) tmin = tzmin;
    if (tzmax < tmax) tmax = tzmax;
    t_enter = tmin;
    return tmax > r.tmin;
}

// The same slab test for a ray with RAY_FINITE_INV and a box with finite
// lo <= hi on every axis (every binary node's child box). Then inv_min == inv_max,
// the near/far plane distances of an axis are min/max of its two plane
// distances (a float subtraction and multiplication round monotonically),
// no value is NaN, and the reference's pairwise comparison chain fails
// exactly when max(near) > min(far); its final tmin is max(near). The verdict
// and t_enter therefore equal slab_intrinsic's (t_enter up to the sign of a
// zero, which no comparison distinguishes).
#ifndef LMGPU_TRACE_FAST_SLAB
#define LMGPU_TRACE_FAST_SLAB 1
#endif
#ifndef LMGPU_TRACE_F32X2
#define LMGPU_TRACE_F32X2 1
#endif
// (lo - o) * inv and (hi - o) * inv: with LMGPU_TRACE_F32X2 as one packed
// sub.rn.f32x2 and one mul.rn.f32x2 (sm_100), each lane rounded to nearest
// on its own, i.e. the same two results as the scalar __fsub_rn/__fmul_rn.
__device__ __forceinline__ void plane_pair(float lo, float hi, float o, float inv, float& a, float& b)
{
#if LMGPU_TRACE_F32X2
    asm("{\n\t.reg .b64 p, q;\n\t"
        "mov.b64 p, {%2, %3};\n\t"
        "mov.b64 q, {%4, %4};\n\t"
        "sub.rn.f32x2 p, p, q;\n\t"
        "mov.b64 q, {%5, %5};\n\t"
        "mul.rn.f32x2 p, p, q;\n\t"
        "mov.b64 {%0, %1}, p;\n\t}"
        : "=f"(a), "=f"(b) : "f"(lo), "f"(hi), "f"(o), "f"(inv));
#else
    a = __fmul_rn(__fsub_rn(lo, o), inv);
    b = __fmul_rn(__fsub_rn(hi, o), inv);
#endif
}

__device__ __forceinline__ bool slab_finite(const TraversalRay& r,
                                            float lox, float hix, float loy, float hiy,
                                            float loz, float hiz, float& t_enter)
{
    float ax, bx, ay, by, az, bz;
    plane_pair(lox, hix, r.o[0], r.inv_min[0], ax, bx);
    plane_pair(loy, hiy, r.o[1], r.inv_min[1], ay, by);
    plane_pair(loz, hiz, r.o[2], r.inv_min[2], az, bz);
    const float tn = fmaxf(fmaxf(fminf(ax, bx), fminf(ay, by)), fminf(az, bz));
    const float tf = fminf(fminf(fmaxf(ax, bx), fmaxf(ay, by)), fmaxf(az, bz));
    t_enter = tn;
    return tn <= tf && tf > r.tmin;
}

// x * s + b and y * s + b, each rounded once (packed, sm_100).
__device__ __forceinline__ void fma_pair(float x, float y, float s, float b, float& a, float& c)
{
    asm("{\n\t.reg .b64 p, q, r;\n\t"
        "mov.b64 p, {%2, %3};\n\t"
        "mov.b64 q, {%4, %4};\n\t"
        "mov.b64 r, {%5, %5};\n\t"
        "fma.rn.f32x2 p, p, q, r;\n\t"
        "mov.b64 {%0, %1}, p;\n\t}"
        : "=f"(a), "=f"(c) : "f"(x), "f"(y), "f"(s), "f"(b));
}

// The slab test of render rays (setup_ray<true>): multiply-adds, near and far planes by
// min and max. The box is hit iff this holds and t_enter < maxT.
__device__ __forceinline__ bool slab_render(const TraversalRay& r, float lox, float hix, float loy, float hiy,
                                            float loz, float hiz, float& t_enter)
{
    float x0, x1, y0, y1, z0, z1;
    fma_pair(lox, hix, r.inv_min[0], r.inv_max[0], x0, x1);
    fma_pair(loy, hiy, r.inv_min[1], r.inv_max[1], y0, y1);
    fma_pair(loz, hiz, r.inv_min[2], r.inv_max[2], z0, z1);
    const float tn = fmaxf(fmaxf(fminf(x0, x1), fminf(y0, y1)), fminf(z0, z1));
    const float tf = fminf(fminf(fmaxf(x0, x1), fmaxf(y0, y1)), fmaxf(z0, z1));
    t_enter = tn;
    return tn <= tf && tf > r.tmin;
}

// Both child boxes of a binary node.
__device__ __forceinline__ void slab_pair(const TraversalRay& r, float4 bx, float4 by, float4 bz,
                                          bool& pl, float& tl, bool& pr, float& tr)
{
    if (LMGPU_TRACE_FAST_SLAB && (r.neg & RAY_FINITE_INV)) {
        pl = slab_finite(r, bx.x, bx.y, by.x, by.y, bz.x, bz.y, tl);
        pr = slab_finite(r, bx.z, bx.w, by.z, by.w, bz.z, bz.w, tr);
    } else {
        pl = slab_intrinsic(r, bx.x, bx.y, by.x, by.y, bz.x, bz.y, tl);
        pr = slab_intrinsic(r, bx.z, bx.w, by.z, by.w, bz.z, bz.w, tr);
    }
}

// TriAccel::Intersect (triaccel.h:100-160) in the reference's order.
// Returns true on a hit within [mint, maxt]; u, v, t are then valid.
__device__ __forceinline__ bool triaccel_intersect(const float4 q0, const float4 q1, const float4 q2,
                                                   const TraversalRay& r, float maxt,
                                                   float& u, float& v, float& t)
{
    const uint32_t k = __float_as_uint(q0.x) & TRI_AXIS_MASK;
    if (k == 3u) return false;
    // (u, v, k) axis permutation: k=0 -> (1,2,0), k=1 -> (2,0,1), k=2 -> (0,1,2)
    const float o_u = k == 0 ? r.o[1] : (k == 1 ? r.o[2] : r.o[0]);
    const float o_v = k == 0 ? r.o[2] : (k == 1 ? r.o[0] : r.o[1]);
    const float o_k = k == 0 ? r.o[0] : (k == 1 ? r.o[1] : r.o[2]);
    const float d_u = k == 0 ? r.d[1] : (k == 1 ? r.d[2] : r.d[0]);
    const float d_v = k == 0 ? r.d[2] : (k == 1 ? r.d[0] : r.d[1]);
    const float d_k = k == 0 ? r.d[0] : (k == 1 ? r.d[1] : r.d[2]);
    const float n_u = q0.y, n_v = q0.z, n_d = q0.w;
    const float a_u = q1.x, a_v = q1.y, b_nu = q1.z, b_nv = q1.w;
    const float c_nu = q2.x, c_nv = q2.y;
    float num = __fsub_rn(n_d, __fmul_rn(o_u, n_u));
    num = __fsub_rn(num, __fmul_rn(o_v, n_v));
    num = __fsub_rn(num, o_k);
    float den = __fadd_rn(__fmul_rn(d_u, n_u), __fmul_rn(d_v, n_v));
    den = __fadd_rn(den, d_k);
    t = __fdiv_rn(num, den);
    if (t < r.tmin || t > maxt) return false;
    const float hu = __fsub_rn(__fadd_rn(o_u, __fmul_rn(t, d_u)), a_u);
    const float hv = __fsub_rn(__fadd_rn(o_v, __fmul_rn(t, d_v)), a_v);
    u = __fadd_rn(__fmul_rn(hv, b_nu), __fmul_rn(hu, b_nv));
    v = __fadd_rn(__fmul_rn(hu, c_nu), __fmul_rn(hv, c_nv));
    return u >= 0.0f && v >= 0.0f && __fadd_rn(u, v) <= 1.0f;
}

// The same TriAccel test for renders, which need the same expected image,
// not bit-identical hits: multiply-adds and an approximate division
// (div.approx: a reciprocal and a multiply) in place of the separately
// rounded products and the correctly rounded division. Hits may differ
// from the exact test's only within rounding of the edges and of t.
__device__ __forceinline__ bool triaccel_intersect_fast(const float4 q0, const float4 q1, const float4 q2,
                                                        const TraversalRay& r, float maxt,
                                                        float& u, float& v, float& t)
{
    const uint32_t k = __float_as_uint(q0.x) & TRI_AXIS_MASK;
    if (k == 3u) return false;
    const float o_u = k == 0 ? r.o[1] : (k == 1 ? r.o[2] : r.o[0]);
    const float o_v = k == 0 ? r.o[2] : (k == 1 ? r.o[0] : r.o[1]);
    const float o_k = k == 0 ? r.o[0] : (k == 1 ? r.o[1] : r.o[2]);
    const float d_u = k == 0 ? r.d[1] : (k == 1 ? r.d[2] : r.d[0]);
    const float d_v = k == 0 ? r.d[2] : (k == 1 ? r.d[0] : r.d[1]);
    const float d_k = k == 0 ? r.d[0] : (k == 1 ? r.d[1] : r.d[2]);
    const float num = __fmaf_rn(-o_v, q0.z, __fmaf_rn(-o_u, q0.y, q0.w)) - o_k;
    const float den = __fmaf_rn(d_v, q0.z, __fmaf_rn(d_u, q0.y, d_k));
    t = __fdividef(num, den);
    if (!(t >= r.tmin && t <= maxt)) return false;
    const float hu = __fmaf_rn(t, d_u, o_u) - q1.x;
    const float hv = __fmaf_rn(t, d_v, o_v) - q1.y;
    u = __fmaf_rn(hv, q1.z, hu * q1.w);
    v = __fmaf_rn(hu, q2.x, hv * q2.y);
    return u >= 0.0f && v >= 0.0f && u + v <= 1.0f;
}

struct Hit {
    int32_t tri;   // reference TriAccel index, -1 = miss
    float t, u, v;
};

struct TraceStats {
    uint32_t nodes;   // binary-node slab tests (reference count)
    uint32_t tris;    // TriAccel tests
};

// Leaf loop: every record of the leaf is tested against the running maxT;
// a hit sets maxT = t so later records need t <= new maxT (scene.bvh.cpp:416-427).
// RENDER: the triangle test of render rays.
template <bool ANY_HIT, bool RENDER = false>
__device__ __forceinline__ bool trace_leaf(const TriRecord* __restrict__ tris, int32_t first,
                                           TraversalRay& r, Hit& h, TraceStats* st)
{
    const float4* p = reinterpret_cast<const float4*>(tris + first);
    for (;;) {
        const float4 q0 = __ldg(p), q1 = __ldg(p + 1), q2 = __ldg(p + 2);
        if (st) st->tris++;
        float u, v, t;
        if (RENDER ? triaccel_intersect_fast(q0, q1, q2, r, r.tmax, u, v, t)
                   : triaccel_intersect(q0, q1, q2, r, r.tmax, u, v, t)) {
            r.tmax = t;
            h.tri = static_cast<int32_t>(__float_as_uint(q2.z));
            h.t = t; h.u = u; h.v = v;
            if (ANY_HIT) return true;
        }
        if (__float_as_uint(q0.x) & TRI_LAST_IN_LEAF) break;
        p += 3;
    }
    return false;
}

// Traversal state: the current reference (internal node >= 0, leaf < 0, or
// REF_DONE) and the deferred far children.
constexpr int32_t REF_DONE = 0x7fffffff;

struct TravState {
    int32_t ref;
    int sp;
};

// Pops the next deferred child whose box is still entered before maxT
// (the reference's far-child test, evaluated with the current maxT).
__device__ __forceinline__ void pop_next(TravState& ts, const int2* stack, const TraversalRay& r, TraceStats* st)
{
    while (ts.sp > 0) {
        const int2 e = stack[--ts.sp];
        if (st) st->nodes++;
        if (__int_as_float(e.y) < r.tmax) { ts.ref = e.x; return; }
    }
    ts.ref = REF_DONE;
}

// Closest hit (or any hit) through the reference's binary tree; the root box
// is tested first (the reference tests every node's own box on entry).
// `stack` is per-thread scratch of `stack_cap` (ref, t_enter) pairs. Returns
// false if the stack bound was exceeded (the caller flags an error).
template <bool ANY_HIT>
__device__ __forceinline__ bool trace_bvh2(const Bvh2Node* __restrict__ nodes,
                                           const TriRecord* __restrict__ tris,
                                           int32_t root_ref, const float* root_box,
                                           TraversalRay& r, Hit& h, int2* stack, int stack_cap,
                                           TraceStats* st)
{
    h.tri = -1;
    TravState ts;
    ts.sp = 0;
    float te;
    if (st) st->nodes++;
    ts.ref = (slab_intrinsic(r, root_box[0], root_box[3], root_box[1], root_box[4], root_box[2], root_box[5], te) &&
              te < r.tmax) ? root_ref : REF_DONE;
    for (;;) {
        while (ts.ref >= 0 && ts.ref != REF_DONE) {
            const float4* np = reinterpret_cast<const float4*>(nodes + ts.ref);
            const float4 bx = __ldg(np), by = __ldg(np + 1), bz = __ldg(np + 2);
            const int4 meta = __ldg(reinterpret_cast<const int4*>(np + 3));
            float tl = 0.f, tr = 0.f;
            bool pl, pr;
            slab_pair(r, bx, by, bz, pl, tl, pr, tr);
            const bool right_first = (r.neg >> meta.z) & 1u;
            const int32_t near_ref = right_first ? meta.y : meta.x;
            const int32_t far_ref = right_first ? meta.x : meta.y;
            const bool near_pass = right_first ? pr : pl;
            const bool far_pass = right_first ? pl : pr;
            const float near_t = right_first ? tr : tl;
            const float far_t = right_first ? tl : tr;
            if (st) st->nodes++;                         // near child's slab test
            if (near_pass && near_t < r.tmax) {
                if (far_pass) {
                    if (ts.sp >= stack_cap) return false;
                    stack[ts.sp++] = make_int2(far_ref, __float_as_int(far_t));
                } else if (st) {
                    st->nodes++;                         // far child's (failing) test
                }
                ts.ref = near_ref;
                continue;
            }
            if (st) st->nodes++;                         // far child's test, same maxT
            if (far_pass && far_t < r.tmax) { ts.ref = far_ref; continue; }
            pop_next(ts, stack, r, st);
        }
        if (ts.ref == REF_DONE) return true;
        if (trace_leaf<ANY_HIT>(tris, ~ts.ref, r, h, st) && ANY_HIT) return true;
        pop_next(ts, stack, r, st);
    }
}

// Closest hit (or any hit) of a render ray (setup_ray<true>) by one thread through a
// binary tree, the child entered first before the other. A visibility ray's maxT does
// not change, so that its deferred children (node references alone) need no test when they
// come up. `stack` holds `stack_cap` entries; returns false if that is exceeded.
template <bool ANY_HIT>
__device__ __forceinline__ bool trace_bvh2_render(const Bvh2Node* __restrict__ nodes, const TriRecord* __restrict__ tris,
                                                  int32_t root_ref, const float* root_box, TraversalRay& r, Hit& h,
                                                  int2* stack, int stack_cap)
{
    int32_t* refs = reinterpret_cast<int32_t*>(stack);
    h.tri = -1;
    TravState ts;
    ts.sp = 0;
    float te;
    ts.ref = (slab_render(r, root_box[0], root_box[3], root_box[1], root_box[4], root_box[2], root_box[5], te) && te < r.tmax)
                 ? root_ref : REF_DONE;
    auto pop = [&] {
        if (!ANY_HIT) pop_next(ts, stack, r, nullptr);
        else ts.ref = ts.sp > 0 ? refs[--ts.sp] : REF_DONE;
    };
    for (;;) {
        while (ts.ref >= 0 && ts.ref != REF_DONE) {
            const float4* np = reinterpret_cast<const float4*>(nodes + ts.ref);
            const float4 bx = __ldg(np), by = __ldg(np + 1), bz = __ldg(np + 2);
            const int4 meta = __ldg(reinterpret_cast<const int4*>(np + 3));
            float tl, tr;
            const bool pl = slab_render(r, bx.x, bx.y, by.x, by.y, bz.x, bz.y, tl) && tl < r.tmax;
            const bool pr = slab_render(r, bx.z, bx.w, by.z, by.w, bz.z, bz.w, tr) && tr < r.tmax;
            const bool right_first = pr && (!pl || tr < tl);
            if (pl && pr) {
                if (ts.sp >= stack_cap) return false;
                const int32_t far_ref = right_first ? meta.x : meta.y;
                if (ANY_HIT) refs[ts.sp++] = far_ref;
                else stack[ts.sp++] = make_int2(far_ref, __float_as_int(right_first ? tl : tr));
            }
            if (pl || pr) ts.ref = right_first ? meta.y : meta.x;
            else pop();
        }
        if (ts.ref == REF_DONE) return true;
        if (trace_leaf<ANY_HIT, true>(tris, ~ts.ref, r, h, nullptr) && ANY_HIT) return true;
        pop();
    }
}

// Brute force over all records in TriAccel order (reference scene.naive.cpp:98-121).
template <bool ANY_HIT>
__device__ __forceinline__ void trace_naive(const TriRecord* __restrict__ tris_in_id_order, int64_t n,
                                            TraversalRay& r, Hit& h, TraceStats* st)
{
    h.tri = -1;
    const float4* p = reinterpret_cast<const float4*>(tris_in_id_order);
    for (int64_t i = 0; i < n; i++, p += 3) {
        const float4 q0 = __ldg(p), q1 = __ldg(p + 1), q2 = __ldg(p + 2);
        if (st) st->tris++;
        float u, v, t;
        if (triaccel_intersect(q0, q1, q2, r, r.tmax, u, v, t)) {
            r.tmax = t;
            h.tri = static_cast<int32_t>(__float_as_uint(q2.z));
            h.t = t; h.u = u; h.v = v;
            if (ANY_HIT) return;
        }
    }
}

}  // namespace lmgpu
