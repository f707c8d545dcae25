// Differentiable rendering: a forward / adjoint pair over the path tracer
// with per-triangle diffuse albedo and per-light emission as parameters.
//
// Both passes run the reference's pt / pt.direct / pt.mis paths (pathtrace*.cpp)
// as waves of the renderers' own kernels (pt_kernels.cuh) under a context that
// replaces albedo and emission. The adjoint pass does not store path vertices from
// the forward pass: it replays every path from its counter-based random
// numbers and, for each radiance contribution c splatted at pixel p, adds
// dL/dI_p * c / R_t to the gradient of the albedo R of every diffuse vertex t
// on the contribution's prefix (c is linear in each of them) and
// dL/dI_p * c / Le to the emission of its light. While a wave runs, each
// path keeps per vertex the triangle and the sum of the weights
// w = dL/dI_p * c whose prefix ends there; once the wave is done the weights are
// turned into suffix sums: one set of atomics per vertex instead of one per
// (contribution, vertex). Emission gradients go to double-precision partial sums
// (EMISSION_COPIES of them, since every path adds to the same few lights).
// Russian-roulette probabilities and MIS weights are held at their sampled
// values, which keeps the estimator unbiased for the diffuse BSDFs (their
// sampling densities do not depend on R).
//
// Waves against one thread per sample (k_diff; measured on the refined Cornell box,
// 512 x 512, 32 samples per pixel, up to 8 vertices, forward + backward):
// one thread per sample over the binary render tree 9.8 + 17.9 ms, over the 8-wide tree
// (more registers, and one ray's leaves hold up its warp) 18.4 + 36.6 ms, waves 14.2 ms in
// all. So one thread walks the binary tree. It stays for the budgets that waves_pay leaves,
// for streams being captured (a wave's workspace is allocated in stream order), and where
// that workspace cannot be had.
//
// The tail of a path of more vertices than a wave records (RECORDED_VERTS;
// UNBOUNDED_VERTS where the depth has no bound) is run by one thread from the path's
// queued ray (k_diff_tail). In k_diff and in that kernel:
//
// Paths deeper than RECORDED_VERTS vertices: the weights of all
// contributions deeper than that are summed into one total W_tail while the
// path runs, and the path's state on arrival at that depth is kept as a
// checkpoint (position, direction, throughput, previous vertex: a few
// registers' worth). When the path has ended, the first vertices' suffix
// sums start from W_tail, and the tail is replayed from the checkpoint a
// second time: a vertex i there is on the prefix of exactly the tail
// contributions deeper than i, so its weight is W_tail minus the running sum
// of the tail contributions met before it; no per-vertex record is needed.
// Only long paths pay for the second replay of their tail. A replay stops at
// MAX_PATH_VERTICES surface vertices and flags LMGPU_ERR_QUEUE_OVERFLOW: paths
// that long occur only in closed scenes without Russian roulette, where the
// reference's own loop (pathtrace*.cpp, `while (true)` with
// max_path_vertices = -1) does not end either.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <cstring>

#include "../../include/lmgpu.h"
#include "internal.h"
#include "pathtrace.cuh"
#include "pt_kernels.cuh"
#include "rng.cuh"
#include "trace.cuh"
#include "trace8.cuh"
#include "trace_kernels.cuh"
#include <memory>
#include <mutex>
#include <unordered_map>

namespace lmgpu {
namespace {

constexpr int RECORDED_VERTS = 32;          // vertices with a per-vertex record
constexpr int MAX_PATH_VERTICES = 4096;     // replay bound (surface vertices)

struct DiffConsts {
    int32_t technique, rr_depth, max_pv, sampling;
    uint64_t seed;
    int64_t sample_offset, num_samples, pixels;
    double inv_pixels;       // 1 / pixels
    SampleOrder order;
    float scale;             // film rescale W*H/num_samples
    const float* albedo;     // 3 per triangle or null
    const float* emission;   // 3 per area light or null
};

template <bool NAIVE, bool ANY, int STACK>
__device__ __forceinline__ int32_t cast_ray(const DeviceScene& s, V3 o, V3 d, float tmin, float tmax, Hit& h,
                                            int2* stack, int32_t* status)
{
    RayIn in;
    in.o[0] = o.x; in.o[1] = o.y; in.o[2] = o.z;
    in.d[0] = d.x; in.d[1] = d.y; in.d[2] = d.z;
    in.tmin = tmin; in.tmax = tmax;
    TraversalRay r;
    setup_ray<!NAIVE>(r, in);   // a render ray (the naive scan keeps the exact setup)
    h.tri = -1;
    if (s.num_tris == 0) return -1;
    bool ok = true;
    // The render tree and arithmetic of the waves, over its binary nodes.
    if (NAIVE) trace_naive<ANY>(s.tris_by_id, s.num_tris, r, h, nullptr);
    else ok = trace_bvh2_render<ANY>(s.bvh2, s.tris, s.root_ref, s.root_box, r, h, stack, s.stack_cap < STACK ? s.stack_cap : STACK);
    if (!ok) { atomicOr(status, STATUS_STACK_OVERFLOW); h.tri = -1; }
    return h.tri;
}

template <bool NAIVE, int STACK>
__device__ __forceinline__ bool visible(const DeviceScene& s, V3 a, V3 b, int2* stack, int32_t* status)
{
    const V3 d = b - a;
    const float len = sqrtf(length2(d));
    const V3 dn = d / len;
    const float maxt = len * (1.0f - EPS_F);
    Hit h;
    if (cast_ray<NAIVE, true, STACK>(s, a, dn, EPS_F, maxt, h, stack, status) >= 0) return false;
    float t;
    if (s.has_env && env_sphere_intersect(s, a, dn, EPS_F, maxt, t)) return false;
    return true;
}

__device__ __forceinline__ Material diff_material(const DeviceScene& s, const DiffConsts& c, int tri)
{
    Material m = material_of(s, s.tri_prim[tri]);
    if (c.albedo && m.type == LMGPU_BSDF_DIFFUSE) m.R = load3(c.albedo + 3 * (int64_t)tri);
    return m;
}

__device__ __forceinline__ V3 light_Le(const DeviceScene& s, const DiffConsts& c, int li)
{
    if (li >= s.num_area_lights) return load3(s.env_Le);
    return c.emission ? load3(c.emission + 3 * li) : load3(s.area_lights[li].Le);
}

// Per-path records of the adjoint. w[i] (i < RECORDED_VERTS): the weights
// of the contributions whose prefix ends at vertex i; w[TAIL_SUM]: all
// contributions deeper than RECORDED_VERTS; w[RUN_SUM]: in the tail replay,
// the tail contributions met so far. (One array, indexed at run time, so
// that the sums stay in local memory rather than in registers.)
constexpr int TAIL_SUM = RECORDED_VERTS, RUN_SUM = RECORDED_VERTS + 1;
struct Replay {
    int32_t tri[RECORDED_VERTS];
    V3 w[RECORDED_VERTS + 2];
};

// A path between two bounces: everything the bounce loop carries, so that
// the loop can resume from it.
struct PathPoint {
    V3 ro, rd, thr, prev_p, prev_n;
    float tmin, prev_pdf;
    int k;                    // index of the next bounce
    int nv;                   // surface vertices so far
    bool prev_deg, prev_spec;
};

// Emission gradient of one light summed by a thread; flushed into the
// block's shared sums (lights below SHARED_LIGHTS) or to global memory.
constexpr int SHARED_LIGHTS = 32;
struct EmissionSum {
    int light;
    V3 g;
};

__device__ __forceinline__ void flush_emission(EmissionSum& e, float* s_de, float* d_emission)
{
    if (e.light < 0) return;
    float* dst = e.light < SHARED_LIGHTS ? s_de + 3 * e.light : d_emission + 3 * e.light;
    if (e.g.x != 0.0f) atomicAdd(dst, e.g.x);
    if (e.g.y != 0.0f) atomicAdd(dst + 1, e.g.y);
    if (e.g.z != 0.0f) atomicAdd(dst + 2, e.g.z);
    e.light = -1;
    e.g = v3(0, 0, 0);
}

// One contribution: forward splats it, the adjoint records dL/dI . c for the
// albedos of its prefix (prefix length `depth`) and for its light. In the
// tail replay (`tail`) only contributions deeper than RECORDED_VERTS count,
// into the running sum; their light's gradient was added by the main replay.
template <bool BACKWARD>
__device__ __forceinline__ void contribute(const DiffConsts& c, const DeviceScene& s, Replay& rp, bool tail, int depth,
                                           int light, int pixel, V3 contrib, float* image, const float* dL,
                                           EmissionSum& es, float* s_de, float* d_emission)
{
    if (pixel < 0 || is_zero(contrib)) return;
    if (!BACKWARD) {
        atomicAdd(image + 3 * pixel, contrib.x * c.scale);
        atomicAdd(image + 3 * pixel + 1, contrib.y * c.scale);
        atomicAdd(image + 3 * pixel + 2, contrib.z * c.scale);
        return;
    }
    const V3 w = v3(dL[3 * pixel] * contrib.x, dL[3 * pixel + 1] * contrib.y, dL[3 * pixel + 2] * contrib.z) * c.scale;
    if (is_zero(w)) return;
    if (tail) {
        if (depth > RECORDED_VERTS) rp.w[RUN_SUM] = rp.w[RUN_SUM] + w;
        return;
    }
    if (depth > 0) {
        const int slot = depth > RECORDED_VERTS ? TAIL_SUM : depth - 1;
        rp.w[slot] = rp.w[slot] + w;
    }
    if (light >= 0 && light < s.num_area_lights) {
        const V3 Le = light_Le(s, c, light);
        const V3 g = v3(Le.x != 0.0f ? w.x / Le.x : 0.0f, Le.y != 0.0f ? w.y / Le.y : 0.0f,
                        Le.z != 0.0f ? w.z / Le.z : 0.0f);
        if (es.light != light) flush_emission(es, s_de, d_emission);
        es.light = light;
        es.g = es.g + g;
    }
}

// The albedo gradient S / R of a vertex of weight S on triangle t (diffuse only, else 0).
__device__ __forceinline__ V3 albedo_grad(const DiffConsts& c, const DeviceScene& s, int t, V3 S)
{
    if (is_zero(S)) return S;
    const Material m = diff_material(s, c, t);
    if (m.type != LMGPU_BSDF_DIFFUSE) return v3(0, 0, 0);
    return v3(m.R.x != 0.0f ? S.x / m.R.x : 0.0f, m.R.y != 0.0f ? S.y / m.R.y : 0.0f, m.R.z != 0.0f ? S.z / m.R.z : 0.0f);
}
__device__ __forceinline__ void add_albedo_grad(const DiffConsts& c, const DeviceScene& s, int t, V3 S, float* d_albedo)
{
    const V3 g = albedo_grad(c, s, t, S);
    if (g.x != 0.0f) atomicAdd(d_albedo + 3 * (int64_t)t, g.x);
    if (g.y != 0.0f) atomicAdd(d_albedo + 3 * (int64_t)t + 1, g.y);
    if (g.z != 0.0f) atomicAdd(d_albedo + 3 * (int64_t)t + 2, g.z);
}

// End of a replayed path: the albedo gradient weight of recorded vertex i is
// the sum of the weights of every contribution whose prefix contains it: the
// suffix sum of the recorded weights plus every deeper contribution.
__device__ __forceinline__ void flush_albedo(const DiffConsts& c, const DeviceScene& s, const Replay& rp, int n,
                                             float* d_albedo)
{
    V3 S = rp.w[TAIL_SUM];
    for (int i = n - 1; i >= 0; i--) {
        S = S + rp.w[i];
        add_albedo_grad(c, s, rp.tri[i], S, d_albedo);
    }
}

// Light sample with the parameterised emission; returns the light index.
__device__ __forceinline__ int sample_light_diff(const DeviceScene& s, const DiffConsts& c, float u0, float u1, LightPoint& lp)
{
    if (!sample_light(s, u0, u1, lp)) return -1;
    const int nl = s.num_lights;
    const int li = min(static_cast<int>(u0 * float(nl)), nl - 1);
    lp.Le = light_Le(s, c, li);
    return li;
}

// Saves the checkpoint. Kept out of line: the copy runs once per deep path,
// and inlined it costs the bounce loop registers (backward 36.6 -> 34.5 ms
// on the refined Cornell box out of line).
__device__ __noinline__ void save_point(PathPoint* dst, const PathPoint& src) { *dst = src; }

// The bounce loop from `pp` until the path ends. TAIL is the adjoint's
// second replay of a deep path's tail; otherwise, in the adjoint, the state
// on arrival at depth RECORDED_VERTS is saved in *ck and *deep set. Both
// instantiations compute the same path from the same state.
template <int TECH, bool NAIVE, int STACK, bool BACKWARD, bool TAIL>
__device__ __forceinline__ void bounce_loop(const DeviceScene& s, const DiffConsts& c, uint64_t key, int path_pixel,
                                            PathPoint& pp, PathPoint* ck, bool* deep, Replay& rp, int2* stack,
                                            float* image, const float* dL, float* d_albedo, EmissionSum& es,
                                            float* s_de, float* d_emission, int32_t* status)
{
    for (;;) {
        if (c.max_pv != -1 && pp.k >= c.max_pv) break;
        if (BACKWARD && !TAIL && pp.nv == RECORDED_VERTS) { save_point(ck, pp); *deep = true; }
        Hit h;
        const int tri = cast_ray<NAIVE, false, STACK>(s, pp.ro, pp.rd, pp.tmin, FLT_MAX, h, stack, status);
        Geom g;
        const V3 wi = -pp.rd;
        V3 Le = v3(0, 0, 0);
        float lpdf = 0.0f;
        int light = -1;
        bool surface = false;
        Material m;
        m.type = LMGPU_BSDF_BLACK;
        m.R = v3(0, 0, 0);
        if (tri < 0) {
            float t;
            if (!(s.has_env && env_sphere_intersect(s, pp.ro, pp.rd, pp.tmin, FLT_MAX, t))) break;
            env_surface(s, pp.ro, pp.rd, t, g);
            Le = emitted(load3(s.env_Le), g.sn, wi);
            lpdf = s.env_inv_area;
            light = s.num_area_lights;
        } else {
            surface_from_hit(s, tri, h.u, h.v, pp.ro, pp.rd, h.t, g);
            const int li = s.prim_light[s.tri_prim[tri]];
            if (li >= 0) {
                Le = emitted(light_Le(s, c, li), g.sn, wi);
                lpdf = s.area_lights[li].inv_area;
                light = li;
            }
            m = diff_material(s, c, tri);
            surface = true;
            if (pp.nv == MAX_PATH_VERTICES) {
                atomicOr(status, STATUS_QUEUE_OVERFLOW);
                break;
            }
            if (BACKWARD && !TAIL && pp.nv < RECORDED_VERTS) {
                rp.tri[pp.nv] = tri;
                rp.w[pp.nv] = v3(0, 0, 0);
            }
            pp.nv++;
        }
        const int depth_here = pp.nv - (surface ? 1 : 0);
        if (!is_zero(Le)) {
            const V3 contrib = pp.thr * Le;
            if (TECH == LMGPU_RENDER_PT || pp.prev_spec) {
                contribute<BACKWARD>(c, s, rp, TAIL, depth_here, light, path_pixel, contrib, image, dL, es, s_de,
                                     d_emission);
            } else if (TECH == LMGPU_RENDER_PT_MIS) {
                const float G = geometry_term(pp.prev_p, pp.prev_n, pp.prev_deg, g.p, g.sn, false);
                const float pdl = G == 0.0f ? 0.0f : lpdf / (float(s.num_lights) * G);
                contribute<BACKWARD>(c, s, rp, TAIL, depth_here, light, path_pixel,
                                     contrib * (pp.prev_pdf / (pp.prev_pdf + pdl)), image, dL, es, s_de, d_emission);
            }
        }
        if (!surface) break;
        // Tail replay: every tail contribution no deeper than this vertex
        // has been met; the rest have it on their prefix.
        if (BACKWARD && TAIL && pp.nv > RECORDED_VERTS) add_albedo_grad(c, s, tri, rp.w[TAIL_SUM] - rp.w[RUN_SUM], d_albedo);
        const int v = pp.k + 1;
        if (TECH != LMGPU_RENDER_PT && c.max_pv != -1 && v >= c.max_pv) break;
        if (TECH != LMGPU_RENDER_PT && has_non_delta(m.type)) {
            LightPoint lp;
            const int li = sample_light_diff(s, c, rng_uniform(key, dim_vertex(v) + DIM_LIGHT),
                                             rng_uniform(key, dim_vertex(v) + DIM_LIGHT + 1), lp);
            if (li >= 0) {
                const V3 ppL = normalize(lp.p - g.p);
                float pb;
                const V3 fs = eval_bsdf(m, g, wi, ppL, pb);
                const float G = geometry_term(g.p, g.sn, false, lp.p, lp.n, false);
                const V3 Lel = emitted(lp.Le, lp.n, -ppL);
                if (G != 0.0f && !is_zero(fs) && !is_zero(Lel) && visible<NAIVE, STACK>(s, g.p, lp.p, stack, status)) {
                    float w = 1.0f;
                    if (TECH == LMGPU_RENDER_PT_MIS) { const float pdl = lp.pdf_area / G; w = pdl / (pdl + pb); }
                    contribute<BACKWARD>(c, s, rp, TAIL, pp.nv, li, path_pixel, pp.thr * fs * Lel * (w * G / lp.pdf_area),
                                         image, dL, es, s_de, d_emission);
                }
            }
        }
        const int kv = TECH == LMGPU_RENDER_PT ? pp.k : v;
        if (TECH != LMGPU_RENDER_PT && c.rr_depth != -1 && kv >= c.rr_depth) {
            const float p = fminf(0.5f, luminance(pp.thr));
            if (rng_uniform(key, dim_vertex(kv) + DIM_RR) > p) break;
            pp.thr = pp.thr / p;
        }
        const BsdfSample bs = sample_bsdf(m, g, wi, rng_uniform(key, dim_vertex(kv) + DIM_BSDF),
                                          rng_uniform(key, dim_vertex(kv) + DIM_BSDF + 1),
                                          rng_uniform(key, dim_vertex(kv) + DIM_COMP));
        if (is_zero(bs.weight)) break;
        pp.thr = pp.thr * bs.weight;
        if (TECH == LMGPU_RENDER_PT && c.rr_depth != -1 && pp.k >= c.rr_depth) {
            const float p = fminf(0.5f, luminance(pp.thr));
            if (rng_uniform(key, dim_vertex(pp.k) + DIM_RR) > p) break;
            pp.thr = pp.thr / p;
        }
        if (TECH == LMGPU_RENDER_PT && c.max_pv != -1 && pp.k + 1 >= c.max_pv) break;
        pp.prev_p = g.p; pp.prev_n = g.sn; pp.prev_deg = false; pp.prev_spec = bs.specular; pp.prev_pdf = bs.pdf;
        pp.ro = g.p; pp.rd = bs.wo; pp.tmin = EPS_F;
        pp.k++;
    }
}

template <int TECH, bool NAIVE, int STACK, bool BACKWARD, int BLOCKS>
// BLOCKS resident blocks per SM. A budget that 4 a SM hold takes 4 (no spills): its time
// is its longest path's, and each spilled value is a trip through local memory on it
// (65 x 49 x 4, both passes with their calls: 315 -> 295 us).
// Larger ones take 8 (64 registers, some spills): on the refined Cornell box, 512 x 512 x
// 32, forward / backward 9.8 / 17.9 ms against 12.3 / 23.0 ms with 4. The passes are
// latency-bound and gain more from resident warps than they lose to spills.
__global__ void __launch_bounds__(128, BLOCKS) k_diff(const DeviceScene s, const DiffConsts c, float* image, const float* dL,
                                              float* d_albedo, float* d_emission, int32_t* status)
{
    int2 stack[STACK];
    Replay rp;
    __shared__ float s_de[3 * SHARED_LIGHTS];
    EmissionSum es;
    es.light = -1;
    es.g = v3(0, 0, 0);
    if (BACKWARD) {
        for (int i = threadIdx.x; i < 3 * SHARED_LIGHTS; i += blockDim.x) s_de[i] = 0.0f;
        __syncthreads();
    }
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < c.num_samples; j += stride) {
        const uint64_t sample = (uint64_t)(c.sample_offset + ordered_sample(c.order, j));
        const uint64_t key = sample_key(c.seed, sample);
        if (BACKWARD) {
            rp.w[TAIL_SUM] = v3(0, 0, 0);
            rp.w[RUN_SUM] = v3(0, 0, 0);
        }
        const float u0 = rng_uniform(key, DIM_RASTER), u1 = rng_uniform(key, DIM_RASTER + 1);
        float rx, ry;
        if (c.sampling == LMGPU_SAMPLING_STRATIFIED) {
            stratified_raster((int64_t)sample, c.pixels, c.inv_pixels, s.cam.width, s.cam.height, u0, u1, rx, ry);
        } else {
            rx = u0; ry = u1;
        }
        const int path_pixel = film_pixel(s.cam, rx, ry);
        float pdf_cam;
        const V3 dir = camera_direction(s.cam, rx, ry, pdf_cam);
        const V3 cp = load3(s.cam.position);
        if (c.max_pv != -1 && c.max_pv <= 1) continue;
        PathPoint pp;
        pp.ro = cp; pp.rd = dir; pp.thr = v3(1, 1, 1);
        pp.prev_p = cp; pp.prev_n = v3(0, 0, 1);
        pp.prev_deg = true; pp.prev_spec = false;
        pp.prev_pdf = pdf_cam;
        pp.tmin = TECH == LMGPU_RENDER_PT ? 0.0f : EPS_F;
        pp.k = 1;
        pp.nv = 0;
        bool alive = true;
        if (TECH != LMGPU_RENDER_PT) {
            LightPoint lp;
            const int li = sample_light_diff(s, c, rng_uniform(key, dim_vertex(1) + DIM_LIGHT),
                                             rng_uniform(key, dim_vertex(1) + DIM_LIGHT + 1), lp);
            if (li >= 0) {
                const V3 ppL = normalize(lp.p - cp);
                float lrx, lry, We;
                if (camera_project(s.cam, cp, ppL, lrx, lry, We) && We > 0.0f) {
                    const float G = geometry_term(cp, v3(0, 0, 1), true, lp.p, lp.n, false);
                    const V3 Le = emitted(lp.Le, lp.n, -ppL);
                    if (G != 0.0f && !is_zero(Le) && visible<NAIVE, STACK>(s, cp, lp.p, stack, status)) {
                        float w = 1.0f;
                        if (TECH == LMGPU_RENDER_PT_MIS) { const float pdl = lp.pdf_area / G; w = pdl / (pdl + We); }
                        contribute<BACKWARD>(c, s, rp, false, 0, li, film_pixel(s.cam, lrx, lry),
                                             Le * (w * We * G / lp.pdf_area), image, dL, es, s_de, d_emission);
                    }
                }
            }
            if (c.rr_depth != -1 && 1 >= c.rr_depth) {
                const float p = fminf(0.5f, luminance(pp.thr));
                if (rng_uniform(key, dim_vertex(1) + DIM_RR) > p) alive = false;
                else pp.thr = pp.thr / p;
            }
        }
        PathPoint ck;
        bool deep = false;
        if (alive)
            bounce_loop<TECH, NAIVE, STACK, BACKWARD, false>(s, c, key, path_pixel, pp, &ck, &deep, rp, stack, image, dL,
                                                              d_albedo, es, s_de, d_emission, status);
        if (BACKWARD) {
            flush_albedo(c, s, rp, min(pp.nv, RECORDED_VERTS), d_albedo);
            // The tail of a path deeper than RECORDED_VERTS: replayed from the
            // checkpoint taken on arrival at that depth.
            if (deep)
                bounce_loop<TECH, NAIVE, STACK, BACKWARD, true>(s, c, key, path_pixel, ck, nullptr, nullptr, rp, stack,
                                                                 image, dL, d_albedo, es, s_de, d_emission, status);
        }
    }
    if (BACKWARD) {
        flush_emission(es, s_de, d_emission);
        __syncthreads();
        const int n = 3 * min(s.num_area_lights, SHARED_LIGHTS);
        for (int i = threadIdx.x; i < n; i += blockDim.x)
            if (s_de[i] != 0.0f) atomicAdd(d_emission + i, s_de[i]);
    }
}

// ------------------------------------------------------------- waves ----

constexpr int64_t WAVE_PATHS = int64_t(1) << 23;   // paths in flight (a workspace of 350 bytes a path at 8 vertices)
constexpr int64_t MIN_WAVE_PATHS = int64_t(1) << 20;   // where memory is short; shorter still: one thread per sample
constexpr uint64_t POOL_KEEP = uint64_t(1) << 32;     // bytes a device's pool keeps; a workspace takes no more
constexpr int UNBOUNDED_VERTS = 20;                // vertices a wave follows a path of unbounded depth
constexpr int EMISSION_COPIES = 512;
// Doubles from one light's partial sum to the next: a 128-byte line each. Packed sums of
// several copies shared lines, and their atomics took their turns: the adjoint's traversals
// of 8.4 M paths took 5.3 or 6.0 ms, by where the workspace lay; now 4.98 ms.
constexpr int EMISSION_LINE = 16;

// The renderers' context with parameters in place of the scene's albedo and
// emission. The adjoint's shadow rays carry the weight dL/dI_p * c in place of c, and
// their light.
template <bool BACKWARD>
struct DiffScene : RenderContext {
    static constexpr bool TABLE = false, STREAM = false;
    DeviceScene s;
    RenderConsts rc;
    float scale;
    const float* albedo;
    const float* emission_of;
    float* image;            // forward
    const float* dL;         // adjoint, from here on
    float4* record;          // [vertex][path]: weight, triangle
    int64_t stride;
    int32_t* vertices;       // surface vertices of each path
    int32_t hit_no;          // shadow pass: the vertex its rays leave from
    double* d_emission;      // [copy][light][EMISSION_LINE]
    int32_t copies;

    __device__ __forceinline__ const DeviceScene& scene(int) const { return s; }
    __device__ __forceinline__ const RenderConsts& consts(int) const { return rc; }
    __device__ __forceinline__ int64_t wave_count(int64_t n) const { return n; }
    __device__ __forceinline__ int64_t sample_of(int, int64_t i) const
    {
        return rc.sample_base + ordered_sample(rc.order, rc.path_base + i);
    }
    __device__ __forceinline__ int begin_path(const PathState&, int64_t j, int64_t& i, int64_t& sample) const
    {
        i = j;
        sample = sample_of(0, j);
        return 0;
    }
    __device__ __forceinline__ int path_depth(const PathState&, int64_t, int k) const { return k; }

    __device__ __forceinline__ V3 Le_of(const DeviceScene&, int li) const
    {
        if (li >= s.num_area_lights) return load3(s.env_Le);
        return emission_of ? load3(emission_of + 3 * li) : load3(s.area_lights[li].Le);
    }
    __device__ __forceinline__ Material material(const DeviceScene&, int prim, int32_t tri) const
    {
        Material m = material_of(s, prim);
        if (albedo && m.type == LMGPU_BSDF_DIFFUSE) m.R = load3(albedo + 3 * (int64_t)tri);
        return m;
    }
    __device__ __forceinline__ V3 area_Le(const DeviceScene&, int li) const { return Le_of(s, li); }
    __device__ __forceinline__ void light_sample(const DeviceScene&, LightPoint& lp) const { lp.Le = Le_of(s, lp.light); }
    __device__ __forceinline__ V3 weight(int pixel, V3 c) const
    {
        return v3(dL[3 * pixel] * c.x, dL[3 * pixel + 1] * c.y, dL[3 * pixel + 2] * c.z) * scale;
    }
    __device__ __forceinline__ V3 path_weight(const PathState& st, int64_t i, V3 c) const
    {
        const float2 r = st.raster[i];
        return weight(film_pixel(s.cam, r.x, r.y), c);
    }
    __device__ __forceinline__ void add_record(int vertex, int64_t i, V3 w) const
    {
        float4& q = record[vertex * stride + i];
        const float4 v = q;
        q = make_float4(v.x + w.x, v.y + w.y, v.z + w.z, v.w);
    }
    __device__ __forceinline__ void add_emission(int li, V3 w) const
    {
        if (li >= s.num_area_lights) return;
        const V3 Le = Le_of(s, li);
        const int copy = (int)((blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) & (unsigned)(copies - 1));
        double* dst = d_emission + EMISSION_LINE * ((int64_t)copy * s.num_area_lights + li);
        if (Le.x != 0.0f) atomicAdd(dst, (double)(w.x / Le.x));
        if (Le.y != 0.0f) atomicAdd(dst + 1, (double)(w.y / Le.y));
        if (Le.z != 0.0f) atomicAdd(dst + 2, (double)(w.z / Le.z));
    }
    __device__ __forceinline__ void start(int64_t i) const { if (BACKWARD) vertices[i] = 0; }
    __device__ __forceinline__ void vertex(const PathState&, int64_t i, int k, int32_t tri) const
    {
        if (!BACKWARD) return;
        record[(int64_t)(k - 1) * stride + i] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(tri));
        vertices[i] = k;
    }
    __device__ __forceinline__ void emission(const PathState& st, int64_t i, int k, int li, V3 c) const
    {
        if (!BACKWARD) { RenderContext::emission(st, i, k, li, c); return; }
        const V3 w = path_weight(st, i, c);
        if (is_zero(w)) return;
        if (k >= 2) add_record(k - 2, i, w);       // its prefix ends at the vertex before the hit
        add_emission(li, w);
    }
    __device__ __forceinline__ V3 nee(const PathState& st, int64_t i, V3 c) const { return BACKWARD ? path_weight(st, i, c) : c; }
    __device__ __forceinline__ V3 camera_nee(int pixel, V3 c) const { return BACKWARD ? weight(pixel, c) : c; }
    __device__ __forceinline__ int shadow_tag(int, int light) const { return BACKWARD ? light : 0; }
    __device__ __forceinline__ void lit(float4* L, int32_t dest, V3 c, int tag) const
    {
        if (!BACKWARD) { RenderContext::lit(L, dest, c, tag); return; }
        add_record(hit_no - 1, dest, c);
        add_emission(tag, c);
    }
    __device__ __forceinline__ void lit_pixel(int tag, int pixel, V3 c) const
    {
        if (BACKWARD) add_emission(tag, c);
        else film_add(image, pixel, c * scale);
    }
};

// Forward, end of a wave: each path's radiance to its pixel.
__global__ void __launch_bounds__(128) k_diff_splat(const DiffScene<false> ctx, const PathState st, int64_t n)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float2 r = st.raster[i];
    film_add(ctx.image, film_pixel(ctx.s.cam, r.x, r.y), f3(st.L[i]) * ctx.scale);
}

// Adjoint, end of a wave: the albedo gradient weight of a vertex is the sum of
// the weights of every contribution whose prefix contains it: the suffix sum of
// the recorded weights plus the tail's (left in st.L by k_diff_tail, else 0).
// Bound by its atomics, three per vertex with a non-zero weight, and neighbouring paths
// mostly begin on the same triangle: the first vertices' gradients are summed over the
// warp's runs of one triangle before they are added. 2^20 paths of a 64 x 64 image of 144
// triangles: 1559 -> 750 us for the kernel.
__global__ void __launch_bounds__(128) k_diff_flush(const DiffScene<true> ctx, const DiffConsts c, const PathState st, int64_t n,
                                                    float* d_albedo)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int m = i < n ? ctx.vertices[i] : 0;
    V3 S = i < n ? f3(st.L[i]) : v3(0, 0, 0);
    for (int v = m - 1; v > 0; v--) {
        const float4 q = ctx.record[v * ctx.stride + i];
        S = S + f3(q);
        add_albedo_grad(c, ctx.s, __float_as_int(q.w), S, d_albedo);
    }
    int tri = -1;
    V3 g = v3(0, 0, 0);
    if (m > 0) {
        const float4 q = ctx.record[i];
        tri = __float_as_int(q.w);
        g = albedo_grad(c, ctx.s, tri, S + f3(q));
    }
    film_add_runs(d_albedo, tri, g);
}

// One warp per light and channel.
__global__ void __launch_bounds__(128) k_diff_emission(const double* part, int copies, int lights, float* d_emission)
{
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= 3 * (int64_t)lights) return;
    double sum = 0.0;
    for (int k = threadIdx.x & 31; k < copies; k += 32) sum += part[EMISSION_LINE * ((int64_t)k * lights + i / 3) + i % 3];
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0 && sum != 0.0) atomicAdd(d_emission + i, (float)sum);
}

// The paths still alive after a wave's last bounce, one thread each from their
// queued ray. Their vertices count from RECORDED_VERTS on, so that every
// contribution is "deeper than the record" (see the head of this file); the one
// found by the first hit belongs to the wave's last vertex.
constexpr int TAIL_STACK = 256;
template <int TECH, bool BACKWARD>
__global__ void __launch_bounds__(128) k_diff_tail(const DiffScene<BACKWARD> ctx, const DiffConsts c, const PathState st, int q, int k0,
                                                   float* d_albedo, float* d_emission, int32_t* status)
{
    int2 stack[TAIL_STACK];
    Replay rp;
    __shared__ float s_de[3 * SHARED_LIGHTS];
    EmissionSum es;
    es.light = -1;
    es.g = v3(0, 0, 0);
    if (BACKWARD) {
        for (int i = threadIdx.x; i < 3 * SHARED_LIGHTS; i += blockDim.x) s_de[i] = 0.0f;
        __syncthreads();
    }
    const int64_t n = (int64_t)st.counters[ring_rays(k0)];
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
        const float4 o4 = st.qo[q][j], d4 = st.qd[q][j], t4 = st.qt[q][j];
        const float4 n4 = TECH == LMGPU_RENDER_PT ? make_float4(0, 0, 1, 0) : st.qn[q][j];
        const int64_t i = queued_path(d4);
        const uint64_t key = sample_key(c.seed, (uint64_t)ctx.sample_of(0, i));
        const float2 rs = st.raster[i];
        const int pixel = film_pixel(ctx.s.cam, rs.x, rs.y);
        PathPoint pp, ck;
        pp.ro = f3(o4); pp.rd = f3(d4); pp.thr = f3(t4);
        pp.prev_p = pp.ro; pp.prev_n = f3(n4);
        pp.prev_deg = (__float_as_uint(n4.w) & PREV_DEGENERATED) != 0;
        pp.prev_spec = (__float_as_uint(n4.w) & PREV_SPECULAR) != 0;
        pp.prev_pdf = t4.w;
        pp.tmin = queued_tmin(d4);
        pp.k = k0;
        pp.nv = BACKWARD ? RECORDED_VERTS : k0 - 1;
        bool deep = false;
        if (BACKWARD) rp.w[RECORDED_VERTS - 1] = rp.w[TAIL_SUM] = rp.w[RUN_SUM] = v3(0, 0, 0);
        bounce_loop<TECH, false, TAIL_STACK, BACKWARD, false>(ctx.s, c, key, pixel, pp, &ck, &deep, rp, stack, ctx.image, ctx.dL, d_albedo,
                                                         es, s_de, d_emission, status);
        if (BACKWARD) {
            st.L[i] = f4(rp.w[TAIL_SUM] + rp.w[RECORDED_VERTS - 1], 0.0f);
            if (deep)
                bounce_loop<TECH, false, TAIL_STACK, BACKWARD, true>(ctx.s, c, key, pixel, ck, nullptr, nullptr, rp, stack, ctx.image, ctx.dL,
                                                                d_albedo, es, s_de, d_emission, status);
        }
    }
    if (BACKWARD) {
        flush_emission(es, s_de, d_emission);
        __syncthreads();
        const int m = 3 * min(ctx.s.num_area_lights, SHARED_LIGHTS);
        for (int i = threadIdx.x; i < m; i += blockDim.x)
            if (s_de[i] != 0.0f) atomicAdd(d_emission + i, s_de[i]);
    }
}

// Stream-ordered memory of the waves' workspaces, one pool per device: calls
// on several streams or threads each get their own, and what they return stays
// in the pool for the next call, up to POOL_KEEP, until lmgpu_render_release or until another
// allocation of this library finds the device full (device_malloc).
struct DiffPool {
    std::mutex mu;
    cudaMemPool_t pool = nullptr;
};
DiffPool& diff_pool(int device)
{
    static std::mutex map_mu;
    static std::unordered_map<int, std::unique_ptr<DiffPool>> all;
    std::lock_guard<std::mutex> lock(map_mu);
    auto& e = all[device];
    if (!e) e.reset(new DiffPool);
    return *e;
}
cudaError_t diff_pool_of(int device, cudaMemPool_t* out)
{
    DiffPool& p = diff_pool(device);
    std::lock_guard<std::mutex> lock(p.mu);
    if (!p.pool) {
        cudaMemPoolProps props;
        std::memset(&props, 0, sizeof(props));
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaError_t e = cudaMemPoolCreate(&p.pool, &props);
        if (e != cudaSuccess) { p.pool = nullptr; return e; }
        uint64_t keep = POOL_KEEP;
        e = cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep);
        if (e != cudaSuccess) { cudaMemPoolDestroy(p.pool); p.pool = nullptr; return e; }
    }
    *out = p.pool;
    return cudaSuccess;
}

// (not a status of the library) nothing was launched: the workspace could not be had
constexpr int WAVES_NO_MEMORY = 1 << 30;

template <int TECH, int STACK, bool BACKWARD>
int run_diff_waves(LmgpuScene* sc, const DiffConsts& c, float* image, const float* dL, float* da, float* de, cudaStream_t stream)
{
    using Ctx = DiffScene<BACKWARD>;
    const DeviceScene& s = sc->rdev;
    if (c.max_pv != -1 && c.max_pv <= 1) return LMGPU_OK;      // no vertex beyond the camera
    const int limit = c.max_pv == -1 ? UNBOUNDED_VERTS : RECORDED_VERTS;
    const int bounces = c.max_pv == -1 ? limit : std::min(c.max_pv - 1, limit);
    const bool tail = c.max_pv == -1 || c.max_pv - 1 > limit;
    const int lights = s.num_area_lights;
    int copies = 1;
    while (2 * copies <= EMISSION_COPIES && 2 * copies * std::max(lights, 1) <= 64 * EMISSION_COPIES) copies *= 2;
    // Workspace: counters, emission partial sums, then the path state.
    const size_t emission_bytes = BACKWARD ? (size_t)copies * lights * EMISSION_LINE * sizeof(double) : 0;
    const size_t head = (256 + emission_bytes + 255) / 256 * 256;
    const size_t per_path = 16 * 13 + 8 + (BACKWARD ? 4 + 16 * (size_t)bounces : 0);
    if (head > POOL_KEEP / 2) return WAVES_NO_MEMORY;
    cudaMemPool_t pool = nullptr;
    LMGPU_CUDA_TRY(diff_pool_of(sc->device, &pool));
    int64_t P = std::min({ c.num_samples, WAVE_PATHS, (int64_t)((POOL_KEEP - head - 256) / per_path) });
    char* mem = nullptr;
    for (;;) {
        const cudaError_t e = cudaMallocFromPoolAsync(reinterpret_cast<void**>(&mem), head + (size_t)P * per_path + 256, pool, stream);
        if (e == cudaSuccess) break;
        cudaGetLastError();
        if (e != cudaErrorMemoryAllocation) return cuda_fail(e, "cudaMallocFromPoolAsync");
        if (P <= MIN_WAVE_PATHS) return WAVES_NO_MEMORY;
        P = (P + 1) / 2;
    }
    PathState st{};
    st.counters = reinterpret_cast<uint32_t*>(mem);
    char* p = mem + head;
    auto take = [&](size_t b) { char* r = p; p += b; return r; };
    Ctx ctx;
    ctx.record = reinterpret_cast<float4*>(take(BACKWARD ? 16 * (size_t)P * bounces : 0));
    for (int q = 0; q < 2; q++) {
        st.qo[q] = reinterpret_cast<float4*>(take(16 * (size_t)P));
        st.qd[q] = reinterpret_cast<float4*>(take(16 * (size_t)P));
        st.qt[q] = reinterpret_cast<float4*>(take(16 * (size_t)P));
        st.qn[q] = reinterpret_cast<float4*>(take(16 * (size_t)P));
    }
    st.hit = reinterpret_cast<float4*>(take(16 * (size_t)P));
    st.L = reinterpret_cast<float4*>(take(16 * (size_t)P));
    st.sh_o = reinterpret_cast<float4*>(take(16 * (size_t)P));
    st.sh_d = reinterpret_cast<float4*>(take(16 * (size_t)P));
    st.sh_c = reinterpret_cast<float4*>(take(16 * (size_t)P));
    st.raster = reinterpret_cast<float2*>(take(8 * (size_t)P));
    ctx.vertices = reinterpret_cast<int32_t*>(take(BACKWARD ? 4 * (size_t)P : 0));
    for (uint32_t& q : st.cap) q = (uint32_t)P;
#if LMGPU_BOUNDS_CHECK
    for (uint32_t& q : st.cap) q = (uint32_t)std::min<int64_t>(P, check_limit_from_env("LMGPU_CHECK_QUEUE_LIMIT"));
#endif
    st.status = sc->d_status;
    ctx.s = s;
    ctx.rc.technique = TECH;
    ctx.rc.rr_depth = c.rr_depth;
    ctx.rc.max_pv = c.max_pv;
    ctx.rc.sampling = c.sampling;
    ctx.rc.seed = c.seed;
    ctx.rc.pixels = c.pixels;
    ctx.rc.inv_pixels = c.inv_pixels;
    ctx.rc.sample_base = c.sample_offset;
    ctx.rc.order = c.order;
    ctx.scale = c.scale;
    ctx.albedo = c.albedo;
    ctx.emission_of = c.emission;
    ctx.image = image;
    ctx.dL = dL;
    ctx.stride = P;
    ctx.hit_no = 0;
    ctx.d_emission = reinterpret_cast<double*>(mem + 256);
    ctx.copies = copies;
    cudaError_t e = emission_bytes ? cudaMemsetAsync(ctx.d_emission, 0, emission_bytes, stream) : cudaSuccess;
    auto closest = k_trace_persistent<STACK, TRACE_CLOSEST, PathRayIO<false>>;
    auto both = k_trace_persistent<STACK, TRACE_MIXED, BounceIO<Ctx>>;
    auto any = k_trace_persistent<STACK, TRACE_ANY, ShadowIO<Ctx>>;
    auto work = [&](int word) { return work_counter(st.counters, word); };
    for (int64_t base = 0; base < c.num_samples && e == cudaSuccess; base += P) {
        const int64_t n = std::min(P, c.num_samples - base);
        const int64_t full = (n + 127) / 128;
        const unsigned shade = (unsigned)std::min<int64_t>(full, 148 * 8);
        auto grid = [&](auto kernel, int64_t blocks) { return (unsigned)std::min<int64_t>(blocks, resident_blocks(kernel)); };
        ctx.rc.path_base = base;
        k_wave_begin<<<1, 128, 0, stream>>>(st.counters);
        k_pt_init<TECH, Ctx><<<(unsigned)full, 128, 0, stream>>>(ctx, st, n, 0);
        for (int k = 1; k <= bounces; k++) {
            const int qin = (k - 1) & 1;
            const auto io = ray_queue<false>(st, qin, ring_rays(k), nullptr);
            ctx.hit_no = k - 1;
            if (TECH == LMGPU_RENDER_PT) {
                closest<<<grid(closest, full), 128, 0, stream>>>(s, io, sc->d_status, work(ring_work(k)), nullptr);
            } else {
                const BounceIO<Ctx> bio{ io, shadow_queue(st, ring_shadow(k - 1), ctx) };
                both<<<grid(both, 2 * full), 128, 0, stream>>>(s, bio, sc->d_status, work(ring_work(k)), nullptr);
            }
            k_pt_shade<TECH, Ctx><<<shade, 128, 0, stream>>>(ctx, st, k, qin, nullptr);
        }
        if (TECH != LMGPU_RENDER_PT) {
            ctx.hit_no = bounces;
            any<<<grid(any, full), 128, 0, stream>>>(s, shadow_queue(st, ring_shadow(bounces), ctx), sc->d_status,
                                                     work(ring_shadow_work(bounces)), nullptr);
        }
        if (tail) k_diff_tail<TECH, BACKWARD><<<shade, 128, 0, stream>>>(ctx, c, st, bounces & 1, bounces + 1, da, de, sc->d_status);
        if constexpr (BACKWARD) k_diff_flush<<<(unsigned)full, 128, 0, stream>>>(ctx, c, st, n, da);
        else k_diff_splat<<<(unsigned)full, 128, 0, stream>>>(ctx, st, n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && emission_bytes) {
        k_diff_emission<<<(unsigned)((3 * (int64_t)lights + 3) / 4), 128, 0, stream>>>(ctx.d_emission, copies, lights, de);
        e = cudaGetLastError();
    }
    const cudaError_t f = cudaFreeAsync(mem, stream);
    if (e != cudaSuccess) return cuda_fail(e, "differentiable render wave");
    if (f != cudaSuccess) return cuda_fail(f, "cudaFreeAsync");
    return LMGPU_OK;
}

// Whether a budget runs as waves. Waves pay for their launches (0.2 ms a pass) and for
// path state in memory; one thread per sample for divergence, which grows with the
// tree. Forward + backward of refined Cornell boxes, one thread -> waves, ms on the device
// (pt: 6 vertices; pt.direct: 6; pt.mis: 9):
//   samples                              2^18         2^19         2^20         2^21         2^23
//   pt      576 triangles, 512 x 512     0.37 -> 0.67 0.58 -> 0.84 1.06 -> 1.20 2.05 -> 1.91 8.20 -> 6.10
//   pt      36,864, 512 x 512            0.53 -> 1.02 0.85 -> 1.24 1.55 -> 1.74 2.94 -> 2.71 11.9 -> 8.38
//   direct  144, 160 x 160                            1.24 -> 1.33 2.49 -> 2.38 4.86 -> 4.51 20.3 -> 17.4
//   direct  576, 160 x 160                            1.01 -> 1.25 2.01 -> 2.16 4.23 -> 3.96 19.1 -> 15.1
//   mis     36,864, 512 x 512            1.11 -> 1.78 1.72 -> 2.20 3.62 -> 3.00 7.06 -> 4.58 29.0 -> 14.0
//   direct  144, 64 x 64                 0.84 -> 1.09 1.43 -> 1.71 2.70 -> 3.01 5.18 -> 5.77 21.1 -> 23.4
//   mis     2,304, 64 x 64               0.86 -> 1.34 1.50 -> 1.89 3.06 -> 3.02 6.14 -> 5.35 25.7 -> 20.8
// Light samples seen from the camera add up in the pixels that see the light, all in one
// launch: on images of few pixels that holds waves up, unless the tree is large.
bool waves_pay(const DiffConsts& c, int64_t triangles)
{
    const bool nee = c.technique != LMGPU_RENDER_PT;
    if (nee && c.pixels < (1 << 13) && triangles < 1024) return false;
    return c.num_samples >= int64_t(1) << (nee && c.pixels >= (1 << 14) ? 20 : 21);
}

bool diff_as_waves(const LmgpuScene* sc, const DiffConsts& c, cudaStream_t stream)
{
    if (sc->dev.layout == LMGPU_LAYOUT_NAIVE || sc->rdev.num_tris == 0 || !waves_pay(c, sc->rdev.num_tris)) return false;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return cap == cudaStreamCaptureStatusNone;
}

// Whether one thread per sample takes samples in the renders' order (SampleOrder). Its
// warps then walk alike, and add to the same pixels and triangles one after the other. Index ->
// renders' order, forward + backward, us:
//   65 x 49 x 4, pt.direct, 144 triangles                     177 -> 186
//   2^15 / 2^18 / 2^20, pt, 2,304 triangles, 256 x 128        323 -> 351 / 565 -> 463 / 1608 -> 1144
//   2^18 / 2^20 / 2^23, pt.mis, 576 triangles, 64 x 64        853 -> 785 / 3125 -> 2756 / 26600 -> 23550
//   2^18 / 2^20 / 2^23, pt.direct, 36 triangles, 64 x 64      1049 -> 1144 / 3358 -> 3870 / 26360 -> 27900
bool ordered_pays(const DiffConsts& c, int64_t triangles)
{
    return c.num_samples >= (int64_t(1) << 18) && (c.technique == LMGPU_RENDER_PT || triangles >= 512);
}

template <int TECH, bool NAIVE, int STACK>
int launch_diff_l(LmgpuScene* sc, DiffConsts c, bool backward, float* image, const float* dL, float* da,
                  float* de, cudaStream_t st)
{
    if (!ordered_pays(c, sc->rdev.num_tris)) c.order.ordered = 0;
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((c.num_samples + 127) / 128, 148 * 16));
    auto launch = [&](auto kernel) { kernel<<<blocks, 128, 0, st>>>(sc->rdev, c, image, dL, da, de, sc->d_status); };
    if (blocks <= 148 * 4) {
        if (backward) launch(k_diff<TECH, NAIVE, STACK, true, 4>);
        else launch(k_diff<TECH, NAIVE, STACK, false, 4>);
    } else {
        if (backward) launch(k_diff<TECH, NAIVE, STACK, true, 8>);
        else launch(k_diff<TECH, NAIVE, STACK, false, 8>);
    }
    LMGPU_CUDA_TRY(cudaGetLastError());
    return LMGPU_OK;
}

template <int TECH, int STACK>
int launch_diff_s(LmgpuScene* sc, const DiffConsts& c, bool backward, float* image, const float* dL, float* da,
                  float* de, cudaStream_t st)
{
    if (sc->dev.layout == LMGPU_LAYOUT_NAIVE) return launch_diff_l<TECH, true, 1>(sc, c, backward, image, dL, da, de, st);
    return launch_diff_l<TECH, false, STACK>(sc, c, backward, image, dL, da, de, st);
}

template <int TECH>
int launch_diff_t(LmgpuScene* sc, const DiffConsts& c, bool backward, float* image, const float* dL, float* da,
                  float* de, cudaStream_t st)
{
    const int cap = sc->rdev.stack_cap, cap8 = sc->rdev.stack8_cap;
    if (cap8 <= 256 && cap <= TAIL_STACK && diff_as_waves(sc, c, st)) {
        int rc;
        if (cap8 <= 32)
            rc = backward ? run_diff_waves<TECH, 32, true>(sc, c, image, dL, da, de, st)
                          : run_diff_waves<TECH, 32, false>(sc, c, image, dL, da, de, st);
        else
            rc = backward ? run_diff_waves<TECH, 256, true>(sc, c, image, dL, da, de, st)
                          : run_diff_waves<TECH, 256, false>(sc, c, image, dL, da, de, st);
        if (rc != WAVES_NO_MEMORY) return rc;
    }
    if (cap <= 32) return launch_diff_s<TECH, 32>(sc, c, backward, image, dL, da, de, st);
    if (cap <= 64) return launch_diff_s<TECH, 64>(sc, c, backward, image, dL, da, de, st);
    if (cap <= 256) return launch_diff_s<TECH, 256>(sc, c, backward, image, dL, da, de, st);
    return fail(LMGPU_ERR_UNSUPPORTED, "BVH too deep for the differentiable path (stack 256)");
}

int launch_diff(LmgpuScene* sc, const LmgpuRenderParams* p, const LmgpuDiffParams* dp, bool backward, float* image,
                const float* dL, float* da, float* de, cudaStream_t st, LmgpuRenderStats* stats)
{
    if (!sc || !p) return fail(LMGPU_ERR_INVALID, "null argument");
    if (const int rc = check_scene_device(sc)) return rc;
    if (!sc->dev.cam.valid) return fail(LMGPU_ERR_INVALID, "scene has no camera");
    if (p->num_samples <= 0) return fail(LMGPU_ERR_INVALID, "num_samples must be positive");
    if (p->sample_offset < 0) return fail(LMGPU_ERR_INVALID, "negative sample offset");
    if (!sample_range_ok(p->sample_offset, p->num_samples)) return fail(LMGPU_ERR_INVALID, "sample indices reach 2^53");
    if (p->technique < LMGPU_RENDER_PT || p->technique > LMGPU_RENDER_PT_MIS) return fail(LMGPU_ERR_INVALID, "unknown technique");
    DiffConsts c;
    std::memset(&c, 0, sizeof(c));
    c.technique = p->technique;
    c.rr_depth = p->rr_depth;
    c.max_pv = p->max_path_vertices;
    c.sampling = p->sampling;
    c.seed = p->seed;
    c.sample_offset = p->sample_offset;
    c.num_samples = p->num_samples;
    c.pixels = (int64_t)sc->dev.cam.width * sc->dev.cam.height;
    c.inv_pixels = 1.0 / double(c.pixels);
    c.order = sample_order(p->num_samples, sc->dev.cam.width, sc->dev.cam.height, p->sampling == LMGPU_SAMPLING_STRATIFIED);
    c.scale = float(double(c.pixels) / double(p->num_samples));
    c.albedo = dp ? dp->albedo : nullptr;
    c.emission = dp ? dp->emission : nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (stats) {
        LMGPU_CUDA_TRY(cudaEventCreate(&e0));
        LMGPU_CUDA_TRY(cudaEventCreate(&e1));
        LMGPU_CUDA_TRY(cudaEventRecord(e0, st));
    }
    int rc;
    switch (p->technique) {
    case LMGPU_RENDER_PT: rc = launch_diff_t<LMGPU_RENDER_PT>(sc, c, backward, image, dL, da, de, st); break;
    case LMGPU_RENDER_PT_DIRECT: rc = launch_diff_t<LMGPU_RENDER_PT_DIRECT>(sc, c, backward, image, dL, da, de, st); break;
    default: rc = launch_diff_t<LMGPU_RENDER_PT_MIS>(sc, c, backward, image, dL, da, de, st); break;
    }
    if (stats) {
        std::memset(stats, 0, sizeof(*stats));
        stats->paths = p->num_samples;
        if (rc == LMGPU_OK) {
            cudaEventRecord(e1, st);
            cudaEventSynchronize(e1);
            float ms = 0.0f;
            cudaEventElapsedTime(&ms, e0, e1);
            stats->device_ms = ms;
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
    }
    return rc;
}

}  // namespace

int release_diff_pool(int device)
{
    DiffPool& p = diff_pool(device);
    std::lock_guard<std::mutex> lock(p.mu);
    if (p.pool) LMGPU_CUDA_TRY(cudaMemPoolTrimTo(p.pool, 0));
    return LMGPU_OK;
}

}  // namespace lmgpu

using namespace lmgpu;

extern "C" {

int lmgpu_adjoint_forward(LmgpuScene* scene, const LmgpuRenderParams* params, const LmgpuDiffParams* diff,
                          float* image_device, void* stream, LmgpuRenderStats* stats)
{
    if (!image_device) return fail(LMGPU_ERR_INVALID, "null image");
    return launch_diff(scene, params, diff, false, image_device, nullptr, nullptr, nullptr,
                       static_cast<cudaStream_t>(stream), stats);
}

int lmgpu_adjoint_backward(LmgpuScene* scene, const LmgpuRenderParams* params, const LmgpuDiffParams* diff,
                           const float* dL_dimage_device, float* d_albedo_device, float* d_emission_device,
                           void* stream, LmgpuRenderStats* stats)
{
    if (!dL_dimage_device || !d_albedo_device || !d_emission_device)
        return fail(LMGPU_ERR_INVALID, "null gradient buffer");
    return launch_diff(scene, params, diff, true, nullptr, dL_dimage_device, d_albedo_device, d_emission_device,
                       static_cast<cudaStream_t>(stream), stats);
}

}  // extern "C"
