// Persistent traversal kernel shared by the intersection API and the path
// tracer's ray and shadow queues. The I/O policy supplies the ray count, the
// rays and what to do with each result.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <mutex>
#include <type_traits>
#include <unordered_map>
#include "internal.h"
#include "trace.cuh"
#include "trace8.cuh"

namespace lmgpu {

// Scheduling constants of the persistent traversal kernel. They change only
// when lanes take new rays and when a descent pauses, never a ray's result.
// Measured on the soup, camera, bounce and shadow rays named in trace8.cuh:
// pausing below 24 descending lanes beat 4, 8, 12 and 16 on all four (2.46, 2.09,
// 1.87, 1.74 -> 1.66 ms on the soup) and 26 / 28 changed 0 / +3 %; refilling at 8 idle
// lanes equals 4 and 6, 12 is slower by 6-12 % on incoherent rays.
#ifndef LMGPU_TRACE_REFILL_MIN
#define LMGPU_TRACE_REFILL_MIN 8      // idle lanes that trigger a refill
#endif
#ifndef LMGPU_TRACE_EXIT_BELOW
#define LMGPU_TRACE_EXIT_BELOW 24     // pause a descent when fewer lanes descend
#endif
// Resident blocks of 128 threads per SM: 8 (64 registers, no spills); 7 and 9
// (71 and 56 registers) were 4 % slower on all four ray sets.
#ifndef LMGPU_TRACE_MIN_BLOCKS
#define LMGPU_TRACE_MIN_BLOCKS 8
#endif
#ifndef LMGPU_TRACE_SHARED_STACK
#define LMGPU_TRACE_SHARED_STACK 10   // stack entries per lane kept in shared memory
#endif

// I/O policies whose rays each belong to their own scene (a multi-scene
// batch) declare PER_RAY_SCENE = true and supply ray_scene(j).
template <class IO, class = void>
struct per_ray_scene : std::false_type {};
template <class IO>
struct per_ray_scene<IO, std::void_t<decltype(IO::PER_RAY_SCENE)>> : std::bool_constant<IO::PER_RAY_SCENE> {};

// Render rays (the path tracer's queues) declare RENDER = true: their
// triangle tests take triaccel_intersect_fast; the intersection API keeps
// the reference's exact arithmetic and answers.
template <class IO, class = void>
struct render_rays : std::false_type {};
template <class IO>
struct render_rays<IO, std::void_t<decltype(IO::RENDER)>> : std::bool_constant<IO::RENDER> {};

// Which question a traversal launch asks of its rays. TRACE_MIXED answers two queues
// in one launch: io.closest's rays first, then io.shadow's (any hit).
constexpr int TRACE_CLOSEST = 0, TRACE_ANY = 1, TRACE_MIXED = 2;
// Added to one of these: a launch of at most 32 rays for each of its warps. Its warps share
// the rays out evenly at the start, without the work counter, on as few lanes as their
// number allows: such a launch takes as long as its slowest warp, and lanes of a warp wait
// for one another. 512 rays x 4,096 triangles, whole call: 49 -> 38 us (with the
// counter's memset gone); a 67 x 45 x 8 preview 290 -> 270 us. (The same as a run-time
// branch of one kernel cost the large launches 2 to 4 %.)
constexpr int TRACE_SPREAD = 4;

// Adds each lane's counts to counts[0] (box tests: eight per node visit) and
// counts[1] (TriAccel tests); the whole warp calls it.
__device__ __forceinline__ void add_trace_stats(const TraceStats& st, unsigned long long* counts)
{
    unsigned long long a = st.nodes, b = st.tris;
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31u) == 0) { atomicAdd(counts, a); atomicAdd(counts + 1, b); }
}

// Rays handed back to the reference's own walk (see HIT_TIED) wait in a list of
// BACK_LIST per warp. A warp whose list is more than half full takes no new
// rays, and walks the list once all its lanes are idle: no lane's state is then live
// across that walk. (Walking each where it came up, through an out-of-line
// function, cost the exact kernel 7 local-memory accesses a ray: 2.82 ms on 2^23
// soup rays.)
constexpr int BACK_LIST = 64;

// The reference's walk of ray `in`; a stack overflow is flagged and gives a miss.
template <bool ANY_HIT, int STACK>
__device__ __forceinline__ void reference_walk(const DeviceScene& s, int32_t* status, const RayIn& in, TraversalRay& r,
                                               Hit& h)
{
    int2 stack[STACK];
    setup_ray(r, in);
    if (!trace_bvh2<ANY_HIT>(s.bvh2, s.tris, s.root_ref, s.root_box, r, h, stack,
                             s.stack_cap < STACK ? s.stack_cap : STACK, nullptr)) {
        atomicOr(status, STATUS_STACK_OVERFLOW);
        h.tri = -1;
    }
}

// Persistent traversal with per-lane ray replacement: a warp keeps tracing
// until the batch is exhausted; lanes whose ray has finished take the next
// rays from a global counter (one warp-aggregated atomic per refill), so short
// rays do not idle behind long ones. Lanes alternate "descend" and "test the
// leaves of one visited node". A lane that finds leaves while it holds none
// postpones them and goes on descending with the rest of the warp; the
// descent ends when every lane still in it holds leaves, and pauses once fewer
// than LMGPU_TRACE_EXIT_BELOW lanes are in it. When a ray's triangles are
// tested thus depends on the warp's other rays; in which order does not, nor does its
// result (see the candidate rules in trace8.cuh). (Without postponing: 1.97 against 1.66 ms on the soup,
// 2.00 / 1.59 and 1.87 / 1.59 ms on the bounce and shadow rays.)
// For a multi-scene I/O policy each lane switches to its new ray's scene at
// refill; an empty scene is a miss. The COUNT instantiation (measurement
// runs only) also adds the rays' box and TriAccel tests to counts[0..1].
template <int STACK, int KIND, class IO, bool COUNT = false>
__global__ void __launch_bounds__(128, LMGPU_TRACE_MIN_BLOCKS)
k_trace_persistent(const __grid_constant__ DeviceScene s, const __grid_constant__ IO io, int32_t* status,
                   unsigned long long* next_ray, unsigned long long* counts)
{
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int MODE = KIND & ~TRACE_SPREAD;
    constexpr bool SPREAD = (KIND & TRACE_SPREAD) != 0;
    constexpr bool RENDER = render_rays<IO>::value;
    constexpr bool TABLE = per_ray_scene<IO>::value;
    constexpr int SH = LMGPU_TRACE_SHARED_STACK;
    __shared__ uint2 stack_sh[SH][128];
    uint2 stack_local[STACK > SH ? STACK - SH : 1];
    __shared__ int64_t back_sh[RENDER ? 1 : 4][RENDER ? 1 : BACK_LIST];   // rays handed back (exact)
    int back = 0;                              // entries in the warp's list
    bool hand_back = false;                    // this lane's ray joins it
    // 32 bits where they save the closest-hit walk its spills: the queues of one-scene waves, also
    // the two of a mixed launch, hold fewer than 2^31 rays (a path's state takes 216 bytes and adds
    // at most two, so that more would need 230 GB).
    using Index = std::conditional_t<RENDER && !TABLE, int32_t, int64_t>;
    Index n_closest = 0;
    if constexpr (MODE == TRACE_MIXED) n_closest = (Index)io.closest.count();
    const Index n = (Index)io.count();
    const unsigned lane = threadIdx.x & 31u;
    const int cap = s.stack8_cap < STACK ? s.stack8_cap : STACK;
    const Bvh8Node* nodes = s.bvh8;
    const TriRecord* tris = s.tris8;
    TraceStats stats{ 0, 0 };
    TraversalRay r;
    Hit h;
    h.tri = -1;
    uint32_t oct = 0;
    Walk8 w;
    w.mask = 0;
    w.leaves = 0;
    w.sp = 0;
    uint32_t pend_node = 0, pend = 0;          // postponed leaves
    Index idx = -1;
    bool live = false;
    bool exhausted = n <= 0;
    bool any = MODE == TRACE_ANY;              // this lane's ray stops at its first hit
    auto load = [&](Index j) -> RayIn {
        if constexpr (MODE == TRACE_MIXED) return any ? io.shadow.load(j - n_closest) : io.closest.load(j);
        else return io.load(j);
    };
    auto store = [&](Index j) {
        if constexpr (MODE == TRACE_MIXED) {
            if (any) io.shadow.store(j - n_closest, h, r);
            else io.closest.store(j, h, r);
        } else io.store(j, h, r);
    };
    auto ray_scene = [&](Index j) -> const DeviceScene& {
        if constexpr (MODE == TRACE_MIXED) return any ? io.shadow.ray_scene(j - n_closest) : io.closest.ray_scene(j);
        else if constexpr (TABLE) return io.ray_scene(j);
        else return s;
    };
    for (;;) {
        const unsigned need = __ballot_sync(FULL, !live);
        if constexpr (!RENDER) {
            const unsigned m = __ballot_sync(FULL, hand_back);
            if (m != 0) {
                if (hand_back) back_sh[threadIdx.x >> 5][back + __popc(m & ((1u << lane) - 1u))] = idx;
                hand_back = false;
                back += __popc(m);
            }
            if (need == FULL && (exhausted ? back > 0 : back > BACK_LIST - 32)) {
                __syncwarp();
                for (int i = (int)lane; i < back; i += 32) {
                    idx = (Index)back_sh[threadIdx.x >> 5][i];
                    reference_walk<MODE == TRACE_ANY, STACK>(s, status, load(idx), r, h);
                    store(idx);
                }
                __syncwarp();
                back = 0;
            }
        }
        if (!exhausted && back <= BACK_LIST - 32 && (__popc(need) >= LMGPU_TRACE_REFILL_MIN || need == FULL)) {
            unsigned long long base = 0;
            bool take = !live;
            if constexpr (SPREAD) {            // once, with every lane idle
                const int64_t warps = (int64_t)gridDim.x * (128 / 32);
                const unsigned share = (unsigned)((n + warps - 1) / warps);
                base = (unsigned long long)(blockIdx.x * (128 / 32) + (threadIdx.x >> 5)) * share;
                take = lane < share;
                exhausted = true;
            } else {
                const int leader = __ffs(need) - 1;
                if ((int)lane == leader) base = atomicAdd(next_ray, (unsigned long long)__popc(need));
                base = __shfl_sync(FULL, base, leader);
                if (base + __popc(need) >= (unsigned long long)n) exhausted = true;
            }
            if (take) {
                idx = (Index)base + __popc(need & ((1u << lane) - 1u));
                if (base < (unsigned long long)n && idx < n) {
                    if constexpr (MODE == TRACE_MIXED) any = idx >= n_closest;
                    const RayIn in = load(idx);
                    setup_ray<true>(r, in);
                    oct = r.neg & 7u;
                    h.tri = -1;
                    live = true;
                    if constexpr (TABLE) {
                        const DeviceScene& rs = ray_scene(idx);
                        nodes = rs.bvh8;
                        tris = rs.tris8;
                        live = rs.num_tris > 0;
                    }
                    if constexpr (!RENDER) {
                        if (!exact_wide_ok(in, s.wide_limit)) {
                            live = false;
                            hand_back = true;
                        }
                    }
                    if (live) walk8_begin(w, oct);
                    else if (!hand_back) store(idx);
                }
            }
        } else if (exhausted && need == FULL && !__any_sync(FULL, hand_back)) {
            break;
        }
        if (!live) continue;
        bool ok = true;
        while (w.leaves == 0 || pend == 0) {
            if (w.leaves != 0) {               // postpone them, go on descending
                pend = w.leaves;
                pend_node = w.leaf_node;
                w.leaves = 0;
            }
            if (__all_sync(__activemask(), pend != 0)) break;
            if ((w.mask & 0xffu) == 0) {
                if (w.sp == 0) break;
                w.sp--;
                const uint2 e = w.sp < SH ? stack_sh[w.sp][threadIdx.x] : stack_local[w.sp - SH];
                w.base = e.x;
                w.mask = e.y;
            }
            const uint32_t node = walk8_next(w, oct);
            if (w.mask & 0xffu) {
                if (w.sp >= cap) { ok = false; break; }
                if (w.sp < SH) stack_sh[w.sp][threadIdx.x] = make_uint2(w.base, w.mask);
                else stack_local[w.sp - SH] = make_uint2(w.base, w.mask);
                w.sp++;
            }
            walk8_visit(w, nodes, node, r, oct);
            if (COUNT) stats.nodes += 8;
            if (!exhausted && __popc(__activemask()) < LMGPU_TRACE_EXIT_BELOW) break;
        }
        if (pend == 0) {
            pend = w.leaves;
            pend_node = w.leaf_node;
            w.leaves = 0;
        }
        bool done = false;
        if (!ok) {
            atomicOr(status, STATUS_STACK_OVERFLOW);
            h.tri = -1;
            done = true;
        } else if (pend != 0) {
            const float4* p = walk8_leaf(nodes, tris, pend_node, pend);
            for (;;) {
                const float4 q0 = __ldg(p), q1 = __ldg(p + 1), q2 = __ldg(p + 2);
                if (COUNT) stats.tris++;
                const int32_t id = static_cast<int32_t>(__float_as_uint(q2.z));
                float u, v, t;
                if constexpr (RENDER) {
                    float window;
                    if (triaccel_intersect_fast(q0, q1, q2, r, r.tmax, u, v, t) &&
                        render_candidate<MODE == TRACE_ANY>(TABLE ? ray_scene(idx) : s, (p - reinterpret_cast<const float4*>(tris)) / 3, id,
                                                            t, u, v, r, h, any, window)) {
                        r.tmax = window;
                        h.tri = id; h.t = t; h.u = u; h.v = v;
                        if (any) { done = true; break; }
                    }
                } else {
                    if (triaccel_intersect(q0, q1, q2, r, r.tmax, u, v, t)) {
                        const int64_t at = (p - reinterpret_cast<const float4*>(tris)) / 3;
                        if (any) {
                            float te;
                            if (leaf_box_exact(s.boxes8, at, r, te) && te < r.tmax) {
                                h.tri = id;
                                done = true;
                                break;
                            }
                        } else {
                            exact_candidate(s.boxes8, at, id, t, u, v, load(idx).tmax, r, h);
                        }
                    }
                }
                if (__float_as_uint(q0.x) & TRI_LAST_IN_LEAF) {
                    if (pend == 0) break;
                    p = walk8_leaf(nodes, tris, pend_node, pend);
                } else {
                    p += 3;
                }
            }
            pend = 0;
            if constexpr (!RENDER && MODE == TRACE_CLOSEST) {
                if (h.tri == HIT_TIED) {
                    hand_back = true;
                    done = true;
                }
            }
        }
        if (done) {
            w.mask = 0;
            w.leaves = 0;
            w.sp = 0;
            pend = 0;
        }
        if (pend == 0 && w.leaves == 0 && (w.mask & 0xffu) == 0 && w.sp == 0) {
            live = false;
            if (!hand_back) store(idx);
        }
    }
    if (COUNT) add_trace_stats(stats, counts);
}

// Brute-force traversal for the naive layout (one thread per ray).
template <bool ANY_HIT, class IO>
__global__ void __launch_bounds__(128) k_trace_naive(const DeviceScene s, const IO io)
{
    const int64_t n = io.count();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        TraversalRay r;
        setup_ray(r, io.load(i));
        Hit h;
        h.tri = -1;
        if (s.num_tris > 0) trace_naive<ANY_HIT>(s.tris_by_id, s.num_tris, r, h, nullptr);
        io.store(i, h, r);
    }
}

// Resident-grid size of a kernel (blocks of 128 threads), cached per kernel.
int resident_blocks_of(const void* kernel);
template <class K>
int resident_blocks(K kernel)
{
    return resident_blocks_of(reinterpret_cast<const void*>(kernel));
}

// Grid of a TRACE_SPREAD launch of at most max_rays rays, 0 if they are too many for one.
inline int64_t spread_blocks(int64_t resident, int64_t max_rays)
{
    return max_rays <= 128 * resident ? std::max<int64_t>(1, std::min<int64_t>(resident, (max_rays + 3) / 4)) : 0;
}

// Launches the traversal for `io` on `stream`: persistent kernel for the
// BVH layouts (with one of the scene's work counters, reset first, unless the
// launch is spread), brute force for the naive layout. `max_rays` is the number
// of rays.
template <bool ANY_HIT, int STACK, class IO>
int launch_trace_stack(LmgpuScene* sc, const DeviceScene& s, const IO& io, int64_t max_rays, cudaStream_t stream)
{
    if (s.layout == LMGPU_LAYOUT_NAIVE || s.num_tris == 0) {
        const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((max_rays + 127) / 128, 148 * 64));
        k_trace_naive<ANY_HIT, IO><<<blocks, 128, 0, stream>>>(s, io);
        LMGPU_CUDA_TRY(cudaGetLastError());
        return LMGPU_OK;
    }
    // Each launch takes its own counter from the scene's ring, so persistent
    // kernels queued on different streams never share one.
    constexpr int MODE = ANY_HIT ? TRACE_ANY : TRACE_CLOSEST;
    auto few = k_trace_persistent<STACK, MODE | TRACE_SPREAD, IO>;
    if (const int64_t blocks = spread_blocks(resident_blocks(few), max_rays)) {
        few<<<blocks, 128, 0, stream>>>(s, io, sc->d_status, nullptr, nullptr);
    } else {
        unsigned long long* work = sc->d_work + (sc->work_slot++ % LmgpuScene::WORK_SLOTS);
        LMGPU_CUDA_TRY(cudaMemsetAsync(work, 0, sizeof(unsigned long long), stream));
        auto k = k_trace_persistent<STACK, MODE, IO>;
        k<<<resident_blocks(k), 128, 0, stream>>>(s, io, sc->d_status, work, nullptr);
    }
    LMGPU_CUDA_TRY(cudaGetLastError());
    return LMGPU_OK;
}

// The intersection API's launch (the reference's tree). The stack bound is the wide
// walk's and that of the reference's walk a ray may be handed to.
template <bool ANY_HIT, class IO>
int launch_trace(LmgpuScene* sc, const IO& io, int64_t max_rays, cudaStream_t stream)
{
    static_assert(!render_rays<IO>::value, "renders launch their own traversals");
    const DeviceScene& s = sc->dev;
    const int cap = std::max(s.stack8_cap, s.stack_cap);
    if (cap <= 32) return launch_trace_stack<ANY_HIT, 32>(sc, s, io, max_rays, stream);
    if (cap <= 64) return launch_trace_stack<ANY_HIT, 64>(sc, s, io, max_rays, stream);
    if (cap <= 128) return launch_trace_stack<ANY_HIT, 128>(sc, s, io, max_rays, stream);
    if (cap <= 256) return launch_trace_stack<ANY_HIT, 256>(sc, s, io, max_rays, stream);
    return fail(LMGPU_ERR_UNSUPPORTED, "BVH deeper than the largest compiled traversal stack (256)");
}

}  // namespace lmgpu
