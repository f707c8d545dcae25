// Device data layout of a built scene, shared by the host builder (g++) and
// the CUDA kernels (nvcc). Plain structs only.
//
// HBM layout of an accelerator:
//   Bvh8Node[]   128 B each, the 8-wide compressed collapse of a binary tree
//                that every traversal walks.
//   TriRecord[]  48 B each, the reference TriAccel constants
//                (triaccel.h:31-47) in the wide tree's leaf order; leaves
//                are contiguous runs ended by TRI_LAST_IN_LEAF.
//   LeafBox[]    32 B each, the binary leaf's box of every triangle.
// and, for the reference's own depth-first walk (rays the wide walk hands back,
// work counts, full hit records) and, of the render tree, for render rays walked by
// one thread and for the order of hits (order_takes):
//   Bvh2Node[]   64 B each, DFS pre-order, both children's boxes stored in
//                the parent; a child reference >= 0 is an internal node index, < 0
//                a leaf whose first TriRecord is ~ref.
//   TriRecord[]  the same records in the binary tree's leaf order
//                (bvhTriIndices of scene.bvh.cpp:193).
#pragma once
#include <stdint.h>

namespace lmgpu {

constexpr uint32_t TRI_AXIS_MASK = 3u;          // TriAccel::k (3 = degenerate)
constexpr uint32_t TRI_LAST_IN_LEAF = 1u << 31; // last record of a leaf

struct alignas(16) Bvh2Node {
    // Per axis: left.lo, left.hi, right.lo, right.hi
    float bx[4];
    float by[4];
    float bz[4];
    int32_t left, right;   // child references
    int32_t axis;          // split axis of this node (near-first order)
    int32_t split;         // position of the right child's first triangle (set_splits)
};
static_assert(sizeof(Bvh2Node) == 64, "Bvh2Node is 64 B");

// 8-wide compressed node (after Ylitie, Karras, Laine, "Efficient Incoherent
// Ray Traversal on GPUs Through Compressed Wide BVHs", HPG 2017): up to eight
// children, each child's box on a per-node grid of 8-bit planes. Axis k's planes sit
// at origin[k] + q * 2^(e_k - 127), e_k byte k of `exps`; collapse_bvh8
// (builder.cpp) rounds them outward with a margin, so a box only grows.
// Slot s holds a child whose centre lies towards the corner of the node given
// by s's bits (bit k set: the high side of axis k), so that the slots taken in
// the order s ^ (signs of the ray's direction) run roughly near to far.
// Internal children are consecutive nodes from `child_base` in slot order; a
// leaf child is the run of TriRecords from start[s], ended by TRI_LAST_IN_LEAF.
// A visit reads the first 96 bytes as three 32-byte loads; start[] is read
// when a leaf is tested.
struct alignas(128) Bvh8Node {
    float origin[3];
    uint32_t exps;         // e_x | e_y << 8 | e_z << 16 | mask of internal children << 24
    uint32_t child_base;
    uint32_t valid;        // mask of the slots in use
    uint32_t pad0[2];
    uint32_t lox[2], loy[2], loz[2], hix[2];   // byte s of each pair: slot s
    uint32_t hiy[2], hiz[2], pad1[4];
    uint32_t start[8];
};
static_assert(sizeof(Bvh8Node) == 128, "Bvh8Node is 128 B");

// Box of a triangle's leaf in the binary tree (lo.xyz hi.x | hi.yz - -), by
// position in the wide tree's triangle array.
struct alignas(16) LeafBox {
    float lo[3], hi[3];
    float pad[2];
};
static_assert(sizeof(LeafBox) == 32, "LeafBox is 32 B");

struct alignas(16) TriRecord {
    uint32_t k_flags;      // TriAccel::k | TRI_LAST_IN_LEAF
    float n_u, n_v, n_d;
    float a_u, a_v, b_nu, b_nv;
    float c_nu, c_nv;
    uint32_t tri_id;       // reference TriAccel index (primitive-major)
    uint32_t prim;         // primitive index
};
static_assert(sizeof(TriRecord) == 48, "TriRecord is 48 B");

}  // namespace lmgpu
