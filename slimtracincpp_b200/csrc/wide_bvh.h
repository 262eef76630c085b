// Four-wide form of a mesh BVH for the persistent mesh walks.
//
// The uploaded binary BVH (scene/bvh.h:5-21) is collapsed, node by node, to
// nodes of up to four children whose boxes are rounded outwards to 16 bits a
// plane.  A walk over it reaches every leaf that the binary walk reaches (a
// box holds its children's boxes, and the slab test is monotonic in the
// planes), and tests each leaf's own, unrounded box before its triangles, so
// both find the same hits.
#pragma once
#include <cstdint>
#include <vector>
#include "slimtracer_b200.h"

namespace slim {

// 80 bytes, five 16-byte loads.  A plane is origin + a 16-bit float (the
// upper half of a float's bits).  Slots 2k and 2k + 1 share word k of an
// axis: the even slot's plane is the word's lower half, shifted up; the odd
// slot's is the whole word read as a float, chosen with the lower half in
// place.  An empty slot's box is inside out.
struct alignas(16) WideNode {
    float origin[3];
    uint32_t _pad;
    uint32_t child[4];              // a node's index, or kWideLeaf | a leaf record's
    uint32_t lo[3][2], hi[3][2];    // by axis
};
static_assert(sizeof(WideNode) == 80, "WideNode is five 16-byte words");

// A leaf: the binary node's 32 bytes (its box, first triangle, count) and the
// 48 hot bytes of its first two triangles, on one 128-byte line.
struct alignas(16) WideLeaf {
    SlimBVHNode node;
    float triangles[2][12];
};
static_assert(sizeof(WideLeaf) == 128, "WideLeaf is one cache line");

constexpr uint32_t kWideLeaf = 0x80000000u;
constexpr uint32_t kNoWideBVH = 0xFFFFFFFFu;   // DevMesh::wide_root of a mesh without the wide form

// The plane that slot s of an axis' words decodes to, relative to the origin.
float wide_offset(const uint32_t words[2], int s);

// Appends the wide form of `nodes` (a checked binary BVH whose root is an
// inner node) to `out` and `leaves` and returns the index of its root.
// `hot` holds 12 floats per triangle.  Returns kNoWideBVH, appending nothing,
// when a node's box does not hold its children's boxes or a plane is not
// finite (or beyond 1e18), which the argument above needs, when a walk could
// have more than `stack` nodes waiting, or when nodes share children, so that
// the form would hold many copies of them.  `extent`: no plane of the form,
// rounded or not, is further from the mesh's origin.
uint32_t build_wide_bvh(const SlimBVHNode *nodes, uint32_t node_count, const float *hot, uint32_t stack,
                        std::vector<WideNode> &out, std::vector<WideLeaf> &leaves, float &extent);

// Most nodes the wide form of a binary BVH can have.  A wide node with four
// children takes the place of three inner nodes, one with fewer has leaves only;
// with F of the former and P of the latter, P <= 3 F + 1 and there are at least
// 3 F + P inner nodes.
uint32_t most_wide_nodes(const SlimBVHNode *nodes, uint32_t node_count);

// Every box finite (within 1e18) and inside its parent's: a slab test that
// passes for a node then passes for everything above it.
bool boxes_nest(const SlimBVHNode *nodes, uint32_t count);

}  // namespace slim
