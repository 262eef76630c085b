// Collapse of a binary mesh BVH to the four-wide form (see wide_bvh.h).
#include "wide_bvh.h"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace slim {

namespace {

void box_of(const SlimBVHNode &n, float lo[3], float hi[3]) {
    lo[0] = n.aabb.min.x; lo[1] = n.aabb.min.y; lo[2] = n.aabb.min.z;
    hi[0] = n.aabb.max.x; hi[1] = n.aabb.max.y; hi[2] = n.aabb.max.z;
}

float from_bits(uint32_t u) {
    float f;
    memcpy(&f, &u, 4);
    return f;
}
uint32_t to_bits(float f) {
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
}

// The 16 bits of a plane at offset x >= 0, its float's lower half being
// `below`: the largest that decodes to x or less, or the smallest that
// decodes to x or more.  (Offset 0 with bits below reads as a denormal,
// which the walk's margin covers.)
uint32_t plane_bits(double x, bool up, uint32_t below) {
    const float f = (float)x;
    uint32_t bits = to_bits(f);                      // floats of one sign order as their bits
    if (up) {
        if ((double)f < x) bits++;
        const uint32_t h = bits >> 16;
        return (h << 16 | below) < bits ? h + 1 : h;
    }
    if ((double)f > x) bits--;
    const uint32_t h = bits >> 16;
    return h && (h << 16 | below) > bits ? h - 1 : h;
}

double surface(const SlimBVHNode &n) {
    const double x = (double)n.aabb.max.x - n.aabb.min.x, y = (double)n.aabb.max.y - n.aabb.min.y,
                 z = (double)n.aabb.max.z - n.aabb.min.z;
    return x * y + y * z + z * x;
}

}  // namespace

bool boxes_nest(const SlimBVHNode *nodes, uint32_t count) {
    for (uint32_t i = 0; i < count; i++) {
        float lo[3], hi[3];
        box_of(nodes[i], lo, hi);
        for (int a = 0; a < 3; a++)
            if (!(std::fabs(lo[a]) < 1e18f && std::fabs(hi[a]) < 1e18f)) return false;
        if (nodes[i].leaf_count) continue;
        for (uint32_t c = nodes[i].first_index; c < nodes[i].first_index + 2; c++) {
            float clo[3], chi[3];
            box_of(nodes[c], clo, chi);
            for (int a = 0; a < 3; a++)
                if (!(clo[a] >= lo[a] && chi[a] <= hi[a])) return false;
        }
    }
    return true;
}

float wide_offset(const uint32_t words[2], int s) {
    return from_bits(s & 1 ? words[s >> 1] : words[s >> 1] << 16);
}

uint32_t most_wide_nodes(const SlimBVHNode *nodes, uint32_t node_count) {
    uint32_t inner = 0;
    for (uint32_t i = 0; i < node_count; i++) inner += !nodes[i].leaf_count;
    return (uint32_t)((2ull * inner + 1) / 3);
}

uint32_t build_wide_bvh(const SlimBVHNode *nodes, uint32_t node_count, const float *hot, uint32_t stack,
                        std::vector<WideNode> &out, std::vector<WideLeaf> &leaves, float &extent) {
    if (!node_count || nodes[0].leaf_count || !boxes_nest(nodes, node_count)) return kNoWideBVH;
    const size_t root = out.size(), first_leaf = leaves.size();
    const size_t most = most_wide_nodes(nodes, node_count);
    size_t leaf_nodes = 0;
    for (uint32_t i = 0; i < node_count; i++) leaf_nodes += nodes[i].leaf_count != 0;
    std::vector<uint32_t> source{0};       // binary node of every wide node from `root` on
    std::vector<uint32_t> waiting{0};      // nodes a walk may have waiting when it enters it
    source.reserve(node_count / 2);
    waiting.reserve(node_count / 2);
    for (size_t w = 0; w < source.size(); w++) {
        // open the largest inner child until four are reached
        uint32_t child[4], count = 0;
        double area[4];                              // of an inner child's box; a leaf is not opened
        auto put = [&](uint32_t k, uint32_t node) {
            child[k] = node;
            area[k] = nodes[node].leaf_count ? -1.0 : surface(nodes[node]);
        };
        put(count++, nodes[source[w]].first_index);
        put(count++, nodes[source[w]].first_index + 1);
        while (count < 4) {
            uint32_t open = 0;
            for (uint32_t k = 1; k < count; k++)
                if (area[k] > area[open]) open = k;
            if (area[open] < 0.0) break;
            const uint32_t first = nodes[child[open]].first_index;
            put(open, first);
            put(count++, first + 1);
        }
        WideNode n{};
        float far_corner[3];
        box_of(nodes[source[w]], n.origin, far_corner);
        for (uint32_t k = 0; k < 4; k++) {
            uint32_t lo_bits[3], hi_bits[3];
            n.child[k] = kWideLeaf;
            for (int a = 0; a < 3; a++) {
                lo_bits[a] = to_bits(1e30f) >> 16;
                hi_bits[a] = to_bits(-1e30f) >> 16;
            }
            if (k < count) {
                const SlimBVHNode &c = nodes[child[k]];
                float lo[3], hi[3];
                box_of(c, lo, hi);
                for (int a = 0; a < 3; a++) {
                    lo_bits[a] = plane_bits((double)lo[a] - n.origin[a], false, k & 1 ? n.lo[a][k >> 1] : 0u);
                    hi_bits[a] = plane_bits((double)hi[a] - n.origin[a], true, k & 1 ? n.hi[a][k >> 1] : 0u);
                }
                if (c.leaf_count) {
                    n.child[k] = kWideLeaf | (uint32_t)leaves.size();
                    WideLeaf leaf{};
                    leaf.node = c;
                    for (uint32_t t = 0; t < c.leaf_count && t < 2; t++)
                        memcpy(leaf.triangles[t], hot + 12 * (size_t)(c.first_index + t), sizeof(leaf.triangles[t]));
                    leaves.push_back(leaf);
                } else {
                    n.child[k] = (uint32_t)(root + source.size());
                    source.push_back(child[k]);
                    waiting.push_back(waiting[w] + count - 1);
                }
            }
            for (int a = 0; a < 3; a++) {
                n.lo[a][k >> 1] |= lo_bits[a] << (16 * (k & 1));
                n.hi[a][k >> 1] |= hi_bits[a] << (16 * (k & 1));
            }
        }
        out.push_back(n);
        if (waiting[w] + count - 1 > stack || leaves.size() >= kWideLeaf || root + source.size() >= kWideLeaf ||
            source.size() > most || leaves.size() - first_leaf > leaf_nodes) {      // no tree
            out.resize(root);
            leaves.resize(first_leaf);
            return kNoWideBVH;
        }
    }
    float lo[3], hi[3], largest = 0.0f;
    box_of(nodes[0], lo, hi);
    for (int a = 0; a < 3; a++) largest = std::max({largest, std::fabs(lo[a]), std::fabs(hi[a])});
    extent = 1.05f * largest + 1e-12f;     // a rounded offset is at most 2^-7 of itself, hence of 2 largest, further out
    return (uint32_t)root;
}

}  // namespace slim
