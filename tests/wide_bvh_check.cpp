// Host check of the four-wide mesh BVH (csrc/wide_bvh.cpp), built and run by
// test_wide_bvh.py: reads a binary BVH, builds the wide form and compares the
// leaves that rays reach through both, with the device's arithmetic.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <set>
#include <vector>

#include "wide_bvh.h"

using namespace slim;

struct V { float x, y, z; };
struct Ray { V o, rcp, so; bool n[3]; };

static float maxr(float a, float b) { return a > b ? a : b; }
static float minr(float a, float b) { return a < b ? a : b; }
static float at(const V &v, int a) { return a == 0 ? v.x : a == 1 ? v.y : v.z; }

static bool slab(const Ray &r, const SlimAABB &b, float &nearD, float &farD) {
    float t0[3], t1[3];
    for (int a = 0; a < 3; a++) {
        const float mn = a == 0 ? b.min.x : a == 1 ? b.min.y : b.min.z, mx = a == 0 ? b.max.x : a == 1 ? b.max.y : b.max.z;
        t0[a] = fmaf(r.n[a] ? mx : mn, at(r.rcp, a), at(r.so, a));
        t1[a] = fmaf(r.n[a] ? mn : mx, at(r.rcp, a), at(r.so, a));
    }
    const float m = maxr(t0[0], maxr(t0[1], t0[2]));
    nearD = 0 > m ? 0.0f : m;
    farD = minr(t1[0], minr(t1[1], t1[2]));
    return nearD <= farD;
}

static uint32_t wide_hits(const WideNode &n, const Ray &r, float extent, float tmax) {
    uint32_t hits = 0;
    for (int s = 0; s < 4; s++) {
        float t0 = 0.0f, t1 = tmax;
        for (int a = 0; a < 3; a++) {
            const bool along = !(fabsf(at(r.rcp, a)) < 1e18f);
            const float rcp = along ? copysignf(1e18f, at(r.rcp, a)) : at(r.rcp, a), so = along ? -at(r.o, a) * rcp : at(r.so, a);
            const float e = fmaf(extent, fabsf(rcp), fabsf(so)) * (along ? 0x1p-16f : 0x1p-21f);
            const float lo = wide_offset(n.lo[a], s), hi = wide_offset(n.hi[a], s);
            t0 = fmaxf(t0, fmaf(r.n[a] ? hi : lo, rcp, fmaf(n.origin[a], rcp, so - e)));
            t1 = fminf(t1, fmaf(r.n[a] ? lo : hi, rcp, fmaf(n.origin[a], rcp, so + e)));
        }
        if (!std::signbit(t1 - t0)) hits |= 1u << s;
    }
    return hits;
}

int main(int argc, char **argv) {
    FILE *f = fopen(argv[1], "rb");
    uint32_t count = 0, triangles = 0;
    if (!f || fread(&count, 4, 1, f) != 1 || fread(&triangles, 4, 1, f) != 1) return 2;
    std::vector<SlimBVHNode> nodes(count);
    if (fread(nodes.data(), sizeof(SlimBVHNode), count, f) != count) return 2;
    fclose(f);
    std::vector<float> hot(12 * (size_t)triangles);
    for (size_t i = 0; i < hot.size(); i++) hot[i] = (float)i;
    std::vector<WideNode> wide(3);             // not at index 0: offsets are absolute
    std::vector<WideLeaf> leaves(5);
    float extent = 0.0f;
    const uint32_t root = build_wide_bvh(nodes.data(), count, hot.data(), argc > 2 ? (uint32_t)atoi(argv[2]) : 64u, wide, leaves, extent);
    if (root == kNoWideBVH) { printf("none\n"); return wide.size() == 3 && leaves.size() == 5 ? 0 : 1; }
    if (root != 3) return 1;
    // every node and leaf once, children in range, planes outside the boxes
    std::vector<int> seen(triangles, 0);
    size_t leaf_total = 0;
    std::vector<int> reached(wide.size(), 0);
    reached[root] = 1;
    for (size_t w = 3; w < wide.size(); w++) {
        const WideNode &n = wide[w];
        for (int s = 0; s < 4; s++) {
            const uint32_t c = n.child[s];
            if (wide_offset(n.lo[0], s) > wide_offset(n.hi[0], s)) continue;     // an empty slot
            if (!(c & kWideLeaf)) {
                if (c <= w || c >= wide.size() || reached[c]++) return 1;
                continue;
            }
            const uint32_t l = c & ~kWideLeaf;
            if (l < 5 || l >= leaves.size()) return 1;
            const SlimBVHNode &b = leaves[l].node;
            for (uint32_t t = 0; t < b.leaf_count; t++) seen[b.first_index + t]++;
            for (uint32_t t = 0; t < b.leaf_count && t < 2; t++)
                if (leaves[l].triangles[t][0] != hot[12 * (size_t)(b.first_index + t)]) return 1;
            const float lo[3] = {b.aabb.min.x, b.aabb.min.y, b.aabb.min.z}, hi[3] = {b.aabb.max.x, b.aabb.max.y, b.aabb.max.z};
            for (int a = 0; a < 3; a++) {
                const double l2 = (double)n.origin[a] + wide_offset(n.lo[a], s), h2 = (double)n.origin[a] + wide_offset(n.hi[a], s);
                if (l2 > lo[a] + 1e-37 || h2 < hi[a] || fabs(l2) > extent || fabs(h2) > extent) return 1;
            }
            leaf_total++;
        }
    }
    if (leaf_total + 5 != leaves.size()) return 1;
    for (int v : seen) if (v != 1) return 1;
    for (size_t w = 3; w < wide.size(); w++) if (reached[w] != 1) return 1;

    std::mt19937 rng(1);
    std::uniform_real_distribution<float> u(-1.0f, 1.0f);
    size_t hits = 0;
    for (int k = 0; k < 4000; k++) {
        // from near and far, some directions almost parallel to an axis,
        // some origins on a box plane
        const float reach = k % 3 == 0 ? 1.5f : k % 3 == 1 ? 20.0f : 300.0f;
        V o{reach * u(rng), reach * u(rng), reach * u(rng)}, d{u(rng) * 0.9f - o.x, u(rng) * 0.9f - o.y, u(rng) * 0.9f - o.z};
        if (k % 5 == 0) d.x *= 1e-6f;
        if (k % 7 == 0) { o.y = nodes[(size_t)k % count].aabb.min.y; d.y = 1e-3f * u(rng); }
        // parallel to an axis, in a box's plane or beside it: the exact test
        // leaves out the axis, the wide walk keeps to the boxes around it
        const bool parallel = k % 11 == 0;
        if (parallel) (k % 2 ? d.x : d.y) = k % 3 ? 0.0f : -0.0f;
        else if (d.x == 0 || d.y == 0 || d.z == 0) continue;
        Ray r{o, {1.0f / d.x, 1.0f / d.y, 1.0f / d.z}, {}, {std::signbit(d.x), std::signbit(d.y), std::signbit(d.z)}};
        r.so = {(-o.x) * r.rcp.x, (-o.y) * r.rcp.y, (-o.z) * r.rcp.z};
        const float tmax = k % 4 == 0 ? INFINITY : fabsf(u(rng)) * 1.5f;
        std::set<uint32_t> binary, through;
        float ln, lf;
        std::vector<uint32_t> stack;
        if (slab(r, nodes[0].aabb, ln, lf) && ln < tmax) stack.push_back(0);
        const bool enters = !stack.empty();
        while (!stack.empty()) {
            const SlimBVHNode &n = nodes[stack.back()];
            stack.pop_back();
            for (uint32_t c = n.first_index; c < n.first_index + 2; c++) {
                if (!slab(r, nodes[c].aabb, ln, lf) || !(ln < tmax)) continue;
                if (nodes[c].leaf_count) binary.insert(nodes[c].first_index);
                else stack.push_back(c);
            }
        }
        // the lane's walk of the persistent kernels: a leaf waits while the
        // walk goes on, and is tested at turns other lanes decide
        constexpr uint32_t kNone = 0xFFFFFFFFu;
        uint32_t next = enters ? root : kNone, waiting = kNone, entries[64], top = 0, turns = 0;
        auto advance = [&]() {
            if (next == kNone && top) next = entries[--top];
            if (next != kNone && (next & kWideLeaf) && waiting == kNone) {
                waiting = next;
                next = top ? entries[--top] : kNone;
            }
        };
        while (next != kNone || waiting != kNone || top) {
            if (++turns > 1000000u) { printf("ray %d does not end\n", k); return 1; }
            if (!(next & kWideLeaf)) {
                const WideNode &n = wide[next];
                const uint32_t h = wide_hits(n, r, extent, tmax);
                next = kNone;
                for (int s = 0; s < 4; s++) {
                    if (!(h >> s & 1)) continue;
                    if (next != kNone) {
                        if (top >= 64) return 1;
                        entries[top++] = next;
                    }
                    next = n.child[s];
                }
                advance();
            }
            if (waiting != kNone && (rng() & 1)) {
                const SlimBVHNode &l = leaves[waiting & ~kWideLeaf].node;
                if (slab(r, l.aabb, ln, lf) && ln < tmax) through.insert(l.first_index);
                waiting = kNone;
                advance();
            }
        }
        if (parallel) {
            std::set<uint32_t> beside;
            for (const SlimBVHNode &n : nodes) {
                if (!n.leaf_count || !binary.count(n.first_index)) continue;
                const float p = k % 2 ? o.x : o.y, lo = k % 2 ? n.aabb.min.x : n.aabb.min.y, hi = k % 2 ? n.aabb.max.x : n.aabb.max.y;
                if (lo <= p && p <= hi) beside.insert(n.first_index);
            }
            for (uint32_t l : beside) if (!through.count(l)) { printf("ray %d misses a leaf it lies in\n", k); return 1; }
            for (uint32_t l : through) if (!binary.count(l)) { printf("ray %d reaches a leaf the binary walk culls\n", k); return 1; }
        } else if (binary != through) { printf("ray %d: %zu leaves, %zu through the wide form\n", k, binary.size(), through.size()); return 1; }
        hits += binary.size();
    }
    printf("%zu nodes, %zu leaves, %zu leaf hits\n", wide.size() - 3, leaf_total, hits);
    return 0;
}
