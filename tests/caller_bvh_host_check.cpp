// Host check of the device form of the 8-wide BVH over binary BVHs as a caller
// may pass them (tracer_scene_desc::tri_nodes), compiled by
// tests/test_caller_bvh_host.py: node arrays with entries that the root does
// not reach, boxes without padding, geometry and rays far from the origin.
//
// Usage: caller_bvh_host_check <plain|range|overlap|tight> <n> <offset> <distance> <seed>
//   range: unreached leaves whose primitives lie beyond the array; overlap:
//   unreached leaves over other leaves' primitives; tight: unpadded boxes.
//   The triangles lie about (offset, offset, offset); half of the rays start
//   `distance` half sides from there.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "bvh_cw8.h"
#include "tracer_abi.h"

namespace {

struct V {
    float x, y, z;
};
V sub(V a, V b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
V cross(V a, V b) { return {a.y * b.z - b.y * a.z, a.z * b.x - b.z * a.x, a.x * b.y - b.x * a.y}; }
float dot(V a, V b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
V of(const float* p) { return {p[0], p[1], p[2]}; }

struct Hit {
    float t;
    uint32_t id;
};

// the device's one-sided triangle test and strict acceptance
void test(const tracer_triangle& t, uint32_t id, V o, V d, Hit& h)
{
    const V e1 = sub(of(t.v1), of(t.v0)), e2 = sub(of(t.v2), of(t.v0)), p = cross(d, e2), s = sub(o, of(t.v0));
    const float det = dot(e1, p);
    if (det < 1e-3f) return;
    const float inv = 1.0f / det, u = dot(s, p) * inv;
    if (u < 0.0f || u > 1.0f) return;
    const V q = cross(s, e1);
    const float v = dot(d, q) * inv;
    if (v < 0.0f || u + v > 1.0f) return;
    const float k = dot(e2, q) * inv;
    if (k > 1e-3f && (k < h.t || (k == h.t && id < h.id))) h = {k, id};
}

float word(const vkt::W8Node& n, int k)
{
    float f;
    std::memcpy(&f, &n.w[k], 4);
    return f;
}
float inverse(float d) { return 1.0f / (std::fabs(d) > 1e-30f ? d : std::copysign(1e-30f, d)); }

[[noreturn]] void fail(const char* what, long a = 0, long b = 0)
{
    std::printf("FAIL %s %ld %ld\n", what, a, b);
    std::exit(1);
}

}  // namespace

int main(int argc, char** argv)
{
    if (argc < 6) return 2;
    const std::string kind = argv[1];
    const uint32_t n = (uint32_t)std::atoi(argv[2]);
    const float offset = (float)std::atof(argv[3]), distance = (float)std::atof(argv[4]), half = 10.0f;
    std::mt19937 g((uint32_t)std::atoi(argv[5]));
    auto uni = [&](float lo, float hi) { return lo + (hi - lo) * (float)((g() >> 8) * 0x1.0p-24); };
    std::vector<tracer_triangle> tris(n);
    for (tracer_triangle& t : tris) {
        const float c[3] = {uni(-half, half), uni(-half, half), uni(-half, half)};
        for (float* v : {t.v0, t.v1, t.v2})
            for (int a = 0; a < 3; ++a) v[a] = c[a] + uni(-0.9f, 0.9f) + offset;
    }
    std::vector<tracer_bvh_node> nodes(2 * (size_t)n), split;
    std::vector<uint32_t> idx(n), slot_of, order;
    uint32_t nn = 0, depth = 0;
    if (tracer_build_bvh(TRACER_BVH_SAH, TRACER_PRIM_TRIANGLE, tris.data(), n, 4, 16, nodes.data(), &nn, idx.data(),
                         &depth) != TRACER_OK)
        fail("binary build");
    nodes.resize(nn);
    if (kind == "tight")
        for (uint32_t i = nn; i-- > 0;)  // the builder's children follow their parents
            for (int a = 0; a < 3; ++a) {
                float lo = HUGE_VALF, hi = -HUGE_VALF;
                for (int k = 0; k < std::max(2, nodes[i].count); ++k) {
                    const uint32_t at = (uint32_t)nodes[i].left_or_first + k;
                    if (nodes[i].count == 0) {
                        lo = std::min(lo, nodes[at].bmin[a]);
                        hi = std::max(hi, nodes[at].bmax[a]);
                    } else if (k < nodes[i].count) {
                        const tracer_triangle& t = tris[idx[at]];
                        lo = std::min({lo, t.v0[a], t.v1[a], t.v2[a]});
                        hi = std::max({hi, t.v0[a], t.v1[a], t.v2[a]});
                    }
                }
                nodes[i].bmin[a] = lo;
                nodes[i].bmax[a] = hi;
            }
    if (kind == "range" || kind == "overlap")
        for (int count = 1; count <= 6; ++count) {
            tracer_bvh_node extra = nodes[0];
            extra.count = count;
            extra.left_or_first = kind == "range" ? (int32_t)(n - 1) + 1000 * count : 3 * count;
            nodes.push_back(extra);
        }
    if (tracer_validate_bvh(TRACER_PRIM_TRIANGLE, tris.data(), n, nodes.data(), (uint32_t)nodes.size(), idx.data(),
                            &depth) != TRACER_OK)
        fail("the caller's BVH is refused");

    std::vector<double> box(6 * (size_t)n);
    for (uint32_t k = 0; k < n; ++k) {
        const tracer_triangle& t = tris[idx[k]];
        for (int a = 0; a < 3; ++a) {
            box[6 * k + a] = std::min({t.v0[a], t.v1[a], t.v2[a]});
            box[6 * k + 3 + a] = std::max({t.v0[a], t.v1[a], t.v2[a]});
        }
    }
    vkt::split_leaves(nodes.data(), (uint32_t)nodes.size(), reinterpret_cast<const double(*)[6]>(box.data()), split,
                      slot_of);
    if (slot_of.size() != n) fail("slots of the split tree", (long)slot_of.size(), n);
    std::vector<uint32_t> tri_of(n);
    for (uint32_t k = 0; k < n; ++k) {
        if (slot_of[k] >= n) fail("slot", k, slot_of[k]);
        tri_of[k] = idx[slot_of[k]];
    }
    if (tracer_validate_bvh(TRACER_PRIM_TRIANGLE, tris.data(), n, split.data(), (uint32_t)split.size(), tri_of.data(),
                            &depth) != TRACER_OK)
        fail("split tree is no valid BVH");
    std::vector<vkt::Cw8Node> coded;
    std::vector<vkt::W8Node> w;
    if (!vkt::build_cw8(split.data(), (uint32_t)split.size(), coded, order, &depth) || !vkt::pack_w8(coded, w))
        fail("8-wide build");

    // the same on any number of host threads
    for (uint32_t threads : {2u, 8u}) {
        std::vector<tracer_bvh_node> split2;
        std::vector<uint32_t> slot2, order2;
        std::vector<vkt::Cw8Node> coded2;
        double cost = 0.0;
        vkt::split_leaves(nodes.data(), (uint32_t)nodes.size(), reinterpret_cast<const double(*)[6]>(box.data()), split2,
                          slot2, threads);
        if (!vkt::build_cw8(split2.data(), (uint32_t)split2.size(), coded2, order2, &depth, &cost, threads) ||
            slot2 != slot_of || order2 != order || coded2.size() != coded.size() ||
            std::memcmp(split2.data(), split.data(), split.size() * sizeof split[0]) ||
            std::memcmp(coded2.data(), coded.data(), coded.size() * sizeof coded[0]))
            fail("another tree on threads", threads);
    }

    // the device's slab test over every node whose parent it enters
    long hits = 0;
    std::vector<uint32_t> stack;
    for (int r = 0; r < 4000; ++r) {
        const V to = {uni(-half, half) + offset, uni(-half, half) + offset, uni(-half, half) + offset};
        V d = {uni(-1, 1), uni(-1, 1), uni(-1, 1)};
        const float len = 1.0f / std::sqrt(dot(d, d));
        d = {d.x * len, d.y * len, d.z * len};
        const float back = r % 2 ? 0.0f : distance * half;
        const V o = {to.x - back * d.x, to.y - back * d.y, to.z - back * d.z};
        Hit brute{1e9f, 0}, h{1e9f, 0};
        for (uint32_t k = 0; k < n; ++k) test(tris[k], k, o, d, brute);
        const float inv[3] = {inverse(d.x), inverse(d.y), inverse(d.z)};
        const float neg[3] = {-(o.x * inv[0]), -(o.y * inv[1]), -(o.z * inv[2])};
        const float slack = 1.0f + 0x1.0p-20f;
        stack.assign(1, 0u);
        while (!stack.empty()) {
            const vkt::W8Node& y = w[stack.back()];
            stack.pop_back();
            uint32_t child = y.w[6], prim = y.w[7];
            for (int k = 0; k < 8; ++k) {
                const bool inner = y.w[8] >> k & 1u, leaf = y.w[8] >> (8 + k) & 1u;
                const uint32_t count = leaf ? 1u + (y.w[8] >> (16 + k) & 1u) : 0u;
                float tn = -HUGE_VALF, tf = HUGE_VALF;
                for (int a = 0; a < 3; ++a)
                    for (int side = 0; side < 2; ++side) {
                        const uint32_t q = y.w[10 + 4 * a + 2 * side + k / 4] >> (8 * (k % 4)) & 0xFFu;
                        const float t = std::fma(32768.0f + (float)q, word(y, 3 + a) * inv[a],
                                                 std::fma(word(y, a), inv[a], neg[a]));
                        if ((side == 1) == (inv[a] < 0)) tn = std::max(tn, t);
                        else tf = std::min(tf, t);
                    }
                const bool in = !std::signbit(std::min(std::min(std::fma(tf, slack, -tn), tf), h.t * slack - tn));
                if (inner && in) stack.push_back(child);
                for (uint32_t q = prim; leaf && in && q < prim + count; ++q)
                    test(tris[tri_of[order[q]]], tri_of[order[q]], o, d, h);
                child += inner;
                prim += count;
            }
        }
        if (h.t != brute.t || h.id != brute.id) fail("closest hit differs", r, (long)h.id);
        hits += brute.t < 1e9f;
    }
    std::printf("ok nodes=%zu hits=%ld\n", w.size(), hits);
    return 0;
}
