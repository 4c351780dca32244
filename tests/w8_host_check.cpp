// Host check of the device form of the 8-wide BVH (split_leaves, build_cw8,
// pack_w8 of vk-renderer_gb300/csrc/bvh_cw8.cpp), compiled by
// tests/test_w8_host.py: every index the kernels read from a node is in
// range, every triangle is referenced once, the boxes equal the 8-bit node's,
// and a host emulation of the device traversal (tracer_cw8.cuh) finds a
// brute-force scan's closest hits.
//
// Usage: w8_host_check <soup|flat|grid> <n> <leaf> <rays> <seed>
//   soup: random triangles; flat: triangles in the plane y = 0 (boxes without
//   extent); grid: a height field of connected triangles
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "bvh_cw8.h"
#include "tracer_abi.h"

using vkt::Cw8Node;
using vkt::W8Node;

namespace {

struct V {
    float x, y, z;
};
V sub(const float* a, const float* b) { return {a[0] - b[0], a[1] - b[1], a[2] - b[2]}; }
V cross(V a, V b) { return {a.y * b.z - b.y * a.z, a.z * b.x - b.z * a.x, a.x * b.y - b.x * a.y}; }
float dot(V a, V b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
float as_float(uint32_t w)
{
    float f;
    std::memcpy(&f, &w, 4);
    return f;
}

[[noreturn]] void fail(const char* what, long a = 0, long b = 0)
{
    std::printf("FAIL %s %ld %ld\n", what, a, b);
    std::exit(1);
}

struct Hit {
    float t;
    uint32_t id;
};

// the device's one-sided triangle test and strict acceptance
void test(const tracer_triangle& t, uint32_t id, V o, V d, Hit& h)
{
    const V e1 = sub(t.v1, t.v0), e2 = sub(t.v2, t.v0), p = cross(d, e2);
    const float det = dot(e1, p);
    if (det < 1e-3f) return;
    const float inv = 1.0f / det;
    const V s = {o.x - t.v0[0], o.y - t.v0[1], o.z - t.v0[2]};
    const float u = dot(s, p) * inv;
    if (u < 0.0f || u > 1.0f) return;
    const V q = cross(s, e1);
    const float v = dot(d, q) * inv;
    if (v < 0.0f || u + v > 1.0f) return;
    const float k = dot(e2, q) * inv;
    if (k > 1e-3f && (k < h.t || (k == h.t && id < h.id))) h = {k, id};
}

float inverse(float d) { return 1.0f / (std::fabs(d) > 1e-30f ? d : std::copysign(1e-30f, d)); }
uint32_t byte_at(const uint32_t* w, int word, int k) { return w[word + k / 4] >> (8 * (k % 4)) & 0xFFu; }
int first_bit(uint32_t x) { return __builtin_ctz(x); }

}  // namespace

int main(int argc, char** argv)
{
    if (argc < 6) return 2;
    const char* kind = argv[1];
    const uint32_t want = (uint32_t)std::atoi(argv[2]), leaf = (uint32_t)std::atoi(argv[3]);
    const int rays = std::atoi(argv[4]);
    std::mt19937 g((uint32_t)std::atoi(argv[5]));
    auto uni = [&](float lo, float hi) { return lo + (hi - lo) * (float)((g() >> 8) * 0x1.0p-24); };
    std::vector<tracer_triangle> tris;
    float extent = 10.0f;
    if (kind[0] == 'g') {
        const int k = std::max(1, (int)std::lround(std::sqrt(want / 2.0)));
        std::vector<float> y((size_t)(k + 1) * (k + 1));
        for (float& v : y) v = uni(-0.3f, 0.3f);
        extent = 0.5f * (float)k;
        for (int i = 0; i < k; ++i)
            for (int j = 0; j < k; ++j)
                for (int half = 0; half < 2; ++half) {
                    const int c[3][2] = {{i + half, j}, {i, j + 1}, {i + 1, j + half}};
                    tracer_triangle t{};
                    float* v[3] = {t.v0, t.v1, t.v2};
                    for (int q = 0; q < 3; ++q) {
                        v[q][0] = (float)c[q][0] - extent;
                        v[q][1] = y[(size_t)c[q][0] * (k + 1) + c[q][1]];
                        v[q][2] = (float)c[q][1] - extent;
                    }
                    tris.push_back(t);
                }
    } else {
        for (uint32_t i = 0; i < want; ++i) {
            const float c[3] = {uni(-extent, extent), uni(-extent, extent), uni(-extent, extent)};
            tracer_triangle t{};
            float* v[3] = {t.v0, t.v1, t.v2};
            for (float* p : v)
                for (int a = 0; a < 3; ++a) p[a] = c[a] + uni(-0.6f, 0.6f);
            if (kind[0] == 'f') t.v0[1] = t.v1[1] = t.v2[1] = 0.0f;
            tris.push_back(t);
        }
    }
    const uint32_t n = (uint32_t)tris.size();
    std::vector<tracer_bvh_node> nodes(2 * (size_t)n), split;
    std::vector<uint32_t> idx(n), slot_of, order;
    uint32_t nn = 0, bdepth = 0, depth = 0;
    if (tracer_build_bvh(TRACER_BVH_SAH, TRACER_PRIM_TRIANGLE, tris.data(), n, leaf, 16, nodes.data(), &nn, idx.data(),
                         &bdepth) != TRACER_OK)
        fail("binary build");
    nodes.resize(nn);
    std::vector<double> box(6 * (size_t)n);
    for (uint32_t k = 0; k < n; ++k) {
        const tracer_triangle& t = tris[idx[k]];
        for (int a = 0; a < 3; ++a) {
            box[6 * k + a] = std::min({t.v0[a], t.v1[a], t.v2[a]});
            box[6 * k + 3 + a] = std::max({t.v0[a], t.v1[a], t.v2[a]});
        }
    }
    vkt::split_leaves(nodes.data(), nn, reinterpret_cast<const double(*)[6]>(box.data()), split, slot_of);
    std::vector<uint32_t> tri_of(n);  // primitive of the split tree -> triangle
    for (uint32_t k = 0; k < n; ++k) tri_of[k] = idx[slot_of[k]];
    uint32_t sdepth = 0;
    if (tracer_validate_bvh(TRACER_PRIM_TRIANGLE, tris.data(), n, split.data(), (uint32_t)split.size(), tri_of.data(),
                            &sdepth) != TRACER_OK)
        fail("split tree is no valid BVH");
    for (const auto& nd : split)
        if (nd.count > 1) fail("leaf not split", nd.count);
    std::vector<Cw8Node> coded;
    std::vector<W8Node> w;
    if (!vkt::build_cw8(split.data(), (uint32_t)split.size(), coded, order, &depth)) fail("build_cw8");
    if (!vkt::pack_w8(coded, w)) fail("pack_w8");
    if (depth > sdepth) fail("8-wide deeper than the split tree", depth, sdepth);
    // structure
    std::vector<int> seen(n, 0), reached(w.size(), 0);
    reached[0] = 1;
    for (size_t i = 0; i < w.size(); ++i) {
        const uint32_t* y = w[i].w;
        const uint32_t imask = y[8] & 0xFFu, lf = y[8] >> 8 & 0xFFu, two = y[8] >> 16 & 0xFFu;
        if ((imask & lf) || (two & ~lf) || (y[8] >> 24)) fail("masks", (long)i);
        for (uint32_t k = 0, c = 0; k < 8; ++k)
            if (imask >> k & 1u) {
                if (y[6] + c >= w.size()) fail("child range", (long)i, k);
                reached[y[6] + c++]++;
            }
        uint32_t p = y[7];
        for (uint32_t k = 0; k < 8; ++k)
            for (uint32_t j = 0; j < (lf >> k & 1u) + (two >> k & 1u); ++j, ++p) {
                if (p >= n) fail("primitive range", (long)i, k);
                seen[order[p]]++;
            }
        for (int a = 0; a < 3; ++a) {
            const double step = as_float(y[3 + a]), p = as_float(y[a]) + 32768.0 * step;
            if (p != as_float(coded[i].w[a])) fail("origin", (long)i, a);
            for (int side = 0; side < 2; ++side)
                for (int k = 0; k < 8; ++k)
                    if (byte_at(y, 10 + 4 * a + 2 * side, k) != byte_at(coded[i].w, 8 + 2 * a + 6 * side, k))
                        fail("plane", (long)i, k);
        }
    }
    for (uint32_t k = 0; k < n; ++k)
        if (seen[k] != 1) fail("triangle count", k, seen[k]);
    for (size_t i = 0; i < w.size(); ++i)
        if (reached[i] != 1) fail("node count", (long)i, reached[i]);
    // traversal
    int hits = 0;
    std::vector<std::pair<uint32_t, uint32_t>> stack;
    for (int r = 0; r < rays; ++r) {
        const V o = {uni(-1.3f, 1.3f) * extent, uni(-1.3f, 1.3f) * extent, uni(-1.3f, 1.3f) * extent};
        V d = {uni(-1, 1), uni(-1, 1), uni(-1, 1)};
        if (r % 7 == 0) (r % 3 == 0 ? d.x : r % 3 == 1 ? d.y : d.z) = 0.0f;
        const float tmax = r % 5 == 0 ? 3.0f : 3000.0f, slack = 1.0f + 0x1.0p-20f;
        Hit brute{tmax, 0}, h{tmax, 0};
        for (uint32_t k = 0; k < n; ++k) test(tris[k], k, o, d, brute);
        const float i3[3] = {inverse(d.x), inverse(d.y), inverse(d.z)};
        const float n3[3] = {-(o.x * i3[0]), -(o.y * i3[1]), -(o.z * i3[2])};
        const uint32_t pref[3] = {i3[2] < 0 ? 0xF0u : 0x0Fu, i3[1] < 0 ? 0xCCu : 0x33u, i3[0] < 0 ? 0xAAu : 0x55u};
        std::pair<uint32_t, uint32_t> G{0u, 0x101u};
        stack.clear();
        for (;;) {
            if (!(G.second & 0xFFu)) {
                if (stack.empty()) break;
                G = stack.back();
                stack.pop_back();
            }
            uint32_t x = G.second & 0xFFu;
            for (uint32_t p : pref) x = (x & p) ? x & p : x;
            if (x & (x - 1)) fail("child choice", x);
            G.second ^= x;
            const uint32_t ci = G.first + (uint32_t)__builtin_popcount(G.second >> 8 & (x - 1u));
            if (ci >= w.size()) fail("visit index", ci);
            if (G.second & 0xFFu) stack.push_back(G);
            if (stack.size() > depth) fail("stack above the tree's depth", (long)stack.size(), depth);
            const uint32_t* y = w[ci].w;
            float b[3];
            float s3[3];
            for (int a = 0; a < 3; ++a) {
                b[a] = std::fma(as_float(y[a]), i3[a], n3[a]);
                s3[a] = as_float(y[3 + a]) * i3[a];
            }
            uint32_t hit = 0;
            for (int k = 0; k < 8; ++k) {
                float tn = -HUGE_VALF, tf = HUGE_VALF;
                for (int a = 0; a < 3; ++a) {
                    auto plane = [&](int side) {
                        return std::fma(32768.0f + (float)byte_at(y, 10 + 4 * a + 2 * side, k), s3[a], b[a]);
                    };
                    tn = std::fmax(tn, plane(i3[a] < 0));
                    tf = std::fmin(tf, plane(!(i3[a] < 0)));
                }
                if (!std::signbit(std::fmin(std::fmin(std::fma(tf, slack, -tn), tf), h.t * slack - tn))) hit |= 1u << k;
            }
            G = {y[6], (hit & y[8] & 0xFFu) | (y[8] & 0xFFu) << 8};
            std::pair<uint32_t, uint32_t> P{y[7], (y[8] >> 8 & hit & 0xFFu) | (y[8] & 0xFFFF00u)};
            while (P.second & 0xFFu) {
                const uint32_t s = 1u << first_bit(P.second);
                P.second ^= s;
                const uint32_t k0 = P.first + (uint32_t)__builtin_popcount(P.second >> 8 & ((s - 1u) * 0x101u));
                const bool two = P.second >> 16 & s;
                for (uint32_t k = k0; k < k0 + 1 + two; ++k) {
                    if (k >= n) fail("primitive index", k);
                    test(tris[tri_of[order[k]]], tri_of[order[k]], o, d, h);
                }
            }
        }
        if (h.t != brute.t || h.id != brute.id) fail("closest hit differs", r, (long)h.id);
        hits += brute.t < tmax;
    }
    std::printf("ok nodes=%zu depth=%u hits=%d\n", w.size(), depth, hits);
    return 0;
}
