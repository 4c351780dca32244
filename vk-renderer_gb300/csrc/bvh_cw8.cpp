// Collapse of a binary BVH into compressed 8-wide nodes (see bvh_cw8.h).
// Host code, deterministic: every choice has a total order (surface area,
// then position in the child list; assignment scores, then child, then slot).
#include "bvh_cw8.h"

#include <algorithm>
#include <array>
#include <atomic>
#include <cmath>
#include <cstring>
#include <memory>

namespace vkt {

namespace {

// Cost of testing one primitive against that of visiting a node, and the most
// primitives of a merged leaf child.  c1 frame / c3 adjoint, ms, with (cost,
// merge): (0.3, 3) 53.5 / 0.69, (0.3, 2) 54.2 / 0.65, (0.3, 1) 57.1 / 0.63, (0.6,
// 3) 55.7 / 0.64, (0.15, 3) 53.7 / 0.71; whole binary leaves, largest area
// first: 58.0 / 0.79.  Two, as the kernels fetch two triangles at a time.
constexpr float kPrimCost = 0.3f;
constexpr uint32_t kMergePrims = 2;
constexpr double kGridMargin = 1.0 / 64;  // see Cw8Node's boxes

double area(const tracer_bvh_node& n)
{
    const double dx = (double)n.bmax[0] - n.bmin[0];
    const double dy = (double)n.bmax[1] - n.bmin[1];
    const double dz = (double)n.bmax[2] - n.bmin[2];
    return 2.0 * (dx * dy + dy * dz + dz * dx);
}

// std::nextafter(f, -inf) of a float without the library call, of which leaf
// splitting makes six a triangle (100k triangles on one Arm core: 16.1 -> 14.6 ms).
float next_below(float f)
{
    uint32_t b;
    std::memcpy(&b, &f, 4);
    if (f != f || b == 0xFF800000u) return f;  // NaN, -inf
    b = b == 0u || b == 0x80000000u ? 0x80000001u : (b >> 31) ? b + 1 : b - 1;
    std::memcpy(&f, &b, 4);
    return f;
}
float next_above(float f) { return -next_below(-f); }

// 2^e for -1022 <= e <= 1023.
double pow2(int e)
{
    const uint64_t b = (uint64_t)(e + 1023) << 52;
    double v;
    std::memcpy(&v, &b, 8);
    return v;
}

// Smallest e (biased float exponent, 1..254) with 2^(e - 127) * 255 >= ext.
int grid_exponent(double ext)
{
    int x = 0;
    std::frexp(ext / 255.0, &x);  // 255 * 2^(x - 1) <= ext < 255 * 2^x, up to the quotient's rounding
    int e = std::min(254, std::max(1, x + 125));
    while (e < 254 && 255.0 * pow2(e - 127) < ext) ++e;
    return e;
}

// The largest float not above v.
float float_below(double v)
{
    const float f = (float)v;
    return (double)f > v ? next_below(f) : f;
}

void put_byte(uint32_t* w, int k, uint32_t v)
{
    w[k / 4] |= (v & 0xFFu) << (8 * (k % 4));
}

// One binary node of the collapse.  cost[i], i = 1..8: least expected cost of
// its subtree given as at most i children of an 8-wide node; split[i]: of a
// cut into i >= 2 parts, how many the left child gets; parts[i]: how many of
// the i parts are used (1 = the node itself is one child).  most: the largest
// number of parts that differ, its binary leaves or 8; beyond it, cost, split and
// parts stay the same, and are not worked out again.
struct Cut {
    float cost[9];
    uint8_t split[9], parts[9];
    uint8_t most;
    bool leaf;       // as one child: a leaf child with all its primitives
    uint32_t prims;  // primitives of the subtree
};

// The plan of node `at`, its children's being there.
void plan_node(const tracer_bvh_node* nodes, uint32_t at, Cut* cuts)
{
    const tracer_bvh_node& n = nodes[at];
    Cut& c = cuts[at];
    const float a = (float)area(n);
    if (n.count > 0) {
        c.leaf = true;
        c.prims = (uint32_t)n.count;
        c.most = 1;
        for (int i = 1; i <= 8; ++i) {
            c.cost[i] = a * (float)c.prims * kPrimCost;
            c.parts[i] = 1;
            c.split[i] = 0;
        }
        return;
    }
    const Cut& l = cuts[(uint32_t)n.left_or_first];
    const Cut& r = cuts[(uint32_t)n.left_or_first + 1];
    float cut[9];
    const int most = std::min(8, l.most + r.most);
    c.most = (uint8_t)most;
    for (int i = 2; i <= most; ++i) {
        cut[i] = l.cost[1] + r.cost[i - 1];
        c.split[i] = 1;
        for (int k = 2; k <= std::min(i - 1, (int)l.most); ++k) {
            const float v = l.cost[k] + r.cost[i - k];
            if (v < cut[i]) {
                cut[i] = v;
                c.split[i] = (uint8_t)k;
            }
        }
    }
    for (int i = most + 1; i <= 8; ++i) {
        cut[i] = cut[most];
        c.split[i] = c.split[most];
    }
    c.prims = l.prims + r.prims;
    c.leaf = false;
    c.cost[1] = a + cut[8];
    c.parts[1] = 1;
    if (c.prims <= kMergePrims && a * (float)c.prims * kPrimCost <= c.cost[1]) {
        c.cost[1] = a * (float)c.prims * kPrimCost;
        c.leaf = true;
    }
    for (int i = 2; i <= 8; ++i) {
        const bool use = cut[i] < c.cost[i - 1];
        c.cost[i] = use ? cut[i] : c.cost[i - 1];
        c.parts[i] = use ? (uint8_t)i : c.parts[i - 1];
    }
}

void plan_subtree(const tracer_bvh_node* nodes, uint32_t at, Cut* cuts)
{
    if (nodes[at].count == 0)
        for (uint32_t h = 0; h < 2; ++h) plan_subtree(nodes, (uint32_t)nodes[at].left_or_first + h, cuts);
    plan_node(nodes, at, cuts);
}

std::unique_ptr<Cut[]> plan_cuts(const tracer_bvh_node* nodes, uint32_t num_nodes, uint32_t threads)
{
    std::unique_ptr<Cut[]> cuts(new Cut[num_nodes]);
    // the top of the tree, parents first, then the subtrees below it
    std::vector<uint32_t> top{0u};
    size_t planned = 0;
    while (planned < top.size() && top.size() - planned < 8 * threads) {
        const tracer_bvh_node& n = nodes[top[planned++]];
        for (uint32_t h = 0; h < 2 && n.count == 0; ++h) top.push_back((uint32_t)n.left_or_first + h);
    }
    over_chunks(top.size() - planned, num_nodes < 4096 ? 1 : threads, [&](size_t from, size_t to) {
        for (size_t k = from; k < to; ++k) plan_subtree(nodes, top[planned + k], cuts.get());
    }, 1);
    while (planned > 0) plan_node(nodes, top[--planned], cuts.get());
    return cuts;
}

// The parts of node n as at most `budget` children (>= 2: n itself is cut).
void cut_children(const tracer_bvh_node* nodes, const Cut* cuts, uint32_t n, int budget, uint32_t* kids, uint32_t& nk)
{
    const uint32_t l = (uint32_t)nodes[n].left_or_first;
    const int left = cuts[n].split[budget], part[2] = {left, budget - left};
    for (int h = 0; h < 2; ++h) {
        const int use = cuts[l + h].parts[part[h]];
        if (use == 1)
            kids[nk++] = l + h;
        else
            cut_children(nodes, cuts, l + h, use, kids, nk);
    }
}

void bounds(const double (*tri)[6], const uint32_t* v, uint32_t n, double* lo, double* hi)
{
    for (int a = 0; a < 3; ++a) {
        lo[a] = tri[v[0]][a];
        hi[a] = tri[v[0]][a + 3];
        for (uint32_t k = 1; k < n; ++k) {
            lo[a] = std::min(lo[a], tri[v[k]][a]);
            hi[a] = std::max(hi[a], tri[v[k]][a + 3]);
        }
    }
}

// area[k]: half the surface area of the box of triangles v[0], v[d], ..., v[k * d].
void running_areas(const double (*tri)[6], const uint32_t* v, uint32_t n, int d, double* area)
{
    double lo[3], hi[3];
    for (uint32_t k = 0; k < n; ++k, v += d) {
        for (int a = 0; a < 3; ++a) {
            lo[a] = k ? std::min(lo[a], tri[*v][a]) : tri[*v][a];
            hi[a] = k ? std::max(hi[a], tri[*v][a + 3]) : tri[*v][a + 3];
        }
        const double x = hi[0] - lo[0], y = hi[1] - lo[1], z = hi[2] - lo[2];
        area[k] = x * y + y * z + z * x;
    }
}

// Shrinks the box to the n triangles', padded outward as the binary
// builder's boxes are (2^-14 of the largest coordinate or side, + 1e-6).
void shrink_box(const double (*tri)[6], const uint32_t* v, uint32_t n, tracer_bvh_node& box)
{
    double lo[3], hi[3], scale = 0.0;
    bounds(tri, v, n, lo, hi);
    for (int a = 0; a < 3; ++a)
        scale = std::max(scale, std::max(std::max(std::fabs(lo[a]), std::fabs(hi[a])), hi[a] - lo[a]));
    const double pad = scale * 0x1.0p-14 + 1e-6;
    for (int a = 0; a < 3; ++a) {
        box.bmin[a] = std::max(box.bmin[a], next_below((float)(lo[a] - pad)));
        box.bmax[a] = std::min(box.bmax[a], next_above((float)(hi[a] + pad)));
    }
}

// Splits leaf i of `out` (2 to kCw8MaxLeafPrims triangles) down to single ones,
// its parts at out[at] and up, its triangles' slots reordered.
void split_leaf(const double (*tri)[6], uint32_t i, uint32_t at, tracer_bvh_node* out, uint32_t* slot)
{
    const tracer_bvh_node leaf = out[i];  // every part's box stays inside it
    uint32_t todo[kCw8MaxLeafPrims], n_todo = 0;
    todo[n_todo++] = i;
    while (n_todo > 0) {
        const uint32_t n = todo[--n_todo];
        const uint32_t first = (uint32_t)out[n].left_or_first, count = (uint32_t)out[n].count;
        uint32_t* s = slot + first;
        // the split of a sorted axis with the least count x area on both sides
        uint32_t best[kCw8MaxLeafPrims], best_at = 1;
        double best_cost = HUGE_VAL;
        for (int a = 0; a < 3 && count > 2; ++a) {
            uint32_t v[kCw8MaxLeafPrims];
            double key[kCw8MaxLeafPrims], left[kCw8MaxLeafPrims], right[kCw8MaxLeafPrims];
            for (uint32_t k = 0; k < count; ++k) {  // by box centre, ties by slot
                const double c = tri[s[k]][a] + tri[s[k]][a + 3];
                uint32_t j = k;
                for (; j > 0 && (c < key[j - 1] || (c == key[j - 1] && s[k] < v[j - 1])); --j) {
                    key[j] = key[j - 1];
                    v[j] = v[j - 1];
                }
                key[j] = c;
                v[j] = s[k];
            }
            running_areas(tri, v, count, 1, left);
            running_areas(tri, v + count - 1, count, -1, right);
            for (uint32_t m = 1; m < count; ++m) {
                const double cost = m * left[m - 1] + (count - m) * right[count - m - 1];
                if (cost < best_cost) {
                    best_cost = cost;
                    best_at = m;
                    std::copy(v, v + count, best);
                }
            }
        }
        if (best_cost < HUGE_VAL) std::copy(best, best + count, s);
        out[n].left_or_first = (int32_t)at;
        out[n].count = 0;
        for (uint32_t h = 0; h < 2; ++h, ++at) {
            tracer_bvh_node c = leaf;
            c.left_or_first = (int32_t)(h ? first + best_at : first);
            c.count = (int32_t)(h ? count - best_at : best_at);
            shrink_box(tri, slot + c.left_or_first, (uint32_t)c.count, c);
            out[at] = c;
            if (c.count > 1) todo[n_todo++] = at;
        }
    }
}

constexpr uint32_t kNoNode = 0xFFFFFFFFu;

// The 8-wide node of binary node `bin`: its children by slot (kNoNode: none), its
// grid, boxes and masks; not where its children and primitives start.
bool fill_node(const tracer_bvh_node* nodes, const Cut* cuts, uint32_t bin, std::array<uint32_t, 8>& in_slot, Cw8Node& node)
{
    // children: the binary node's cut into at most 8 (or the root itself,
    // when it is a leaf child), fewer if their leaves hold too many
    uint32_t kids[8], nk = 0, prims = 0;
    if (cuts[bin].leaf) {
        kids[nk++] = bin;
    } else {
        for (int budget = 8; budget >= 2; --budget) {
            nk = prims = 0;
            cut_children(nodes, cuts, bin, budget, kids, nk);
            for (uint32_t k = 0; k < nk; ++k)
                if (cuts[kids[k]].leaf) prims += cuts[kids[k]].prims;
            if (prims <= kCw8MaxNodePrims) break;
        }
        if (prims > kCw8MaxNodePrims) return false;
    }
    // slot assignment: slot s takes the child whose centroid lies furthest
    // toward the side where rays of octant s enter (greedy on the scores)
    double ulo[3] = {HUGE_VAL, HUGE_VAL, HUGE_VAL}, uhi[3] = {-HUGE_VAL, -HUGE_VAL, -HUGE_VAL};
    for (uint32_t k = 0; k < nk; ++k)
        for (int a = 0; a < 3; ++a) {
            ulo[a] = std::min(ulo[a], (double)nodes[kids[k]].bmin[a]);
            uhi[a] = std::max(uhi[a], (double)nodes[kids[k]].bmax[a]);
        }
    double score[8][8];
    int best[8];  // each child's best free slot, the first of equals
    for (size_t k = 0; k < nk; ++k) {
        double c[3];
        for (int a = 0; a < 3; ++a)
            c[a] = 0.5 * ((double)nodes[kids[k]].bmin[a] + nodes[kids[k]].bmax[a]) - 0.5 * (ulo[a] + uhi[a]);
        best[k] = 0;
        for (int s = 0; s < 8; ++s) {
            score[k][s] = ((s & 1 ? c[0] : -c[0]) + (s & 2 ? c[1] : -c[1])) + (s & 4 ? c[2] : -c[2]);
            if (score[k][s] > score[k][best[k]]) best[k] = s;
        }
    }
    int kid_in[8] = {-1, -1, -1, -1, -1, -1, -1, -1};  // slot -> child
    uint32_t left = (1u << nk) - 1u;                   // children without a slot
    for (size_t n = 0; n < nk; ++n) {
        int bk = -1;
        for (size_t k = 0; k < nk; ++k) {
            if (!(left >> k & 1u)) continue;
            if (kid_in[best[k]] >= 0) {
                int b = -1;
                for (int s = 0; s < 8; ++s)
                    if (kid_in[s] < 0 && (b < 0 || score[k][s] > score[k][b])) b = s;
                best[k] = b;
            }
            if (bk < 0 || score[k][best[k]] > score[bk][best[bk]]) bk = (int)k;
        }
        kid_in[best[bk]] = bk;
        left &= ~(1u << bk);
    }
    // quantisation grid: step = a power of two, origin a little below the
    // union's low corner, such that 255 steps cover the union and the
    // margins, and origin - 2^15 steps is a float
    float p[3];
    double steps[3], per_step[3];
    int ex[3];
    for (int a = 0; a < 3; ++a) {
        for (ex[a] = grid_exponent(uhi[a] - ulo[a]);; ++ex[a]) {
            const double step = pow2(ex[a] - 127), shift = pow2(ex[a] - 127 + 15);
            const float below = float_below(float_below(ulo[a] - step / 16) - shift);
            p[a] = (float)((double)below + shift);  // exact: a multiple of a step of `below`, and no larger
            if (ex[a] == 254 || uhi[a] - p[a] <= (255.0 - kGridMargin) * step) break;
        }
        steps[a] = pow2(ex[a] - 127);
        per_step[a] = pow2(127 - ex[a]);  // exact: x * per_step is x / step
    }
    node = Cw8Node{};
    for (int a = 0; a < 3; ++a) {
        std::memcpy(&node.w[a], &p[a], 4);
        node.w[3] |= (uint32_t)ex[a] << (8 * a);
    }
    for (uint32_t s = 0, first = 0; s < 8; ++s) {
        in_slot[s] = kid_in[s] < 0 ? kNoNode : kids[kid_in[s]];
        if (kid_in[s] < 0) continue;
        const tracer_bvh_node& n = nodes[in_slot[s]];
        for (int a = 0; a < 3; ++a) {
            const double step = steps[a];
            double qlo = std::floor(((double)n.bmin[a] - p[a]) * per_step[a] - kGridMargin);
            double qhi = std::ceil(((double)n.bmax[a] - p[a]) * per_step[a] + kGridMargin);
            qlo = std::min(255.0, std::max(0.0, qlo));
            qhi = std::min(255.0, std::max(0.0, qhi));
            // the decoded box must contain the child's box (exact in double)
            if (!((double)p[a] + qlo * step <= (double)n.bmin[a] && (double)p[a] + qhi * step >= (double)n.bmax[a]))
                return false;
            put_byte(node.w + 8 + 2 * a, s, (uint32_t)qlo);
            put_byte(node.w + 14 + 2 * a, s, (uint32_t)qhi);
        }
        if (cuts[in_slot[s]].leaf) {
            put_byte(node.w + 20, s, (1u << cuts[in_slot[s]].prims) - 1u);
            put_byte(node.w + 22, s, first);
            first += cuts[in_slot[s]].prims;
        } else {
            node.w[3] |= 1u << (24 + s);
            put_byte(node.w + 6, s, 7u);
            put_byte(node.w + 20, s, 1u);
            put_byte(node.w + 22, s, 24u + s);
        }
    }
    return true;
}

void append_prims(const tracer_bvh_node* nodes, uint32_t n, std::vector<uint32_t>& order)
{
    if (nodes[n].count > 0) {
        for (int32_t j = 0; j < nodes[n].count; ++j) order.push_back((uint32_t)(nodes[n].left_or_first + j));
        return;
    }
    append_prims(nodes, (uint32_t)nodes[n].left_or_first, order);
    append_prims(nodes, (uint32_t)nodes[n].left_or_first + 1, order);
}

}  // namespace

bool build_cw8(const tracer_bvh_node* nodes, uint32_t num_nodes, std::vector<Cw8Node>& out,
               std::vector<uint32_t>& order_out, uint32_t* depth_out, double* cost_out, uint32_t threads)
{
    out.clear();
    order_out.clear();
    if (depth_out) *depth_out = 0;
    if (cost_out) *cost_out = 0.0;
    if (!nodes || num_nodes == 0) return true;
    std::atomic<bool> ok{true};
    over_chunks(num_nodes, threads, [&](size_t from, size_t to) {
        for (size_t i = from; i < to; ++i) {
            const tracer_bvh_node& n = nodes[i];
            bool fits = n.count >= 0 && (uint32_t)n.count <= kCw8MaxLeafPrims;
            if (n.count == 0 && (n.left_or_first <= 0 || (uint32_t)n.left_or_first + 1 >= num_nodes)) fits = false;
            for (int a = 0; a < 3; ++a) fits = fits && std::fabs(n.bmin[a]) <= 1e6f && std::fabs(n.bmax[a]) <= 1e6f;
            if (!fits) ok = false;
        }
    });
    if (!ok) return false;
    // Which binary nodes become 8-wide nodes, which leaf children: the least
    // expected cost, bottom up.
    const std::unique_ptr<Cut[]> cuts = plan_cuts(nodes, num_nodes, threads);
    const double root_area = area(nodes[0]);
    if (cost_out && root_area > 0.0) *cost_out = cuts[0].cost[1] / root_area;
    // level by level: a level's nodes, then where their children and primitives start
    std::vector<uint32_t> bin{0u};                  // the binary node of each 8-wide one
    std::vector<std::array<uint32_t, 8>> in_slot;  // of the level's nodes
    uint32_t depth = 0;
    for (size_t lo = 0; lo < bin.size(); ++depth) {
        const size_t n = bin.size() - lo;
        out.resize(lo + n);
        in_slot.resize(n);
        over_chunks(n, threads, [&](size_t from, size_t to) {
            for (size_t k = from; k < to; ++k)
                if (!fill_node(nodes, cuts.get(), bin[lo + k], in_slot[k], out[lo + k])) ok = false;
        }, 256);
        if (!ok) return false;
        for (size_t k = 0; k < n; ++k) {
            out[lo + k].w[4] = (uint32_t)bin.size();
            out[lo + k].w[5] = (uint32_t)order_out.size();
            for (uint32_t c : in_slot[k]) {
                if (c == kNoNode) continue;
                if (cuts[c].leaf)
                    append_prims(nodes, c, order_out);
                else
                    bin.push_back(c);
            }
        }
        lo += n;
    }
    if (depth_out) *depth_out = depth;
    return true;
}

bool pack_w8(const std::vector<Cw8Node>& in, std::vector<W8Node>& out)
{
    out.assign(in.size(), W8Node{});
    for (size_t i = 0; i < in.size(); ++i) {
        const uint32_t* x = in[i].w;
        uint32_t* y = out[i].w;
        auto byte_of = [&](int word, int k) { return (x[word + k / 4] >> (8 * (k % 4))) & 0xFFu; };
        const uint32_t imask = x[3] >> 24;
        uint32_t leaf = 0, two = 0;
        for (int k = 0; k < 8; ++k) {
            const uint32_t bits = byte_of(20, k);
            if (((imask >> k) & 1u) || bits == 0) continue;
            if (bits > 3u) return false;
            leaf |= 1u << k;
            if (bits == 3u) two |= 1u << k;
        }
        for (int a = 0; a < 3; ++a) {
            const int e = (int)((x[3] >> (8 * a)) & 0xFFu);
            float p;
            std::memcpy(&p, &x[a], 4);
            const float step = std::ldexp(1.0f, e - 127), shifted = (float)((double)p - std::ldexp(1.0, e - 127 + 15));
            std::memcpy(&y[a], &shifted, 4);
            std::memcpy(&y[3 + a], &step, 4);
            for (int h = 0; h < 2; ++h) {
                y[10 + 4 * a + h] = x[8 + 2 * a + h];
                y[12 + 4 * a + h] = x[14 + 2 * a + h];
            }
        }
        y[6] = x[4];
        y[7] = x[5];
        y[8] = imask | leaf << 8 | two << 16;
    }
    return true;
}

void split_leaves(const tracer_bvh_node* nodes, uint32_t num_nodes, const double (*tri)[6],
                  std::vector<tracer_bvh_node>& out, std::vector<uint32_t>& slot_out, uint32_t threads)
{
    // Only what the root reaches is split: a caller's array may hold other
    // entries, whose ranges nobody has checked.
    std::vector<uint8_t> reached(num_nodes, 0);
    std::vector<uint32_t> todo(1, 0u);
    uint32_t n_prims = 0;
    while (!todo.empty()) {
        const uint32_t i = todo.back();
        todo.pop_back();
        reached[i] = 1;
        if (nodes[i].count > 0) {
            n_prims += (uint32_t)nodes[i].count;
        } else {
            todo.push_back((uint32_t)nodes[i].left_or_first);
            todo.push_back((uint32_t)nodes[i].left_or_first + 1);
        }
    }
    struct Leaf {
        uint32_t node, parts;  // its entry, and where its parts go
    };
    std::vector<Leaf> leaves;
    uint32_t end = num_nodes;
    for (uint32_t i = 0; i < num_nodes; ++i)
        if (reached[i] && nodes[i].count > 1) {
            leaves.push_back({i, end});
            end += 2 * (uint32_t)nodes[i].count - 2;
        }
    out.resize(end);
    slot_out.resize(n_prims);
    over_chunks(n_prims, threads, [&](size_t from, size_t to) {
        for (size_t k = from; k < to; ++k) slot_out[k] = (uint32_t)k;
    });
    std::copy(nodes, nodes + num_nodes, out.begin());
    over_chunks(leaves.size(), threads, [&](size_t from, size_t to) {
        for (size_t k = from; k < to; ++k) split_leaf(tri, leaves[k].node, leaves[k].parts, out.data(), slot_out.data());
    }, 256);
}

}  // namespace vkt
