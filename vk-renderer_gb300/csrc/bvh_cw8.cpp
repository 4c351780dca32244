// Collapse of a binary BVH into compressed 8-wide nodes (see bvh_cw8.h).
// Host code, deterministic: every choice has a total order (surface area,
// then position in the child list; assignment scores, then child, then slot).
#include "bvh_cw8.h"

#include <algorithm>
#include <cmath>
#include <cstring>

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

// Smallest e (biased float exponent, 1..254) with 2^(e - 127) * 255 >= ext.
int grid_exponent(double ext)
{
    int x = 0;
    std::frexp(ext / 255.0, &x);  // 255 * 2^(x - 1) <= ext < 255 * 2^x, up to the quotient's rounding
    int e = std::min(254, std::max(1, x + 125));
    while (e < 254 && std::ldexp(255.0, e - 127) < ext) ++e;
    return e;
}

// The largest float not above v.
float float_below(double v)
{
    const float f = (float)v;
    return (double)f > v ? std::nextafter(f, -HUGE_VALF) : f;
}

void put_byte(uint32_t* w, int k, uint32_t v)
{
    w[k / 4] |= (v & 0xFFu) << (8 * (k % 4));
}

// One binary node of the collapse.  cost[i], i = 1..8: least expected cost of
// its subtree given as at most i children of an 8-wide node; split[i]: of a
// cut into i >= 2 parts, how many the left child gets; parts[i]: how many of
// the i parts are used (1 = the node itself is one child).
struct Cut {
    float cost[9];
    uint8_t split[9], parts[9];
    bool leaf;       // as one child: a leaf child with all its primitives
    uint32_t prims;  // primitives of the subtree
};

std::vector<Cut> plan_cuts(const tracer_bvh_node* nodes, uint32_t num_nodes)
{
    // children before parents: a builder's nodes have larger indices than
    // their parent, a caller's need not
    std::vector<uint32_t> order, todo{0u};
    order.reserve(num_nodes);
    while (!todo.empty()) {
        const uint32_t n = todo.back();
        todo.pop_back();
        order.push_back(n);
        if (nodes[n].count == 0) {
            todo.push_back((uint32_t)nodes[n].left_or_first);
            todo.push_back((uint32_t)nodes[n].left_or_first + 1);
        }
    }
    std::vector<Cut> cuts(num_nodes);
    for (size_t q = order.size(); q-- > 0;) {
        const tracer_bvh_node& n = nodes[order[q]];
        Cut& c = cuts[order[q]];
        const float a = (float)area(n);
        if (n.count > 0) {
            c.leaf = true;
            c.prims = (uint32_t)n.count;
            for (int i = 1; i <= 8; ++i) {
                c.cost[i] = a * (float)c.prims * kPrimCost;
                c.parts[i] = 1;
                c.split[i] = 0;
            }
            continue;
        }
        const Cut& l = cuts[(uint32_t)n.left_or_first];
        const Cut& r = cuts[(uint32_t)n.left_or_first + 1];
        float cut[9];
        for (int i = 2; i <= 8; ++i) {
            cut[i] = l.cost[1] + r.cost[i - 1];
            c.split[i] = 1;
            for (int k = 2; k < i; ++k) {
                const float v = l.cost[k] + r.cost[i - k];
                if (v < cut[i]) {
                    cut[i] = v;
                    c.split[i] = (uint8_t)k;
                }
            }
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
    return cuts;
}

// The parts of node n as at most `budget` children (>= 2: n itself is cut).
void cut_children(const tracer_bvh_node* nodes, const std::vector<Cut>& cuts, uint32_t n, int budget,
                  std::vector<uint32_t>& kids)
{
    const uint32_t l = (uint32_t)nodes[n].left_or_first;
    const int left = cuts[n].split[budget], part[2] = {left, budget - left};
    for (int h = 0; h < 2; ++h) {
        const int use = cuts[l + h].parts[part[h]];
        if (use == 1)
            kids.push_back(l + h);
        else
            cut_children(nodes, cuts, l + h, use, kids);
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
        box.bmin[a] = std::max(box.bmin[a], std::nextafter((float)(lo[a] - pad), -HUGE_VALF));
        box.bmax[a] = std::min(box.bmax[a], std::nextafter((float)(hi[a] + pad), HUGE_VALF));
    }
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
               std::vector<uint32_t>& order_out, uint32_t* depth_out, double* cost_out)
{
    out.clear();
    order_out.clear();
    if (depth_out) *depth_out = 0;
    if (cost_out) *cost_out = 0.0;
    if (!nodes || num_nodes == 0) return true;
    for (uint32_t i = 0; i < num_nodes; ++i) {
        const tracer_bvh_node& n = nodes[i];
        if (n.count < 0 || (uint32_t)n.count > kCw8MaxLeafPrims) return false;
        if (n.count == 0 && (n.left_or_first <= 0 || (uint32_t)n.left_or_first + 1 >= num_nodes)) return false;
        for (int a = 0; a < 3; ++a)
            if (!(std::fabs(n.bmin[a]) <= 1e6f && std::fabs(n.bmax[a]) <= 1e6f)) return false;
    }
    // Which binary nodes become 8-wide nodes, which leaf children: the least
    // expected cost, bottom up (children are stored after their parents).
    const std::vector<Cut> cuts = plan_cuts(nodes, num_nodes);
    const double root_area = area(nodes[0]);
    if (cost_out && root_area > 0.0) *cost_out = cuts[0].cost[1] / root_area;
    struct Work {
        uint32_t wide, bin, level;
    };
    std::vector<Work> work{{0u, 0u, 1u}};
    out.push_back(Cw8Node{});
    uint32_t depth = 1;
    std::vector<uint32_t> leaf_prims;
    for (size_t wi = 0; wi < work.size(); ++wi) {
        const Work W = work[wi];
        depth = std::max(depth, W.level);
        // children: the binary node's cut into at most 8 (or the root itself,
        // when it is a leaf child), fewer if their leaves hold too many
        std::vector<uint32_t> kids;
        if (cuts[W.bin].leaf) {
            kids.push_back(W.bin);
        } else {
            for (int budget = 8; budget >= 2; --budget) {
                kids.clear();
                cut_children(nodes, cuts, W.bin, budget, kids);
                uint32_t prims = 0;
                for (uint32_t k : kids)
                    if (cuts[k].leaf) prims += cuts[k].prims;
                if (prims <= kCw8MaxNodePrims) break;
            }
        }
        // slot assignment: slot s takes the child whose centroid lies furthest
        // toward the side where rays of octant s enter (greedy on the scores)
        double ulo[3] = {HUGE_VAL, HUGE_VAL, HUGE_VAL}, uhi[3] = {-HUGE_VAL, -HUGE_VAL, -HUGE_VAL};
        for (uint32_t k : kids)
            for (int a = 0; a < 3; ++a) {
                ulo[a] = std::min(ulo[a], (double)nodes[k].bmin[a]);
                uhi[a] = std::max(uhi[a], (double)nodes[k].bmax[a]);
            }
        const size_t nk = kids.size();
        std::vector<double> score(nk * 8);
        for (size_t k = 0; k < nk; ++k)
            for (int s = 0; s < 8; ++s) {
                double v = 0.0;
                for (int a = 0; a < 3; ++a) {
                    const double c = 0.5 * ((double)nodes[kids[k]].bmin[a] + nodes[kids[k]].bmax[a]) -
                                     0.5 * (ulo[a] + uhi[a]);
                    v += ((s >> a) & 1) ? c : -c;
                }
                score[k * 8 + s] = v;
            }
        int slot_of[8] = {-1, -1, -1, -1, -1, -1, -1, -1};  // child -> slot
        int kid_in[8] = {-1, -1, -1, -1, -1, -1, -1, -1};   // slot -> child
        for (size_t n = 0; n < nk; ++n) {
            int bk = -1, bs = -1;
            double bv = -HUGE_VAL;
            for (size_t k = 0; k < nk; ++k) {
                if (slot_of[k] >= 0) continue;
                for (int s = 0; s < 8; ++s) {
                    if (kid_in[s] >= 0) continue;
                    if (score[k * 8 + s] > bv) {
                        bv = score[k * 8 + s];
                        bk = (int)k;
                        bs = s;
                    }
                }
            }
            slot_of[bk] = bs;
            kid_in[bs] = bk;
        }
        // quantisation grid: step = a power of two, origin a little below the
        // union's low corner, such that 255 steps cover the union and the
        // margins, and origin - 2^15 steps is a float
        Cw8Node node{};
        float p[3];
        double steps[3];
        int ex[3];
        for (int a = 0; a < 3; ++a) {
            for (ex[a] = grid_exponent(uhi[a] - ulo[a]);; ++ex[a]) {
                const double step = std::ldexp(1.0, ex[a] - 127), shift = std::ldexp(1.0, ex[a] - 127 + 15);
                const float below = float_below(float_below(ulo[a] - step / 16) - shift);
                p[a] = (float)((double)below + shift);  // exact: a multiple of a step of `below`, and no larger
                if (ex[a] == 254 || uhi[a] - p[a] <= (255.0 - kGridMargin) * step) break;
            }
            steps[a] = std::ldexp(1.0, ex[a] - 127);
            std::memcpy(&node.w[a], &p[a], 4);
        }
        uint32_t imask = 0, n_int = 0;
        for (int s = 0; s < 8; ++s)
            if (kid_in[s] >= 0 && !cuts[kids[kid_in[s]]].leaf) {
                imask |= 1u << s;
                ++n_int;
            }
        node.w[3] = (uint32_t)ex[0] | (uint32_t)ex[1] << 8 | (uint32_t)ex[2] << 16 | imask << 24;
        const uint32_t child_base = (uint32_t)out.size();
        const uint32_t prim_base = (uint32_t)order_out.size();
        node.w[4] = child_base;
        node.w[5] = prim_base;
        uint32_t next_child = child_base;
        for (int s = 0; s < 8; ++s) {
            if (kid_in[s] < 0) continue;
            const tracer_bvh_node& n = nodes[kids[kid_in[s]]];
            for (int a = 0; a < 3; ++a) {
                const double step = steps[a];  // a power of two: x * (1 / step) is x / step
                double qlo = std::floor(((double)n.bmin[a] - p[a]) * (1.0 / step) - kGridMargin);
                double qhi = std::ceil(((double)n.bmax[a] - p[a]) * (1.0 / step) + kGridMargin);
                qlo = std::min(255.0, std::max(0.0, qlo));
                qhi = std::min(255.0, std::max(0.0, qhi));
                // the decoded box must contain the child's box (exact in double)
                if (!((double)p[a] + qlo * step <= (double)n.bmin[a] && (double)p[a] + qhi * step >= (double)n.bmax[a]))
                    return false;
                put_byte(node.w + 8 + 2 * a, s, (uint32_t)qlo);
                put_byte(node.w + 14 + 2 * a, s, (uint32_t)qhi);
            }
            if (cuts[kids[kid_in[s]]].leaf) {
                const uint32_t o = (uint32_t)order_out.size() - prim_base;
                put_byte(node.w + 20, s, (1u << cuts[kids[kid_in[s]]].prims) - 1u);
                put_byte(node.w + 22, s, o);
                append_prims(nodes, kids[kid_in[s]], order_out);
            } else {
                put_byte(node.w + 6, s, 7u);
                put_byte(node.w + 20, s, 1u);
                put_byte(node.w + 22, s, 24u + (uint32_t)s);
                work.push_back({next_child++, kids[kid_in[s]], W.level + 1});
            }
        }
        if ((uint32_t)order_out.size() - prim_base > kCw8MaxNodePrims) return false;
        out[W.wide] = node;
        out.resize(out.size() + n_int);
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
                  std::vector<tracer_bvh_node>& out, std::vector<uint32_t>& slot_out)
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
    out.assign(nodes, nodes + num_nodes);
    out.reserve(2 * (size_t)n_prims + num_nodes);
    slot_out.resize(n_prims);
    for (uint32_t k = 0; k < n_prims; ++k) slot_out[k] = k;
    for (uint32_t i = 0; i < num_nodes; ++i) {
        if (!reached[i] || nodes[i].count <= 1) continue;
        const tracer_bvh_node leaf = nodes[i];  // every part's box stays inside it
        todo.assign(1, i);
        while (!todo.empty()) {
            const uint32_t n = todo.back();
            todo.pop_back();
            const uint32_t first = (uint32_t)out[n].left_or_first, count = (uint32_t)out[n].count;
            uint32_t* s = slot_out.data() + first;
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
                for (uint32_t at = 1; at < count; ++at) {
                    const double cost = at * left[at - 1] + (count - at) * right[count - at - 1];
                    if (cost < best_cost) {
                        best_cost = cost;
                        best_at = at;
                        std::copy(v, v + count, best);
                    }
                }
            }
            if (best_cost < HUGE_VAL) std::copy(best, best + count, s);
            const uint32_t l = (uint32_t)out.size();
            out[n].left_or_first = (int32_t)l;
            out[n].count = 0;
            for (uint32_t h = 0; h < 2; ++h) {
                tracer_bvh_node c = leaf;
                c.left_or_first = (int32_t)(h ? first + best_at : first);
                c.count = (int32_t)(h ? count - best_at : best_at);
                shrink_box(tri, slot_out.data() + c.left_or_first, (uint32_t)c.count, c);
                out.push_back(c);
                if (c.count > 1) todo.push_back(l + h);
            }
        }
    }
}

}  // namespace vkt
