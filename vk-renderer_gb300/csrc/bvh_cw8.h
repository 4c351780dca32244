// Compressed 8-wide BVH for the wavefront's extend kernel, collapsed from the
// binary BVH (the traversal scheme of Ylitie, Karras and Laine, "Efficient
// Incoherent Ray Traversal on GPUs Through Compressed Wide BVHs", HPG 2017:
// quantised child boxes, child slots ordered by ray octant, node groups with
// a hit mask on the traversal stack; the layout below is this project's).
#pragma once

#include <algorithm>
#include <cstdint>
#include <thread>
#include <vector>

#include "tracer_abi.h"

namespace vkt {

// One node = 96 bytes (three 256-bit loads), as 24 little-endian words:
//   w0..w2   p: origin of the quantisation grid (float x, y, z)
//   w3       ex | ey << 8 | ez << 16 | imask << 24: grid steps 2^(e - 127)
//            per axis (e is a float's biased exponent), imask bit k = slot k
//            holds an interior child
//   w4       child_base: node index of the first interior child; the
//            interior children are stored consecutively in slot order
//   w5       prim_base: index (in the 8-wide primitive order) of the first
//            primitive of the node's leaf children, stored consecutively in
//            slot order (at most 24 per node)
//   w6, w7   octant mask byte of slot k (byte k % 4 of w6 + k / 4): 7 for an
//            interior child, else 0
//   w8..w19  quantised box bytes, slot k in byte k % 4 of the word pair:
//            lo x (w8, w9), lo y (w10, w11), lo z (w12, w13),
//            hi x (w14, w15), hi y (w16, w17), hi z (w18, w19);
//            box = [p + lo * 2^(e - 127), p + hi * 2^(e - 127)] per axis,
//            which contains the binary child's box with a margin of 1/64
//            grid step on each side: the kernel's slab distances, with 2^15
//            steps added and taken off, round by some 1/512 step and by 2^-23
//            of the distance from the ray's origin to p.  The second part, for
//            origins more than 2^16 steps away the larger one, is covered by
//            the acceptance's 2^-20, as in the binary test;
//            p - 2^15 * 2^(e - 127) is a float too
//   w20, w21 hit-mask bits of slot k: a leaf of c primitives (1..6) ->
//            (1 << c) - 1; an interior child -> 1; an empty slot -> 0
//   w22, w23 bit position of slot k: a leaf -> o, its first primitive being
//            prim_base + o (o + c <= 24); an interior child -> 24 + slot
// The kernels read it as a W8Node (below), without w6, w7 and w20..w23's
// positions; those are for a traversal that keeps one mask of a node's hits: a
// child hit by a ray of octant s (bit a set for a negative direction
// component on axis a) adds its bits at position (position ^ (mask & s ^ 7)).
// Slot order: slot s holds the child met first by rays of octant s.
struct alignas(32) Cw8Node {
    uint32_t w[24];
};
static_assert(sizeof(Cw8Node) == 96, "8-wide node is 96 bytes");

constexpr uint32_t kCw8MaxLeafPrims = 6;
constexpr uint32_t kCw8MaxNodePrims = 24;

// fn(from, to) over parts of [0, n), `least` or more each, on up to `threads`
// host threads, this one among them.  fn allocates nothing and throws nothing; a
// part whose thread cannot be started runs here.
template <class F> void over_chunks(size_t n, uint32_t threads, const F& fn, size_t least = 2048)
{
    const size_t parts = std::max<size_t>(1, std::min<size_t>(threads, n / least));
    std::vector<std::thread> pool;
    pool.reserve(parts - 1);
    try {
        for (size_t p = 1; p < parts; ++p) pool.emplace_back([&fn, n, p, parts] { fn(n * p / parts, n * (p + 1) / parts); });
    } catch (...) {
    }
    fn(0, n / parts);
    for (size_t p = pool.size() + 1; p < parts; ++p) fn(n * p / parts, n * (p + 1) / parts);
    for (std::thread& t : pool) t.join();
}

// Collapses a binary BVH (tracer_bvh_node, root 0, children side by side,
// leaves = ranges of the leaf-ordered primitive array) into 8-wide nodes:
// the cut of the binary tree with the least expected cost (the dynamic
// programme of Ylitie et al., section 3.1: surface area x 1 for a node
// visit, x kPrimCost for a primitive of a leaf child), where a subtree of at
// most kMergePrims primitives may become one leaf child and a node's leaf
// children hold at most 24 primitives.  order_out[k] = leaf-ordered slot of the 8-wide order's
// primitive k.  *depth_out = levels of 8-wide nodes (the traversal stack
// holds at most one entry per level).  Returns false (no 8-wide BVH) when a
// leaf holds more than 6 primitives or a coordinate's magnitude exceeds 1e6
// (the quantised slab test's range).  *cost_out = the plan's cost over the
// root's surface area: what a random ray through the root box is expected to
// visit, in nodes.
// threads: host threads to use; the tree is the same on any number.
bool build_cw8(const tracer_bvh_node* nodes, uint32_t num_nodes, std::vector<Cw8Node>& out,
               std::vector<uint32_t>& order_out, uint32_t* depth_out, double* cost_out = nullptr,
               uint32_t threads = 1);

// The node the kernels read, 96 bytes (three 256-bit loads), as 24
// little-endian words: a Cw8Node's boxes with the grid written out as floats
// and its masks gathered.
//   w0..w2   p - 2^15 * step per axis (float, exact): the kernel makes a byte
//            q the float 2^15 + q with one byte permute, so that a plane is
//            w0 + (2^15 + q) * step
//   w3..w5   the grid steps (float x, y, z)
//   w6       child_base, w7 prim_base: as Cw8Node's; slot k's primitives start
//            at prim_base + popc(leaf mask below k) + popc(two mask below k)
//   w8       imask | leaf mask << 8 | two mask << 16: bit k of each = slot k
//            holds an interior child / a leaf child / a leaf child of two
//            primitives (leaf children hold one or two); w9 0
//   w10..w21 quantised box bytes, slot k in byte k % 4 of the word pair:
//            lo x, hi x, lo y, hi y, lo z, hi z; w22, w23 0
struct alignas(32) W8Node {
    uint32_t w[24];
};
static_assert(sizeof(W8Node) == 96, "device node is 96 bytes");

// One W8Node per node of an 8-wide BVH whose leaf children hold at most two
// primitives each; false otherwise.
bool pack_w8(const std::vector<Cw8Node>& in, std::vector<W8Node>& out);

// Splits every leaf that the root of a valid binary BVH over triangles reaches
// down to single triangles (kCw8MaxLeafPrims at most per leaf), keeping the
// nodes above and whatever else the array holds.  tri[k]: low
// and high corner of the box of leaf-ordered triangle k.  out: the deeper
// tree, its leaves ranges of a new order whose entry j is leaf-ordered slot
// slot_out[j].  A part's box is that of its triangles, padded as the binary
// builder's, and inside the leaf's.  threads: as build_cw8.
void split_leaves(const tracer_bvh_node* nodes, uint32_t num_nodes, const double (*tri)[6],
                  std::vector<tracer_bvh_node>& out, std::vector<uint32_t>& slot_out, uint32_t threads = 1);

}  // namespace vkt
