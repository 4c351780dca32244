// Device side of the 8-wide BVH (node layout: W8Node in bvh_cw8.h): one
// node's eight slab tests and the groups a traversal keeps.
//
// A node group is (child_base, interior children hit and not yet visited |
// imask << 8), bit k = slot k: slot k's node index is
// child_base + popc(imask & ((1 << k) - 1)).  A leaf group is (prim_base,
// leaf children hit and not yet tested | leaf mask << 8 | two mask << 16).
#pragma once

#include "tracer_traverse.cuh"

namespace vkt {

// The ray's quantities for the 8-wide slab test.  Octant s of the direction:
// bit a set for a negative inverse direction on axis a.  pref4, pref2, pref1:
// the slots whose bit 2, 1, 0 equals s's, i.e. the half to visit first.
struct W8Ray {
    BoxRay br;
    uint32_t pref4, pref2, pref1;
};

__device__ __forceinline__ W8Ray make_w8ray(const Ray& r)
{
    W8Ray c;
    c.br = make_boxray(r);
    const bool fx = c.br.ix < 0.0f, fy = c.br.iy < 0.0f, fz = c.br.iz < 0.0f;
    c.pref1 = fx ? 0xAAu : 0x55u;
    c.pref2 = fy ? 0xCCu : 0x33u;
    c.pref4 = fz ? 0xF0u : 0x0Fu;
    return c;
}

// Byte k of w as the float 2^15 + byte: one byte permute into the bits of
// 2^15 (an integer-to-float conversion takes as many instructions, or a
// slower pipe).
__device__ __forceinline__ float byte_f(uint32_t w, int k)
{
    return __uint_as_float(__byte_perm(w, 0x47000000u, 0x7404u | (uint32_t)k << 4));
}

// The group of the root alone: the one interior child (slot 0) of a group of
// its own.
__device__ __forceinline__ uint2 w8_root() { return make_uint2(0u, 1u | 1u << 8); }
__device__ __forceinline__ bool w8_any(uint2 G) { return (G.y & 0xFFu) != 0u; }

// Visits node `idx`: tests its children's boxes against the ray with the
// current best distance tbest and returns the node group of the interior
// children hit (G) and the leaf group of the leaf children hit (P).  The slab
// distances are fma(2^15 + q, step * ix, fma(p - 2^15 * step, ix, -o * ix)); a
// child is hit iff max(near distances, 0) <= min(far distances, tbest), the
// right side times (1 + 2^-20): the binary test's acceptance, on a box that
// contains the binary box with a margin (Cw8Node).  A box that a ray passes
// through is entered; of boxes that it only touches within rounding, a caller's
// unpadded ones far from the origin among them, the two tests may enter
// different ones.
__device__ __forceinline__ void w8_visit(const float4* nodes, uint32_t idx, const W8Ray& r, float tbest, uint2& G,
                                         uint2& P)
{
    uint32_t u[8], v[8], w[8];
    const float4* n = nodes + 6 * (size_t)idx;
    ldg256u(n, u);
    ldg256u(n + 2, v);
    ldg256u(n + 4, w);
    const float ax = __uint_as_float(u[3]) * r.br.ix, bx = __fmaf_rn(__uint_as_float(u[0]), r.br.ix, r.br.nx);
    const float ay = __uint_as_float(u[4]) * r.br.iy, by = __fmaf_rn(__uint_as_float(u[1]), r.br.iy, r.br.ny);
    const float az = __uint_as_float(u[5]) * r.br.iz, bz = __fmaf_rn(__uint_as_float(u[2]), r.br.iz, r.br.nz);
    const float tb = tbest * BOX_SLACK;
    const float2 ax2 = make_float2(ax, ax), ay2 = make_float2(ay, ay), az2 = make_float2(az, az);
    const float2 bx2 = make_float2(bx, bx), by2 = make_float2(by, by), bz2 = make_float2(bz, bz);
    const bool fx = r.br.ix < 0.0f, fy = r.br.iy < 0.0f, fz = r.br.iz < 0.0f;
    uint32_t miss = 0;
#pragma unroll
    for (int h = 1; h >= 0; --h) {
        // near / far plane words per axis, four slots each
        const uint32_t nx = fx ? v[4 + h] : v[2 + h], qx = fx ? v[2 + h] : v[4 + h];
        const uint32_t ny = fy ? w[h] : v[6 + h], qy = fy ? v[6 + h] : w[h];
        const uint32_t nz = fz ? w[4 + h] : w[2 + h], qz = fz ? w[2 + h] : w[4 + h];
#pragma unroll
        for (int k = 2; k >= 0; k -= 2) {
            auto two = [&](uint32_t q, float2 a, float2 c) {
                return __ffma2_rn(make_float2(byte_f(q, k), byte_f(q, k + 1)), a, c);
            };
            const float2 x0 = two(nx, ax2, bx2), y0 = two(ny, ay2, by2), z0 = two(nz, az2, bz2);
            const float2 x1 = two(qx, ax2, bx2), y1 = two(qy, ay2, by2), z1 = two(qz, az2, bz2);
            const float2 tn = make_float2(fmax3(x0.x, y0.x, z0.x), fmax3(x0.y, y0.y, z0.y));
            const float2 tf = make_float2(fmin3(x1.x, y1.x, z1.x), fmin3(x1.y, y1.y, z1.y));
            const float2 mn = make_float2(-tn.x, -tn.y);
            const float2 d1 = __ffma2_rn(tf, make_float2(BOX_SLACK, BOX_SLACK), mn);
            const float2 d3 = __fadd2_rn(make_float2(tb, tb), mn);
            miss = __funnelshift_l(__float_as_uint(fmin3(d1.y, tf.y, d3.y)), miss, 1);
            miss = __funnelshift_l(__float_as_uint(fmin3(d1.x, tf.x, d3.x)), miss, 1);
        }
    }
    const uint32_t hit = ~miss;
    const uint32_t imask = v[0] & 0xFFu;
    G = make_uint2(u[6], (hit & imask) | imask << 8);
    P = make_uint2(u[7], (v[0] >> 8 & hit & 0xFFu) | (v[0] & 0x00FFFF00u));
}

// Takes the next child of a node group (which has one), the one the ray's
// octant meets first: its node index; the group keeps the others.
__device__ __forceinline__ uint32_t w8_next(uint2& G, const W8Ray& r)
{
    uint32_t x = G.y & 0xFFu, p;
    p = x & r.pref4;
    x = p ? p : x;
    p = x & r.pref2;
    x = p ? p : x;
    p = x & r.pref1;
    x = p ? p : x;  // one bit
    G.y ^= x;
    return G.x + __popc((G.y >> 8) & (x - 1u));
}

// Takes the next leaf child of a leaf group (which has one): its first
// primitive, and whether it has a second.
__device__ __forceinline__ uint32_t w8_next_leaf(uint2& P, bool& two)
{
    const uint32_t x = P.y & (0u - P.y) & 0xFFu;  // lowest of the bits below 8
    P.y ^= x;
    const uint32_t below = (x - 1u) * 0x0101u;  // x - 1 in both bytes
    two = ((P.y >> 16) & x) != 0u;
    return P.x + __popc((P.y >> 8) & below);
}

// Tests primitive k0 of the 8-wide order and, if two, the next.  A record is
// 64 bytes (v0, original id) (v1 - v0, leaf-ordered slot) (v2 - v0, 0) (0),
// read as a 256-bit and a 128-bit load; both records are fetched before
// either test, so the two L2 round trips overlap.  On acceptance the hit
// records the leaf-ordered slot (the storage slot every other kernel indexes).
template <bool STATS>
__device__ __forceinline__ void cw8_test_tri2(const float4* tris, uint32_t k0, bool two, const Ray& ray, Hit& h,
                                              Counters& cnt)
{
    if (STATS) cnt.c[C_TRIS] += two ? 2 : 1;
    float4 a0, b0, a1, b1;
    ldg256(tris + 4 * (size_t)k0, a0, b0);
    const float4 c0 = __ldg(tris + 4 * (size_t)k0 + 2);
    const uint32_t k = two ? k0 + 1u : k0;
    ldg256(tris + 4 * (size_t)k, a1, b1);
    const float4 c1 = __ldg(tris + 4 * (size_t)k + 2);
    const float t0 = tri_intersect(ray, v3(a0), v3(b0), v3(c0));
    const float t1 = tri_intersect(ray, v3(a1), v3(b1), v3(c1));
    if (accept_strict(t0, __float_as_uint(a0.w), h)) {
        h.t = t0;
        h.prim = __float_as_uint(a0.w);
        h.kind = 1;
        h.slot = __float_as_uint(b0.w);
    }
    if (two && accept_strict(t1, __float_as_uint(a1.w), h)) {
        h.t = t1;
        h.prim = __float_as_uint(a1.w);
        h.kind = 1;
        h.slot = __float_as_uint(b1.w);
    }
}

// Per-lane record of the extend kernel in shared memory: what a lane does not
// need while it visits nodes (its registers then hold a node).
struct alignas(16) W8Lane {
    float4 o, d;         // the ray; .w: scene, path slot
    const float4* tris;  // the lane's scene's primitives (8-wide order)
    uint32_t prim, slot; // best hit so far: id, storage slot (NO_PRIM: none)
};
static_assert(sizeof(W8Lane) == 48, "lane record is 48 bytes");

// One ray's pass over the triangles' 8-wide BVH by one thread: the extend
// kernel's node visit and triangle test, a node's leaves tested right after
// the visit.  any: stop at the first hit.
template <bool STATS>
__device__ __forceinline__ void w8_pass(const DevScene& sc, const Ray& ray, const W8Ray& cr, Hit& h, bool any,
                                        const PairStack& stk, int* status, uint32_t trav_limit, Counters& cnt)
{
    uint2 G = w8_root();
    int sp = 0;
    uint32_t steps = 0;
    for (;;) {
        if (!w8_any(G)) {
            if (sp == 0) break;
            --sp;
            const int2 e = stk.e[sp * stk.stride];
            G = make_uint2((uint32_t)e.x, (uint32_t)e.y);
        }
        if (++steps > trav_limit) {
            atomicCAS(status, ST_OK, ST_TRAVERSAL_LIMIT);
            break;
        }
        const uint32_t idx = w8_next(G, cr);
        if (w8_any(G)) {
            if (sp >= stk.cap) {
                atomicCAS(status, ST_OK, ST_STACK_OVERFLOW);
            } else {
                stk.e[sp * stk.stride] = make_int2((int)G.x, (int)G.y);
                ++sp;
            }
        }
        uint2 P;
        w8_visit(sc.tri_cw8, idx, cr, h.t, G, P);
        if (STATS) cnt.c[C_NODES] += 3;
        while (w8_any(P)) {
            bool two;
            const uint32_t k = w8_next_leaf(P, two);
            cw8_test_tri2<STATS>(sc.tri_cw8_prims, k, two, ray, h, cnt);
        }
        if (any && h.kind) break;
    }
}

// trace_ray of one ray by one thread over a scene with BVHs (strict ties):
// the triangles over the 8-wide BVH where the scene has one, else, and the
// spheres, over the binary BVHs, then the planes.  The same hit as every
// other traversal.  h.t holds tmax on entry; on a miss h.kind = 0 and h.prim =
// NO_PRIM.  shadow: any hit will do.  stk: the thread's stack (8-byte entries,
// interleaved by thread), at least as deep as either BVH.
// W8: a triangle-only scene with an 8-wide BVH and a closest hit: no binary
// passes, whose code and registers cost the finishing kernels a tenth (256^2
// adjoint 593 against 527 us).
template <bool STATS, bool W8>
__device__ __forceinline__ bool trace_bvh(const DevScene& sc, const Ray& ray, Hit& h, bool shadow, const PairStack& stk,
                                          int* status, uint32_t trav_limit, Counters& cnt)
{
    if (STATS) {
        cnt.c[C_SHADOW] += shadow ? 1 : 0;
        cnt.c[C_CLOSEST] += shadow ? 0 : 1;
    }
    Lane L;
    L.h.t = h.t;
    L.h.prim = 0;  // see accept_strict
    L.h.kind = 0;
    L.h.slot = 0;
    if (!isnan3(ray.d)) {
        const W8Ray cr = make_w8ray(ray);
        const bool wide = W8 || sc.tri_cw8 != nullptr;
        if (wide) w8_pass<STATS>(sc, ray, cr, L.h, shadow, stk, status, trav_limit, cnt);
        if (!W8) {
            L.br = cr.br;
            for (L.pass = wide ? 1 : 0; L.pass < 2 && !(shadow && L.h.kind); ++L.pass) {
                const bool any = L.pass == 0 ? (sc.n_tri_nodes > 0 && sc.nt > 0) : (sc.n_sph_nodes > 0 && sc.ns > 0);
                if (any) enc_pass<STATS>(sc, ray, L, shadow, stk, status, trav_limit, cnt);
            }
        }
        planes_pass<STATS>(sc, ray, L.h, cnt, shadow);
    }
    h = L.h;
    if (h.kind == 0) {
        h.prim = NO_PRIM;
        return false;
    }
    if (STATS && !shadow) cnt.c[C_HITS]++;
    return true;
}

// The per-thread trace_ray of the path kernels: trace_bvh on scenes with
// BVHs, else the linear scan.
template <int TIE, bool BVH, bool STATS, bool W8 = false, bool SHORT = false>
struct PathTracer : Tracer<TIE, false, STATS, SHORT> {
    PairStack pstk;
    __device__ __forceinline__ PathTracer(const DevScene& sc, const PairStack& p, Counters& cnt, int* status,
                                          uint32_t trav_limit)
        : Tracer<TIE, false, STATS, SHORT>{sc, Stack{nullptr, nullptr, 0, 0}, cnt, status, trav_limit}, pstk(p)
    {
    }
    __device__ __forceinline__ bool trace(const Ray& ray, Hit& h, bool shadow)
    {
        if (BVH)
            return trace_bvh<STATS, W8>(this->sc, ray, h, shadow, pstk, this->status, this->trav_limit, this->cnt);
        return Tracer<TIE, false, STATS, SHORT>::trace(ray, h, shadow);
    }
};

// A thread's stack in a block's dynamic shared memory: depth 8-byte entries a thread.
__device__ __forceinline__ PairStack thread_stack(int* smem, uint32_t depth)
{
    return PairStack{reinterpret_cast<int2*>(smem) + threadIdx.x, (int)blockDim.x, (int)depth};
}

}  // namespace vkt
