// Wavefront path tracing for sm_103a: the radiance loop of Assets/Tracer.comp
// split into stages that each run as their own kernel over a queue of live
// paths, one path per pixel.
//
//   wf_generate  seeds every pixel's RNG (Tracer.comp:563-566), writes its
//                primary ray (:568-574) and queues all pixels.
//   wf_extend    persistent warps trace the queued rays (trace_ray,
//                :374-431).  Each lane owns one ray at a time and takes the
//                next ray from the queue as soon as its ray is finished
//                (warp-aggregated fetch: ballot + popc + one atomicAdd).
//                BVH traversal is the speculative while-while scheme: all
//                lanes step through interior nodes together, each holding
//                back up to four leaves it finds, then all test their held
//                leaves together, one primitive per lane and step; stacks
//                and held leaves live in shared memory.  Small register
//                footprint, so many warps per SM hide the L1/L2 latency of
//                node fetches.
//   wf_shade     one thread per queued path: the rest of the depth iteration
//                (:441-549: clamp, sky, scatter, next-event estimation, Russian
//                roulette).  A surviving path appends itself to the next queue
//                (warp-aggregated atomics = warp-level ray compaction); a
//                finished sample starts the pixel's next sample, whose RNG
//                continues where the last one stopped (the shader's rand_salt
//                runs across samples, :578-581); a finished pixel is resolved
//                (:585-592).
//   wf_finish    for the last rounds, when few paths are live: each thread
//                runs queued paths to the end of their pixels (all remaining
//                bounces and samples), without per-round launches.
//
// MULTI = true runs many scenes of different size and resolution in the same
// queues (the batched form): every path slot belongs to one scene, whose
// TraceArgs (scene pointers into one device arena, camera, image size,
// parameters, output pointers) live in a device table.
//
// Per pixel the operations are exactly those of the plain kernel, in the same
// order, so images and hits are identical to it and to the oracle.  Only the
// order of node visits inside one ray's traversal differs (it depends on the
// warp), which changes no result under strict ties but does change the node
// counters.

#include <cuda_runtime.h>

#include "tracer_core.cuh"
#include "tracer_cw8.cuh"
#include "tracer_traverse.cuh"
#include "tracer_wavefront.h"

namespace vkt {

// The TraceArgs a path belongs to: the launch's own (single scene) or its
// scene's entry in the table (batched).
#define SCENE_ARGS(MULTI, a, slots, sid) ((MULTI) ? (slots)[(sid)] : (a))

// ---------------------------------------------------------------- generate --
template <bool MULTI>
__global__ void __launch_bounds__(256) wf_generate(TraceArgs a, WfState s, const TraceArgs* slots, uint32_t nslots)
{
    const uint32_t n = a.num_slots;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) {
        s.count[0] = n;
        s.count[1] = 0;
        s.count[2] = 0;
    }
    if (i >= n) return;
    uint32_t sid = 0;
    if (MULTI) {  // the scene whose slot range holds i: last pixel_base <= i
        uint32_t lo = 0, hi = nslots;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (slots[mid].pixel_base <= i)
                lo = mid;
            else
                hi = mid;
        }
        sid = lo;
        s.scene_of[i] = sid;
    }
    const TraceArgs& A = SCENE_ARGS(MULTI, a, slots, sid);
    const uint32_t p = i - A.pixel_base;
    const uint32_t x = p % A.width, y = p / A.width;
    Rng g;
    seed_rng(A, x, y, g);
    const Ray r = primary_ray(A, x, y);
    s.ray_o[i] = make_float4(r.o.x, r.o.y, r.o.z, depth_tmax(0));
    s.ray_d[i] = make_float4(r.d.x, r.d.y, r.d.z, 0.0f);
    s.acc[i] = make_float4(0.0f, 0.0f, 0.0f, g.salt);
    s.mask[i] = make_float4(1.0f, 1.0f, 1.0f, -1.0f);
    s.accum[i] = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(0u));
    s.prim0[i] = NO_PRIM;
    s.queue[0][i] = i;
}

// ------------------------------------------------------------------ extend --
__device__ __forceinline__ void order2(float& ta, int& ra, float& tb, int& rb)
{
    if (tb < ta) {
        const float t = ta;
        ta = tb;
        tb = t;
        const int r = ra;
        ra = rb;
        rb = r;
    }
}

// One 4-wide node: the slab test of each child's box (the binary node's box,
// the same test as box_hit), the nearest child hit becomes the next
// reference, the others are pushed farthest first.  Which boxes are tested
// differs from the binary traversal only in order and in skipping interior
// boxes, so the closest hit under strict ties is the same.
template <bool STATS>
__device__ __forceinline__ void visit_wide(Lane& L, int w, const PairStack& stk, int* status, Counters& cnt)
{
    // node = four (box min, reference) (box max, 0) records
    const float4* n = L.nodes + 8 * (size_t)w;
    const float INF = __int_as_float(0x7f800000);
    float t0, t1, t2, t3;
    int r0, r1, r2, r3;
    auto child = [&](int k, float& t, int& r) {
        const float4 lo = __ldg(n + 2 * k), hi = __ldg(n + 2 * k + 1);
        r = __float_as_int(lo.w);
        if (STATS) cnt.c[C_NODES] += r != 0;
        if (!(r != 0 && box_hit(L.br, lo, hi, L.h.t, t))) {
            t = INF;
            r = 0;
        }
    };
    child(0, t0, r0);
    child(1, t1, r1);
    child(2, t2, r2);
    child(3, t3, r3);
    // sorting network: ascending distance (misses last)
    order2(t0, r0, t1, r1);
    order2(t2, r2, t3, r3);
    order2(t0, r0, t2, r2);
    order2(t1, r1, t3, r3);
    order2(t1, r1, t2, r2);
    if (r3) push(L, stk, r3, t3, status);
    if (r2) push(L, stk, r2, t2, status);
    if (r1) push(L, stk, r1, t1, status);
    L.cur = r0 ? r0 : pop(L, stk);
}

// Leaves a lane may hold back while the warp's slowest lane is still looking
// for its first (measured on c1: 2 -> 95.8 ms, 4 -> 91.0, 6 -> 91.0, 8 -> 91.2).
constexpr int kPostpone = 4;

// Moves leaf references from L.cur into the lane's buffer of postponed leaves
// (entry j at lbuf[j * stride]), taking the next stack entry after each,
// until L.cur is an interior node or empty or the buffer is full.
__device__ __forceinline__ void postpone_leaves(Lane& L, const PairStack& stk, int* lbuf, int stride, int& nl)
{
    while (L.cur < 0 && nl < kPostpone) {
        lbuf[nl * stride] = L.cur;
        ++nl;
        L.cur = pop(L, stk);
    }
}

template <bool STATS, bool WIDE>
__device__ __forceinline__ void start_pass(const DevScene& sc, Lane& L, Counters& cnt, const PairStack& stk,
                                           int* lbuf, int stride, int& nl, int* status)
{
    L.prims = L.pass == 0 ? sc.tri : sc.sph_geo;
    L.sp = 0;
    if (WIDE) {
        L.nodes = L.pass == 0 ? sc.tri_wide : sc.sph_wide;
        visit_wide<STATS>(L, 0, stk, status, cnt);
    } else {
        L.nodes = L.pass == 0 ? sc.tri_enc : sc.sph_enc;  // references pre-encoded in bmin.w
        float4 lo, hi;
        ldg256(L.nodes, lo, hi);
        if (STATS) cnt.c[C_NODES]++;
        float tn;
        L.cur = box_hit(L.br, lo, hi, L.h.t, tn) ? __float_as_int(lo.w) : 0;  // the root may be a leaf
    }
    postpone_leaves(L, stk, lbuf, stride, nl);
}

// Tests primitive `slot` of the current pass for the lane's ray.
template <bool STATS, bool MULTI>
__device__ __forceinline__ void test_prim(const TraceArgs& a, const TraceArgs* slots, Lane& L, const Ray& ray,
                                          int slot, Counters& cnt)
{
    if (L.pass == 0) {
        if (STATS) cnt.c[C_TRIS]++;
        const float4* t = L.prims + 3 * (size_t)slot;
        const float4 ta = __ldg(t), tb = __ldg(t + 1), tc = __ldg(t + 2);
        const float tt = tri_intersect(ray, v3(ta), v3(tb), v3(tc));
        const uint32_t id = __float_as_uint(tb.w);
        if (accept_strict(tt, id, L.h)) {
            L.h.t = tt;
            L.h.prim = id;
            L.h.kind = 1;
            L.h.slot = slot;
        }
    } else {
        const DevScene& sc = SCENE_ARGS(MULTI, a, slots, L.scene).sc;
        if (STATS) cnt.c[C_SPHERES]++;
        const float4 gg = __ldg(L.prims + slot);
        const float tt = sphere_intersect(ray, v3(gg), gg.w);
        const uint32_t id = sc.nt + __ldg(sc.sph_id + slot);
        if (accept_strict(tt, id, L.h)) {
            L.h.t = tt;
            L.h.prim = id;
            L.h.kind = 2;
            L.h.slot = slot;
        }
    }
}

// 1024 resident threads per SM (63 registers).  Each outer iteration: idle
// lanes fetch rays; all lanes step through interior nodes until every lane
// still tracing holds a leaf, lanes that already hold some keep going (up to
// kPostpone leaves, speculatively: their best hit is not yet updated by
// them); then all lanes test their held leaves' primitives, one primitive per
// lane and iteration.
template <int TIE, bool STATS, bool MULTI, int BLOCK, bool WIDE>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK)
    wf_extend_bvh(TraceArgs a, WfState s, int qsel, const TraceArgs* slots)
{
    extern __shared__ int smem[];
    const unsigned full = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const PairStack stk{reinterpret_cast<int2*>(smem) + threadIdx.x, BLOCK, (int)a.stack_depth};
    int* lbuf = smem + 2 * (size_t)a.stack_depth * BLOCK + threadIdx.x;  // postponed leaves, stride BLOCK
    const uint32_t total = s.count[qsel];
    const uint32_t* queue = qsel ? s.queue[1] : s.queue[0];
    if (blockIdx.x == 0 && threadIdx.x == 0) s.count[qsel ^ 1] = 0;
    Counters cnt;
#pragma unroll
    for (int k = 0; k < C_COUNT; ++k) cnt.c[k] = 0;
    Lane L;
    L.has = false;
    int nl = 0;  // postponed leaves held
    bool exhausted = false;
    for (;;) {
        // 1) idle lanes take the next rays of the queue
        const unsigned need = __ballot_sync(full, !L.has && !exhausted);
        if (need) {
            const int leader = __ffs(need) - 1;
            uint32_t base = 0;
            if (lane == leader) base = atomicAdd(&s.count[2], (uint32_t)__popc(need));
            base = __shfl_sync(full, base, leader);
            if (!L.has && !exhausted) {
                const uint32_t qi = base + __popc(need & ((1u << lane) - 1u));
                if (qi >= total) {
                    exhausted = true;
                } else {
                    L.pid = queue[qi];
                    L.scene = MULTI ? s.scene_of[L.pid] : 0;
                    const DevScene& sc = SCENE_ARGS(MULTI, a, slots, L.scene).sc;
                    const float4 ro = s.ray_o[L.pid];
                    const float4 rd = s.ray_d[L.pid];
                    L.o = v3(ro);
                    L.d = v3(rd);
                    L.h.t = ro.w;
                    L.h.prim = 0;  // see accept_strict
                    L.h.kind = 0;
                    L.h.slot = 0;
                    L.steps = 0;
                    if (STATS) cnt.c[C_CLOSEST]++;
                    L.has = true;
                    const bool has_tri = sc.n_tri_nodes > 0 && sc.nt > 0;
                    const bool has_sph = sc.n_sph_nodes > 0 && sc.ns > 0;
                    if (isnan3(L.d) || (!has_tri && !has_sph)) {
                        // no BVH work: NaN directions hit nothing; planes only
                        if (!isnan3(L.d)) planes_pass<STATS>(sc, Ray{L.o, L.d}, L.h, cnt);
                        if (STATS && L.h.kind) cnt.c[C_HITS]++;
                        s.hit[L.pid] = make_uint4(__float_as_uint(L.h.t), L.h.prim, L.h.slot, (uint32_t)L.h.kind);
                        L.has = false;
                    } else {
                        L.br = make_boxray(Ray{L.o, L.d});
                        L.pass = has_tri ? 0 : 1;
                        start_pass<STATS, WIDE>(sc, L, cnt, stk, lbuf, BLOCK, nl, a.status);
                    }
                }
            }
        }
        if (!__any_sync(full, L.has)) {
            if (__all_sync(full, exhausted)) break;
            continue;
        }
        // 2) interior nodes, until every lane still tracing holds a leaf
        for (;;) {
            const bool can = L.has && L.cur > 0 && nl < kPostpone;
            if (!__any_sync(full, can && nl == 0)) break;
            if (can) {
                if (++L.steps > a.trav_limit) {
                    atomicCAS(a.status, ST_OK, ST_TRAVERSAL_LIMIT);
                    L.cur = 0;
                    L.sp = 0;
                } else if (WIDE) {
                    visit_wide<STATS>(L, L.cur, stk, a.status, cnt);
                } else {
                    const float4* c = L.nodes + 2 * (size_t)L.cur;
                    float4 lo0, hi0, lo1, hi1;
                    ldg256(c, lo0, hi0);
                    ldg256(c + 2, lo1, hi1);
                    if (STATS) cnt.c[C_NODES] += 2;
                    float t0, t1;
                    const bool h0 = box_hit(L.br, lo0, hi0, L.h.t, t0);
                    const bool h1 = box_hit(L.br, lo1, hi1, L.h.t, t1);
                    const int e0 = __float_as_int(lo0.w), e1 = __float_as_int(lo1.w);
                    if (!h0 && !h1) {
                        L.cur = pop(L, stk);
                    } else {
                        const bool swap = h1 && (!h0 || t1 < t0);
                        L.cur = swap ? e1 : e0;
                        if (h0 && h1) push(L, stk, swap ? e0 : e1, swap ? t0 : t1, a.status);
                    }
                }
                postpone_leaves(L, stk, lbuf, BLOCK, nl);
            }
        }
        // 3) the held leaves, one primitive per lane and iteration
        {
            int lj = 0, lfirst = 0, lcount = 0;
            const Ray ray{L.o, L.d};
            for (;;) {
                const bool lf = L.has && (lcount > 0 || lj < nl);
                if (!__any_sync(full, lf)) break;
                if (lf) {
                    if (lcount == 0) {
                        leaf_dec(lbuf[lj * BLOCK], lfirst, lcount);
                        ++lj;
                    }
                    test_prim<STATS, MULTI>(a, slots, L, ray, lfirst, cnt);
                    ++lfirst;
                    --lcount;
                }
            }
        }
        nl = 0;
        if (L.has) postpone_leaves(L, stk, lbuf, BLOCK, nl);  // a leaf met with the buffer full
        // 4) finished passes: next primitive kind, or planes and the result
        if (L.has && L.cur == 0 && nl == 0) {
            const DevScene& sc = SCENE_ARGS(MULTI, a, slots, L.scene).sc;
            if (L.pass == 0 && sc.n_sph_nodes > 0 && sc.ns > 0) {
                L.pass = 1;
                start_pass<STATS, WIDE>(sc, L, cnt, stk, lbuf, BLOCK, nl, a.status);
            } else {
                planes_pass<STATS>(sc, Ray{L.o, L.d}, L.h, cnt);
                if (STATS && L.h.kind) cnt.c[C_HITS]++;
                s.hit[L.pid] = make_uint4(__float_as_uint(L.h.t), L.h.prim, L.h.slot, (uint32_t)L.h.kind);
                L.has = false;
            }
        }
    }
    if (STATS) flush_counters(a, cnt);
}

// Leaf groups a lane of the 8-wide traversal may hold back while the warp's
// slowest lane is still looking for its first (c1 frame, ms: 4 -> 43.9, 6 ->
// 42.4, 8 -> 42.4, 12 -> 42.3; each takes 8 bytes of shared memory a thread).
constexpr int kCw8Postpone = 6;

// The extend kernel over the 8-wide BVH (triangle scenes; strict ties).
// Phases as in wf_extend_bvh: idle lanes fetch rays; all lanes visit 8-wide
// nodes (one per lane and step: eight quantised slab tests, the hit interior
// children become a node group on the stack, the hit leaves a leaf group held
// back) until every lane still tracing holds some leaves, lanes that hold
// fewer than kCw8Postpone groups going on; then all lanes test their held
// leaves, one leaf (at most two triangles, both records fetched before
// either test) per lane and step.  Node groups are visited nearest-octant
// first; which boxes are entered depends on the order, the closest hit under
// strict ties does not.
//
// What bounds it (c1 scene, ncu): L1's data pipe 68 %, the integer pipe 62 %,
// issue 60 %, all three by the node visits (36 a ray, 5-10 triangle tests).
// So the node is three 256-bit loads, not more and narrower ones: a 128-byte
// node with its planes as 16-bit floats saves the byte conversions but was
// slower here, c1 frame 52.0 ms against 46.3 (seven or eight loads a visit,
// L1 83 %), though faster in the finishing kernels.  Pairs of slots share one
// packed multiply-add (43.1 against 46.3 ms).  c1 frame over the steps: 58.0
// ms with binary leaves as leaf children (43 tests a ray), 54.2 with leaves
// split and the collapse planned by cost, 42.4 with this node and kernel.
// Sharing the last leaves of a phase out over the warp no longer pays (43.1;
// it needs 16 more bytes and the phase is a sixth of the work now), nor does
// ending the node phase once 4, 6, 8 or 12 lanes idle (45.1, 44.1, 43.8, 44.0).
// 72 registers, seven 128-thread blocks per SM (64 registers and eight
// blocks: 34 bytes spilled, 43.8 ms; 80 and six: 42.8).
template <bool STATS, bool MULTI, int BLOCK>
__global__ void __launch_bounds__(BLOCK, 896 / BLOCK)
    wf_extend_cw8(TraceArgs a, WfState s, int qsel, const TraceArgs* slots)
{
    extern __shared__ int smem[];
    const unsigned full = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    // stack of node groups, then held leaf groups (entry j of a thread at
    // j * BLOCK + threadIdx.x), then the threads' records.  The stack holds at
    // most one group per level of the tree (siblings left behind on the way
    // down), and stack_depth is at least its number of levels.
    uint2* stk = reinterpret_cast<uint2*>(smem) + threadIdx.x;
    uint2* held = reinterpret_cast<uint2*>(smem) + (size_t)a.stack_depth * BLOCK + threadIdx.x;
    W8Lane* rec =
        reinterpret_cast<W8Lane*>(reinterpret_cast<uint2*>(smem) + ((size_t)a.stack_depth + kCw8Postpone) * BLOCK) +
        threadIdx.x;
    const uint32_t total = s.count[qsel];
    const uint32_t* queue = qsel ? s.queue[1] : s.queue[0];
    if (blockIdx.x == 0 && threadIdx.x == 0) s.count[qsel ^ 1] = 0;
    Counters cnt;
#pragma unroll
    for (int k = 0; k < C_COUNT; ++k) cnt.c[k] = 0;
    bool has = false, exhausted = false;
    uint32_t steps = 0;
    W8Ray cr{};
    float tbest = 0.0f;
    uint2 G = make_uint2(0u, 0u);
    int sp = 0, nh = 0;
    // one scene: its nodes (a kernel argument); batched: the lane's scene's
    const float4* my_nodes = nullptr;
    // idle lanes take the next rays of the queue (warp-aggregated: one
    // atomic per warp and call)
    auto fetch = [&]() {
        const unsigned need = __ballot_sync(full, !has && !exhausted);
        if (!need) return;
        const int leader = __ffs(need) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(&s.count[2], (uint32_t)__popc(need));
        base = __shfl_sync(full, base, leader);
        if (has || exhausted) return;
        const uint32_t qi = base + __popc(need & ((1u << lane) - 1u));
        if (qi >= total) {
            exhausted = true;
            return;
        }
        const uint32_t pid = queue[qi];
        const uint32_t scene = MULTI ? s.scene_of[pid] : 0;
        const DevScene& sc = SCENE_ARGS(MULTI, a, slots, scene).sc;
        const float4 ro = s.ray_o[pid];
        const float4 rd = s.ray_d[pid];
        const Ray ray{v3(ro), v3(rd)};
        steps = 0;
        if (STATS) cnt.c[C_CLOSEST]++;
        has = true;
        if (isnan3(ray.d) || !(sc.n_tri_nodes > 0 && sc.nt > 0)) {
            // no BVH work: NaN directions hit nothing; planes only
            Hit h{ro.w, 0u, 0, 0u};
            if (!isnan3(ray.d)) planes_pass<STATS>(sc, ray, h, cnt);
            if (STATS && h.kind) cnt.c[C_HITS]++;
            s.hit[pid] = make_uint4(__float_as_uint(h.t), h.prim, h.slot, (uint32_t)h.kind);
            has = false;
        } else {
            rec->o = make_float4(ro.x, ro.y, ro.z, __uint_as_float(scene));
            rec->d = make_float4(rd.x, rd.y, rd.z, __uint_as_float(pid));
            rec->tris = sc.tri_cw8_prims;
            rec->prim = 0u;  // see accept_strict
            rec->slot = NO_PRIM;
            tbest = ro.w;
            cr = make_w8ray(ray);
            if (MULTI) my_nodes = sc.tri_cw8;
            G = w8_root();
            sp = 0;
        }
    };
    // a ray whose traversal is over and whose primitives are all tested:
    // planes, then its result
    auto finish_ray = [&]() {
        const float4 o = rec->o, d = rec->d;
        const uint32_t pid = __float_as_uint(d.w), slot = rec->slot;
        Hit h{tbest, rec->prim, slot != NO_PRIM ? 1 : 0, slot != NO_PRIM ? slot : 0u};
        const DevScene& sc = SCENE_ARGS(MULTI, a, slots, __float_as_uint(o.w)).sc;
        planes_pass<STATS>(sc, Ray{v3(o), v3(d)}, h, cnt);
        if (STATS && h.kind) cnt.c[C_HITS]++;
        s.hit[pid] = make_uint4(__float_as_uint(h.t), h.prim, h.slot, (uint32_t)h.kind);
        has = false;
    };
    for (;;) {
        // 1) idle lanes take the next rays of the queue
        fetch();
        if (!__any_sync(full, has)) {
            if (__all_sync(full, exhausted)) break;
            continue;
        }
        // 2) nodes, until every lane still tracing holds primitives
        for (;;) {
            const bool search = has && nh < kCw8Postpone && (w8_any(G) || sp > 0) && steps < a.trav_limit;
            if (!__any_sync(full, search && nh == 0)) break;
            if (search) {
                ++steps;
                if (!w8_any(G)) {
                    --sp;
                    G = stk[sp * BLOCK];
                }
                const uint32_t idx = w8_next(G, cr);
                if (w8_any(G)) {
                    stk[sp * BLOCK] = G;
                    ++sp;
                }
                uint2 P;
                w8_visit(MULTI ? my_nodes : a.sc.tri_cw8, idx, cr, tbest, G, P);
                if (STATS) cnt.c[C_NODES] += 3;
                held[nh * BLOCK] = P;
                nh += w8_any(P) ? 1 : 0;
            }
        }
        if (has && steps >= a.trav_limit && (w8_any(G) || sp > 0)) {  // give up the rest of this ray's nodes
            atomicCAS(a.status, ST_OK, ST_TRAVERSAL_LIMIT);
            G = make_uint2(0u, 0u);
            sp = 0;
        }
        // 3) the held leaves: one leaf (two primitives at most) per lane and step
        if (nh > 0) {
            int j = 0;
            uint2 cur = make_uint2(0u, 0u);
            const Ray ray{v3(rec->o), v3(rec->d)};
            const float4* tris = MULTI ? rec->tris : a.sc.tri_cw8_prims;
            Hit h{tbest, rec->prim, 1, rec->slot};
            for (;;) {
                if (!w8_any(cur)) {
                    if (j == nh) break;
                    cur = held[j * BLOCK];
                    ++j;
                }
                bool two;
                const uint32_t k = w8_next_leaf(cur, two);
                cw8_test_tri2<STATS>(tris, k, two, ray, h, cnt);
            }
            tbest = h.t;
            rec->prim = h.prim;
            rec->slot = h.slot;
            nh = 0;
        }
        // 4) finished rays: planes and the result
        if (has && !w8_any(G) && sp == 0) finish_ray();
    }
    if (STATS) flush_counters(a, cnt);
}

// Linear-scan scenes (the reference's own trace_ray, reference or strict ties):
// persistent lanes with a per-warp fetch.  Single scene only.
template <int TIE, bool STATS>
__global__ void __launch_bounds__(128) wf_extend_linear(TraceArgs a, WfState s, int qsel)
{
    const unsigned full = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const uint32_t total = s.count[qsel];
    const uint32_t* queue = qsel ? s.queue[1] : s.queue[0];
    if (blockIdx.x == 0 && threadIdx.x == 0) s.count[qsel ^ 1] = 0;
    Counters cnt;
#pragma unroll
    for (int k = 0; k < C_COUNT; ++k) cnt.c[k] = 0;
    Tracer<TIE, false, STATS> tr{a.sc, Stack{nullptr, nullptr, 0, 0}, cnt, a.status, a.trav_limit};
    for (;;) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&s.count[2], 32u);
        base = __shfl_sync(full, base, 0);
        if (base >= total) break;
        const uint32_t qi = base + lane;
        if (qi < total) {
            const uint32_t pid = queue[qi];
            const float4 ro = s.ray_o[pid];
            const float4 rd = s.ray_d[pid];
            Hit h;
            h.t = ro.w;
            tr.trace(Ray{v3(ro), v3(rd)}, h, false);
            s.hit[pid] = make_uint4(__float_as_uint(h.t), h.prim, h.slot, (uint32_t)h.kind);
        }
    }
    if (STATS) flush_counters(a, cnt);
}

// ------------------------------------------------------------- path state --
// One path slot between rounds, unpacked from the WfState arrays.
struct PathRegs {
    Ray ray;
    V3 acc, mask, accum;
    float t0;  // t of the pixel's primary hit (-1: none)
    uint32_t prim0, sample, depth;
    Rng g;
};

__device__ __forceinline__ void load_path(const WfState& s, const TraceArgs& A, uint32_t pid, uint32_t x, uint32_t y,
                                          PathRegs& p)
{
    const float4 ro = s.ray_o[pid], rd = s.ray_d[pid];
    const float4 acc4 = s.acc[pid], mask4 = s.mask[pid], accum4 = s.accum[pid];
    p.ray = Ray{v3(ro), v3(rd)};
    p.acc = v3(acc4);
    p.mask = v3(mask4);
    p.accum = v3(accum4);
    p.t0 = mask4.w;
    p.prim0 = s.prim0[pid];
    const uint32_t sd = __float_as_uint(accum4.w);
    p.sample = sd >> 16;
    p.depth = sd & 0xFFFFu;
    p.g.salt = acc4.w;
    p.g.cx = (float)x / (float)A.width;
    p.g.cy = (float)y / (float)A.height;
}

__device__ __forceinline__ void store_path(const WfState& s, uint32_t pid, const PathRegs& p)
{
    s.ray_o[pid] = make_float4(p.ray.o.x, p.ray.o.y, p.ray.o.z, depth_tmax(p.depth));
    s.ray_d[pid] = make_float4(p.ray.d.x, p.ray.d.y, p.ray.d.z, 0.0f);
    s.acc[pid] = make_float4(p.acc.x, p.acc.y, p.acc.z, p.g.salt);
    s.mask[pid] = make_float4(p.mask.x, p.mask.y, p.mask.z, p.t0);
    s.accum[pid] = make_float4(p.accum.x, p.accum.y, p.accum.z, __uint_as_float((p.sample << 16) | p.depth));
    s.prim0[pid] = p.prim0;
}

// The pixel's primary hit, for the primary-hit image.
__device__ __forceinline__ void note_primary(PathRegs& p, bool found, const Hit& h)
{
    if (p.sample == 0 && p.depth == 0) {
        p.prim0 = found ? h.prim : NO_PRIM;
        p.t0 = found ? h.t : -1.0f;
    }
}

// After a bounce (cont: its path goes on): the next depth, else the pixel's
// next sample, else the resolve.  Returns true while the pixel has a ray.
__device__ __forceinline__ bool next_ray(const TraceArgs& A, uint32_t x, uint32_t y, bool cont, PathRegs& p)
{
    p.depth++;
    if (cont && p.depth < A.max_depth) return true;
    p.accum = p.accum + p.acc;
    p.sample++;
    p.depth = 0;
    if (p.sample < A.spp) {
        p.ray = primary_ray(A, x, y);
        p.acc = splat(0.0f);
        p.mask = splat(1.0f);
        return true;
    }
    resolve_pixel(A, x, y, p.accum, p.g, p.prim0, p.t0);
    return false;
}

// The rest of one depth iteration after its closest hit h (Tracer.comp:441-549:
// clamp, sky, scatter, next-event estimation, Russian roulette), then the
// sample and pixel bookkeeping (:578-592): the next depth, else the pixel's
// next sample (its RNG continues where the last sample stopped), else the
// resolve.  Returns true while the pixel has another ray to trace: p.ray, with
// tmax depth_tmax(p.depth).  NEE, SYNC: as shade_bounce; with SYNC every lane of
// the warp calls this together, those with a path being on.
template <bool NEE, bool SYNC, class TR>
__device__ __forceinline__ bool advance_path(TR& tr, const TraceArgs& A, bool on, uint32_t x, uint32_t y, const Hit& h,
                                             PathRegs& p)
{
    const bool found = on && h.kind != 0;
    if (on) {
        note_primary(p, found, h);
        p.acc = vclamp01(p.acc);
    }
    const bool cont = shade_bounce<NEE, SYNC>(tr, A, on, p.depth, found, h, p.ray, p.acc, p.mask, p.g);
    return on && next_ray(A, x, y, cont, p);
}

// The next sample of pixel pid starts with its primary ray, whose hit sample 0
// kept (s.hit0): h = that hit, and no ray to trace.  False with p elsewhere.
__device__ __forceinline__ bool known_hit(const WfState& s, uint32_t pid, const PathRegs& p, Hit& h)
{
    if (!s.hit0 || p.depth > 0 || p.sample == 0) return false;
    h = hit_unpack(s.hit0[pid]);
    return true;
}

// ------------------------------------------------------------------- shade --
// KEEP: a pixel's next sample goes on from its kept primary hit here, without a
// round.  A form of its own, as the loop costs the others 8 % (2000 spheres,
// 1920x1080 x 1 spp, all shade launches: 0.40 ms, 0.37 without).
template <int TIE, bool BVH, bool STATS, bool MULTI, bool NEE, bool KEEP>
__global__ void __launch_bounds__(256) wf_shade(TraceArgs a, WfState s, int qsel, const TraceArgs* slots)
{
    extern __shared__ int smem[];
    const uint32_t n = s.count[qsel];
    const uint32_t* queue = qsel ? s.queue[1] : s.queue[0];
    uint32_t* next = qsel ? s.queue[0] : s.queue[1];
    if (blockIdx.x == 0 && threadIdx.x == 0) s.count[2] = 0;  // fetch cursor of the next round
    Counters cnt;
#pragma unroll
    for (int k = 0; k < C_COUNT; ++k) cnt.c[k] = 0;
    const PairStack stk = thread_stack(smem, a.stack_depth);  // shadow rays'
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
        const uint32_t qi = base + threadIdx.x;
        bool on = qi < n;
        const uint32_t pid = on ? queue[qi] : 0;
        const TraceArgs& A = SCENE_ARGS(MULTI, a, slots, MULTI && on ? s.scene_of[pid] : 0);
        PathTracer<TIE, BVH, STATS> tr(A.sc, stk, cnt, a.status, A.trav_limit);
        const uint32_t p = pid - (on ? A.pixel_base : 0);
        const uint32_t x = p % A.width, y = p / A.width;
        PathRegs ps;
        Hit h;
        if (on) {
            load_path(s, A, pid, x, y, ps);
            h = hit_unpack(s.hit[pid]);
            if (s.hit0 && ps.sample == 0 && ps.depth == 0) s.hit0[pid] = hit_pack(h);
        }
        bool again = false;
        while (NEE ? __any_sync(0xFFFFFFFFu, on) : on) {
            const bool more = advance_path<NEE, NEE>(tr, A, on, x, y, h, ps);
            again = on ? more : again;
            if (!KEEP) break;
            on = on && more && known_hit(s, pid, ps, h);
        }
        if (again) store_path(s, pid, ps);
        warp_append(again, pid, next, &s.count[qsel ^ 1]);
    }
    if (STATS) flush_counters(a, cnt);
}

// ------------------------------------------------------------------ finish --
// Runs every queued path to the end of its pixel in one launch: a thread takes
// a path and traces and shades it bounce after bounce, sample after sample,
// with the per-thread traversal, until the pixel is resolved; then it takes
// the next.  For the last rounds of a wavefront, when few paths are live, and
// for whole frames with fewer pixels than that: the paths then need no
// launches per round and do not wait each round for that round's slowest ray.
// The operations per pixel are those of extend + shade, in the same order, so
// the results are identical.  A warp's lanes go from bounce to bounce
// together (640x360 x 4 frame with two lights: 2.25 ms, 7.18 each on its own).
// First path of a thread: queue entry = its global index; later ones from the
// cursor count[2] (zeroed by the generate or shade that wrote the queue),
// offset by the number of threads.
// W8: triangle-only scenes with an 8-wide BVH, without lights.  (Lanes with
// finished rays shading while the others' walks wait, once 13, 10 or 8 of 16
// are finished, instead of all: 720p mesh 3354, 3449, 3554 against 3481 us, but
// a 10k-triangle soup 1240, 1377, 1384 against 1146.)
template <int TIE, bool BVH, bool STATS, bool MULTI, bool NEE, bool W8>
__global__ void __launch_bounds__(128) wf_finish(TraceArgs a, WfState s, int qsel, const TraceArgs* slots)
{
    extern __shared__ int smem[];
    const uint32_t n = s.count[qsel];
    const uint32_t* queue = qsel ? s.queue[1] : s.queue[0];
    Counters cnt;
#pragma unroll
    for (int k = 0; k < C_COUNT; ++k) cnt.c[k] = 0;
    const PairStack stk = thread_stack(smem, a.stack_depth);
    const uint32_t threads = gridDim.x * blockDim.x;
    uint32_t qi = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t pid = 0, scene = 0, x = 0, y = 0;
    PathRegs ps;
    bool on = false;
    auto take = [&]() {  // the path of queue entry qi, if there is one
        on = qi < n;
        if (!on) return;
        pid = queue[qi];
        scene = MULTI ? s.scene_of[pid] : 0;
        const TraceArgs& A = SCENE_ARGS(MULTI, a, slots, scene);
        const uint32_t p = pid - A.pixel_base;
        x = p % A.width;
        y = p / A.width;
        load_path(s, A, pid, x, y, ps);
    };
    take();
    // Linear scans, but for long ones with lights: each lane on its own, as a bounce
    // is mostly shading (the reference's scene without its light, 320x180 x 4: 0.10
    // ms, 0.16 in step, with it 800x600 1.41, 1.52; 100 spheres with two lights 320x180
    // 0.96, 1.06; 204 primitives with lights, 800x600, 4.85, 4.46).
    const bool alone = !BVH && (!NEE || a.sc.nt + a.sc.ns + a.sc.np <= 128u);
    while (alone && on) {
        PathTracer<TIE, BVH, STATS, W8> tr(a.sc, stk, cnt, a.status, a.trav_limit);
        Hit h;
        do {
            if (known_hit(s, pid, ps, h)) continue;
            h.t = depth_tmax(ps.depth);
            tr.trace(ps.ray, h, false);
            if (s.hit0 && ps.sample == 0 && ps.depth == 0) s.hit0[pid] = hit_pack(h);
        } while (advance_path<NEE, false>(tr, a, true, x, y, h, ps));
        qi = n > threads ? threads + atomicAdd(&s.count[2], 1u) : n;
        take();
    }
    while (!alone && __any_sync(0xFFFFFFFFu, on)) {
        const TraceArgs& A = SCENE_ARGS(MULTI, a, slots, scene);
        PathTracer<TIE, BVH, STATS, W8> tr(A.sc, stk, cnt, a.status, A.trav_limit);
        Hit h;
        h.t = on ? depth_tmax(ps.depth) : 0.0f;
        bool again = false;
        const auto first_hit = [&](bool found, const Hit& first) {
            note_primary(ps, found, first);
            if (s.hit0 && ps.sample == 0 && ps.depth == 0) s.hit0[pid] = hit_pack(first);
        };
        if (NEE) {
            const bool given = on && known_hit(s, pid, ps, h);
            if (on) ps.acc = vclamp01(ps.acc);
            const bool cont = trace_bounce(tr, A, on, given, given && h.kind != 0, h, ps.depth, ps.ray, ps.acc, ps.mask,
                                           ps.g, first_hit);
            again = on && next_ray(A, x, y, cont, ps);
        } else {
            if (on) first_hit(tr.trace(ps.ray, h, false), h);
            __syncwarp();
            for (bool go = on; go; go = again && known_hit(s, pid, ps, h))
                again = advance_path<false, false>(tr, A, true, x, y, h, ps);
            __syncwarp();
        }
        if (on && !again) {
            qi = n > threads ? threads + atomicAdd(&s.count[2], 1u) : n;
            take();
        }
    }
    if (STATS) flush_counters(a, cnt);
}

// ---------------------------------------------------------------- dispatch --
template <class K>
static void smem_attr(K k, size_t smem)
{
    if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

// Dynamic shared memory of the extend kernel: every thread's traversal stack
// (8 B per entry) and its held leaves (binary and 4-wide: 4 B per leaf
// reference) or held primitive groups (8-wide: 8 B per group).
static size_t wf_extend_smem(size_t stack_depth, uint32_t block, int wide)
{
    return (stack_depth * 8 + (wide == WF_WIDTH_8 ? kCw8Postpone * 8 + sizeof(W8Lane) : kPostpone * 4)) * block;
}

template <int TIE, bool STATS, bool MULTI, int BLOCK>
static cudaError_t extend_bvh_b(const TraceArgs& a, const WfState& s, const WfConfig& c, int qsel, cudaStream_t st)
{
    auto k = c.wide == WF_WIDTH_8   ? wf_extend_cw8<STATS, MULTI, BLOCK>
             : c.wide == WF_WIDTH_4 ? wf_extend_bvh<TIE, STATS, MULTI, BLOCK, true>
                                    : wf_extend_bvh<TIE, STATS, MULTI, BLOCK, false>;
    if (c.wide == WF_WIDTH_8 && c.cw8_stack != 0) {
        TraceArgs a8 = a;
        a8.stack_depth = c.cw8_stack;
        const size_t smem = wf_extend_smem(a8.stack_depth, BLOCK, c.wide);
        smem_attr(k, smem);
        k<<<c.extend_grid, BLOCK, smem, st>>>(a8, s, qsel, c.slots);
        return cudaGetLastError();
    }
    const size_t smem = wf_extend_smem(a.stack_depth, BLOCK, c.wide);
    smem_attr(k, smem);
    k<<<c.extend_grid, BLOCK, smem, st>>>(a, s, qsel, c.slots);
    return cudaGetLastError();
}

template <int TIE, bool BVH, bool STATS, bool MULTI>
static cudaError_t extend_t(const TraceArgs& a, const WfState& s, const WfConfig& c, int qsel, cudaStream_t st)
{
    if (BVH) {
        if (c.block == 64) return extend_bvh_b<TIE, STATS, MULTI, 64>(a, s, c, qsel, st);
        if (c.block == 256) return extend_bvh_b<TIE, STATS, MULTI, 256>(a, s, c, qsel, st);
        return extend_bvh_b<TIE, STATS, MULTI, 128>(a, s, c, qsel, st);
    }
    wf_extend_linear<TIE, STATS><<<c.extend_grid, 128, 0, st>>>(a, s, qsel);
    return cudaGetLastError();
}

template <int TIE, bool BVH, bool STATS, bool MULTI>
static cudaError_t shade_t(const TraceArgs& a, const WfState& s, const WfConfig& c, int qsel, cudaStream_t st)
{
    auto k = c.has_emitters ? wf_shade<TIE, BVH, STATS, MULTI, true, false> : wf_shade<TIE, BVH, STATS, MULTI, false, false>;
    if constexpr (!STATS)
        if (c.shade_samples)
            k = c.has_emitters ? wf_shade<TIE, BVH, STATS, MULTI, true, true> : wf_shade<TIE, BVH, STATS, MULTI, false, true>;
    const size_t smem = (BVH && c.has_emitters) ? (size_t)a.stack_depth * 256 * 8 : 0;  // shadow rays' stack
    smem_attr(k, smem);
    k<<<c.shade_grid, 256, smem, st>>>(a, s, qsel, c.slots);
    return cudaGetLastError();
}

// Dynamic shared memory of the finishing kernel (128 threads): the stacks.
static size_t wf_finish_smem(bool bvh, size_t stack_depth) { return bvh ? stack_depth * 128 * 8 : 0; }

using FinishKernel = void (*)(TraceArgs, WfState, int, const TraceArgs*);

template <int TIE, bool BVH, bool STATS, bool MULTI>
static FinishKernel finish_kernel(const WfConfig& c)
{
    if (c.has_emitters) return wf_finish<TIE, BVH, STATS, MULTI, true, false>;
    if (BVH && c.finish_w8) return wf_finish<TIE, BVH, STATS, MULTI, false, BVH>;
    return wf_finish<TIE, BVH, STATS, MULTI, false, false>;
}

template <int TIE, bool BVH, bool STATS, bool MULTI>
static cudaError_t finish_t(const TraceArgs& a, const WfState& s, const WfConfig& c, int qsel, cudaStream_t st)
{
    const FinishKernel k = finish_kernel<TIE, BVH, STATS, MULTI>(c);
    const size_t smem = wf_finish_smem(BVH, a.stack_depth);
    smem_attr(k, smem);
    k<<<c.finish_grid, 128, smem, st>>>(a, s, qsel, c.slots);
    return cudaGetLastError();
}

template <int TIE, bool BVH, bool STATS, bool MULTI>
static int finish_occ(size_t smem, const WfConfig& c)
{
    const FinishKernel k = finish_kernel<TIE, BVH, STATS, MULTI>(c);
    smem_attr(k, smem);
    int n = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, 128, smem) == cudaSuccess ? n : 0;
}

// Template selection: ties, BVH (strict only), statistics, multi-scene (BVH only).
#define WF_DISPATCH(fn)                                                                                    \
    if (c.multi) {                                                                                         \
        return c.stats ? fn<TIE_STRICT, true, true, true>(a, s, c, qsel, st)                              \
                       : fn<TIE_STRICT, true, false, true>(a, s, c, qsel, st);                            \
    }                                                                                                      \
    if (c.tie == TIE_REFERENCE)                                                                            \
        return c.stats ? fn<TIE_REFERENCE, false, true, false>(a, s, c, qsel, st)                         \
                       : fn<TIE_REFERENCE, false, false, false>(a, s, c, qsel, st);                       \
    if (c.bvh)                                                                                             \
        return c.stats ? fn<TIE_STRICT, true, true, false>(a, s, c, qsel, st)                             \
                       : fn<TIE_STRICT, true, false, false>(a, s, c, qsel, st);                           \
    return c.stats ? fn<TIE_STRICT, false, true, false>(a, s, c, qsel, st)                                \
                   : fn<TIE_STRICT, false, false, false>(a, s, c, qsel, st);

cudaError_t wf_launch_generate(const TraceArgs& a, const WfState& s, const WfConfig& c, cudaStream_t st)
{
    const uint32_t n = a.num_slots;
    if (c.multi)
        wf_generate<true><<<(n + 255) / 256, 256, 0, st>>>(a, s, c.slots, c.nslots);
    else
        wf_generate<false><<<(n + 255) / 256, 256, 0, st>>>(a, s, nullptr, 0);
    return cudaGetLastError();
}

cudaError_t wf_launch_extend(const TraceArgs& a, const WfState& s, const WfConfig& c, int qsel, cudaStream_t st)
{
    WF_DISPATCH(extend_t)
}

cudaError_t wf_launch_shade(const TraceArgs& a, const WfState& s, const WfConfig& c, int qsel, cudaStream_t st)
{
    WF_DISPATCH(shade_t)
}

cudaError_t wf_launch_finish(const TraceArgs& a, const WfState& s, const WfConfig& c, int qsel, cudaStream_t st)
{
    WF_DISPATCH(finish_t)
}

int wf_finish_blocks_per_sm(const WfConfig& c, uint32_t stack_depth)
{
    const size_t smem = wf_finish_smem(c.bvh != 0, stack_depth);
    if (c.multi) return c.stats ? finish_occ<TIE_STRICT, true, true, true>(smem, c)
                                : finish_occ<TIE_STRICT, true, false, true>(smem, c);
    if (c.tie == TIE_REFERENCE) return c.stats ? finish_occ<TIE_REFERENCE, false, true, false>(smem, c)
                                               : finish_occ<TIE_REFERENCE, false, false, false>(smem, c);
    if (c.bvh) return c.stats ? finish_occ<TIE_STRICT, true, true, false>(smem, c)
                              : finish_occ<TIE_STRICT, true, false, false>(smem, c);
    return c.stats ? finish_occ<TIE_STRICT, false, true, false>(smem, c)
                   : finish_occ<TIE_STRICT, false, false, false>(smem, c);
}

template <int TIE, bool STATS, bool MULTI, int BLOCK>
static cudaError_t occ_bvh_b(int& n, int wide, size_t smem)
{
    auto k = wide == WF_WIDTH_8   ? wf_extend_cw8<STATS, MULTI, BLOCK>
             : wide == WF_WIDTH_4 ? wf_extend_bvh<TIE, STATS, MULTI, BLOCK, true>
                                  : wf_extend_bvh<TIE, STATS, MULTI, BLOCK, false>;
    smem_attr(k, smem);
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, BLOCK, smem);
}

template <int TIE, bool STATS, bool MULTI>
static int occ_bvh(uint32_t block, size_t stack_depth, int wide)
{
    int n = 0;
    const size_t smem = wf_extend_smem(stack_depth, block, wide);
    cudaError_t e;
    if (block == 64)
        e = occ_bvh_b<TIE, STATS, MULTI, 64>(n, wide, smem);
    else if (block == 256)
        e = occ_bvh_b<TIE, STATS, MULTI, 256>(n, wide, smem);
    else
        e = occ_bvh_b<TIE, STATS, MULTI, 128>(n, wide, smem);
    return e == cudaSuccess ? n : 0;
}

int wf_extend_blocks_per_sm(const WfConfig& c, uint32_t stack_depth)
{
    const int w = c.wide;
    if (w == WF_WIDTH_8 && c.cw8_stack != 0) stack_depth = c.cw8_stack;
    if (c.multi) return c.stats ? occ_bvh<TIE_STRICT, true, true>(c.block, stack_depth, w)
                                : occ_bvh<TIE_STRICT, false, true>(c.block, stack_depth, w);
    if (c.bvh) return c.stats ? occ_bvh<TIE_STRICT, true, false>(c.block, stack_depth, w)
                              : occ_bvh<TIE_STRICT, false, false>(c.block, stack_depth, w);
    int n = 0;
    cudaError_t e;
    if (c.tie == TIE_REFERENCE)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &n, c.stats ? wf_extend_linear<TIE_REFERENCE, true> : wf_extend_linear<TIE_REFERENCE, false>, 128, 0);
    else
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &n, c.stats ? wf_extend_linear<TIE_STRICT, true> : wf_extend_linear<TIE_STRICT, false>, 128, 0);
    return e == cudaSuccess ? n : 0;
}

}  // namespace vkt
