// Plain forward kernel for sm_103a: one thread per pixel, 16-pixel-wide
// tiles, one launch -- the reference dispatch's own form (vkCmdDispatch(
// res/16, res/16, 1), GraphicsDevice.cpp:1266).  For linear-scan scenes and
// small frames, the 1x bar for the wavefront and batched paths and, with
// statistics, the canonical definition of the traversal counters.

#include <cuda_runtime.h>

#include <type_traits>

#include "tracer_core.cuh"
#include "tracer_cw8.cuh"
#include "tracer_launch.h"

namespace vkt {

// With statistics, the canonical traversal (its node visiting order is the
// oracle's); without, the path kernels' faster one, which finds the same hits.
template <int TIE, bool BVH, bool STATS, bool W8, bool SHORT>
using PlainTracer = std::conditional_t<STATS, Tracer<TIE, BVH, STATS, SHORT>, PathTracer<TIE, BVH, STATS, W8, SHORT>>;

template <int TIE, bool BVH, bool STATS, bool W8, bool SHORT>
__device__ __forceinline__ PlainTracer<TIE, BVH, STATS, W8, SHORT> plain_tracer(const TraceArgs& a, int* smem, Counters& cnt)
{
    if constexpr (STATS) {
        const int n = blockDim.x, tid = threadIdx.x;
        return Tracer<TIE, BVH, STATS, SHORT>{
            a.sc, Stack{smem + tid, reinterpret_cast<float*>(smem + (size_t)a.stack_depth * n) + tid, n, (int)a.stack_depth},
            cnt, a.status, a.trav_limit};
    } else {
        return PathTracer<TIE, BVH, STATS, W8, SHORT>(a.sc, thread_stack(smem, a.stack_depth), cnt, a.status, a.trav_limit);
    }
}

// The bounces of a warp's paths run in step: every live lane traces one
// closest hit, then the lanes shade together (shadow rays too).  All lanes
// finish a sample before any starts the next (the reference's frame: 1.56 ms
// against 1.76 for lanes that go straight on, as measured when every sample
// still traced its primary ray).  Every sample of a pixel starts with
// the same ray (no jitter, Tracer.comp:568-574), so its hit is found once (not
// with statistics, which count the reference's rays): 1280x720 x 4 spp, soup of
// 10k triangles 1.15 -> 0.64 ms, height field of 200k 1.65 -> 1.31, 20k
// triangles and 30 spheres 3.52 -> 2.65, lit scene of 12k 14.3 -> 13.4; 1 to 3 %
// slower at 1 spp, by registers.
//
// Bound by issue and instruction fetches, so a kernel holds only what its
// scenes need: no next-event code without lights (NEE; 1280x720 x 4 spp of 20k
// triangles, 30 spheres: 3.42 ms, 3.70 with it), no binary traversal on
// triangle-only scenes (W8), and with BVHs and lights one copy of the
// traversal (trace_rays: 12k triangles, 200 spheres, 2 lights: 14.2 ms, 29.1
// with two).
template <int TIE, bool BVH, bool STATS, bool NEE, bool W8, int BLOCKS>
__global__ void __launch_bounds__(256, BLOCKS) k_plain(TraceArgs a)
{
    extern __shared__ int smem[];
    const int tid = threadIdx.x;
    const int nthreads = blockDim.x;
    Counters cnt;
#pragma unroll
    for (int k = 0; k < C_COUNT; ++k) cnt.c[k] = 0;
    constexpr bool kShort = !BVH && NEE;
    PlainTracer<TIE, BVH, STATS, W8, kShort> tr = plain_tracer<TIE, BVH, STATS, W8, kShort>(a, smem, cnt);
    const uint32_t x = blockIdx.x * 16 + (tid & 15);
    const uint32_t y = blockIdx.y * (nthreads >> 4) + (tid >> 4);
    bool alive = x < a.width && y < a.height;
    std::conditional_t<!BVH && NEE && BLOCKS >= 4, RngCall, Rng> g;
    seed_rng(a, x, y, g);
    const Ray pr = primary_ray(a, x, y);
    Ray ray = pr;
    V3 accum = splat(0.0f), acc = splat(0.0f), mask = splat(1.0f);
    uint32_t prim0 = NO_PRIM, sample = 0, depth = 0;
    float t0 = -1.0f;  // with prim0, kind0, slot0: the primary hit
    int kind0 = 0;
    uint32_t slot0 = 0;
    for (; sample < a.spp; ++sample) {
        bool on = alive;
        ray = pr;
        acc = splat(0.0f);
        mask = splat(1.0f);
        for (depth = 0; depth < a.max_depth; ++depth) {
            if (!__any_sync(0xFFFFFFFFu, on)) break;
            // the primary ray is the same in every sample: traced once
            const bool given = !STATS && sample > 0 && depth == 0;
            const auto primary = [&](bool found, const Hit& h) {
                if (sample == 0 && depth == 0) {
                    prim0 = found ? h.prim : NO_PRIM;
                    t0 = found ? h.t : -1.0f;
                    kind0 = h.kind;
                    slot0 = h.slot;
                }
            };
            Hit h{given ? t0 : depth_tmax(depth), prim0, kind0, slot0};
            if (on) acc = vclamp01(acc);
            if (BVH && NEE) {
                on = trace_bounce(tr, a, on, given, kind0 != 0, h, depth, ray, acc, mask, g, primary);
            } else {
                bool found = kind0 != 0;
                if (on && !given) {
                    found = tr.trace(ray, h, false);
                    primary(found, h);
                }
                __syncwarp();
                on = shade_bounce<NEE, NEE>(tr, a, on, depth, found, h, ray, acc, mask, g);
            }
        }
        accum = accum + acc;
    }
    if (alive) resolve_pixel(a, x, y, accum, g, prim0, t0);
    if (STATS) flush_counters(a, cnt);
}

template <int TIE, bool BVH, bool STATS, bool NEE, bool W8, int BLOCKS>
static cudaError_t launch_k(const TraceArgs& a, const LaunchConfig& lc, cudaStream_t s)
{
    const size_t smem = (size_t)a.stack_depth * lc.block * 8;
    auto k = k_plain<TIE, BVH, STATS, NEE, W8, BLOCKS>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    dim3 grid((a.width + 15) / 16, (a.height + (lc.block / 16) - 1) / (lc.block / 16));
    k<<<grid, lc.block, smem, s>>>(a);
    return cudaGetLastError();
}

// The register budget, as resident blocks of 256.  Frames that fit two such
// blocks per SM have no use for a third: 104-127 registers with BVHs, where a
// soup of 10k triangles at 320x180 x 4 spp took 225 us (232 at three blocks,
// 247 at four), a lit scene of 12.7k primitives 2.79 ms (3.09, 3.16); linear
// scans with lights too, the reference's scene at that size 206 us (229 at four).
// (Counted traversals of BVHs, 100k triangles: 3.3 ms without a bound, 3.5 at
// three.)  Larger ones: four, three on triangle-only scenes (1280x720 x 4 spp, three /
// four: height field of 20k triangles 0.86 / 0.90 ms; 64 spheres 1.23 / 1.11,
// the lit scene 15.3 / 14.2).
template <int TIE, bool BVH, bool STATS, bool NEE, bool W8>
static cudaError_t launch_sized(const TraceArgs& a, const LaunchConfig& lc, cudaStream_t s)
{
    constexpr int kSmall = STATS && BVH ? 1 : BVH || NEE ? 2 : 4, kLarge = W8 || (STATS && BVH) ? 3 : 4;
    if ((uint64_t)a.width * a.height <= 512ull * lc.sms) return launch_k<TIE, BVH, STATS, NEE, W8, kSmall>(a, lc, s);
    return launch_k<TIE, BVH, STATS, NEE, W8, kLarge>(a, lc, s);
}

template <int TIE, bool BVH>
static cudaError_t launch_s(const TraceArgs& a, const LaunchConfig& lc, cudaStream_t s)
{
    if (lc.stats)
        return a.sc.ne ? launch_sized<TIE, BVH, true, true, false>(a, lc, s)
                       : launch_sized<TIE, BVH, true, false, false>(a, lc, s);
    if (a.sc.ne) return launch_sized<TIE, BVH, false, true, false>(a, lc, s);
    if constexpr (BVH)
        if (lc.w8) return launch_sized<TIE, BVH, false, false, true>(a, lc, s);
    return launch_sized<TIE, BVH, false, false, false>(a, lc, s);
}

// Reads n 16-byte words `passes` times with loads that are cached in L2 only
// (ld.global.cg), so a buffer smaller than L2 is served by L2 after the first
// pass; one word per thread is written so the loads are not optimised away.
__global__ void __launch_bounds__(256) k_l2_read(const uint4* __restrict__ buf, size_t n, uint32_t passes,
                                                 uint32_t* __restrict__ sink)
{
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t acc = 0;
    for (uint32_t p = 0; p < passes; ++p) {
        for (size_t i = tid; i < n; i += stride) {
            const uint4 v = __ldcg(buf + i);
            acc ^= v.x ^ v.y ^ v.z ^ v.w;
        }
    }
    sink[tid] = acc;
}

cudaError_t launch_l2_read(const void* buf, size_t bytes, uint32_t passes, uint32_t* sink, uint32_t blocks,
                           cudaStream_t s)
{
    k_l2_read<<<blocks, 256, 0, s>>>(static_cast<const uint4*>(buf), bytes / 16, passes, sink);
    return cudaGetLastError();
}

cudaError_t launch_plain(const TraceArgs& a, const LaunchConfig& lc, cudaStream_t s)
{
    if (lc.tie == TIE_REFERENCE) return launch_s<TIE_REFERENCE, false>(a, lc, s);
    if (lc.bvh) return launch_s<TIE_STRICT, true>(a, lc, s);
    return launch_s<TIE_STRICT, false>(a, lc, s);
}

}  // namespace vkt
