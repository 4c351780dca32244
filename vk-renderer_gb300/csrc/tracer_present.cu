// The steps after the compute dispatch, for sm_103a:
//
//   k_present     the reference's present pass, Assets/Fullscreen.frag, over
//                 a headless framebuffer: per output pixel, the fragment's
//                 uv (Fullscreen.vert:8-10 draws one triangle over the
//                 viewport), flipped vertically (:16), five bilinear taps of
//                 the current image and one of the previous image (:18-24),
//                 the temporal variance vT (:26) and either the four-tap
//                 average or the centre tap (:28).
//   k_accumulate  progressive accumulation: the running sum of the frames'
//                 linear radiance and its tonemapped mean, which the present
//                 pass then reads in place of the two frame images.
//
// Sampling restates the reference's sampler (Source/GraphicsDevice.cpp:
// 770-790: linear filter, clamp-to-border with opaque black) from the texel
// filtering equations of the Vulkan specification, with exact float weights:
//   u = s * width - 0.5, i0 = floor(u), alpha = u - i0 (likewise v, j0, beta)
//   tau = (1-a)(1-b) T[i0,j0] + a(1-b) T[i0+1,j0] + (1-a) b T[i0,j0+1] + a b T[i0+1,j0+1]
// An RGBA8 UNORM texel c reads as c / 255.  Every operation is one IEEE
// single-precision operation in the order written (--fmad=false), so the
// output is bit-identical to the oracle's.
//
// k_present reads each source texel from DRAM once (taps of neighbouring
// threads share texels through L1) and is bound by instruction issue: six
// bilinear taps of twelve texel channels each.  So the arithmetic is packed
// two floats to an instruction (each rounds as its scalar form does), a tap's
// column and row are worked out once and shared by the taps they have in
// common, the conversion unit (an eighth of the FMA pipe's rate) is avoided,
// and the four neighbour taps are only evaluated where the variance test
// needs them.  1024^2 -> 1920x1080, RGBA8, half of the picture above the
// threshold: 44 us with scalar arithmetic, 32 packed.

#include <cuda_runtime.h>

#include "tracer_core.cuh"
#include "tracer_present.h"

namespace vkt {

// Two products in one instruction.  Their sums are scalar: the assembler fuses
// a packed product and a packed sum into a packed multiply-add, also where
// both ask for their own rounding and --fmad=false is given.
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }

// A texel's channels (r, g) and b.
struct Texel {
    float2 rg;
    float b;
};

// Byte K of word as a float without the conversion unit: one byte permute
// builds the float 2^23 + c, and subtracting 2^23 leaves c exactly.
template <int K>
__device__ __forceinline__ float byte_bits(uint32_t word)
{
    return __uint_as_float(__byte_perm(word, 0x4B000000u, K | (4 << 4) | (4 << 8) | (7 << 12)));
}
// c / 255, correctly rounded, for two UNORM8 codes c given as 2^23 + c: with
// 1 / 255 = hi + lo, fma(c, hi, c * lo).  Equal to the IEEE quotient for all
// 256 codes (checked exhaustively with exact rational arithmetic).
__device__ __forceinline__ float2 unorm2(float2 f)
{
    const float hi = 1.0f / 255.0f, lo = -0x1.fdfdfep-33f;
    const float2 c = __fadd2_rn(f, both(-8388608.0f));
    return __ffma2_rn(c, both(hi), mul2(c, both(lo)));
}

// Four texels of a bilinear tap.
__device__ __forceinline__ void decode4(const uint32_t (&w)[4], Texel (&t)[4])
{
#pragma unroll
    for (int k = 0; k < 4; ++k) t[k].rg = unorm2(make_float2(byte_bits<0>(w[k]), byte_bits<1>(w[k])));
#pragma unroll
    for (int k = 0; k < 4; k += 2) {
        const float2 b = unorm2(make_float2(byte_bits<2>(w[k]), byte_bits<2>(w[k + 1])));
        t[k].b = b.x;
        t[k + 1].b = b.y;
    }
}
__device__ __forceinline__ void fetch4(const uchar4* im, const size_t (&at)[4], const bool (&in)[4], Texel (&t)[4])
{
    uint32_t w[4];  // R in the low byte; 0 (black) outside
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = in[k] ? __ldg(reinterpret_cast<const uint32_t*>(im) + at[k]) : 0u;
    decode4(w, t);
}

// floor(x) and (int)x of an integer-valued x, for |x| < 2^22, on the FMA and
// integer pipes (adding 1.5 x 2^23 rounds x to an integer in the low mantissa
// bits): the same values as floorf and the float-to-int conversion.
__device__ __forceinline__ float floor_small(float x)
{
    const float r = (x + 12582912.0f) - 12582912.0f;  // x rounded to the nearest integer
    return r > x ? r - 1.0f : r;
}
__device__ __forceinline__ int int_of_small(float x) { return __float_as_int(x + 12582912.0f) - 0x4B400000; }

// A tap's position along one axis: first texel, and the second's weight.
struct Axis {
    int i;
    float f;
};
__device__ __forceinline__ Axis axis(float s, float size)
{
    const float u = s * size - 0.5f;
    const float fi = floor_small(u);
    return Axis{int_of_small(fi), u - fi};
}

// Float texels, four loads from one base but at the border and scalar products:
// nothing is decoded, and the packed form below takes longer (1920x1080 to
// 3840x2160, pictures alike: 82 us, scalar 72).
__device__ __forceinline__ V3 bilinear(const float4* im, uint32_t w, uint32_t h, Axis x, Axis y)
{
    const float w00 = (1.0f - x.f) * (1.0f - y.f), w10 = x.f * (1.0f - y.f);
    const float w01 = (1.0f - x.f) * y.f, w11 = x.f * y.f;
    V3 t[4];
    if (x.i >= 0 && y.i >= 0 && x.i + 1 < (int)w && y.i + 1 < (int)h) {
        const float4* p = im + ((size_t)y.i * w + x.i);
        t[0] = v3(__ldg(p));
        t[1] = v3(__ldg(p + 1));
        t[2] = v3(__ldg(p + w));
        t[3] = v3(__ldg(p + w + 1));
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = x.i + (k & 1), j = y.i + (k >> 1);
            const bool in = i >= 0 && j >= 0 && i < (int)w && j < (int)h;
            t[k] = in ? v3(__ldg(im + ((size_t)j * w + i))) : splat(0.0f);  // border: black
        }
    }
    return ((t[0] * w00 + t[1] * w10) + t[2] * w01) + t[3] * w11;
}

__device__ __forceinline__ V3 bilinear(const uchar4* im, uint32_t w, uint32_t h, Axis x, Axis y)
{
    const float2 cx = make_float2(1.0f - x.f, x.f);
    const float2 w0 = mul2(cx, both(1.0f - y.f)), w1 = mul2(cx, both(y.f));  // (w00, w10), (w01, w11)
    const bool x0 = x.i >= 0 && x.i < (int)w, x1 = x.i + 1 >= 0 && x.i + 1 < (int)w;
    const bool y0 = y.i >= 0 && y.i < (int)h, y1 = y.i + 1 >= 0 && y.i + 1 < (int)h;
    Texel t[4];
    const size_t k = (size_t)((long long)y.i * (int)w + x.i);  // used where its texel is inside
    const size_t at[4] = {k, k + 1, k + w, k + w + 1};
    const bool in[4] = {x0 && y0, x1 && y0, x0 && y1, x1 && y1};
    fetch4(im, at, in, t);
    const float2 p0 = mul2(t[0].rg, both(w0.x)), p1 = mul2(t[1].rg, both(w0.y));
    const float2 p2 = mul2(t[2].rg, both(w1.x)), p3 = mul2(t[3].rg, both(w1.y));
    const float2 b0 = mul2(make_float2(t[0].b, t[1].b), w0), b1 = mul2(make_float2(t[2].b, t[3].b), w1);
    return v3(((p0.x + p1.x) + p2.x) + p3.x, ((p0.y + p1.y) + p2.y) + p3.y, ((b0.x + b0.y) + b1.x) + b1.y);
}

template <class T>
__global__ void __launch_bounds__(256) k_present(PresentArgs p, const T* __restrict__ img0, const T* __restrict__ img1)
{
    const uint32_t x = blockIdx.x * 32 + (threadIdx.x & 31);
    const uint32_t y = blockIdx.y * 8 + (threadIdx.x >> 5);
    if (x >= p.width || y >= p.height) return;
    const float s = ((float)x + 0.5f) / (float)p.width;
    const float t = 1.0f - ((float)y + 0.5f) / (float)p.height;
    const float inv = 1.0f / 2048.0f;  // Fullscreen.frag:12, half a texel of the reference's 1024^2 image
    const float fw = (float)p.src_w, fh = (float)p.src_h;  // exact below 2^24
    const Axis cx = axis(s, fw), cy = axis(t, fh);
    const V3 c0 = bilinear(img0, p.src_w, p.src_h, cx, cy);
    const V3 c1 = bilinear(img1, p.src_w, p.src_h, cx, cy);
    const V3 d = c0 - c1;
    const float vT = dot(d, d);
    V3 f = c0;
    if (vT > 0.0005f) {  // the four taps are only read where the variance test fires
        const V3 n = bilinear(img0, p.src_w, p.src_h, cx, axis(t + inv, fh));
        const V3 so = bilinear(img0, p.src_w, p.src_h, cx, axis(t - inv, fh));
        const V3 e = bilinear(img0, p.src_w, p.src_h, axis(s + inv, fw), cy);
        const V3 w = bilinear(img0, p.src_w, p.src_h, axis(s - inv, fw), cy);
        f = (((n + so) + e) + w) / 4.0f;
    }
    const size_t o = (size_t)y * p.width + x;
    if (p.out8) p.out8[o] = make_uchar4(unorm8(f.x), unorm8(f.y), unorm8(f.z), 255);
    if (p.out32) p.out32[o] = make_float4(f.x, f.y, f.z, 1.0f);
}

// sum += linear; display = tonemap(sum / n) (Tracer.comp:586-588 without the
// dither).  Grid-stride over pixels.
__global__ void __launch_bounds__(256) k_accumulate(const float4* __restrict__ lin, float4* __restrict__ sum,
                                                    float4* __restrict__ disp, uint32_t npx, uint32_t n)
{
    const float gam = 1.0f / 2.2f;
    const float fn = (float)n;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < npx; i += gridDim.x * blockDim.x) {
        const float4 l = lin[i];
        float4 s = sum[i];
        s.x = s.x + l.x;
        s.y = s.y + l.y;
        s.z = s.z + l.z;
        s.w = 1.0f;
        sum[i] = s;
        V3 m = v3(s.x / fn, s.y / fn, s.z / fn);
        m = m / (m + splat(1.0f));
        disp[i] = make_float4(powf(m.x, gam), powf(m.y, gam), powf(m.z, gam), 1.0f);
    }
}

cudaError_t launch_present(const PresentArgs& p, const void* img0, const void* img1, int src_float, cudaStream_t st)
{
    const dim3 grid((p.width + 31) / 32, (p.height + 7) / 8);
    if (src_float)
        k_present<float4><<<grid, 256, 0, st>>>(p, static_cast<const float4*>(img0), static_cast<const float4*>(img1));
    else
        k_present<uchar4><<<grid, 256, 0, st>>>(p, static_cast<const uchar4*>(img0), static_cast<const uchar4*>(img1));
    return cudaGetLastError();
}

cudaError_t launch_accumulate(const float4* lin, float4* sum, float4* disp, uint32_t npx, uint32_t n, int sm_count,
                              cudaStream_t st)
{
    const uint32_t need = (npx + 255) / 256;
    const uint32_t cap = 8u * (uint32_t)sm_count;
    k_accumulate<<<need < cap ? need : cap, 256, 0, st>>>(lin, sum, disp, npx, n);
    return cudaGetLastError();
}

}  // namespace vkt
