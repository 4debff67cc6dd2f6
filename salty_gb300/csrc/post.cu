// post.cu -- tonemapping, sRGB8 and the NLM denoisers.
//
//   ToneMapper::Map (src/s3d_tonemapper.cpp:206-353): a log-average / max-luminance
//   reduction, then a per-pixel curve (Reinhard, Uncharted2, ACES) fused with the clamp,
//   OETF and 8-bit rounding of PathTracer::Capture (src/s3d_pt.cpp:145-171).  Both passes
//   stream the image once (HBM bound); per-pixel arithmetic keeps the reference's
//   operation order with separately rounded products.  The reduction adds log terms in pairs
//   of FP32 numbers and the pairs in double (salty_tonemap), or four by four and then in double
//   (salty_tonemap_noalloc), where the reference adds them one by one in single precision.
//   FilterNLM (src/s3d_denoiser.cpp:19-95): each block stages its tile plus halo in
//   shared memory; overlapping patches share their squared differences.
#include <algorithm>
#include <cfloat>
#include <cstring>

#include "internal.h"

namespace salty {
namespace {

__device__ __forceinline__ int f2o(float f) {
    int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float o2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }
struct LumAcc {
    double sum;
    int maxo;
    int pad;
};

// RGBToY (src/s3d_tonemapper.cpp:31-33)
__device__ __forceinline__ float rgb_to_y(float r, float g, float b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(0.299f, r), __fmul_rn(0.587f, g)), __fmul_rn(0.114f, b));
}

constexpr int kRedBlock = 256;

__device__ __forceinline__ float u2_curve(float x) {
    const float A = 0.15f, B = 0.50f, C = 0.10f, D = 0.20f, E = 0.01f, F = 0.30f;
    // ((x*(A*x + C*B) + D*E) / (x*(A*x + B) + D*F)) - E/F
    float num = __fadd_rn(__fmul_rn(x, __fadd_rn(__fmul_rn(A, x), __fmul_rn(C, B))), __fmul_rn(D, E));
    float den = __fadd_rn(__fmul_rn(x, __fadd_rn(__fmul_rn(A, x), B)), __fmul_rn(D, F));
    return __fsub_rn(__fdiv_rn(num, den), __fdiv_rn(E, F));
}

__device__ __forceinline__ float saturate(float x) { return x < 0.0f ? 0.0f : (x > 1.0f ? 1.0f : x); }

// a / 12 rounded to nearest, for |a| in [2^-100, 2^100]: a quotient estimate, its exact remainder
// and one correction, which rounds correctly when the reciprocal is itself correctly rounded
// (Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990).
__device__ __forceinline__ float div12(float a) {
    constexpr float r = 1.0f / 12.0f;
    const float q = __fmul_rn(a, r);
    return fmaf(fmaf(-12.0f, q, a), r, q);
}

// ACESFilm (src/s3d_tonemapper.cpp:117-130)
__device__ __forceinline__ float aces_curve(float x) {
    const float a = 2.51f, b = 0.03f, c = 2.43f, d = 0.59f, e = 0.14f, f = 0.665406f, g = 12.0f;
    const float axf = __fmul_rn(__fmul_rn(a, x), f), xf = __fmul_rn(x, f);
    float axf12, xf12;
    if (fabsf(x) > 0x1p-90f && fabsf(x) < 0x1p90f) {
        axf12 = div12(axf);
        xf12 = div12(xf);
    } else {
        axf12 = __fdiv_rn(axf, g);
        xf12 = __fdiv_rn(xf, g);
    }
    float num = __fmul_rn(x, __fadd_rn(axf12, b));
    float den = __fadd_rn(__fmul_rn(xf12, __fadd_rn(__fmul_rn(__fmul_rn(c, x), f), d)), e);
    return saturate(__fdiv_rn(num, den));
}

// 8-bit code of a tonemapped value: clamp to [0, 1], the OETF (the reference's
// 1.055^(1/2.4)-scaled variant or the standard one), then x * 255 + 0.5 truncated.  The power
// is first taken with the hardware approximation (__powf); only when the scaled value lies
// within 2^-10 of a code boundary is it recomputed with powf, so the code always equals
// the all-powf formula's: the approximation moves x * 255 + 0.5 by less than 1e-4 (from
// the documented errors of the hardware log2 and exp2 on [0.0031308, 1.055]), a tenth of
// the margin.  Most values skip powf entirely.
__device__ __forceinline__ float oetf_scaled(float x, int ref_oetf, bool exact) {
    const float b = ref_oetf ? __fmul_rn(1.055f, x) : x;
    const float p = exact ? powf(b, 1.0f / 2.4f) : __powf(b, 1.0f / 2.4f);
    const float v = ref_oetf ? __fsub_rn(p, 0.055f) : __fsub_rn(__fmul_rn(1.055f, p), 0.055f);
    return __fadd_rn(__fmul_rn(v, 255.0f), 0.5f);
}

__device__ __forceinline__ unsigned char to_srgb8(float x, int ref_oetf) {
    if (x > 1.0f) x = 1.0f;
    if (x < 0.0f) x = 0.0f;
    if (x != x) x = 0.0f;
    if (x <= 0.0031308f) return (unsigned char)__fadd_rn(__fmul_rn(__fmul_rn(12.92f, x), 255.0f), 0.5f);
    float t = oetf_scaled(x, ref_oetf, false);
    const float fr = t - floorf(t);
    if (fr < 0x1p-10f || fr > 1.0f - 0x1p-10f) t = oetf_scaled(x, ref_oetf, true);
    return (unsigned char)t;
}

struct TmParams {
    int type;
    float coeff;
    float m2;      // Reinhard (maxLw * coeff)^2
    float white;   // Uncharted2 curve at LinearWhite
    int ref_oetf;
};

__device__ __forceinline__ float tm_curve(float v, const TmParams& p) {
    const float x = __fmul_rn(v, p.coeff);
    if (p.type == SALTY_TM_ACES) return aces_curve(x);
    if (p.type == SALTY_TM_UNCHARTED2) return __fdiv_rn(u2_curve(__fmul_rn(2.0f, x)), p.white);
    // L * (1 + L / maxLw2) / (1 + L)  (src/s3d_tonemapper.cpp:256-268)
    return __fdiv_rn(__fmul_rn(x, __fadd_rn(1.0f, __fdiv_rn(x, p.m2))), __fadd_rn(1.0f, x));
}

__device__ __forceinline__ void map_value(const float* in, long long i, const TmParams& p, float* out,
                                          unsigned char* srgb) {
    const float y = tm_curve(in[i], p);
    if (out) out[i] = y;
    if (srgb) srgb[i] = to_srgb8(y, p.ref_oetf);
}

__global__ void k_tonemap_params(const float* in, long long n, const TmParams* pp, float* out, unsigned char* srgb) {
    cudaGridDependencySynchronize();
    const TmParams p = *pp;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        map_value(in, i, p, out, srgb);
}

// The same map, four pixels (twelve values) per step: three 16-byte loads and stores and
// three 4-byte sRGB8 words, and the values past the last whole group one by one.  in/out 16-byte
// aligned, srgb 4-byte aligned.  Launched over the reduction before it, it waits for the
// parameters with its first pixels loaded.
// Bound: issue (three divisions, the power and the clamps of each value).
__global__ void __launch_bounds__(256) k_tonemap_params4(const float* rgb, long long n, const TmParams* pp, float* out,
                                                         unsigned char* srgb) {
    const float4* in = reinterpret_cast<const float4*>(rgb);
    float4* o4 = reinterpret_cast<float4*>(out);
    uint32_t* s4 = reinterpret_cast<uint32_t*>(srgb);
    const long long groups = n / 12, step = (long long)gridDim.x * blockDim.x;
    const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    float4 q[3] = {};
    if (t0 < groups) q[0] = in[3 * t0], q[1] = in[3 * t0 + 1], q[2] = in[3 * t0 + 2];
    cudaGridDependencySynchronize();
    const TmParams p = *pp;
    for (long long g = t0; g < groups; g += step) {
        if (g != t0) q[0] = in[3 * g], q[1] = in[3 * g + 1], q[2] = in[3 * g + 2];
        float* v = reinterpret_cast<float*>(q);
#pragma unroll
        for (int k = 0; k < 12; ++k) v[k] = tm_curve(v[k], p);
        if (out) {
            o4[3 * g] = q[0];
            o4[3 * g + 1] = q[1];
            o4[3 * g + 2] = q[2];
        }
        if (srgb) {
#pragma unroll
            for (int w = 0; w < 3; ++w)
                s4[3 * g + w] = (uint32_t)to_srgb8(v[4 * w], p.ref_oetf) |
                                ((uint32_t)to_srgb8(v[4 * w + 1], p.ref_oetf) << 8) |
                                ((uint32_t)to_srgb8(v[4 * w + 2], p.ref_oetf) << 16) |
                                ((uint32_t)to_srgb8(v[4 * w + 3], p.ref_oetf) << 24);
        }
    }
    if (t0 < n - 12 * groups) map_value(rgb, 12 * groups + t0, p, out, srgb);
}

bool aligned_to(const void* p, uintptr_t a) { return p == nullptr || reinterpret_cast<uintptr_t>(p) % a == 0; }

// Maps the whole image: groups of four pixels where the arrays' alignment allows it, else value
// by value.  early: the launch may begin while the reduction that writes *pp still runs.
cudaError_t launch_tonemap(const salty_ctx* ctx, cudaStream_t st, const float* rgb, long long npx, const TmParams* pp,
                           float* out, uint8_t* srgb, bool early) {
    const bool vec = aligned_to(rgb, 16) && aligned_to(out, 16) && aligned_to(srgb, 4);
    const long long n = npx * 3, work = vec ? (npx + 3) / 4 : n;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)std::min((work + 255) / 256, (long long)ctx->num_sms * 14));
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, vec ? k_tonemap_params4 : k_tonemap_params, rgb, n, pp, out, srgb);
}

// log(eps + Lw) of one pixel, with the reference's guards, and the running maximum of Lw.
__device__ __forceinline__ float lum_log(float r, float g, float b, float& mx) {
    const float eps = 0.00001f;
    float lw = rgb_to_y(r, g, b);
    if (lw != lw) lw = eps;
    if (lw < FLT_EPSILON) lw = eps;
    mx = fmaxf(mx, lw);
    return logf(__fadd_rn(eps, lw));
}

// The block's (s, mx) in its first thread: shuffles, then the warps' values in order.
__device__ __forceinline__ void block_lum(double& s, float& mx) {
    for (int off = 16; off > 0; off >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, off);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    }
    __shared__ double ss[kRedBlock / 32];
    __shared__ float sm[kRedBlock / 32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) { ss[w] = s; sm[w] = mx; }
    __syncthreads();
    if (threadIdx.x == 0) {
        s = 0.0;
        mx = -FLT_MAX;
        for (int k = 0; k < kRedBlock / 32; ++k) { s += ss[k]; mx = fmaxf(mx, sm[k]); }
    }
}

// What the luminance reduction leaves: for the host (pinned), and the map's parameters.
struct LumResult {
    double sum;
    float max_lw, coeff;
};
struct LumScratch {
    unsigned ticket;  // zero between calls
    TmParams params;
    LumAcc part[1];   // one per block
};

// Log-average and maximum luminance, and the map's parameters from them: a partial per block, and
// the block that finishes last adds them in index order, so one launch does it and the sum does
// not depend on the order of the blocks.  rgb 16-byte aligned (vec): four pixels per step.  A
// thread's logarithms are added as an unevaluated FP32 pair (Knuth's TwoSum, 48 bits), since FP64
// runs at a 64th of the rate; pairs meet in FP64.  A thread adds 18 terms at 1080p and 72 at 4K,
// which a pair holds without any error (FP32 logarithms of images; 2,300 terms at 16,384^2: 1e-9
// of the FP32 mean's rounding).  The average is exp of the FP32 mean; taken in
// FP64 and rounded it is nearly always the host's expf (the caller compares).
// Bound: the logarithms' and additions' issue and the latency of a handful of loads.
__device__ __forceinline__ void two_sum(float& hi, float& lo, float x) {
    const float t = __fadd_rn(hi, x), z = __fsub_rn(t, hi);
    lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(t, z)), __fsub_rn(x, z)));
    hi = t;
}

__global__ void __launch_bounds__(kRedBlock) k_lum(const float* __restrict__ rgb, long long npx, int vec, TmParams p,
                                                   LumScratch* sc, LumResult* host) {
    cudaTriggerProgrammaticLaunchCompletion();  // every block runs by then: the map's may come in
    float mx = -FLT_MAX, hi = 0.0f, lo = 0.0f;
    const long long t0 = blockIdx.x * (long long)kRedBlock + threadIdx.x, nt = (long long)gridDim.x * kRedBlock;
    long long i0 = 0;
    if (vec) {
        const float4* q = reinterpret_cast<const float4*>(rgb);
        for (long long g = t0; g < npx / 4; g += nt) {
            const float4 a = __ldg(q + 3 * g), b = __ldg(q + 3 * g + 1), c = __ldg(q + 3 * g + 2);
            two_sum(hi, lo, lum_log(a.x, a.y, a.z, mx));
            two_sum(hi, lo, lum_log(a.w, b.x, b.y, mx));
            two_sum(hi, lo, lum_log(b.z, b.w, c.x, mx));
            two_sum(hi, lo, lum_log(c.y, c.z, c.w, mx));
        }
        i0 = npx / 4 * 4;
    }
    for (long long i = i0 + t0; i < npx; i += nt) two_sum(hi, lo, lum_log(rgb[3 * i], rgb[3 * i + 1], rgb[3 * i + 2], mx));
    double s = mx < INFINITY ? (double)hi + (double)lo : (double)INFINITY;
    block_lum(s, mx);
    __shared__ bool last;
    if (threadIdx.x == 0) {
        sc->part[blockIdx.x] = LumAcc{s, f2o(mx), 0};
        __threadfence();
        last = atomicAdd(&sc->ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    s = 0.0;
    mx = -FLT_MAX;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += kRedBlock) {
        s += __ldcg(&sc->part[i].sum);
        mx = fmaxf(mx, o2f(__ldcg(&sc->part[i].maxo)));
    }
    block_lum(s, mx);
    if (threadIdx.x != 0) return;
    sc->ticket = 0;
    const float ave = (float)exp((double)(float)(s / (double)npx));
    p.coeff = __fdiv_rn(p.coeff, ave);
    const float m2 = __fmul_rn(mx, p.coeff);
    p.m2 = __fmul_rn(m2, m2);
    sc->params = p;
    *host = LumResult{s, mx, p.coeff};
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// ---------------------------------------------------------------- NLM by column walks
// Both NLM filters weigh a pixel's neighbours by patch distances that are (2P+1)^2 box sums
// of a per-pixel term, so for one search offset the terms are computed once and summed
// separably.  One warp owns a tile of 32 - 2P columns (one lane per column, P more on either
// side for the patch) and kNlmRows rows, and walks its columns downwards: the vertical sums
// come from the lane's own last terms, the horizontal ones from shuffles, and the centre
// pixels and the accumulators stay in registers for the whole search, so a step loads only
// the neighbour pixel from the staged tile.  The block's warps share the tile and take the
// search offsets in turn (their accumulators are added at the end, in warp order), which
// gives small images four times as many warps as tiles.  Nothing is clamped in the walk: the
// staged tile holds the border-clamped pixels.  A tile of r rows costs 1 + 2P/r of the terms of an
// ideal walk; 16 (kNlmRows) keep the reference filter's centre and accumulators within 255
// registers (8 warps per SM), and 12 (kVarRows) leave the variance-scaled one's room to load
// ahead (1080p, radius 3: 16 rows 2.71 ms, 13 2.49, 12 2.39-2.45, 11 2.64, 10 2.58, 8 2.74, 8 at three
// blocks per SM 2.82).
// Bound: instruction issue and the latency that 2 warps per scheduler leave (packed FP32
// operations 20 % slower, one reciprocal for three quotients 2 % faster and not kept).
// Measured (GB300), against one thread per pixel with the terms and row sums in shared memory
// (variance-scaled) or all 25 taps per offset (reference): 1920 x 1080, 21 x 21 search, 7 x 7
// patch 10.25 -> 2.42 ms; 1279 x 719 FilterNLM 3.26 -> 0.27 ms.
constexpr int kNlmRows = 16;
constexpr int kVarRows = 12;
constexpr int kNlmWarps = 4;

// Sum of the 2P+1 terms v - 2P .. v of one column, from the sums of shorter runs.
template <int P, int N>
struct ColumnSums {
    float d[N], s2[N], s3[N], s4[N];
    __device__ __forceinline__ float push(int v, float x) {
        d[v] = x;
        if (v >= 1) s2[v] = x + d[v - 1];
        if (P == 3 && v >= 2) s3[v] = s2[v] + d[v - 2];
        if (P >= 2 && v >= 3) s4[v] = s2[v] + s2[v - 2];
        if (P == 1) return v >= 2 ? s2[v] + d[v - 2] : 0.0f;
        if (P == 2) return v >= 4 ? s4[v] + d[v - 4] : 0.0f;
        return v >= 6 ? s4[v] + s3[v - 4] : 0.0f;
    }
};

// x / y by the hardware reciprocal (1 ulp) and a product, for y >= 1e-10: the compiler's own
// approximate division would also rescale denormal divisors, which cannot occur here.
__device__ __forceinline__ float quick_div(float x, float y) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
    return x * r;
}
// 2^x for x <= 0 by the hardware exponential (2 ulp); results below 2^-126 are zero, against a
// sum of weights of at least 1 (the pixel's own).
__device__ __forceinline__ float quick_exp2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
constexpr float kLog2e = 1.4426950408889634f;

// Sum over the lanes l - P .. l + P (meaningless in the outer P lanes of either side).
template <int P>
__device__ __forceinline__ float lane_sum(float v) {
    constexpr unsigned m = 0xffffffffu;
    const float r1 = __shfl_down_sync(m, v, 1);
    if (P == 1) return __shfl_up_sync(m, v, 1) + v + r1;
    const float a = v + r1;  // l, l + 1
    if (P == 2) return __shfl_up_sync(m, a, 2) + a + __shfl_down_sync(m, v, 2);
    const float b = a + __shfl_down_sync(m, a, 2);  // l .. l + 3
    return __shfl_up_sync(m, a, 2) + b + __shfl_up_sync(m, v, 3);
}

// Adds the warps' accumulators acc[kNlmRows][C] in warp order into warp 0's, through shared
// memory (C * 32 floats per row; the staged tile is dead by then).
template <int C, int ROWS>
__device__ __forceinline__ void add_warps(float (&acc)[ROWS][C], float* sm, int warp, int lane, int warps) {
    for (int k = 1; k < warps; ++k) {
        __syncthreads();
        if (warp == k) {
#pragma unroll
            for (int y = 0; y < ROWS; ++y)
#pragma unroll
                for (int c = 0; c < C; ++c) sm[(y * C + c) * 32 + lane] = acc[y][c];
        }
        __syncthreads();
        if (warp == 0) {
#pragma unroll
            for (int y = 0; y < ROWS; ++y)
#pragma unroll
                for (int c = 0; c < C; ++c) acc[y][c] += sm[(y * C + c) * 32 + lane];
        }
    }
}

// ---------------------------------------------------------------- NLM (reference)
// FilterNLM's 13x13 search and 5x5 patch.  The reference adds the 25 squared differences of
// a patch one by one; here they are shared between the patches that overlap.
constexpr int kRefR = 6, kRefP = 2;

__global__ void __launch_bounds__(32 * kNlmWarps, 2) k_nlm_ref(const float4* __restrict__ src, int w, int h, float inv_h2,
                                                               float two_s2, float4* __restrict__ dst) {
    constexpr int P = kRefP, R = kRefR, N = kNlmRows + 2 * P, S = 32 + 2 * R, SR = N + 2 * R;
    __shared__ float4 tile[SR * S];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int bx = blockIdx.x * (32 - 2 * P), by = blockIdx.y * kNlmRows;
    for (int i = threadIdx.x; i < SR * S; i += 32 * kNlmWarps)
        tile[i] = __ldg(src + (size_t)clampi(by - P - R + i / S, 0, h - 1) * w + clampi(bx - P - R + i % S, 0, w - 1));
    __syncthreads();
    float4 a[N];
#pragma unroll
    for (int v = 0; v < N; ++v) a[v] = tile[(v + R) * S + lane + R];
    float acc[kNlmRows][5];
#pragma unroll
    for (int y = 0; y < kNlmRows; ++y)
#pragma unroll
        for (int c = 0; c < 5; ++c) acc[y][c] = 0.0f;
#pragma unroll 1
    for (int o = warp; o < (2 * R + 1) * (2 * R + 1); o += kNlmWarps) {
        const float4* q = tile + (o / (2 * R + 1)) * S + lane + o % (2 * R + 1);
        ColumnSums<P, N> cs;
        float4 b[N];
#pragma unroll
        for (int v = 0; v < N; ++v) {
            b[v] = q[v * S];
            const float d0 = a[v].x - b[v].x, d1 = a[v].y - b[v].y, d2 = a[v].z - b[v].z, d3 = a[v].w - b[v].w;
            const float col = cs.push(v, fmaf(d3, d3, d2 * d2) + fmaf(d1, d1, d0 * d0));
            if (v < 2 * P) continue;
            const float sum = lane_sum<P>(col);
            const float wt = quick_exp2(-fmaxf(sum - two_s2, 0.0f) * (inv_h2 * kLog2e));
            const float4 c = b[v - P];
            float(&A)[5] = acc[v - 2 * P];
            A[0] = fmaf(c.x, wt, A[0]);
            A[1] = fmaf(c.y, wt, A[1]);
            A[2] = fmaf(c.z, wt, A[2]);
            A[3] = fmaf(c.w, wt, A[3]);
            A[4] += wt;
        }
    }
    add_warps(acc, reinterpret_cast<float*>(tile), warp, lane, kNlmWarps);
    const int x = bx + lane - P;
    if (warp != 0 || lane < P || lane >= 32 - P || x >= w) return;
#pragma unroll
    for (int y = 0; y < kNlmRows; ++y)
        if (by + y < h)
            dst[(size_t)(by + y) * w + x] = make_float4(__fdiv_rn(acc[y][0], acc[y][4]), __fdiv_rn(acc[y][1], acc[y][4]),
                                                        __fdiv_rn(acc[y][2], acc[y][4]), __fdiv_rn(acc[y][3], acc[y][4]));
}

// ---------------------------------------------------------------- NLM (variance scaled)
// Rousselle, Knaus, Zwicker, "Adaptive rendering with non-local means filtering"
// (SIGGRAPH Asia 2012): patch distance normalised by the pixels' variances.
//
// Separable form: for one search offset (dx, dy) the patch distance of every pixel is a
// (2P+1)^2 box sum of the per-pixel term
//   D(x) = sum_c [(I_c(x) - I_c(x+d))^2 - (V_c(x) + min(V_c(x), V_c(x+d)))] / (eps + k^2 (V_c(x) + V_c(x+d)))
// (each coordinate clamped to the image), so a CTA computes D once over its tile plus the
// patch border, sums it along rows and then columns in shared memory, and every pixel reads
// its distance: O(1) work per pixel and offset instead of O(patch).  The same sums as the
// direct double loop in a different order, with quotients within 2 ulp.  Patch radii 1..3 run
// as column walks (k_nlm_var_cols, 4.2x faster at radius 3); k_nlm_var keeps the others, whose
// centre pixels would not fit the registers (radius >= 4) or need no box sum (radius 0), and
// the search of one pixel (radius 0; 640 x 480 27 us against 36 by column walks, radius 1 54
// against 46), where three of a walk's four warps would find no offset.
constexpr int kVTile = 16;

__global__ void __launch_bounds__(kVTile* kVTile) k_nlm_var(const float* __restrict__ rgb, const float* __restrict__ var,
                                                            int w, int h, int R, int P, float k2, float norm,
                                                            float* __restrict__ out) {
    extern __shared__ float sm[];
    const int H = R + P;
    const int S = kVTile + 2 * H;   // staged halo side
    const int E = kVTile + 2 * P;   // tile plus patch border
    float* tc = sm;                 // S*S*3 colours
    float* tv = tc + S * S * 3;     // S*S*3 variances
    float* dd = tv + S * S * 3;     // E*E per-pixel terms D
    float* hs = dd + E * E;         // E rows x kVTile columns of row sums
    const int tid = threadIdx.y * kVTile + threadIdx.x, nt = kVTile * kVTile;
    const int bx = blockIdx.x * kVTile, by = blockIdx.y * kVTile;
    const int x0 = bx - H, y0 = by - H;
    for (int i = tid; i < S * S; i += nt) {
        const int ty = i / S, tx = i % S;
        const size_t g = ((size_t)clampi(y0 + ty, 0, h - 1) * w + clampi(x0 + tx, 0, w - 1)) * 3;
        for (int c = 0; c < 3; ++c) {
            tc[i * 3 + c] = rgb[g + c];
            tv[i * 3 + c] = var[g + c];
        }
    }
    __syncthreads();
    const int x = bx + threadIdx.x, y = by + threadIdx.y;
    const float eps = 1e-10f;
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, sw = 0.f;
    for (int dy = -R; dy <= R; ++dy) {
        for (int dx = -R; dx <= R; ++dx) {
            // D over the tile plus its patch border (image coordinates bx - P .. bx + kVTile + P)
            for (int i = tid; i < E * E; i += nt) {
                const int u = i % E, v = i / E;
                const int ax = clampi(bx - P + u, 0, w - 1), ay = clampi(by - P + v, 0, h - 1);
                const int qx = clampi(bx - P + u + dx, 0, w - 1), qy = clampi(by - P + v + dy, 0, h - 1);
                const int ia = ((ay - y0) * S + (ax - x0)) * 3, ib = ((qy - y0) * S + (qx - x0)) * 3;
                float d = 0.0f;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const float a = tc[ia + c], b = tc[ib + c], va = tv[ia + c], vb = tv[ib + c];
                    const float num = (a - b) * (a - b) - (va + fminf(va, vb));
                    d += __fdividef(num, eps + k2 * (va + vb));  // 2-ulp division: the weights need no IEEE quotient
                }
                dd[i] = d;
            }
            __syncthreads();
            // row sums over the patch width
            for (int i = tid; i < E * kVTile; i += nt) {
                const int u = i % kVTile, v = i / kVTile;
                const float* r = dd + v * E + u;
                float t = 0.0f;
                for (int k = 0; k <= 2 * P; ++k) t += r[k];
                hs[i] = t;
            }
            __syncthreads();
            // column sum over the patch height: this pixel's patch distance
            float d2 = 0.0f;
            for (int k = 0; k <= 2 * P; ++k) d2 += hs[(threadIdx.y + k) * kVTile + threadIdx.x];
            const float wt = expf(-fmaxf(0.0f, d2 * norm));
            const int iq = ((clampi(y + dy, 0, h - 1) - y0) * S + (clampi(x + dx, 0, w - 1) - x0)) * 3;
            sw += wt;
            s0 += wt * tc[iq];
            s1 += wt * tc[iq + 1];
            s2 += wt * tc[iq + 2];
        }
    }
    if (x >= w || y >= h) return;
    const size_t o = ((size_t)y * w + x) * 3;
    out[o] = s0 / sw;
    out[o + 1] = s1 / sw;
    out[o + 2] = s2 / sw;
}

// The same filter by column walks, for patch radii up to 3 (centre pixels and variances of
// ROWS + 2P rows in registers).  RM: largest search radius, the staged tile's column pitch
// is fixed by it.
template <int P, int RM, int ROWS>
__global__ void __launch_bounds__(32 * kNlmWarps, 2)
k_nlm_var_cols(const float* __restrict__ rgb, const float* __restrict__ var, int w, int h, int R, float k2, float norm,
               float* __restrict__ out) {
    constexpr int N = ROWS + 2 * P, S = 32 + 2 * RM;
    extern __shared__ __align__(16) float sm[];
    const int rows = N + 2 * R, cols = 32 + 2 * R;
    float2* t0 = reinterpret_cast<float2*>(sm);  // (r, g), (b, var r), (var g, var b)
    float2* t1 = t0 + rows * S;
    float2* t2 = t1 + rows * S;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // blocks in one dimension: the second has room for 65,535 only
    const int tiles_x = (w + 31 - 2 * P) / (32 - 2 * P);
    const int bx = (int)(blockIdx.x % tiles_x) * (32 - 2 * P), by = (int)(blockIdx.x / tiles_x) * ROWS;
    for (int i = threadIdx.x; i < rows * cols; i += 32 * kNlmWarps) {
        const int ty = i / cols, tx = i - ty * cols;
        const size_t g = ((size_t)clampi(by - P - R + ty, 0, h - 1) * w + clampi(bx - P - R + tx, 0, w - 1)) * 3;
        const int o = ty * S + tx;
        t0[o] = make_float2(__ldg(rgb + g), __ldg(rgb + g + 1));
        t1[o] = make_float2(__ldg(rgb + g + 2), __ldg(var + g));
        t2[o] = make_float2(__ldg(var + g + 1), __ldg(var + g + 2));
    }
    __syncthreads();
    const float eps = 1e-10f;
    float a[N][3], va[N][3];
#pragma unroll
    for (int v = 0; v < N; ++v) {
        const int o = (v + R) * S + lane + R;
        const float2 p0 = t0[o], p1 = t1[o], p2 = t2[o];
        a[v][0] = p0.x; a[v][1] = p0.y; a[v][2] = p1.x;
        va[v][0] = p1.y; va[v][1] = p2.x; va[v][2] = p2.y;
    }
    float acc[ROWS][4];
#pragma unroll
    for (int y = 0; y < ROWS; ++y)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[y][c] = 0.0f;
    const int side = 2 * R + 1;
#pragma unroll 1
    for (int o = warp; o < side * side; o += kNlmWarps) {
        const int q = (o / side) * S + lane + o % side;
        ColumnSums<P, N> cs;
        float b[N][3];
#pragma unroll
        for (int v = 0; v < N; ++v) {
            const float2 p0 = t0[q + v * S], p1 = t1[q + v * S], p2 = t2[q + v * S];
            b[v][0] = p0.x; b[v][1] = p0.y; b[v][2] = p1.x;
            const float vb[3] = {p1.y, p2.x, p2.y};
            float d = 0.0f;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float t = a[v][c] - b[v][c];
                const float num = t * t - (va[v][c] + fminf(va[v][c], vb[c]));
                d += quick_div(num, eps + k2 * (va[v][c] + vb[c]));
            }
            const float col = cs.push(v, d);
            if (v < 2 * P) continue;
            const float wt = quick_exp2(-fmaxf(0.0f, lane_sum<P>(col) * (norm * kLog2e)));
            float(&A)[4] = acc[v - 2 * P];
#pragma unroll
            for (int c = 0; c < 3; ++c) A[c] = fmaf(wt, b[v - P][c], A[c]);
            A[3] += wt;
        }
    }
    add_warps(acc, sm, warp, lane, kNlmWarps);
    const int x = bx + lane - P;
    if (warp != 0 || lane < P || lane >= 32 - P || x >= w) return;
#pragma unroll
    for (int y = 0; y < ROWS; ++y)
        if (by + y < h) {
            const size_t o = ((size_t)(by + y) * w + x) * 3;
#pragma unroll
            for (int c = 0; c < 3; ++c) out[o + c] = acc[y][c] / acc[y][3];
        }
}

template <int P, int RM, int ROWS>
salty_status launch_nlm_var_cols(salty_ctx* ctx, int w, int h, int R, float k2, float norm, const float* rgb,
                                 const float* var, float* out) {
    const long long tiles = (long long)((w + 31 - 2 * P) / (32 - 2 * P)) * ((h + ROWS - 1) / ROWS);
    // fewer tiles than SMs: shorter ones, more of them (200 x 150, radius 3: 89 -> 72 us)
    if (ROWS > 8 && tiles <= ctx->num_sms)
        return launch_nlm_var_cols<P, RM, 8>(ctx, w, h, R, k2, norm, rgb, var, out);
    const size_t tile = (size_t)(ROWS + 2 * P + 2 * R) * (32 + 2 * RM) * 3 * sizeof(float2);
    const size_t smem = std::max(tile, (size_t)ROWS * 4 * 32 * sizeof(float));
    auto kern = k_nlm_var_cols<P, RM, ROWS>;
    SALTY_TRY_CUDA(ctx->err, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<(unsigned)tiles, 32 * kNlmWarps, smem, ctx->stream>>>(rgb, var, w, h, R, k2, norm, out);
    SALTY_TRY_CUDA(ctx->err, cudaGetLastError());
    return SALTY_OK;
}

}  // namespace

// Blocks of the luminance reduction: more cost more in tickets than they hide (8 per SM: 2 us).
static int lum_blocks(const salty_ctx* ctx) { return ctx->num_sms * 3; }

// The reduction's scratch (19 KB), made with the context so that no tonemap allocates it.
salty_status tonemap_prepare(salty_ctx* ctx) {
    const size_t bytes = sizeof(LumScratch) + (size_t)lum_blocks(ctx) * sizeof(LumAcc);
    SALTY_TRY_CUDA(ctx->err, ctx->lum_ws.ensure(bytes));
    SALTY_TRY_CUDA(ctx->err, cudaMemsetAsync(ctx->lum_ws.p, 0, bytes, ctx->stream));
    return SALTY_OK;
}

// One round trip: the reduction derives the map's parameters on the device, the map follows
// without waiting, and the host then checks the one value that its own arithmetic defines, the
// exponential of the mean (expf).  Where the device's differs in the last place, or where an
// output overlaps the input, the map runs (again) with the host's.  Measured (GB300, ACES, device
// arrays), against two round trips with scalar loads, an initialising copy and FP64 atomics:
// 1920 x 1080 70 -> 47 us, 640 x 480 48 -> 28 us.
salty_status tonemap_device(salty_ctx* ctx, int type, int w, int h, const float* d_rgb, float* d_out,
                            uint8_t* d_srgb, int ref_oetf, float* ave, float* mx) {
    auto& E = ctx->err;
    cudaStream_t st = ctx->stream;
    const long long npx = (long long)w * h;
    LumScratch* sc = reinterpret_cast<LumScratch*>(ctx->lum_ws.p);
    LumResult* res = static_cast<LumResult*>(ctx->pinned);
    TmParams p{};
    p.type = type;
    p.ref_oetf = ref_oetf;
    p.coeff = type == SALTY_TM_ACES ? 0.27f : 0.18f;
    {
        // Uncharted2Tonemap(LinearWhite = 11.2), host evaluation in the same order
        const float A = 0.15f, B = 0.50f, C = 0.10f, D = 0.20f, Ee = 0.01f, F = 0.30f, x = 11.2f;
        float num = x * (A * x + C * B) + D * Ee;
        float den = x * (A * x + B) + D * F;
        p.white = num / den - Ee / F;
    }
    const bool vec = aligned_to(d_rgb, 16);
    const long long need = ((vec ? (npx + 3) / 4 : npx) + kRedBlock - 1) / kRedBlock;
    k_lum<<<(unsigned)std::min<long long>(lum_blocks(ctx), need), kRedBlock, 0, st>>>(d_rgb, npx, vec, p, sc, res);
    auto apart = [&](const void* q, size_t len) {
        const auto a = reinterpret_cast<uintptr_t>(d_rgb), b = reinterpret_cast<uintptr_t>(q);
        return !q || b >= a + (size_t)npx * 12 || b + len <= a;
    };
    const bool ahead = apart(d_out, (size_t)npx * 12) && apart(d_srgb, (size_t)npx * 3);
    SALTY_TRY_CUDA(E, cudaGetLastError());
    if ((d_out || d_srgb) && ahead)
        SALTY_TRY_CUDA(E, launch_tonemap(ctx, st, d_rgb, npx, &sc->params, d_out, d_srgb, true));
    SALTY_TRY_CUDA(E, cudaStreamSynchronize(st));
    // ComputeLogarithmicAverage (src/s3d_tonemapper.cpp:84-94)
    const float ave_lw = expf((float)(res->sum / (double)npx));
    if (ave) *ave = ave_lw;
    if (mx) *mx = res->max_lw;
    const float dev_coeff = res->coeff;
    p.coeff /= ave_lw;
    const float m2 = res->max_lw * p.coeff;
    p.m2 = m2 * m2;
    if ((d_out || d_srgb) && !(ahead && std::memcmp(&dev_coeff, &p.coeff, 4) == 0)) {
        SALTY_TRY_CUDA(E, cudaMemcpyAsync(&sc->params, &p, sizeof p, cudaMemcpyHostToDevice, st));
        SALTY_TRY_CUDA(E, launch_tonemap(ctx, st, d_rgb, npx, &sc->params, d_out, d_srgb, false));
    }
    return SALTY_OK;
}

salty_status nlm_ref_device(salty_ctx* ctx, int w, int h, float coeff, const float* d_in, float* d_out) {
    // FilterNLM parameters (src/s3d_denoiser.cpp:22-25)
    float ph = fmaxf(0.0001f, coeff), sigma = fmaxf(0.0001f, coeff);
    float inv_h2 = 1.0f / (ph * ph);
    float two_s2 = 2.0f * (sigma * sigma);
    constexpr int cols = 32 - 2 * kRefP;
    const dim3 grd((w + cols - 1) / cols, (h + kNlmRows - 1) / kNlmRows);
    k_nlm_ref<<<grd, 32 * kNlmWarps, 0, ctx->stream>>>((const float4*)d_in, w, h, inv_h2, two_s2, (float4*)d_out);
    SALTY_TRY_CUDA(ctx->err, cudaGetLastError());
    return SALTY_OK;
}

salty_status nlm_var_device(salty_ctx* ctx, int w, int h, int search_r, int patch_r, float k, const float* d_rgb,
                            const float* d_var, float* d_out) {
    const float norm = 1.0f / (3.0f * (float)((2 * patch_r + 1) * (2 * patch_r + 1)));
#define SALTY_NLM(P)                                                                                       \
    if (patch_r == P && search_r > 0)                                                                      \
        return search_r <= 10 ? launch_nlm_var_cols<P, 10, kVarRows>(ctx, w, h, search_r, k * k, norm, d_rgb, d_var, d_out) \
                              : launch_nlm_var_cols<P, 32, kVarRows>(ctx, w, h, search_r, k * k, norm, d_rgb, d_var, d_out)
    SALTY_NLM(1);
    SALTY_NLM(2);
    SALTY_NLM(3);
#undef SALTY_NLM
    const int H = search_r + patch_r, S = kVTile + 2 * H, Eb = kVTile + 2 * patch_r;
    size_t smem = ((size_t)S * S * 6 + (size_t)Eb * Eb + (size_t)Eb * kVTile) * sizeof(float);
    if (smem > 200 * 1024) return ctx->err.fail(SALTY_ERR_CAPACITY, "NLM window too large");
    SALTY_TRY_CUDA(ctx->err, cudaFuncSetAttribute(k_nlm_var, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 blk(kVTile, kVTile), grd((w + kVTile - 1) / kVTile, (h + kVTile - 1) / kVTile);
    k_nlm_var<<<grd, blk, smem, ctx->stream>>>(d_rgb, d_var, w, h, search_r, patch_r, k * k, norm, d_out);
    SALTY_TRY_CUDA(ctx->err, cudaGetLastError());
    return SALTY_OK;
}

}  // namespace salty

// ---------------------------------------------------------------- no-allocation tonemap
// salty_tonemap_noalloc: the same tonemap for callers that must not allocate device memory
// when they tonemap (see include/salty_gpu.h).  Its scratch is the fixed array below,
// part of the library image, so it exists on every device that loads the library until
// the process exits.  Layout: kNoAllocPartials partial sums (one per block of
// kNoAllocPixelsPerBlock pixels), then the tonemap parameters.  Every call overwrites what
// it reads, so nothing has to be cleared between calls; calls that overlap on the GPU share
// the array and race.
namespace salty {
namespace {

constexpr int kNoAllocPartials = 4096;
constexpr int kNoAllocPixelsPerBlock = 4096;
constexpr long long kNoAllocMaxPixels = (long long)kNoAllocPartials * kNoAllocPixelsPerBlock;

struct NoAllocScratch {
    LumAcc part[kNoAllocPartials];
    TmParams params;
    float ave_max[2];
};

static __device__ __align__(256) unsigned char g_noalloc_scratch[sizeof(NoAllocScratch)];

// Per-block luminance partials in a fixed pixel-to-block mapping (deterministic).
// vec: rgb is 16-byte aligned -- four pixels (three float4) per load step, their four logs
// summed in FP32 before the FP64 running sum (a quarter of the FP64 additions).
__global__ void __launch_bounds__(kRedBlock) k_lum_partials(const float* __restrict__ rgb, long long npx,
                                                            NoAllocScratch* sc, int vec) {
    const long long b0 = (long long)blockIdx.x * kNoAllocPixelsPerBlock;
    const long long b1 = min(npx, b0 + kNoAllocPixelsPerBlock);
    double s = 0.0;
    float mx = -FLT_MAX;
    long long i0 = b0;
    if (vec) {
        const float4* q = reinterpret_cast<const float4*>(rgb);
        const long long ge = b1 / 4;  // b0 is a multiple of 4
        for (long long gi = b0 / 4 + threadIdx.x; gi < ge; gi += blockDim.x) {
            const float4 a = __ldg(q + 3 * gi), b = __ldg(q + 3 * gi + 1), c = __ldg(q + 3 * gi + 2);
            const float l4 = lum_log(a.x, a.y, a.z, mx) + lum_log(a.w, b.x, b.y, mx) + lum_log(b.z, b.w, c.x, mx) +
                             lum_log(c.y, c.z, c.w, mx);
            s += (double)l4;
        }
        i0 = ge * 4;
    }
    for (long long i = i0 + threadIdx.x; i < b1; i += blockDim.x)
        s += (double)lum_log(rgb[3 * i], rgb[3 * i + 1], rgb[3 * i + 2], mx);
    for (int off = 16; off > 0; off >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, off);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    }
    __shared__ double ss[kRedBlock / 32];
    __shared__ float sm[kRedBlock / 32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { ss[w] = s; sm[w] = mx; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        float m = -FLT_MAX;
        for (int k = 0; k < kRedBlock / 32; ++k) { t += ss[k]; m = fmaxf(m, sm[k]); }
        sc->part[blockIdx.x].sum = t;
        sc->part[blockIdx.x].maxo = f2o(m);
    }
}

// Reduces the partials in index order and derives the curve parameters on the device, so
// the three launches need no host round trip.  ComputeLogarithmicAverage and the
// per-operator constants: src/s3d_tonemapper.cpp:84-94, :246-250, :291-297, :331-335.
__global__ void __launch_bounds__(kRedBlock) k_lum_finalize(NoAllocScratch* sc, int nparts, long long npx, int type,
                                                            int ref_oetf) {
    double s = 0.0;
    float mx = -FLT_MAX;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
        s += sc->part[i].sum;
        mx = fmaxf(mx, o2f(sc->part[i].maxo));
    }
    __shared__ double ss[kRedBlock];
    __shared__ float sm[kRedBlock];
    ss[threadIdx.x] = s;
    sm[threadIdx.x] = mx;
    __syncthreads();
    for (int h = kRedBlock / 2; h > 0; h >>= 1) {
        if (threadIdx.x < h) {
            ss[threadIdx.x] += ss[threadIdx.x + h];
            sm[threadIdx.x] = fmaxf(sm[threadIdx.x], sm[threadIdx.x + h]);
        }
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    const float mean = (float)(ss[0] / (double)npx);
    const float ave = expf(mean);
    const float max_lw = sm[0];
    TmParams p;
    p.type = type;
    p.ref_oetf = ref_oetf;
    p.coeff = __fdiv_rn(type == SALTY_TM_ACES ? 0.27f : 0.18f, ave);
    const float m2 = __fmul_rn(max_lw, p.coeff);
    p.m2 = __fmul_rn(m2, m2);
    p.white = u2_curve(11.2f);
    sc->params = p;
    sc->ave_max[0] = ave;
    sc->ave_max[1] = max_lw;
}

// Device address of g_noalloc_scratch per device, looked up once per device with that
// device current (the array's name is only a host-side stand-in in host code).
constexpr int kMaxDevices = 64;
void* g_noalloc_addr[kMaxDevices] = {};

cudaError_t noalloc_scratch(int device, NoAllocScratch** out) {
    if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
    void* p = __atomic_load_n(&g_noalloc_addr[device], __ATOMIC_ACQUIRE);
    if (!p) {
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        __atomic_store_n(&g_noalloc_addr[device], p, __ATOMIC_RELEASE);
    }
    *out = static_cast<NoAllocScratch*>(p);
    return cudaSuccess;
}

// true for device memory of `device` itself, or managed memory; an array on another GPU
// would be read as peer memory (a fault without peer access), so it is refused
bool on_device(const void* p, int device) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (a.type == cudaMemoryTypeManaged) return true;
    return a.type == cudaMemoryTypeDevice && a.device == device;
}

}  // namespace
}  // namespace salty

extern "C" salty_status salty_tonemap_noalloc(salty_ctx* ctx, void* stream, int32_t type, int32_t width,
                                              int32_t height, const float* d_rgb, float* d_out_rgb,
                                              uint8_t* d_out_srgb8, int32_t ref_oetf) {
    using namespace salty;
    if (!ctx) return SALTY_ERR_INVALID_ARG;
    auto& E = ctx->err;
    if (width <= 0 || height <= 0) return E.fail(SALTY_ERR_INVALID_ARG, "tonemap_noalloc: bad image size");
    const long long npx = (long long)width * height;
    if (npx > kNoAllocMaxPixels)
        return E.fail(SALTY_ERR_CAPACITY, "tonemap_noalloc: %lld pixels exceed the fixed scratch limit of %lld",
                      npx, kNoAllocMaxPixels);
    if (type < SALTY_TM_REINHARD || type > SALTY_TM_ACES) return E.fail(SALTY_ERR_INVALID_ARG, "bad tonemap type");
    if (!d_out_rgb && !d_out_srgb8) return E.fail(SALTY_ERR_INVALID_ARG, "tonemap_noalloc: no output");
    SALTY_TRY_CUDA(E, cudaSetDevice(ctx->device));
    const int dv = ctx->device;
    if (!on_device(d_rgb, dv) || (d_out_rgb && !on_device(d_out_rgb, dv)) ||
        (d_out_srgb8 && !on_device(d_out_srgb8, dv)))
        return E.fail(SALTY_ERR_INVALID_ARG, "tonemap_noalloc: arrays must be device memory of the context's GPU");
    NoAllocScratch* sc = nullptr;
    SALTY_TRY_CUDA(E, noalloc_scratch(ctx->device, &sc));
    cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : ctx->stream;
    const int nparts = (int)((npx + kNoAllocPixelsPerBlock - 1) / kNoAllocPixelsPerBlock);
    k_lum_partials<<<nparts, kRedBlock, 0, st>>>(d_rgb, npx, sc, aligned_to(d_rgb, 16) ? 1 : 0);
    k_lum_finalize<<<1, kRedBlock, 0, st>>>(sc, nparts, npx, type, ref_oetf);
    SALTY_TRY_CUDA(E, cudaGetLastError());
    SALTY_TRY_CUDA(E, launch_tonemap(ctx, st, d_rgb, npx, &sc->params, d_out_rgb, d_out_srgb8, false));
    return SALTY_OK;
}
