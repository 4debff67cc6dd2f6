// unet.cu -- the learned denoiser: a 5-level U-Net trained and run by these kernels.
//
// The reference has an NLM filter (src/s3d_denoiser.cpp:19-95) and no learned denoiser;
// this network is new.  Input: 11 features per pixel (log(1 + colour), first-hit albedo,
// normal, 1/(1 + distance), the colour's noise level), padded to 16 channels.  Architecture (NHWC, BF16 activations):
//   enc: conv 16->32, 32->32 | pool | 32->48, 48->48 | pool | 48->64, 64->64 | pool |
//        64->80, 80->80 | pool | 80->96
//   dec: up + concat(96+80) -> 80 | up + concat(80+64) -> 64 | up + concat(64+48) -> 48 |
//        up + concat(48+32) -> 32 | conv 32->8 (channels 0..2: a correction r of the input's
//        log colour; the prediction is log(1 + colour) = x + r)
// every conv 3x3, stride 1, zero padding, ReLU except the last; 2x2 max-pool; nearest 2x
// up-sampling.  Loss: mean |x + r - log(1 + target)| (L1 in log space).  Optimiser: Adam.
//
// Convolutions are implicit GEMMs on the tensor cores (mma.sync m16n8k16, BF16 operands,
// FP32 accumulation):
//   forward       M = pixels, N = Cout, K = 9*Cin: a CTA stages an 8x16-pixel tile plus halo
//                 in shared memory; A fragments come from it, B fragments from the weights.
//   backward data the same kernel on dY with the weights flipped and transposed.
//   backward wts  M = Cout, N = Cin, K = pixels: ldmatrix.trans turns the NHWC tiles of dY and
//                 of the shifted input into fragments with pixels along K; a CTA covers all
//                 nine taps of a 16-channel input slice (one dY fragment serves nine taps),
//                 sums its pixel tiles in registers and adds the partial into FP32 gradients.
// All three convolutions run by default on tcgen05 (conv_tc.cu: TMEM accumulators; the
// forward and backward-data ones over 128-pixel strips staged by TMA in a persistent
// warp-specialised kernel, where the decoder's coarse level is expanded by warps of its own; the
// weight gradient over strips of 2 rows x 64 pixels with dY transposed as the MMA's A, the
// input's halo as B and the taps as descriptor offsets, summed over CTAs in a fixed order);
// the mma.sync kernels below stay selectable (salty_unet_set_conv_kernel) and are the
// reference the tcgen05 kernels are tested against.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "internal.h"
#include "unet_src.cuh"

namespace salty {
namespace {

using bf16 = __nv_bfloat16;

constexpr int kTileX = 16, kTileY = 8;          // output tile of one CTA
constexpr int kHaloX = kTileX + 2, kHaloY = kTileY + 2;
constexpr int kConvThreads = 128;
constexpr int kFeatures = 11;                   // input floats per pixel

__device__ __forceinline__ void mma_bf16(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ unsigned smem_addr(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void ldmatrix_x4_trans(unsigned (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_addr(p)));
}

// ---------------------------------------------------------------- conv3x3 (forward, backward data)
// in:  BF16 NHWC input channels 0..Cin-1 (Cin % 16 == 0) from one or two sources (ConvSrc)
// wt:  [9][wrows][Cin] BF16 (tap-major, input channel contiguous); output channel co reads row co
// out: [N][H][W][out_cs] BF16 at channel offset out_co (channels co < Cout written)
// NT n8-tiles per CTA; blockIdx.y selects output channels [blockIdx.y*NT*8, +NT*8).
// Shared memory: the 18x10-pixel halo tile, then one tap's weight slice [NT*8][Cin], both
// with rows padded by 8 halves so the 8 row addresses of an ldmatrix fall in distinct banks.
// Per 16-channel k-step a warp issues 2 ldmatrix.x4 for A (its two 16-pixel rows), NT/2
// ldmatrix.x4 for B and 2*NT mma.
__device__ __forceinline__ void ldmatrix_x4(unsigned (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_addr(p)));
}
__device__ __forceinline__ void ldmatrix_x2(unsigned& r0, unsigned& r1, const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(r0), "=r"(r1) : "r"(smem_addr(p)));
}

template <int NT>
__global__ void __launch_bounds__(kConvThreads) k_conv3x3(const ConvSrc in, int Cin, const bf16* __restrict__ wt, const float* __restrict__ bias,
                                                          bf16* __restrict__ out, int out_cs, int out_co, int Cout,
                                                          int N, int H, int W, int relu) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    bf16* tile = reinterpret_cast<bf16*>(smem_raw);
    const int stride = Cin + 8;  // halves per halo pixel and per weight row
    bf16* wsm = tile + kHaloX * kHaloY * stride;
    const int tiles_x = (W + kTileX - 1) / kTileX, tiles_y = (H + kTileY - 1) / kTileY;
    int t = blockIdx.x;
    const int tx = t % tiles_x;
    t /= tiles_x;
    const int ty = t % tiles_y;
    const int n = t / tiles_y;
    const int x0 = tx * kTileX, y0 = ty * kTileY;
    // stage the halo tile
    const int chunks = Cin / 8;
    for (int i = threadIdx.x; i < kHaloX * kHaloY * chunks; i += kConvThreads) {
        const int pix = i / chunks, c = i % chunks;
        const int gy = y0 - 1 + pix / kHaloX, gx = x0 - 1 + pix % kHaloX;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (gy >= 0 && gy < H && gx >= 0 && gx < W) v = __ldg(reinterpret_cast<const uint4*>(src_at(in, n, gy, gx, H, W, c * 8)));
        *reinterpret_cast<uint4*>(tile + pix * stride + c * 8) = v;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tq = lane & 3;
    const int co_base = blockIdx.y * NT * 8;
    // ldmatrix lane roles: matrix lane >> 3, row lane & 7
    const int lm = lane >> 3, lr = lane & 7;
    float acc[2][NT][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[m][j][k] = 0.0f;
    for (int tap = 0; tap < 9; ++tap) {
        const int ky = tap / 3, kx = tap % 3;
        // this tap's weight rows [co_base, co_base + NT*8)
        __syncthreads();  // the previous tap's reads of wsm are done (and, for tap 0, the halo is in)
        const bf16* wtap = wt + ((size_t)tap * gridDim.y * NT * 8 + co_base) * Cin;
        for (int i = threadIdx.x; i < NT * 8 * chunks; i += kConvThreads) {
            const int r = i / chunks, c = i % chunks;
            *reinterpret_cast<uint4*>(wsm + r * stride + c * 8) =
                __ldg(reinterpret_cast<const uint4*>(wtap + (size_t)r * Cin + c * 8));
        }
        __syncthreads();
        for (int cb = 0; cb < Cin; cb += 16) {
            // B: n-tiles j, j+1 from one x4 (matrices: rows n, k 0-7 | n, k 8-15 | n+8, k 0-7 | n+8, k 8-15)
            unsigned b[NT][2];
#pragma unroll
            for (int j = 0; j + 1 < NT; j += 2) {
                unsigned r4[4];
                ldmatrix_x4(r4, wsm + ((j + (lm >> 1)) * 8 + lr) * stride + cb + (lm & 1) * 8);
                b[j][0] = r4[0];
                b[j][1] = r4[1];
                b[j + 1][0] = r4[2];
                b[j + 1][1] = r4[3];
            }
            if (NT & 1) ldmatrix_x2(b[NT - 1][0], b[NT - 1][1], wsm + ((NT - 1) * 8 + lr) * stride + cb + (lm & 1) * 8);
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                // A: the 16 pixels of tile row 2*warp + m (matrices: px 0-7, k 0-7 | px 8-15, k 0-7 |
                // px 0-7, k 8-15 | px 8-15, k 8-15)
                const int row = 2 * warp + m;
                unsigned a[4];
                ldmatrix_x4(a, tile + ((row + ky) * kHaloX + lr + (lm & 1) * 8 + kx) * stride + cb + (lm >> 1) * 8);
#pragma unroll
                for (int j = 0; j < NT; ++j) mma_bf16(acc[m][j], a, b[j][0], b[j][1]);
            }
        }
    }
    // epilogue: bias, ReLU, BF16
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const int y = y0 + 2 * warp + m;
        if (y >= H) continue;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            const int co = co_base + j * 8 + 2 * tq;
            if (co >= Cout) continue;
            const float b0 = bias ? bias[co] : 0.0f, b1 = bias ? bias[co + 1] : 0.0f;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int x = x0 + g + 8 * h;
                if (x >= W) continue;
                float v0 = acc[m][j][2 * h] + b0, v1 = acc[m][j][2 * h + 1] + b1;
                if (relu) { v0 = fmaxf(v0, 0.0f); v1 = fmaxf(v1, 0.0f); }
                *reinterpret_cast<__nv_bfloat162*>(out + (((size_t)n * H + y) * W + x) * out_cs + out_co + co) =
                    __floats2bfloat162_rn(v0, v1);
            }
        }
    }
}

// ---------------------------------------------------------------- conv3x3 backward weights
// dW[tap][co][ci] += sum_p dY[p][co] * X[p + (ky-1, kx-1)][ci] for all nine taps, a group of
// up to four 16-row output-channel tiles (blockIdx.y) and a 16-wide input-channel slice
// (blockIdx.z); CTAs stride over 8x16 pixel tiles (blockIdx.x).  With nm output tiles in the
// group, warp w takes tile w % nm and the tile rows s = w / nm, w / nm + 4 / nm, ... (all
// four warps busy for 1, 2 or 4 tiles).  Per tile the CTA stages its dY columns and the X halo once; per 16-pixel
// k-step a warp loads its dY^T fragment once and reuses it for the nine taps' X fragments,
// keeping 9 x 2 accumulator tiles in registers until the end, then adds them into the FP32
// gradients.  dY: [N][H][W][Cpad] (Cpad multiple of 16, zero beyond the layer's real
// outputs); rows co >= cout_real are not written.  X: the layer's input (ConvSrc),
// Cin % 16 == 0.
constexpr int kWgradCo = 64;  // output channels per CTA (4 warps x 16)
__global__ void __launch_bounds__(kConvThreads) k_conv3x3_wgrad(const bf16* __restrict__ dy, int Cpad, int cout_real,
                                                                const ConvSrc x, int Cin, float* __restrict__ dw,
                                                                int N, int H, int W) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int dstride = kWgradCo + 8;
    constexpr int xstride = 16 + 8;
    bf16* dys = reinterpret_cast<bf16*>(smem_raw);         // [128][dstride]
    bf16* xs = dys + kTileX * kTileY * dstride;            // [10*18][xstride]
    const int co0 = blockIdx.y * kWgradCo;
    const int ci0 = blockIdx.z * 16;
    const int cw = min(kWgradCo, Cpad - co0);             // this CTA's output channels (multiple of 16)
    const int tiles_x = (W + kTileX - 1) / kTileX, tiles_y = (H + kTileY - 1) / kTileY;
    const int ntiles = N * tiles_x * tiles_y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nm = cw / 16, ngrp = 4 / nm;                 // output tiles, row groups
    const int mt = warp % nm, kgrp = warp / nm;
    const bool active = kgrp < ngrp;
    float acc[9][2][4];
#pragma unroll
    for (int t = 0; t < 9; ++t)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[t][j][k] = 0.0f;
    const int kk = lane & 7, which = lane >> 3;  // ldmatrix: row within matrix, matrix index
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        int tt = t;
        const int tx = tt % tiles_x;
        tt /= tiles_x;
        const int ty = tt % tiles_y;
        const int n = tt / tiles_y;
        const int x0 = tx * kTileX, y0 = ty * kTileY;
        __syncthreads();
        const int dchunks = cw / 8;
        for (int i = threadIdx.x; i < kTileX * kTileY * dchunks; i += kConvThreads) {
            const int pix = i / dchunks, c = i % dchunks;
            const int gy = y0 + pix / kTileX, gx = x0 + pix % kTileX;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (gy < H && gx < W)
                v = __ldg(reinterpret_cast<const uint4*>(dy + (((size_t)n * H + gy) * W + gx) * Cpad + co0 + c * 8));
            *reinterpret_cast<uint4*>(dys + pix * dstride + c * 8) = v;
        }
        for (int i = threadIdx.x; i < kHaloX * kHaloY * 2; i += kConvThreads) {
            const int pix = i / 2, c = i % 2;
            const int gy = y0 - 1 + pix / kHaloX, gx = x0 - 1 + pix % kHaloX;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (gy >= 0 && gy < H && gx >= 0 && gx < W)
                v = __ldg(reinterpret_cast<const uint4*>(src_at(x, n, gy, gx, H, W, ci0 + c * 8)));
            *reinterpret_cast<uint4*>(xs + pix * xstride + c * 8) = v;
        }
        __syncthreads();
        if (!active) continue;
        // K = the tile's 128 pixels in 8 steps of 16 (one tile row each)
#pragma unroll 1
        for (int s = kgrp; s < kTileY; s += ngrp) {
            // A: output channels (rows) x pixels (k).  Matrices: 0 = (co 0-7, px 0-7),
            // 1 = (co 8-15, px 0-7), 2 = (co 0-7, px 8-15), 3 = (co 8-15, px 8-15)
            unsigned a[4];
            {
                const int px = kk + ((which & 2) ? 8 : 0);
                const int co = mt * 16 + ((which & 1) ? 8 : 0);
                ldmatrix_x4_trans(a, dys + (s * kTileX + px) * dstride + co);
            }
#pragma unroll
            for (int tap = 0; tap < 9; ++tap) {
                const int ky = tap / 3, kx = tap % 3;
                // B: pixels (row s, cols 0..15) shifted by the tap x 16 input channels.  Matrices:
                // 0 = (px 0-7, ci 0-7), 1 = (px 8-15, ci 0-7), 2 = (px 0-7, ci 8-15), 3 = (px 8-15, ci 8-15)
                unsigned bq[4];
                const int px = kk + ((which & 1) ? 8 : 0);
                const int cc = (which & 2) ? 8 : 0;
                ldmatrix_x4_trans(bq, xs + ((s + ky) * kHaloX + px + kx) * xstride + cc);
                mma_bf16(acc[tap][0], a, bq[0], bq[1]);
                mma_bf16(acc[tap][1], a, bq[2], bq[3]);
            }
        }
    }
    if (!active) return;
    const int g = lane >> 2, tq = lane & 3;
#pragma unroll
    for (int tap = 0; tap < 9; ++tap)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int ci = ci0 + j * 8 + 2 * tq;
            const int c0 = co0 + mt * 16 + g, c1 = c0 + 8;
            if (c0 < cout_real) {
                float* r0 = dw + ((size_t)tap * cout_real + c0) * Cin + ci;
                atomicAdd(r0, acc[tap][j][0]);
                atomicAdd(r0 + 1, acc[tap][j][1]);
            }
            if (c1 < cout_real) {
                float* r1 = dw + ((size_t)tap * cout_real + c1) * Cin + ci;
                atomicAdd(r1, acc[tap][j][2]);
                atomicAdd(r1 + 1, acc[tap][j][3]);
            }
        }
}

// ---------------------------------------------------------------- elementwise / layout
// Packs 8 floats into 8 BF16 (round to nearest) in one 16-byte word.
__device__ __forceinline__ uint4 pack_bf16x8(const float (&v)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
        w[k] = *reinterpret_cast<const uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ void unpack_bf16x8(uint4 q, float (&v)[8]) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 f = __bfloat1622float2(h[k]);
        v[2 * k] = f.x;
        v[2 * k + 1] = f.y;
    }
}

// features (kFeatures floats per pixel: colour, albedo, normal, 1/(1+t), noise level)
// -> 16-channel BF16 input, colour as log(1 + colour)
__global__ void k_prep_input(const float* __restrict__ f, long long npx, bf16* __restrict__ x) {
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < npx; p += (long long)gridDim.x * blockDim.x) {
        const float* s = f + p * kFeatures;
        float v[16];
#pragma unroll
        for (int c = 0; c < 3; ++c) v[c] = log1pf(fmaxf(__ldg(s + c), 0.0f));
#pragma unroll
        for (int c = 3; c < kFeatures; ++c) v[c] = __ldg(s + c);
#pragma unroll
        for (int c = kFeatures; c < 16; ++c) v[c] = 0.0f;
        uint32_t w[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
            w[k] = *reinterpret_cast<const uint32_t*>(&h);
        }
        uint4* d = reinterpret_cast<uint4*>(x + p * 16);
        d[0] = make_uint4(w[0], w[1], w[2], w[3]);
        d[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
}

// 2x2 max-pool: in [N][H][W][C] -> out [N][H/2][W/2][C], C % 8 == 0; one thread per output
// pixel and 8 channels (16-byte loads and store; max of BF16 values is exact)
__global__ void k_pool(const bf16* __restrict__ in, bf16* __restrict__ out, int N, int H, int W, int C) {
    const int Ho = H / 2, Wo = W / 2, G = C / 8;
    const long long total = (long long)N * Ho * Wo * G;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int g = (int)(i % G);
        long long p = i / G;
        const int xo = (int)(p % Wo);
        p /= Wo;
        const int yo = (int)(p % Ho);
        const int n = (int)(p / Ho);
        const bf16* s = in + (((size_t)n * H + 2 * yo) * W + 2 * xo) * C + g * 8;
        uint4 q[4] = {__ldg(reinterpret_cast<const uint4*>(s)), __ldg(reinterpret_cast<const uint4*>(s + C)),
                      __ldg(reinterpret_cast<const uint4*>(s + (size_t)W * C)),
                      __ldg(reinterpret_cast<const uint4*>(s + (size_t)W * C + C))};
        __nv_bfloat162* m = reinterpret_cast<__nv_bfloat162*>(&q[0]);
#pragma unroll
        for (int k = 1; k < 4; ++k) {
            const __nv_bfloat162* o = reinterpret_cast<const __nv_bfloat162*>(&q[k]);
#pragma unroll
            for (int e = 0; e < 4; ++e) m[e] = __hmax2(m[e], o[e]);
        }
        *reinterpret_cast<uint4*>(out + i * 8) = q[0];
    }
}

// Block sums of the bias gradient: per-thread sums s[8] (8-channel group j of G, thread row r of
// `per`) added in shared memory in row order into part[blockIdx.x][c], c < C; k_grad_reduce adds
// the blocks' partials.
__device__ __forceinline__ void bias_partials(float* sb, const float (&s)[8], int j, int r, int per, int C,
                                              float* __restrict__ part) {
    if (r < per && j * 8 < C) {
#pragma unroll
        for (int k = 0; k < 8; ++k) sb[r * C + j * 8 + k] = s[k];
    }
    __syncthreads();
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
        float t = 0.0f;
        for (int i = 0; i < per; ++i) t += sb[i * C + c];
        part[(size_t)blockIdx.x * C + c] = t;
    }
}

// L1 loss in log space on channels 0..2 of the prediction y = out + x (the network predicts
// a correction of the input's log colour x, channels 0..2 of the 16-channel input [npx][16]),
// and its gradient as the next GEMMs' operand: g [npx][16] BF16, zero beyond channel 2, with
// the output layer's bias partial sums (8 channels).
__global__ void __launch_bounds__(256) k_loss_bwd(const bf16* __restrict__ out, const bf16* __restrict__ x,
                                                  const float* __restrict__ target, long long npx, bf16* __restrict__ g,
                                                  float* __restrict__ part, double* __restrict__ loss_sum) {
    extern __shared__ float sb[];  // [256][8]
    double s = 0.0;
    float bs[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const float scale = 1.0f / (3.0f * (float)npx);
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < npx; p += (long long)gridDim.x * blockDim.x) {
        const uint2 o = __ldg(reinterpret_cast<const uint2*>(out + p * 8)), xi = __ldg(reinterpret_cast<const uint2*>(x + p * 16));
        const float2 o01 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&o.x)),
                     o2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&o.y)),
                     x01 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&xi.x)),
                     x2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&xi.y));
        const float y[3] = {o01.x + x01.x, o01.y + x01.y, o2.x + x2.x};
        float v[8] = {0, 0, 0, 0, 0, 0, 0, 0}, w[8];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float d = y[c] - log1pf(fmaxf(target[p * 3 + c], 0.0f));
            s += fabsf(d);
            v[c] = (d > 0.0f ? 1.0f : (d < 0.0f ? -1.0f : 0.0f)) * scale;
        }
        const uint4 pk = pack_bf16x8(v);
        reinterpret_cast<uint4*>(g + p * 16)[0] = pk;
        reinterpret_cast<uint4*>(g + p * 16)[1] = make_uint4(0, 0, 0, 0);
        unpack_bf16x8(pk, w);
#pragma unroll
        for (int c = 0; c < 3; ++c) bs[c] += w[c];
    }
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss_sum, s);
    bias_partials(sb, bs, 0, threadIdx.x, blockDim.x, 8, part);
}

// Where a layer's output gradient comes from: backward-data outputs in BF16, read in place.
//   GRAD_PLAIN  a [npx][a_cs], channels 0..C-1
//   GRAD_UP     the layer was up-sampled: the sum of its four children's gradients, channels
//               0..C-1 of a [N][2h][2w][a_cs]
//   GRAD_SKIP   the layer fed a skip connection and a max pool: channels a_off.. of
//               a [npx][a_cs], plus at a 2x2 block's first maximum (of the layer's output) the
//               block's gradient b [N][h/2][w/2][C]
enum GradKind { GRAD_PLAIN, GRAD_UP, GRAD_SKIP };
struct GradSrc {
    const bf16* a;
    int a_cs, a_off;
    const bf16* b;
};

// A layer's output gradient summed in FP32, its ReLU mask (y > 0), the rounding to BF16 that
// the next GEMMs read (g [npx][C]) and the bias gradient's partial sums, in one pass: the
// FP32 copies of the gradients that three kernels wrote and read before are never stored
// (gradients of 16 x 256 x 256: element-wise kernels 0.55 -> 0.26 ms).  Thread t of a block takes
// 8-channel group t % G of the pixels (2x2 blocks for GRAD_SKIP) t / G, t / G + per, ... of
// the block's grid stride.  C and the strides are multiples of 8.
template <int KIND>
__global__ void __launch_bounds__(256) k_grad_in(const bf16* y, GradSrc src, int C, int N, int H, int W, bf16* g,
                                                 float* part) {
    extern __shared__ float sb[];  // [per][C]
    grid_turn();
    const int G = C / 8, per = blockDim.x / G;
    const int j = threadIdx.x % G, r = threadIdx.x / G, c = j * 8;
    float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    auto finish = [&](long long p, const float (&yv)[8], float (&v)[8]) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (!(yv[k] > 0.0f)) v[k] = 0.0f;
        const uint4 pk = pack_bf16x8(v);
        *reinterpret_cast<uint4*>(g + p * C + c) = pk;
        float w[8];
        unpack_bf16x8(pk, w);
#pragma unroll
        for (int k = 0; k < 8; ++k) s[k] += w[k];
    };
    auto ld = [](const bf16* p) { return *reinterpret_cast<const uint4*>(p); };
    if (r < per) {
        if (KIND == GRAD_SKIP) {
            const int Ho = H / 2, Wo = W / 2;
            const long long nb = (long long)N * Ho * Wo;
            for (long long b = (long long)blockIdx.x * per + r; b < nb; b += (long long)gridDim.x * per) {
                const int xo = (int)(b % Wo);
                const long long t = b / Wo;
                const int yo = (int)(t % Ho), n = (int)(t / Ho);
                const long long p0 = ((long long)n * H + 2 * yo) * W + 2 * xo;
                const long long px[4] = {p0, p0 + 1, p0 + W, p0 + W + 1};
                uint4 yq[4], aq[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) yq[k] = ld(y + px[k] * C + c);
#pragma unroll
                for (int k = 0; k < 4; ++k) aq[k] = ld(src.a + px[k] * src.a_cs + src.a_off + c);
                float d[8], m[8], yv[8];
                int arg[8];
                unpack_bf16x8(ld(src.b + b * C + c), d);
#pragma unroll
                for (int e = 0; e < 8; ++e) { m[e] = -INFINITY; arg[e] = 0; }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    unpack_bf16x8(yq[k], yv);
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        if (yv[e] > m[e]) { m[e] = yv[e]; arg[e] = k; }
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    float v[8];
                    unpack_bf16x8(yq[k], yv);
                    unpack_bf16x8(aq[k], v);
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] += arg[e] == k ? d[e] : 0.0f;
                    finish(px[k], yv, v);
                }
            }
        } else {
            const long long npx = (long long)N * H * W, step = (long long)gridDim.x * per;
            for (long long p = (long long)blockIdx.x * per + r; p < npx; p += step) {
                float v[8], yv[8];
                const uint4 yq = ld(y + p * C + c);
                if (KIND == GRAD_UP) {
                    const int x = (int)(p % W);
                    const long long t = p / W;
                    const int yy = (int)(t % H), n = (int)(t / H);
                    const bf16* a = src.a + (((long long)n * 2 * H + 2 * yy) * 2 * W + 2 * x) * src.a_cs + c;
                    const uint4 q[4] = {ld(a), ld(a + src.a_cs), ld(a + (size_t)2 * W * src.a_cs),
                                        ld(a + (size_t)2 * W * src.a_cs + src.a_cs)};
#pragma unroll
                    for (int k = 0; k < 8; ++k) v[k] = 0.0f;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        float w[8];
                        unpack_bf16x8(q[i], w);
#pragma unroll
                        for (int k = 0; k < 8; ++k) v[k] += w[k];
                    }
                } else {
                    unpack_bf16x8(ld(src.a + p * src.a_cs + c), v);
                }
                unpack_bf16x8(yq, yv);
                finish(p, yv, v);
            }
        }
    }
    bias_partials(sb, s, j, r, per, C, part);
}

// Up to four symmetries of one shape, as the self-ensemble's forward passes take them.
struct FlipSet {
    int n, flip[4];
};

// Adds the predictions of a batch of images to rgb [H][W][3]: image j's prediction of pixel
// (px, py) stands at its mirrored place in the padded Wp x Hp output, or, with flip bit 2, at
// the transposed place of the Hp-wide transposed output; it is added times `weight`, in the
// order of the images.  rec: the film's input records, whose first channels are the log
// colour the network corrects.  Blocks of 16 x 16 pixels: transposed images are read down
// columns of 16 neighbours.
__global__ void __launch_bounds__(256) k_output_images(const bf16* __restrict__ out, const uint4* __restrict__ rec, int W,
                                                       int H, int Wp, int Hp, FlipSet fs, float weight, int first,
                                                       float* __restrict__ rgb) {
    const int bw = (W + 15) / 16;
    const int px = (int)(blockIdx.x % bw) * 16 + (threadIdx.x & 15), py = (int)(blockIdx.x / bw) * 16 + (threadIdx.x >> 4);
    if (px >= W || py >= H) return;
    const long long p = (long long)py * W + px;
    const uint2 xr = *reinterpret_cast<const uint2*>(rec + 2 * p);
    const __nv_bfloat162 x01 = *reinterpret_cast<const __nv_bfloat162*>(&xr.x),
                         x2 = *reinterpret_cast<const __nv_bfloat162*>(&xr.y);
    const float x[3] = {__low2float(x01), __high2float(x01), __low2float(x2)};
    float v[3] = {0.0f, 0.0f, 0.0f};
    if (!first)
        for (int c = 0; c < 3; ++c) v[c] = rgb[3 * p + c];
    uint2 o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (j >= fs.n) break;
        const int f = fs.flip[j], qx = (f & 1) ? W - 1 - px : px, qy = (f & 2) ? H - 1 - py : py;
        const long long q = (long long)j * Wp * Hp + ((f & 4) ? (long long)qx * Hp + qy : (long long)qy * Wp + qx);
        o[j] = __ldg(reinterpret_cast<const uint2*>(out + q * 8));
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (j >= fs.n) break;
        const __nv_bfloat162 r01 = *reinterpret_cast<const __nv_bfloat162*>(&o[j].x),
                             r2 = *reinterpret_cast<const __nv_bfloat162*>(&o[j].y);
        const float r[3] = {__low2float(r01), __high2float(r01), __low2float(r2)};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float y = __fmul_rn(weight, fmaxf(expm1f(r[c] + x[c]), 0.0f));
            v[c] = first && j == 0 ? y : __fadd_rn(v[c], y);
        }
    }
    for (int c = 0; c < 3; ++c) rgb[3 * p + c] = v[c];
}

// prediction (input log colour + network correction) -> linear colour
__global__ void k_output(const bf16* __restrict__ out, const bf16* __restrict__ x, long long npx,
                         float* __restrict__ rgb) {
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < npx; p += (long long)gridDim.x * blockDim.x)
        for (int c = 0; c < 3; ++c)
            rgb[p * 3 + c] =
                fmaxf(expm1f(__bfloat162float(out[p * 8 + c]) + __bfloat162float(x[p * 16 + c])), 0.0f);
}

// Adam on FP32 masters, then the BF16 copies: forward layout [tap][co][ci] and the
// backward-data layout [tap][ci][co] with taps flipped (8 - tap).
struct AdamArgs {
    float lr, b1, b2, eps, c1, c2;  // c1 = 1/(1-b1^t), c2 = 1/(1-b2^t)
};
__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       long long n, AdamArgs a) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = a.b1 * m[i] + (1.0f - a.b1) * gi;
        const float vi = a.b2 * v[i] + (1.0f - a.b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= a.lr * (mi * a.c1) / (sqrtf(vi * a.c2) + a.eps);
    }
}

__global__ void k_weights_to_bf16(const float* __restrict__ w, int Cout, int Cin, int rows_fwd, int rows_bwd,
                                  int cout_pad, bf16* __restrict__ wf, bf16* __restrict__ wb) {
    const int total = 9 * Cout * Cin;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int ci = i % Cin, co = (i / Cin) % Cout, tap = i / (Cin * Cout);
        const bf16 v = __float2bfloat16(w[i]);
        wf[((size_t)tap * rows_fwd + co) * Cin + ci] = v;
        if (wb) wb[((size_t)(8 - tap) * rows_bwd + ci) * cout_pad + co] = v;
    }
}

// The film's input records (W x H, 32 bytes per pixel) placed as a batch of network inputs
// (Wp x Hp, multiples of 16) with reflected borders.  With flip bit 0 (1) the frame is
// mirrored left-right (top-bottom) first; with bit 2 the input is the transposed frame, Hp wide
// and Wp tall.  Two threads per pixel, 16 x 8 pixels per block; the records (66 MB at 1080p)
// are read from L2.
__global__ void __launch_bounds__(256) k_place_inputs(const uint4* __restrict__ rec, int W, int H, int Wp, int Hp,
                                                      FlipSet fs, uint4* __restrict__ x) {
    const int half = threadIdx.x & 1, t = threadIdx.x >> 1, f = fs.flip[blockIdx.y];
    // blocks run along the output's rows, in one grid dimension: (u, v) is the output pixel
    const int Wo = (f & 4) ? Hp : Wp, Ho = (f & 4) ? Wp : Hp, bw = Wo / 16;
    const int u = (int)(blockIdx.x % bw) * 16 + (t & 15), v = (int)(blockIdx.x / bw) * 8 + (t >> 4);
    if (u >= Wo || v >= Ho) return;
    const int px = (f & 4) ? v : u, py = (f & 4) ? u : v;
    int sx = px < W ? px : max(2 * W - 2 - px, 0), sy = py < H ? py : max(2 * H - 2 - py, 0);
    if (f & 1) sx = W - 1 - sx;
    if (f & 2) sy = H - 1 - sy;
    x[(((long long)blockIdx.y * Ho + v) * Wo + u) * 2 + half] = __ldg(rec + ((long long)sy * W + sx) * 2 + half);
}

inline int gsz(long long n, int block = 256) {
    long long g = (n + block - 1) / block;
    return (int)(g > 4096 ? 4096 : (g < 1 ? 1 : g));
}

// ---------------------------------------------------------------- network
struct UnetLayer {
    int cin, cout, relu;  // cin % 16 == 0 (input padded); cout % 8 == 0
    int cout_pad;         // cout rounded up to 16 (gradient operand channels)
    long long w_off, b_off;  // parameter vector: w [9][cout][cin], then b [cout]
    int nt, rows_fwd;     // forward conv: n8 tiles per CTA, BF16 weight rows
    int nt_b, rows_bwd;   // backward-data conv (outputs cin channels)
    long long wf_off, wb_off;  // BF16 weight copies
};

// Layer table: input padded to 16 channels, output 8 channels of which 3 are used.
const int kLayers[][3] = {
    {16, 32, 1}, {32, 32, 1},   // enc0 -> e0
    {32, 48, 1}, {48, 48, 1},   // enc1 -> e1
    {48, 64, 1}, {64, 64, 1},   // enc2 -> e2
    {64, 80, 1}, {80, 80, 1},   // enc3 -> e3
    {80, 96, 1},                // bottleneck -> b
    {176, 80, 1},               // dec3: up(b) + e3 -> d3
    {144, 64, 1},               // dec2: up(d3) + e2 -> d2
    {112, 48, 1},               // dec1: up(d2) + e1 -> d1
    {80, 32, 1},                // dec0: up(d1) + e0 -> d0
    {32, 8, 0},                 // output
};
// pyramid level (resolution H >> level) each layer runs at
const int kLayerLevel[] = {0, 0, 1, 1, 2, 2, 3, 3, 4, 3, 2, 1, 0, 0};
constexpr int kNumLayers = 14;

int pick_nt(int c) {
    if (c <= 64) return c / 8;  // the whole channel count in one CTA
    for (int nt = 6; nt >= 2; --nt)
        if (c % (nt * 8) == 0) return nt;
    return 2;
}

inline int round_up(int a, int b) { return (a + b - 1) / b * b; }

// Workspace (BF16), by name; sizes in elements for N x H x W inputs.  T_G: a layer's output
// gradient, T_G2: its input gradient, T_C0..3: the decoder layers' input gradients (read twice,
// as the coarse level's and the skip connection's).
enum {
    T_X, T_A0, T_E0, T_P0, T_A1, T_E1, T_P1, T_A2, T_E2, T_P2, T_A3, T_E3, T_P3, T_B,
    T_D3, T_D2, T_D1, T_D0, T_OUT, T_G, T_G2, T_C3, T_C2, T_C1, T_C0, T_COUNT
};
}  // namespace

struct Unet {
    std::vector<UnetLayer> layers;
    long long n_params = 0;
    DevBuf<float> params, grads, adam_m, adam_v;
    DevBuf<bf16> wf, wb;
    long long step = 0;
    int N = 0, H = 0, W = 0;
    DevBuf<bf16> act;
    long long act_off[T_COUNT];
    DevBuf<float> io;       // device copies of host features / targets / outputs
    DevBuf<float> film_ws;  // a film's input records and the denoised image (salty_denoise_unet)
    DevBuf<double> loss;
    DevBuf<float> wg_ws;    // per-CTA partial weight and bias gradients (fixed-order sums)
    size_t wg_off[kNumLayers], wg_len[kNumLayers], bias_off[kNumLayers], wg_floats;  // each layer's, in floats
    int conv_kind = SALTY_CONV_TCGEN05;  // convolution kernels (forward, backward-data, weights)
};

namespace {

void init_layers(Unet& u) {
    u.layers.clear();
    long long off = 0, wf = 0, wb = 0;
    for (int i = 0; i < kNumLayers; ++i) {
        UnetLayer L;
        L.cin = kLayers[i][0];
        L.cout = kLayers[i][1];
        L.relu = kLayers[i][2];
        L.cout_pad = round_up(L.cout, 16);
        L.w_off = off;
        off += 9LL * L.cin * L.cout;
        L.b_off = off;
        off += L.cout;
        L.nt = pick_nt(L.cout);
        L.rows_fwd = round_up(L.cout, L.nt * 8);
        L.nt_b = pick_nt(L.cin);
        L.rows_bwd = round_up(L.cin, L.nt_b * 8);
        L.wf_off = wf;
        wf += 9LL * L.rows_fwd * L.cin;
        L.wb_off = wb;
        wb += 9LL * L.rows_bwd * L.cout_pad;
        u.layers.push_back(L);
    }
    u.n_params = off;
}

salty_status launch_conv(salty_ctx* ctx, int kind, const ConvSrc& in, int cin, const bf16* w, int rows, int nt,
                         const float* bias, bf16* out, int out_cs, int cout, int N, int H, int W, int relu,
                         bf16* pool = nullptr) {
    if (kind == SALTY_CONV_TCGEN05)
        return conv3x3_tma(ctx, in, cin, w, rows, bias, out, pool, out_cs, cout, N, H, W, relu, ctx->status.p + 8);
    if (pool) {
        SALTY_TRY(launch_conv(ctx, kind, in, cin, w, rows, nt, bias, out, out_cs, cout, N, H, W, relu));
        const long long groups = (long long)N * (H / 2) * (W / 2) * (cout / 8);
        k_pool<<<gsz(groups), 256, 0, ctx->stream>>>(out, pool, N, H, W, cout);
        SALTY_TRY_CUDA(ctx->err, cudaGetLastError());
        return SALTY_OK;
    }
    if (kind == SALTY_CONV_TCGEN05_CP_ASYNC)
        return conv3x3_tc(ctx, in, cin, w, rows, bias, out, out_cs, 0, cout, N, H, W, relu, ctx->status.p + 8);
    const int tiles = N * ((W + kTileX - 1) / kTileX) * ((H + kTileY - 1) / kTileY);
    dim3 grid(tiles, rows / (nt * 8));
    const size_t smem = ((size_t)kHaloX * kHaloY + (size_t)nt * 8) * (cin + 8) * sizeof(bf16);
#define SALTY_CONV_CASE(NTV)                                                                                         \
    case NTV: {                                                                                                     \
        SALTY_TRY_CUDA(ctx->err,                                                                                    \
                       cudaFuncSetAttribute(k_conv3x3<NTV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
        k_conv3x3<NTV><<<grid, kConvThreads, smem, ctx->stream>>>(in, cin, w, bias, out, out_cs, 0, cout, N, H, W,   \
                                                                  relu);                                            \
        break;                                                                                                      \
    }
    switch (nt) {
        SALTY_CONV_CASE(1) SALTY_CONV_CASE(2) SALTY_CONV_CASE(4) SALTY_CONV_CASE(5) SALTY_CONV_CASE(6)
        SALTY_CONV_CASE(8)
        default:
            return ctx->err.fail(SALTY_ERR_INVALID_ARG, "unsupported conv tile %d", nt);
    }
#undef SALTY_CONV_CASE
    SALTY_TRY_CUDA(ctx->err, cudaGetLastError());
    return SALTY_OK;
}

salty_status launch_wgrad(salty_ctx* ctx, Unet& u, int li, const bf16* dy, int cpad, int cout, const ConvSrc& x, int cin,
                          float* dw, int N, int H, int W, GradReduceTable& table) {
    if (u.conv_kind != SALTY_CONV_MMA_SYNC)
        return conv_wgrad_tc(ctx, dy, cpad, cout, x, cin, dw, N, H, W, u.wg_ws.p + u.wg_off[li], u.wg_len[li],
                             ctx->status.p + 8, table);
    const size_t smem = ((size_t)kTileX * kTileY * (kWgradCo + 8) + (size_t)kHaloX * kHaloY * 24) * sizeof(bf16);
    const int tiles = N * ((W + kTileX - 1) / kTileX) * ((H + kTileY - 1) / kTileY);
    const int mg = (cpad + kWgradCo - 1) / kWgradCo;
    // about four resident CTAs per SM over all (output-channel group, input slice) pairs
    int gx = ctx->num_sms * 4 / (mg * (cin / 16));
    if (gx < 1) gx = 1;
    if (gx > tiles) gx = tiles;
    dim3 grid(gx, mg, cin / 16);
    k_conv3x3_wgrad<<<grid, kConvThreads, smem, ctx->stream>>>(dy, cpad, cout, x, cin, dw, N, H, W);
    SALTY_TRY_CUDA(ctx->err, cudaGetLastError());
    return SALTY_OK;
}

salty_status ensure_workspace(salty_ctx* ctx, Unet& u, int N, int H, int W) {
    if (u.N == N && u.H == H && u.W == W && u.act.p) return SALTY_OK;
    const long long P0 = (long long)N * H * W, P1 = P0 / 4, P2 = P0 / 16, P3 = P0 / 64, P4 = P0 / 256;
    const long long asz[T_COUNT] = {P0 * 16, P0 * 32, P0 * 32, P1 * 32, P1 * 48, P1 * 48, P2 * 48, P2 * 64, P2 * 64,
                                    P3 * 64, P3 * 80, P3 * 80, P4 * 80, P4 * 96, P3 * 80, P2 * 64, P1 * 48, P0 * 32,
                                    P0 * 8, P0 * 32, P0 * 32, P3 * 176, P2 * 144, P1 * 112, P0 * 80};
    long long o = 0;
    for (int i = 0; i < T_COUNT; ++i) { u.act_off[i] = o; o += (asz[i] + 63) / 64 * 64; }
    SALTY_TRY_CUDA(ctx->err, u.act.ensure((size_t)o));
    // per layer: the weight gradient's slices, and 4 blocks per SM of bias partials
    size_t ws = 0;
    for (int i = 0; i < kNumLayers; ++i) {
        const UnetLayer& L = u.layers[i];
        const int lv = kLayerLevel[i];
        u.wg_off[i] = ws;
        u.wg_len[i] = conv_wgrad_tc_workspace(ctx->num_sms, L.cin, L.cout_pad, N, H >> lv, W >> lv);
        ws += (u.wg_len[i] + 63) / 64 * 64;
        u.bias_off[i] = ws;
        ws += ((size_t)ctx->num_sms * 4 * L.cout + 63) / 64 * 64;
    }
    u.wg_floats = ws;
    u.N = N; u.H = H; u.W = W;
    return SALTY_OK;
}

salty_status refresh_bf16(salty_ctx* ctx, Unet& u) {
    for (const UnetLayer& L : u.layers)
        k_weights_to_bf16<<<gsz(9LL * L.cout * L.cin), 256, 0, ctx->stream>>>(
            u.params.p + L.w_off, L.cout, L.cin, L.rows_fwd, L.rows_bwd, L.cout_pad, u.wf.p + L.wf_off, u.wb.p + L.wb_off);
    SALTY_TRY_CUDA(ctx->err, cudaGetLastError());
    return SALTY_OK;
}

struct Fwd {
    bf16* t[T_COUNT];
};

// d_feat: the input features, or null when the input tensor T_X is in place already.
salty_status forward(salty_ctx* ctx, Unet& u, const float* d_feat, int N, int H, int W, Fwd& F) {
    SALTY_TRY(ensure_workspace(ctx, u, N, H, W));
    for (int i = 0; i < T_COUNT; ++i) F.t[i] = u.act.p + u.act_off[i];
    cudaStream_t st = ctx->stream;
    const long long P0 = (long long)N * H * W;
    if (d_feat) k_prep_input<<<gsz(P0), 256, 0, st>>>(d_feat, P0, F.t[T_X]);
    // pool: the tensor that takes the 2x2 max-pooled output too, or -1
    auto conv = [&](int li, const ConvSrc& in, int out, int h, int w, int pool = -1) {
        const UnetLayer& L = u.layers[li];
        return launch_conv(ctx, u.conv_kind, in, L.cin, u.wf.p + L.wf_off, L.rows_fwd, L.nt, u.params.p + L.b_off,
                           F.t[out], L.cout, L.cout, N, h, w, L.relu, pool >= 0 ? F.t[pool] : nullptr);
    };
    auto x = [&](int t, int c) { return conv_src(F.t[t], c, c); };
    // decoder inputs: [up2(coarse) | skip], read by the convolutions from both tensors
    auto cat = [&](int coarse, int cc, int skip, int cs) { return conv_src_cat(F.t[coarse], cc, F.t[skip], cs); };
    const int H1 = H / 2, W1 = W / 2, H2 = H / 4, W2 = W / 4, H3 = H / 8, W3 = W / 8, H4 = H / 16, W4 = W / 16;
    SALTY_TRY(conv(0, x(T_X, 16), T_A0, H, W));
    SALTY_TRY(conv(1, x(T_A0, 32), T_E0, H, W, T_P0));
    SALTY_TRY(conv(2, x(T_P0, 32), T_A1, H1, W1));
    SALTY_TRY(conv(3, x(T_A1, 48), T_E1, H1, W1, T_P1));
    SALTY_TRY(conv(4, x(T_P1, 48), T_A2, H2, W2));
    SALTY_TRY(conv(5, x(T_A2, 64), T_E2, H2, W2, T_P2));
    SALTY_TRY(conv(6, x(T_P2, 64), T_A3, H3, W3));
    SALTY_TRY(conv(7, x(T_A3, 80), T_E3, H3, W3, T_P3));
    SALTY_TRY(conv(8, x(T_P3, 80), T_B, H4, W4));
    SALTY_TRY(conv(9, cat(T_B, 96, T_E3, 80), T_D3, H3, W3));
    SALTY_TRY(conv(10, cat(T_D3, 80, T_E2, 64), T_D2, H2, W2));
    SALTY_TRY(conv(11, cat(T_D2, 64, T_E1, 48), T_D1, H1, W1));
    SALTY_TRY(conv(12, cat(T_D1, 48, T_E0, 32), T_D0, H, W));
    SALTY_TRY(conv(13, x(T_D0, 32), T_OUT, H, W));
    SALTY_TRY_CUDA(ctx->err, cudaGetLastError());
    return SALTY_OK;
}

// Blocks of a gradient pass over `work` units of 8 channels x C / 8 groups (4 per SM: the bias
// partials of 4 blocks per SM are what the workspace holds).
int grad_blocks(salty_ctx* ctx, long long work, int per) {
    return (int)std::min<long long>((long long)ctx->num_sms * 4, (work + per - 1) / per);
}

salty_status bias_reduce_add(salty_ctx* ctx, Unet& u, int li, int blocks, GradReduceTable& table) {
    const UnetLayer& L = u.layers[li];
    return grad_reduce_add(ctx, table, {u.wg_ws.p + u.bias_off[li], u.grads.p + L.b_off, blocks, L.cout, L.cout / 4, 1, 1,
                                        L.cout / 4, 0});
}

// The output gradient of layer li in T_G (BF16) and its bias gradient's partial sums.
template <int KIND>
salty_status grad_in(salty_ctx* ctx, Unet& u, Fwd& F, int li, int y, const GradSrc& src, int N, int h, int w,
                     GradReduceTable& table) {
    const UnetLayer& L = u.layers[li];
    const long long npx = (long long)N * h * w, work = KIND == GRAD_SKIP ? npx / 4 : npx;
    const int per = 256 / (L.cout / 8), blocks = grad_blocks(ctx, work, per);
    SALTY_TRY_CUDA(ctx->err, launch_early(k_grad_in<KIND>, blocks, 256, (size_t)per * L.cout * sizeof(float), ctx->stream,
                                          F.t[y], src, L.cout, N, h, w, F.t[T_G], u.wg_ws.p + u.bias_off[li]));
    return bias_reduce_add(ctx, u, li, blocks, table);
}

// Weight gradient of layer li from its output gradient in T_G, and, with dx >= 0, the gradient
// of its input in that tensor ([npx][cin], BF16).
salty_status conv_backward(salty_ctx* ctx, Unet& u, Fwd& F, int li, const ConvSrc& x, int N, int h, int w, int dx,
                           GradReduceTable& table) {
    const UnetLayer& L = u.layers[li];
    bf16* g = F.t[T_G];
    SALTY_TRY(launch_wgrad(ctx, u, li, g, L.cout_pad, L.cout, x, L.cin, u.grads.p + L.w_off, N, h, w, table));
    if (dx >= 0)
        SALTY_TRY(launch_conv(ctx, u.conv_kind, conv_src(g, L.cout_pad, L.cout_pad), L.cout_pad, u.wb.p + L.wb_off,
                              L.rows_bwd, L.nt_b, nullptr, F.t[dx], L.cin, L.cin, N, h, w, 0));
    return SALTY_OK;
}

// Loss and all gradients for the batch in F (after forward); grads are zeroed first.
salty_status backward(salty_ctx* ctx, Unet& u, Fwd& F, const float* d_target, int N, int H, int W, double* loss) {
    cudaStream_t st = ctx->stream;
    const long long P0 = (long long)N * H * W;
    GradReduceTable table;
    SALTY_TRY_CUDA(ctx->err, u.wg_ws.ensure(u.wg_floats));
    SALTY_TRY_CUDA(ctx->err, cudaMemsetAsync(u.grads.p, 0, u.n_params * sizeof(float), st));
    SALTY_TRY_CUDA(ctx->err, u.loss.ensure(1));
    SALTY_TRY_CUDA(ctx->err, cudaMemsetAsync(u.loss.p, 0, sizeof(double), st));
    const int H1 = H / 2, W1 = W / 2, H2 = H / 4, W2 = W / 4, H3 = H / 8, W3 = W / 8, H4 = H / 16, W4 = W / 16;
    auto x = [&](int t, int c) { return conv_src(F.t[t], c, c); };
    auto cat = [&](int coarse, int cc, int skip, int cs) { return conv_src_cat(F.t[coarse], cc, F.t[skip], cs); };
    auto plain = [&](int li, int y, int h, int w) {
        return grad_in<GRAD_PLAIN>(ctx, u, F, li, y, GradSrc{F.t[T_G2], u.layers[li].cout, 0, nullptr}, N, h, w, table);
    };
    auto up = [&](int li, int y, int dcat, int ch, int h, int w) {
        return grad_in<GRAD_UP>(ctx, u, F, li, y, GradSrc{F.t[dcat], ch, 0, nullptr}, N, h, w, table);
    };
    auto skip = [&](int li, int y, int dcat, int ch, int off, int h, int w) {
        return grad_in<GRAD_SKIP>(ctx, u, F, li, y, GradSrc{F.t[dcat], ch, off, F.t[T_G2]}, N, h, w, table);
    };
    auto back = [&](int li, const ConvSrc& in, int h, int w, int dx) {
        return conv_backward(ctx, u, F, li, in, N, h, w, dx, table);
    };
    // the loss, its gradient and the output layer's bias gradient
    const int lb = grad_blocks(ctx, P0, 256);
    k_loss_bwd<<<lb, 256, 256 * 8 * sizeof(float), st>>>(F.t[T_OUT], F.t[T_X], d_target, P0, F.t[T_G],
                                                         u.wg_ws.p + u.bias_off[13], u.loss.p);
    SALTY_TRY(bias_reduce_add(ctx, u, 13, lb, table));
    SALTY_TRY(back(13, x(T_D0, 32), H, W, T_G2));
    SALTY_TRY(plain(12, T_D0, H, W));
    SALTY_TRY(back(12, cat(T_D1, 48, T_E0, 32), H, W, T_C0));
    SALTY_TRY(up(11, T_D1, T_C0, 80, H1, W1));
    SALTY_TRY(back(11, cat(T_D2, 64, T_E1, 48), H1, W1, T_C1));
    SALTY_TRY(up(10, T_D2, T_C1, 112, H2, W2));
    SALTY_TRY(back(10, cat(T_D3, 80, T_E2, 64), H2, W2, T_C2));
    SALTY_TRY(up(9, T_D3, T_C2, 144, H3, W3));
    SALTY_TRY(back(9, cat(T_B, 96, T_E3, 80), H3, W3, T_C3));
    SALTY_TRY(up(8, T_B, T_C3, 176, H4, W4));
    SALTY_TRY(back(8, x(T_P3, 80), H4, W4, T_G2));
    SALTY_TRY(skip(7, T_E3, T_C3, 176, 96, H3, W3));
    SALTY_TRY(back(7, x(T_A3, 80), H3, W3, T_G2));
    SALTY_TRY(plain(6, T_A3, H3, W3));
    SALTY_TRY(back(6, x(T_P2, 64), H3, W3, T_G2));
    SALTY_TRY(skip(5, T_E2, T_C2, 144, 80, H2, W2));
    SALTY_TRY(back(5, x(T_A2, 64), H2, W2, T_G2));
    SALTY_TRY(plain(4, T_A2, H2, W2));
    SALTY_TRY(back(4, x(T_P1, 48), H2, W2, T_G2));
    SALTY_TRY(skip(3, T_E1, T_C1, 112, 64, H1, W1));
    SALTY_TRY(back(3, x(T_A1, 48), H1, W1, T_G2));
    SALTY_TRY(plain(2, T_A1, H1, W1));
    SALTY_TRY(back(2, x(T_P0, 32), H1, W1, T_G2));
    SALTY_TRY(skip(1, T_E0, T_C0, 80, 48, H, W));
    SALTY_TRY(back(1, x(T_A0, 32), H, W, T_G2));
    SALTY_TRY(plain(0, T_A0, H, W));
    SALTY_TRY(back(0, x(T_X, 16), H, W, -1));
    SALTY_TRY(grad_reduce_run(ctx, table));
    SALTY_TRY_CUDA(ctx->err, cudaGetLastError());
    double l = 0.0;
    SALTY_TRY_CUDA(ctx->err, cudaMemcpyAsync(&l, u.loss.p, sizeof(double), cudaMemcpyDeviceToHost, st));
    SALTY_TRY_CUDA(ctx->err, cudaStreamSynchronize(st));
    *loss = l / (3.0 * (double)P0);
    return SALTY_OK;
}

// Copies n floats of a host-or-device array to the device workspace at `off`.
salty_status stage(salty_ctx* ctx, Unet& u, const float* src, long long n, long long off, const float** out) {
    if (is_device_ptr(src)) {
        *out = src;
        return SALTY_OK;
    }
    SALTY_TRY_CUDA(ctx->err, cudaMemcpyAsync(u.io.p + off, src, n * sizeof(float), cudaMemcpyHostToDevice, ctx->stream));
    *out = u.io.p + off;
    return SALTY_OK;
}

// The tensor-core convolutions' status word: zeroed before a call's first launch, read
// after its last synchronisation.
salty_status conv_status_reset(salty_ctx* ctx) {
    SALTY_TRY_CUDA(ctx->err, cudaMemsetAsync(ctx->status.p + 8, 0, sizeof(int), ctx->stream));
    return SALTY_OK;
}
salty_status conv_status_check(salty_ctx* ctx) {
    int s = 0;
    SALTY_TRY_CUDA(ctx->err, cudaMemcpy(&s, ctx->status.p + 8, sizeof(int), cudaMemcpyDeviceToHost));
    if (s & 1) return ctx->err.fail(SALTY_ERR_TIMEOUT, "unet: a tensor-core convolution gave up waiting");
    if (s) return ctx->err.fail(SALTY_ERR_CUDA, "unet: a tensor-core convolution found its shared memory misaligned");
    return SALTY_OK;
}

salty_status check_shape(salty_ctx* ctx, int n, int h, int w) {
    if (n <= 0 || h <= 0 || w <= 0 || h % 16 || w % 16)
        return ctx->err.fail(SALTY_ERR_INVALID_ARG, "unet: n, h, w must be positive and h, w multiples of 16");
    if ((long long)n * h * w > (1ll << 26)) return ctx->err.fail(SALTY_ERR_CAPACITY, "unet: batch too large");
    return SALTY_OK;
}

}  // namespace
}  // namespace salty

struct salty_unet {
    salty::Unet net;
};

extern "C" {

salty_status salty_unet_create(salty_ctx* ctx, uint64_t seed, salty_unet** out) {
    using namespace salty;
    if (!ctx || !out) return SALTY_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    auto* h = new (std::nothrow) salty_unet();
    if (!h) return ctx->err.fail(SALTY_ERR_OOM, "host allocation failed");
    Unet& u = h->net;
    init_layers(u);
    long long wf = 0, wb = 0;
    for (const UnetLayer& L : u.layers) {
        wf = L.wf_off + 9LL * L.rows_fwd * L.cin;
        wb = L.wb_off + 9LL * L.rows_bwd * L.cout_pad;
    }
    auto fail = [&](salty_status s) { delete h; return s; };
    if (u.params.ensure(u.n_params) != cudaSuccess || u.grads.ensure(u.n_params) != cudaSuccess ||
        u.adam_m.ensure(u.n_params) != cudaSuccess || u.adam_v.ensure(u.n_params) != cudaSuccess ||
        u.wf.ensure(wf) != cudaSuccess || u.wb.ensure(wb) != cudaSuccess)
        return fail(ctx->err.fail(SALTY_ERR_OOM, "unet parameters"));
    // He-uniform weights from a PCG stream (seeded), zero biases
    std::vector<float> p(u.n_params, 0.0f);
    uint64_t s = seed + 1442695040888963407ull;
    auto next = [&]() {
        uint64_t old = s;
        s = old * 6364136223846793005ull + 1442695040888963407ull;
        uint32_t xs = (uint32_t)(((old >> 18) ^ old) >> 27), rot = (uint32_t)(old >> 59);
        return (float)((xs >> rot) | (xs << ((~rot + 1u) & 31u))) / 4294967296.0f;
    };
    for (size_t li = 0; li < u.layers.size(); ++li) {
        const UnetLayer& L = u.layers[li];
        const int real_cin = li == 0 ? kFeatures : L.cin;
        // the output layer starts small: the initial prediction is close to the input
        const float bound = std::sqrt(6.0f / (9.0f * real_cin)) * (L.relu ? 1.0f : 0.1f);
        for (long long i = 0; i < 9LL * L.cin * L.cout; ++i) {
            const int ci = (int)(i % L.cin);
            p[L.w_off + i] = (li == 0 && ci >= kFeatures) ? 0.0f : (2.0f * next() - 1.0f) * bound;
        }
    }
    cudaStream_t st = ctx->stream;
    if (cudaMemcpyAsync(u.params.p, p.data(), p.size() * sizeof(float), cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemsetAsync(u.adam_m.p, 0, u.n_params * sizeof(float), st) != cudaSuccess ||
        cudaMemsetAsync(u.adam_v.p, 0, u.n_params * sizeof(float), st) != cudaSuccess ||
        cudaMemsetAsync(u.wf.p, 0, wf * sizeof(bf16), st) != cudaSuccess ||
        cudaMemsetAsync(u.wb.p, 0, wb * sizeof(bf16), st) != cudaSuccess)
        return fail(ctx->err.fail(SALTY_ERR_CUDA, "unet init copies"));
    if (refresh_bf16(ctx, u) != SALTY_OK) return fail(SALTY_ERR_CUDA);
    if (cudaStreamSynchronize(st) != cudaSuccess) return fail(ctx->err.fail(SALTY_ERR_CUDA, "unet init"));
    *out = h;
    return SALTY_OK;
}

void salty_unet_destroy(salty_ctx* ctx, salty_unet* net) {
    if (ctx) {
        cudaSetDevice(ctx->device);
        cudaStreamSynchronize(ctx->stream);
    }
    delete net;
}

int64_t salty_unet_param_count(const salty_unet* net) { return net ? net->net.n_params : 0; }

salty_status salty_unet_get_params(salty_ctx* ctx, salty_unet* net, float* params, float* grads) {
    using namespace salty;
    if (!ctx || !net) return SALTY_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    Unet& u = net->net;
    if (params) SALTY_TRY_CUDA(ctx->err, cudaMemcpy(params, u.params.p, u.n_params * sizeof(float), cudaMemcpyDefault));
    if (grads) SALTY_TRY_CUDA(ctx->err, cudaMemcpy(grads, u.grads.p, u.n_params * sizeof(float), cudaMemcpyDefault));
    return SALTY_OK;
}

salty_status salty_unet_get_adam(salty_ctx* ctx, salty_unet* net, float* m, float* v, int64_t* step) {
    using namespace salty;
    if (!ctx || !net) return SALTY_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    Unet& u = net->net;
    if (m) SALTY_TRY_CUDA(ctx->err, cudaMemcpy(m, u.adam_m.p, u.n_params * sizeof(float), cudaMemcpyDefault));
    if (v) SALTY_TRY_CUDA(ctx->err, cudaMemcpy(v, u.adam_v.p, u.n_params * sizeof(float), cudaMemcpyDefault));
    if (step) *step = u.step;
    return SALTY_OK;
}

salty_status salty_unet_set_adam(salty_ctx* ctx, salty_unet* net, const float* m, const float* v, int64_t step) {
    using namespace salty;
    if (!ctx || !net || !m || !v || step < 0) return SALTY_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    Unet& u = net->net;
    SALTY_TRY_CUDA(ctx->err, cudaMemcpy(u.adam_m.p, m, u.n_params * sizeof(float), cudaMemcpyDefault));
    SALTY_TRY_CUDA(ctx->err, cudaMemcpy(u.adam_v.p, v, u.n_params * sizeof(float), cudaMemcpyDefault));
    u.step = step;
    return SALTY_OK;
}

salty_status salty_unet_set_params(salty_ctx* ctx, salty_unet* net, const float* params) {
    using namespace salty;
    if (!ctx || !net || !params) return SALTY_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    Unet& u = net->net;
    SALTY_TRY_CUDA(ctx->err, cudaMemcpy(u.params.p, params, u.n_params * sizeof(float), cudaMemcpyDefault));
    SALTY_TRY(refresh_bf16(ctx, u));
    SALTY_TRY_CUDA(ctx->err, cudaStreamSynchronize(ctx->stream));
    return SALTY_OK;
}

salty_status salty_unet_forward(salty_ctx* ctx, salty_unet* net, const float* features, int32_t n, int32_t h,
                                int32_t w, float* out_rgb) {
    using namespace salty;
    if (!ctx || !net || !features || !out_rgb) return SALTY_ERR_INVALID_ARG;
    SALTY_TRY(check_shape(ctx, n, h, w));
    cudaSetDevice(ctx->device);
    Unet& u = net->net;
    const long long P0 = (long long)n * h * w;
    SALTY_TRY_CUDA(ctx->err, u.io.ensure((size_t)P0 * 16));
    const float* df;
    SALTY_TRY(stage(ctx, u, features, P0 * kFeatures, 0, &df));
    SALTY_TRY(conv_status_reset(ctx));
    Fwd F;
    SALTY_TRY(forward(ctx, u, df, n, h, w, F));
    const bool dev_out = is_device_ptr(out_rgb);
    float* dout = dev_out ? out_rgb : u.io.p + P0 * kFeatures;
    k_output<<<gsz(P0), 256, 0, ctx->stream>>>(F.t[T_OUT], F.t[T_X], P0, dout);
    if (!dev_out)
        SALTY_TRY_CUDA(ctx->err, cudaMemcpyAsync(out_rgb, dout, P0 * 3 * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    SALTY_TRY_CUDA(ctx->err, cudaStreamSynchronize(ctx->stream));
    SALTY_TRY_CUDA(ctx->err, cudaGetLastError());
    return conv_status_check(ctx);
}

salty_status salty_unet_train_step(salty_ctx* ctx, salty_unet* net, const float* features, const float* target_rgb,
                                   int32_t n, int32_t h, int32_t w, float lr, float* loss) {
    using namespace salty;
    if (!ctx || !net || !features || !target_rgb) return SALTY_ERR_INVALID_ARG;
    SALTY_TRY(check_shape(ctx, n, h, w));
    cudaSetDevice(ctx->device);
    Unet& u = net->net;
    const long long P0 = (long long)n * h * w;
    SALTY_TRY_CUDA(ctx->err, u.io.ensure((size_t)P0 * 16));
    const float *df, *dt;
    SALTY_TRY(stage(ctx, u, features, P0 * kFeatures, 0, &df));
    SALTY_TRY(stage(ctx, u, target_rgb, P0 * 3, P0 * kFeatures, &dt));
    SALTY_TRY(conv_status_reset(ctx));
    Fwd F;
    SALTY_TRY(forward(ctx, u, df, n, h, w, F));
    double l = 0.0;
    SALTY_TRY(backward(ctx, u, F, dt, n, h, w, &l));
    if (loss) *loss = (float)l;
    if (lr > 0.0f) {
        ++u.step;
        AdamArgs a;
        a.lr = lr;
        a.b1 = 0.9f;
        a.b2 = 0.999f;
        a.eps = 1e-8f;
        a.c1 = (float)(1.0 / (1.0 - std::pow(0.9, (double)u.step)));
        a.c2 = (float)(1.0 / (1.0 - std::pow(0.999, (double)u.step)));
        k_adam<<<gsz(u.n_params), 256, 0, ctx->stream>>>(u.params.p, u.grads.p, u.adam_m.p, u.adam_v.p, u.n_params, a);
        SALTY_TRY(refresh_bf16(ctx, u));
    }
    SALTY_TRY_CUDA(ctx->err, cudaStreamSynchronize(ctx->stream));
    SALTY_TRY_CUDA(ctx->err, cudaGetLastError());
    return conv_status_check(ctx);
}

salty_status salty_denoise_unet_ensemble(salty_ctx* ctx, salty_unet* net, salty_scene* scene, int32_t mirrors,
                                        float* out_rgb) {
    using namespace salty;
    if (!ctx || !net || !scene || !out_rgb) return SALTY_ERR_INVALID_ARG;
    if (mirrors != 1 && mirrors != 2 && mirrors != 4 && mirrors != 8)
        return ctx->err.fail(SALTY_ERR_INVALID_ARG, "mirrors must be 1, 2, 4 or 8");
    cudaSetDevice(ctx->device);
    Unet& u = net->net;
    const Film& Fm = scene->film;
    const int W = Fm.width, H = Fm.height;
    if ((long long)W * H == 0 || Fm.samples == 0) return ctx->err.fail(SALTY_ERR_NOT_BUILT, "the film is empty");
    const int Wp = (W + 15) / 16 * 16, Hp = (H + 15) / 16 * 16;
    SALTY_TRY(check_shape(ctx, 1, Hp, Wp));
    const long long npx = (long long)W * H;
    // The symmetries run as batches of images of one shape: the mirror images (up to 4) in
    // one forward pass, their transposes in a second -- each convolution launch then has
    // that many times more strips to spread over the SMs.  An image's outputs do not depend
    // on the batch it runs in (tests/test_unet_gpu.py), and the images are added to the
    // result in the order k = 0..mirrors-1, as one pass per image would add them.
    const int per = mirrors < 4 ? mirrors : 4;
    SALTY_TRY(check_shape(ctx, per, Hp, Wp));
    // the film's input records (8 floats' worth of BF16 per pixel), then the image
    SALTY_TRY_CUDA(ctx->err, u.film_ws.ensure((size_t)npx * 11));
    uint4* rec = reinterpret_cast<uint4*>(u.film_ws.p);
    float* img = u.film_ws.p + npx * 8;
    SALTY_TRY(film_records(ctx, scene, rec));
    SALTY_TRY(conv_status_reset(ctx));
    for (int k0 = 0; k0 < mirrors; k0 += per) {
        FlipSet fs{per, {0, 0, 0, 0}};
        for (int j = 0; j < per; ++j) fs.flip[j] = k0 + j;
        const bool tr = (k0 & 4) != 0;  // the transposed frames: Hp wide, Wp tall
        const int h = tr ? Wp : Hp, w = tr ? Hp : Wp;
        SALTY_TRY(ensure_workspace(ctx, u, per, h, w));
        k_place_inputs<<<dim3((w / 16) * ((h + 7) / 8), per), 256, 0, ctx->stream>>>(
            rec, W, H, Wp, Hp, fs, reinterpret_cast<uint4*>(u.act.p + u.act_off[T_X]));
        Fwd F;
        SALTY_TRY(forward(ctx, u, nullptr, per, h, w, F));
        k_output_images<<<((W + 15) / 16) * ((H + 15) / 16), 256, 0, ctx->stream>>>(
            F.t[T_OUT], rec, W, H, Wp, Hp, fs, 1.0f / (float)mirrors, k0 == 0, img);
    }
    SALTY_TRY_CUDA(ctx->err, cudaGetLastError());
    SALTY_TRY_CUDA(ctx->err, cudaMemcpyAsync(out_rgb, img, (size_t)npx * 3 * sizeof(float), cudaMemcpyDefault,
                                             ctx->stream));
    SALTY_TRY_CUDA(ctx->err, cudaStreamSynchronize(ctx->stream));
    return conv_status_check(ctx);
}

salty_status salty_unet_set_conv_kernel(salty_ctx* ctx, salty_unet* net, int32_t kind) {
    if (!ctx || !net) return SALTY_ERR_INVALID_ARG;
    if (kind != SALTY_CONV_TCGEN05 && kind != SALTY_CONV_MMA_SYNC && kind != SALTY_CONV_TCGEN05_CP_ASYNC)
        return ctx->err.fail(SALTY_ERR_INVALID_ARG, "unknown convolution kernel %d", (int)kind);
    net->net.conv_kind = kind;
    return SALTY_OK;
}

salty_status salty_denoise_unet(salty_ctx* ctx, salty_unet* net, salty_scene* scene, float* out_rgb) {
    return salty_denoise_unet_ensemble(ctx, net, scene, 1, out_rgb);
}

}  // extern "C"

