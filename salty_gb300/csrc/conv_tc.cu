// conv_tc.cu -- the denoiser's 3x3 convolutions on the fifth-generation tensor cores.
//
// Implicit GEMM with the accumulators in tensor memory (TMEM).  One CTA computes a strip of
// R image rows x 128 pixels and all output channels:
//   M = 128 pixels of one image row (TMEM lane i holds pixel x0 + i),
//   N = output channels, padded to a multiple of 16 (16..256),
//   K = 9 taps x Cin, walked 16 input channels (one MMA's K) at a time.
// Operands sit in shared memory in the tensor core's K-major layout without swizzle: "core
// matrices" of 8 rows x 16 bytes (8 BF16 channels), 128 contiguous bytes each.  The
// descriptors' leading byte offset is the distance between the two 8-channel halves of K,
// the stride byte offset the distance between consecutive 8-row groups (128 B here).
//   halo  [2 channel octets][R + 2 rows][130 pixels][8 channels] -- output row r, tap
//         (ky, kx) reads the 128-pixel window starting at halo pixel (r + ky, kx), so the A
//         descriptor of every tap is the same tile with its start moved 16 B per pixel
//   wts   [9 taps][2 channel octets][Npad rows][8 channels]
// Both are staged per 16-channel chunk into one of two buffers with cp.async (zero fill
// outside the image and beyond the real output channels).  Lane 0 of each warp issues the
// chunk's MMAs for its rows (tcgen05.mma kind::f16, BF16 x BF16 -> FP32) and commits them
// to that buffer's mbarrier (4 arrivals); the loaders wait on it before refilling the
// buffer.  R x Npad <= 256
// FP32 accumulator columns are allocated per CTA.  Epilogue: tcgen05.ld of each row's
// columns, bias, ReLU, BF16, 16-byte stores.
//
// Every wait is bounded (2 s of the global timer); a wait that gives up sets
// status[0] |= 1, skips the rest of the strip, frees the CTA's TMEM and returns.
//
// k_conv3x3_tma is the same convolution as a persistent, warp-specialised kernel (one CTA per
// SM looping over strips):
//   warp 0    one lane issues TMA tensor copies (cp.async.bulk.tensor): per 16-channel
//             chunk the halo (a box of 16 channels x 130 pixels x R+2 rows, the image
//             border zero-filled by the copy engine) and the weights (per kx the three
//             vertical taps' Npad rows, one after the other) into a ring of up to 4 stages, each
//             guarded by a "full" (transaction bytes) and an "empty" (MMAs done) mbarrier.  A
//             layer whose weights fit in kResidentMaxBytes has them copied once, chunk by
//             chunk, into a region of their own, and its stages hold only halos.  Both land
//             in the tensor core's 32-byte-swizzled K-major layout: one 32-byte row per pixel
//             (or weight row), the two 16-byte halves of a row exchanged where address bit 7
//             is set.  The MMA unit undoes the exchange from the absolute shared-memory
//             address, so a tap's A operand still starts at any pixel of the halo (32-byte
//             steps, descriptor base offset 0) -- measured on this GPU with exact integer
//             products at row offsets 0-131.
//   warp 1    issues the MMAs.  A 128 x N x 16 MMA takes max(32 + N/4, N/2) cycles (measured:
//             its operands are read from shared memory at 128 bytes a cycle, 4 KB of pixels
//             and 32 N bytes of weights), so at N = 32 most of it is the pixel operand; the
//             vertical taps of one halo row therefore run as one MMA of N = up to 3 x Npad
//             whose columns are three neighbouring rows' accumulators (rows stored in
//             descending order, so ky ascends with the columns).  Every accumulator still sees
//             its products in the order chunk, ky, kx.  The whole warp stays converged and one
//             elected lane issues, which keeps the descriptors in uniform registers: issued
//             from a single diverged lane an MMA cost 233 cycles, and eight such lanes 46.
//   warps 2-9 the epilogue: TMEM -> bias, ReLU, BF16 -> global, two warps per TMEM lane
//             quarter, then release the accumulator; optionally also the 2x2 max-pooled
//             output (rows paired in the strip, columns by a shuffle)
//   warps 10-17 (decoder layers only) fill the chunks that come from the coarse level: each
//             coarse pixel is loaded once and stored to its up to four places in the
//             swizzled halo, so the up-sampled tensor is never written
// Two accumulators of R x Npad columns (512 TMEM columns) let the epilogue of one strip
// overlap the MMAs of the next.  Waits are bounded as above; a wait that gives up raises
// a shared abort flag that ends every role's loop.
// Measured (GB300; film denoise at 1080p, 8 symmetries as two batches of 4 images): all
// convolutions 5.81 -> 2.64 ms against one N = Npad MMA per tap and row from eight diverged
// lanes, with the decoder inputs staged by k_conv3x3_tc.  The full-resolution 32 -> 32 layer
// with its pooled output moves 1.2 GB in 196 us (6.1 TB/s, 0.90 of the copy peak); the
// decoder's up(48) + 32 -> 32 takes 310 us, bound by the MMAs' operand reads.
#include <cuda.h>  // CUtensorMap and its enums (the encoder is fetched from the driver at run time)
#include <cuda_bf16.h>

#include <cstdint>

#include "internal.h"
#include "unet_src.cuh"

namespace salty {
namespace {

using bf16 = __nv_bfloat16;

constexpr int kTcThreads = 128;
constexpr int kStrip = 128;              // pixels per image row of a strip (the MMA's M)
constexpr int kHaloW = kStrip + 2;       // staged pixels per halo row
constexpr int kTmemCols = 256;           // accumulator columns per CTA
constexpr int kBarBytes = 128;           // mbarriers + TMEM address at the start of shared memory
constexpr unsigned long long kWaitNs = 2000000000ull;

__host__ __device__ constexpr int halo_bytes(int R) { return 2 * (R + 2) * kHaloW * 16; }
__host__ __device__ constexpr int wts_bytes(int npad) { return 9 * 2 * npad * 16; }
__host__ __device__ constexpr int stage_bytes(int R, int npad) { return (halo_bytes(R) + wts_bytes(npad) + 127) / 128 * 128; }

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor: start, leading and stride byte offsets (all >> 4), the
// descriptor version bit of this architecture (bit 46), no swizzle.
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor, kind::f16: FP32 accumulator (bits 4-5 = 1), A and B BF16
// (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__device__ __forceinline__ uint32_t idesc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
        :: "r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}

// Waits for the phase with the given parity to complete; false after kWaitNs.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    if (mbar_try(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    while (!mbar_try(bar, parity))
        if (global_ns() - t0 > kWaitNs) return false;
    return true;
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// The same load without its wait, and the wait, which the values depend on.
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :: "memory");
}

struct TcConvArgs {
    ConvSrc src;           // the input's channels (one tensor, or [up2(coarse) | skip])
    int cin;               // cin % 16 == 0
    const bf16* wt;        // [9][wrows][cin]
    int wrows;
    const float* bias;     // [cout] or null
    bf16* out;
    int out_cs, out_co, cout;
    int npad, R;           // MMA N (cout rounded up to 16) and image rows per strip
    int N, H, W, relu;
    int* status;
};

__global__ void __launch_bounds__(kTcThreads, 1) k_conv3x3_tc(const TcConvArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);           // [2] chunk buffers consumed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + 16);
    unsigned char* stage0 = smem + kBarBytes;
    const int R = a.R, npad = a.npad;
    const int sbytes = stage_bytes(R, npad), hbytes = halo_bytes(R);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    const int strips_x = (a.W + kStrip - 1) / kStrip, strips_y = (a.H + R - 1) / R;
    int t = blockIdx.x;
    const int sx = t % strips_x;
    t /= strips_x;
    const int sy = t % strips_y;
    const int n = t / strips_y;
    const int x0 = sx * kStrip, y0 = sy * R;

    if (tid == 0) {  // one commit per warp's issuing thread
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(saddr(bars + 0)), "n"(kTcThreads / 32) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(saddr(bars + 1)), "n"(kTcThreads / 32) : "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(saddr(tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }

    // stages chunk c (input channels 16c .. 16c + 15) into buffer b
    const int hrow = (R + 2) * kHaloW;
    auto load = [&](int c, int b) {
        unsigned char* hs = stage0 + b * sbytes;
        unsigned char* ws = hs + hbytes;
        const int c0 = c * 16;
        for (int i = tid; i < 2 * hrow; i += kTcThreads) {
            const int k8 = i & 1, p = i >> 1;             // neighbouring threads: the two octets of a pixel
            const int hy = p / kHaloW, hx = p - hy * kHaloW;
            const int gy = y0 - 1 + hy, gx = x0 - 1 + hx;
            const bool ok = gy >= 0 && gy < a.H && gx >= 0 && gx < a.W;
            const bf16* src = ok ? src_at(a.src, n, gy, gx, a.H, a.W, c0 + k8 * 8) : a.src.a;
            cp_async16(saddr(hs + (k8 * hrow + p) * 16), src, ok ? 16u : 0u);
        }
        const int live = a.cout < a.wrows ? a.cout : a.wrows;
        for (int i = tid; i < 9 * 2 * npad; i += kTcThreads) {
            const int k8 = i & 1, q = i >> 1;
            const int tap = q / npad, row = q - tap * npad;
            const bool ok = row < live;
            const bf16* src = ok ? a.wt + ((size_t)tap * a.wrows + row) * a.cin + c0 + k8 * 8 : a.wt;
            cp_async16(saddr(ws + ((tap * 2 + k8) * npad + row) * 16), src, ok ? 16u : 0u);
        }
    };

    const int nchunks = a.cin / 16;
    load(0, 0);
    cp_async_commit();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();  // barriers initialised, TMEM address written
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    const uint32_t idesc = idesc_bf16(kStrip, npad);
    bool failed = false;
    for (int c = 0; c < nchunks; ++c) {
        const int b = c & 1;
        if (c + 1 < nchunks) {
            bool ok = true;
            if (c >= 1) ok = mbar_wait(saddr(bars + (b ^ 1)), ((c - 1) >> 1) & 1);  // chunk c-1's MMAs are done
            if (__syncthreads_or(!ok)) {
                failed = true;
                break;
            }
            load(c + 1, b ^ 1);
            cp_async_commit();
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // cp.async data -> tensor core reads
        __syncthreads();
        if (lane == 0) {  // four issuing threads, one per warp: rows r = warp, warp + 4, ...
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t hs = saddr(stage0 + b * sbytes), ws = hs + hbytes;
            const uint32_t lbo_a = (uint32_t)hrow * 16, lbo_b = (uint32_t)npad * 16;
            for (int tap = 0; tap < 9; ++tap) {
                const int ky = tap / 3, kx = tap - ky * 3;
                const uint64_t bd = sdesc(ws + tap * 2 * npad * 16, lbo_b, 128);
                for (int r = warp; r < R; r += kTcThreads / 32) {
                    const uint64_t ad = sdesc(hs + ((r + ky) * kHaloW + kx) * 16, lbo_a, 128);
                    umma_bf16(tmem + r * npad, ad, bd, idesc, (c > 0 || tap > 0) ? 1u : 0u);
                }
            }
            umma_commit(saddr(bars + b));
        }
    }
    cp_async_wait<0>();
    // the last commit completes when every MMA issued before it has
    bool ok = !failed && mbar_wait(saddr(bars + ((nchunks - 1) & 1)), ((nchunks - 1) >> 1) & 1);
    if (__syncthreads_or(!ok)) failed = true;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (!failed) {
        const int x = x0 + warp * 32 + lane;
        for (int r = 0; r < R; ++r) {
            const int y = y0 + r;
            for (int j = 0; j < npad / 16; ++j) {
                uint32_t v[16];
                tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + r * npad + j * 16, v);
                if (y >= a.H || x >= a.W) continue;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int co = j * 16 + h * 8;
                    if (co >= a.cout) continue;
                    uint32_t pk[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        float v0 = __uint_as_float(v[h * 8 + 2 * e]), v1 = __uint_as_float(v[h * 8 + 2 * e + 1]);
                        if (a.bias) { v0 += a.bias[co + 2 * e]; v1 += a.bias[co + 2 * e + 1]; }
                        if (a.relu) { v0 = fmaxf(v0, 0.0f); v1 = fmaxf(v1, 0.0f); }
                        const __nv_bfloat162 p2 = __floats2bfloat162_rn(v0, v1);
                        pk[e] = *reinterpret_cast<const uint32_t*>(&p2);
                    }
                    *reinterpret_cast<uint4*>(a.out + (((size_t)n * a.H + y) * a.W + x) * a.out_cs + a.out_co + co) =
                        make_uint4(pk[0], pk[1], pk[2], pk[3]);
                }
            }
        }
    } else if (tid == 0) {
        atomicOr(a.status, 1);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(kTmemCols) : "memory");
}

// ---------------------------------------------------------------- persistent TMA kernel
constexpr int kMaxStages = 4;
constexpr int kTmaMmaWarps = 1;
constexpr int kTmaEpiWarps = 8;            // two per TMEM lane quarter
constexpr int kTmaCoarseWarps = 8;         // expand the coarse level (decoder layers)
constexpr int kTmaThreads = 32 * (1 + kTmaMmaWarps + kTmaEpiWarps);
constexpr int kTmaMaxChunks = 16;          // input channel chunks with their own weight barrier
constexpr int kTmaHeader = 2048;   // barriers, TMEM address, abort flag, bias
constexpr int kTmaMinSmem = 120 * 1024;  // above half an SM's shared memory: one CTA per SM owns all 512 TMEM columns
constexpr int kResidentMaxBytes = 100 * 1024;  // weights kept resident up to this size

__host__ __device__ constexpr int tma_halo(int R) { return ((R + 2) * kHaloW * 32 + 1023) / 1024 * 1024; }
__host__ __device__ constexpr int tma_wts(int npad) { return (9 * npad * 32 + 1023) / 1024 * 1024; }
__host__ __device__ constexpr int tma_stage(int R, int npad) { return tma_halo(R) + tma_wts(npad); }

// Shared-memory descriptor of a K-major operand in the 32-byte swizzle: rows of 32 bytes,
// 8-row groups 256 bytes apart (stride byte offset), leading byte offset unused (1), base
// offset 0, layout type 6 (bits 61-63).
__device__ __forceinline__ uint64_t sdesc_sw32(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(256u >> 4) << 32) | (1ull << 46) | (6ull << 61);
}

struct TmaConvArgs {
    int cin, npad, R, cout, relu, out_cs;
    int N, H, W, tiles, stages;
    int resident, wres;  // weights staged once for the whole kernel; bytes reserved for them
    const float* bias;
    bf16* out;
    bf16* pool;          // 2x2 max-pooled output [N][H/2][W/2][out_cs] or null (R even then)
    const bf16* coarse;  // decoder layers: input channels [0, coarse_ch) at half resolution
    int coarse_cs, coarse_ch;
    int* status;
};

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        :: "r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar) : "memory");
}

// Bounded wait that also gives up when another role has raised the abort flag.
__device__ __forceinline__ bool wait_or_abort(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status) {
    if (mbar_try(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    for (;;) {
        if (mbar_try(bar, parity)) return true;
        if (*abort_flag) return false;
        if (global_ns() - t0 > kWaitNs) {
            *abort_flag = 1;
            atomicOr(status, 1);
            return false;
        }
    }
}

// One lane of the converged warp (always the same one).
__device__ __forceinline__ uint32_t elect_lane() {
    uint32_t e;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(e));
    return e;
}

// An MMA issued by the elected lane of a converged warp; descriptors as their low words and
// the common high word.
__device__ __forceinline__ void umma_elect(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t desc_hi, uint32_t idesc,
                                           uint32_t elected, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred q, p;\n.reg .b64 a, b;\nsetp.ne.b32 q, %5, 0;\nsetp.ne.b32 p, %6, 0;\n"
        "mov.b64 a, {%1, %3};\nmov.b64 b, {%2, %3};\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p;\n}\n"
        :: "r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(elected), "r"(accumulate));
}
__device__ __forceinline__ void umma_commit_elect(uint32_t bar, uint32_t elected) {
    asm volatile(
        "{\n.reg .pred q;\nsetp.ne.b32 q, %1, 0;\n"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n"
        :: "r"(bar), "r"(elected) : "memory");
}
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status) {
    return __all_sync(0xffffffffu, wait_or_abort(bar, parity, abort_flag, status));
}

// 16 BF16 channels of a pixel (32-byte aligned) or 8 of them
__device__ __forceinline__ void store_pixel16(bf16* p, const uint32_t (&v)[8], bool full) {
    if (full)
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                     :: "l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                     : "memory");
    else
        *reinterpret_cast<uint4*>(p) = make_uint4(v[0], v[1], v[2], v[3]);
}

struct TmaHeader {
    uint64_t full[kMaxStages], empty[kMaxStages];
    uint64_t acc_full[2], acc_empty[2];
    uint64_t wbar[kTmaMaxChunks];  // a resident chunk's weights landed
    uint32_t tmem;
    int abort_flag;
};
static_assert(sizeof(TmaHeader) <= 512, "the bias table starts at byte 512");

template <bool COARSE>
__global__ void __launch_bounds__(kTmaThreads + (COARSE ? 32 * kTmaCoarseWarps : 0), 1)
k_conv3x3_tma(const __grid_constant__ CUtensorMap tm_in, const __grid_constant__ CUtensorMap tm_w, const TmaConvArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    TmaHeader& hd = *reinterpret_cast<TmaHeader*>(smem);
    volatile int* abort_flag = &hd.abort_flag;
    float* sbias = reinterpret_cast<float*>(smem + 512);  // [npad]
    unsigned char* wres = smem + kTmaHeader;
    unsigned char* ring = smem + kTmaHeader + a.wres;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    // TMA destinations and the descriptors below assume a 1024-byte aligned base
    if (saddr(smem) & 1023u) {
        grid_turn();
        if (tid == 0) atomicOr(a.status, 2);
        return;
    }
    constexpr int kFullCount = COARSE ? kTmaCoarseWarps : 1;  // arrivals per "full" phase
    const int R = a.R, npad = a.npad, S = a.stages;
    const int hbytes = tma_halo(R), sbytes = a.resident ? tma_halo(R) : tma_stage(R, npad);
    const uint32_t wchunk = 9u * npad * 32u;                  // one chunk's weights
    const uint32_t halo_tx = (uint32_t)(R + 2) * kHaloW * 32u;
    const int nchunks = a.cin / 16, ncoarse = COARSE ? a.coarse_ch / 16 : 0;
    const int strips_x = (a.W + kStrip - 1) / kStrip, strips_y = (a.H + R - 1) / R;
    if (tid == 0) {
        for (int s = 0; s < kMaxStages; ++s) {
            mbar_init(saddr(hd.full + s), kFullCount);
            mbar_init(saddr(hd.empty + s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(saddr(hd.acc_full + b), 1);
            mbar_init(saddr(hd.acc_empty + b), kTmaEpiWarps);
        }
        for (int c = 0; c < kTmaMaxChunks; ++c) mbar_init(saddr(hd.wbar + c), 1);
        hd.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" :: "r"(saddr(&hd.tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    grid_turn();
    for (int i = tid; i < npad; i += blockDim.x) sbias[i] = (a.bias && i < a.cout) ? a.bias[i] : 0.0f;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, hd.tmem, 0);

    // weights of chunk c: per kx the three vertical taps' rows
    auto load_weights = [&](uint32_t dst, int c, uint32_t bar) {
        for (int kx = 0; kx < 3; ++kx) tma_load_4d(dst + kx * 3 * npad * 32, &tm_w, c * 16, 0, kx, 0, bar);
    };

    if (warp == 0) {
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" :: "l"(reinterpret_cast<uint64_t>(&tm_in)) : "memory");
            asm volatile("prefetch.tensormap [%0];" :: "l"(reinterpret_cast<uint64_t>(&tm_w)) : "memory");
            int s = 0;
            uint32_t ph = 0;
            auto next = [&]() { if (++s == S) { s = 0; ph ^= 1u; } };
            for (int t = blockIdx.x; t < a.tiles; t += gridDim.x) {
                int tt = t;
                const int sx = tt % strips_x;
                tt /= strips_x;
                const int sy = tt % strips_y;
                const int n = tt / strips_y;
                const int x0 = sx * kStrip, y0 = sy * R;
                bool ok = true;
                for (int c = 0; c < nchunks; ++c, next()) {
                    if (a.resident && t == (int)blockIdx.x) {  // the chunk's weights, once
                        const uint32_t wb = saddr(hd.wbar + c);
                        mbar_expect_tx(wb, wchunk);
                        load_weights(saddr(wres) + c * wchunk, c, wb);
                    }
                    // every chunk's stage is waited for, whoever fills it: a parity tells two
                    // successive uses of a stage apart, not a use from the next but one
                    if (!wait_or_abort(saddr(hd.empty + s), ph ^ 1u, abort_flag, a.status)) { ok = false; break; }
                    if (c < ncoarse) continue;  // filled by the coarse warps
                    const uint32_t bar = saddr(hd.full + s);
                    mbar_expect_tx(bar, halo_tx + (a.resident ? 0u : wchunk));
                    const uint32_t dst = saddr(ring + s * sbytes);
                    tma_load_4d(dst, &tm_in, c * 16 - (COARSE ? a.coarse_ch : 0), x0 - 1, y0 - 1, n, bar);
                    if (!a.resident) load_weights(dst + hbytes, c, bar);
                    for (int i = 1; i < kFullCount; ++i) mbar_arrive(bar);
                }
                if (!ok) break;
            }
        }
    } else if (warp == 1) {
        const uint32_t el = elect_lane();
        const uint64_t d0 = sdesc_sw32(0);
        const uint32_t dlo = (uint32_t)d0, dhi = (uint32_t)(d0 >> 32);
        const uint32_t idesc = idesc_bf16(kStrip, 0), nbit = (uint32_t)(npad >> 3) << 17;  // + n * nbit: N = n * npad
        int s = 0, i = 0;
        uint32_t ph = 0;  // parity of the ring position's use
        for (int t = blockIdx.x; t < a.tiles; t += gridDim.x, ++i) {
            const int ab = i & 1;
            if (!warp_wait(saddr(hd.acc_empty + ab), ((uint32_t)(i >> 1) & 1u) ^ 1u, abort_flag, a.status)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = tmem + (uint32_t)ab * 256u;  // row r in columns (R - 1 - r) npad ..
            bool ok = true;
            for (int c = 0; c < nchunks; ++c) {
                if (a.resident && i == 0) ok = warp_wait(saddr(hd.wbar + c), 0u, abort_flag, a.status);
                if (!ok || !warp_wait(saddr(hd.full + s), ph, abort_flag, a.status)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t hs = saddr(ring + s * sbytes);
                const uint32_t ws = a.resident ? saddr(wres) + c * wchunk : hs + hbytes;
                const uint32_t a0 = dlo + (hs >> 4), b0 = dlo + (ws >> 4);
                for (int h = 0; h < R + 2; ++h) {
                    // halo row h is tap ky of output row h - ky
                    const int ky0 = h < R ? 0 : h - R + 1, n = (h < 2 ? h : 2) - ky0 + 1;
                    const uint32_t col = acc + (uint32_t)((R - 1 - h + ky0) * npad);
                    const uint32_t ah = a0 + (uint32_t)(h * kHaloW) * 2u, bh = b0 + (uint32_t)(ky0 * npad) * 2u;
                    const uint32_t kxs = (uint32_t)(3 * npad) * 2u;
                    if (c == 0 && ky0 == 0) {  // row h's first products overwrite its columns
                        umma_elect(col, ah, bh, dhi, idesc + nbit, el, 0u);
                        if (n > 1)
                            umma_elect(col + npad, ah, bh + (uint32_t)npad * 2u, dhi, idesc + (uint32_t)(n - 1) * nbit, el, 1u);
                    } else {
                        umma_elect(col, ah, bh, dhi, idesc + (uint32_t)n * nbit, el, 1u);
                    }
                    umma_elect(col, ah + 2u, bh + kxs, dhi, idesc + (uint32_t)n * nbit, el, 1u);
                    umma_elect(col, ah + 4u, bh + 2u * kxs, dhi, idesc + (uint32_t)n * nbit, el, 1u);
                }
                umma_commit_elect(saddr(hd.empty + s), el);
                if (++s == S) { s = 0; ph ^= 1u; }
            }
            if (!ok) break;
            umma_commit_elect(saddr(hd.acc_full + ab), el);
        }
    } else if (!COARSE || warp < 2 + kTmaEpiWarps) {
        // The operand reads of the MMAs keep shared memory busy, so a load from it takes hundreds
        // of cycles here: the bias stays in registers for a strip's rows of 16 channels.
        const int q = warp & 3, sub = (warp - 2) >> 2;  // TMEM lane quarter; which of its two warps
        const int J = npad / 16;
        // the quarter's two warps share the rows (pooled: row pairs), or the channels of a single one
        const int rstep = a.pool ? 2 : 1, units = R / rstep;
        const int u0 = units > 1 ? sub : 0, ustep = units > 1 ? 2 : 1, j0 = units > 1 ? 0 : sub, jstep = units > 1 ? 1 : 2;
        int i = 0;
        for (int t = blockIdx.x; t < a.tiles; t += gridDim.x, ++i) {
            const int ab = i & 1;
            if (!warp_wait(saddr(hd.acc_full + ab), (uint32_t)(i >> 1) & 1u, abort_flag, a.status)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            int tt = t;
            const int sx = tt % strips_x;
            tt /= strips_x;
            const int sy = tt % strips_y;
            const int n = tt / strips_y;
            const int x = sx * kStrip + q * 32 + lane;
            const uint32_t acc = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)ab * 256u;
            bf16* const orow = a.out + (((size_t)n * a.H + sy * R) * a.W + x) * a.out_cs;
            const size_t rpitch = (size_t)a.W * a.out_cs;
            for (int j = j0; j < J; j += jstep) {
                float bias[16];
                const float4* b4 = reinterpret_cast<const float4*>(sbias + j * 16);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float4 b = b4[e];
                    bias[4 * e] = b.x; bias[4 * e + 1] = b.y; bias[4 * e + 2] = b.z; bias[4 * e + 3] = b.w;
                }
                const bool live = x < a.W && j * 16 < a.cout, full = j * 16 + 16 <= a.cout;
                auto finish = [&](const uint32_t (&v)[16], int r, uint32_t (&pk)[8]) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        float f0 = __uint_as_float(v[2 * e]) + bias[2 * e], f1 = __uint_as_float(v[2 * e + 1]) + bias[2 * e + 1];
                        if (a.relu) { f0 = fmaxf(f0, 0.0f); f1 = fmaxf(f1, 0.0f); }
                        const __nv_bfloat162 p2 = __floats2bfloat162_rn(f0, f1);
                        pk[e] = *reinterpret_cast<const uint32_t*>(&p2);
                    }
                    if (live && sy * R + r < a.H) store_pixel16(orow + r * rpitch + j * 16, pk, full);
                };
                const uint32_t col = acc + (uint32_t)((R - 1) * npad + j * 16);  // row r: npad columns further down each
                if (a.pool) {
                    for (int r = 2 * u0; r < R; r += 2 * ustep) {
                        uint32_t v0[16], v1[16], p0[8], p1[8];
                        tmem_ld16_issue(col - (uint32_t)(r * npad), v0);
                        tmem_ld16_issue(col - (uint32_t)((r + 1) * npad), v1);
                        tmem_ld_wait(v0);
                        tmem_ld_wait(v1);
                        finish(v0, r, p0);
                        finish(v1, r + 1, p1);
                        const int y = sy * R + r;
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            __nv_bfloat162 m = __hmax2(*reinterpret_cast<__nv_bfloat162*>(&p0[e]),
                                                       *reinterpret_cast<__nv_bfloat162*>(&p1[e]));
                            const uint32_t o = __shfl_xor_sync(0xffffffffu, *reinterpret_cast<uint32_t*>(&m), 1);
                            m = __hmax2(m, *reinterpret_cast<const __nv_bfloat162*>(&o));
                            p0[e] = *reinterpret_cast<uint32_t*>(&m);
                        }
                        if (live && y < a.H && !(lane & 1))
                            store_pixel16(a.pool + (((size_t)n * (a.H / 2) + y / 2) * (a.W / 2) + x / 2) * a.out_cs + j * 16,
                                          p0, full);
                    }
                } else {
                    for (int r = u0; r < R; r += 2 * ustep) {  // two rows' loads in flight
                        const int r1 = r + ustep;
                        uint32_t v0[16], v1[16], pk[8];
                        tmem_ld16_issue(col - (uint32_t)(r * npad), v0);
                        if (r1 < R) tmem_ld16_issue(col - (uint32_t)(r1 * npad), v1);
                        tmem_ld_wait(v0);
                        finish(v0, r, pk);
                        if (r1 < R) {
                            tmem_ld_wait(v1);
                            finish(v1, r1, pk);
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(saddr(hd.acc_empty + ab));
        }
    } else {
        // coarse chunks: halo pixel (hy, hx) shows coarse pixel ((y0 - 1 + hy) >> 1, (x0 - 1 + hx) >> 1)
        constexpr int kJobs = 4;  // coarse pixel halves per thread: up to 6 rows x 66 pixels x 2 halves / 256 threads
        constexpr int kCoarseW = kStrip / 2 + 2;
        const int ct = tid - kTmaThreads;
        const int Hc = a.H >> 1, Wc = a.W >> 1;
        int s = 0;
        uint32_t ph = 0;
        for (int t = blockIdx.x; t < a.tiles; t += gridDim.x) {
            int tt = t;
            const int sx = tt % strips_x;
            tt /= strips_x;
            const int sy = tt % strips_y;
            const int n = tt / strips_y;
            const int x0 = sx * kStrip, y0 = sy * R;
            const int cy0 = (y0 - 1) >> 1, cx0 = (x0 - 1) >> 1, ncy = ((y0 + R) >> 1) - cy0 + 1;
            // this strip's coarse pixels (-1: outside the image) and the places of their copies (-1: none)
            int from[kJobs], to[kJobs][4];
#pragma unroll
            for (int u = 0; u < kJobs; ++u) {
                const int i = ct + u * 32 * kTmaCoarseWarps, half = i & 1, p = i >> 1, ry = p / kCoarseW, rx = p % kCoarseW;
                const int cy = cy0 + ry, cx = cx0 + rx;
                from[u] = ry < ncy && cy >= 0 && cy < Hc && cx >= 0 && cx < Wc ? (cy * Wc + cx) * a.coarse_cs + half * 8 : -1;
                const int hy0 = 2 * cy - (y0 - 1), hx0 = 2 * cx - (x0 - 1);
#pragma unroll
                for (int d = 0; d < 4; ++d) {
                    // pairs of pixels swap their left and right copies, so that a warp's 512 bytes cover all banks
                    const int hy = hy0 + (d >> 1), hx = hx0 + ((d ^ (p >> 1)) & 1), px = hy * kHaloW + hx;
                    const bool in = ry < ncy && hy >= 0 && hy < R + 2 && hx >= 0 && hx < kHaloW;
                    to[u][d] = in ? px * 32 + ((half ^ ((px >> 2) & 1)) << 4) : -1;
                }
            }
            const bf16* img = a.coarse + (size_t)n * Hc * Wc * a.coarse_cs;
            bool ok = true;
            for (int c = 0; c < nchunks; ++c) {
                const bool mine = c < ncoarse;  // the others are filled by TMA; waited for here too (see warp 0)
                uint4 v[kJobs];
                if (mine) {
#pragma unroll
                    for (int u = 0; u < kJobs; ++u)
                        v[u] = from[u] >= 0 ? *reinterpret_cast<const uint4*>(img + from[u] + c * 16) : make_uint4(0, 0, 0, 0);
                }
                if (!warp_wait(saddr(hd.empty + s), ph ^ 1u, abort_flag, a.status)) { ok = false; break; }
                if (mine) {
                    const uint32_t bar = saddr(hd.full + s);
                    unsigned char* dst = ring + s * sbytes;
                    if (!a.resident && ct == 0) {
                        asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" :: "r"(bar), "r"(wchunk) : "memory");
                        load_weights(saddr(dst + hbytes), c, bar);
                    }
#pragma unroll
                    for (int u = 0; u < kJobs; ++u)
#pragma unroll
                        for (int d = 0; d < 4; ++d)
                            if (to[u][d] >= 0) *reinterpret_cast<uint4*>(dst + to[u][d]) = v[u];
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // these stores -> tensor core reads
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar);
                }
                if (++s == S) { s = 0; ph ^= 1u; }
            }
            if (!ok) break;
        }
    }
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" :: "r"(tmem) : "memory");
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn tensor_map_encoder() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
        else
            cudaGetLastError();
    }
    return fn;
}

// ---------------------------------------------------------------- weight gradient
// dW[tap][co][ci] = sum over pixels p of dY[p][co] * X[p + d(tap)][ci]: per tap a GEMM on
// the tensor cores with the pixels as its K dimension,
//   M = output channels (dY transposed; 64 rows when they fit, else 128, of which cout
//       are real),
//   N = 16 input channels at a row's three horizontal taps (48), for each vertical tap and
//       16-channel box of a CTA group's share of up to 48 channels: up to 9 x 48 <= 512 TMEM
//       columns,
//   K = pixels: a strip of kWgRows image rows x 64 pixels per stage, 16 per MMA.
// A stage holds the strip's dY (boxes of 16 channels x 64 pixels x kWgRows rows) and the
// input's halo (boxes of 16 channels x 66 pixels x kWgRows + 2 rows), both copied by TMA in
// the 32-byte swizzle, which is the tensor core's MN-major layout: one 32-byte row (16
// channels) per pixel, 8-pixel groups 256 bytes apart (stride byte offset), the next 16
// channels one box further (leading byte offset).  The B operand of vertical tap ky is the same
// halo from row r + ky, and its three 16-column groups, the horizontal taps, lie one pixel apart
// (a leading byte offset of 32) -- the copy engine has zero-filled the image border -- so the input
// is read once per strip, not once per tap, and dY once per vertical tap: an MMA costs its
// operand reads, 16 + N / 4 cycles at M = 64, so a 32-channel chunk takes 6 x 28 instead of the
// 9 x 24 of one MMA per tap (gradients of 16 x 256 x 256: a training step 1,436 -> 1,410 us).  CTAs of a group split
// the strips between them (K-split): each writes its partial sums to its own slice of a
// workspace, and k_grad_reduce adds the slices in a fixed order -- the result does not depend on
// scheduling, unlike atomics.
//
// Warp roles: one lane of warp 0 issues the TMA copies of each strip into a ring of
// kWgStages buffers (a "full" barrier per buffer counts the bytes), warp 1, converged, issues
// the MMAs from one elected lane (a diverged lane took about 75 cycles per MMA against 28 of
// operand reads at M = 64, N = 48; gradients of 16 x 256 x 256: 2.81 -> 2.38 ms) and commits them to the buffer's "empty" barrier, and after the last
// strip to the accumulator barrier; then all four warps move the accumulators from TMEM to
// this CTA's slice.  Every wait is bounded.
constexpr int kWgStrip = 64;
constexpr int kWgRows = 2;
constexpr int kWgHaloW = kWgStrip + 2;
constexpr int kWgChunk = 48;
constexpr int kWgStages = 3;
constexpr int kWgThreads = 128;
constexpr int kWgCoarseWarps = 8;  // warps 2 .. 9 of a decoder layer's blocks expand the coarse level
constexpr int kWgCoarseThreads = 64 + 32 * kWgCoarseWarps;
constexpr int kWgHeader = 1024;
constexpr int kWgDyBox = kWgRows * kWgStrip * 32;                                   // 16 channels
constexpr int kWgXBox = ((kWgRows + 2) * kWgHaloW * 32 + 1023) / 1024 * 1024;  // 16 channels, padded
constexpr int kWgStage = 8 * kWgDyBox + (kWgChunk / 16) * kWgXBox;  // dY sized for M = 128 rows

// Descriptor of an MN-major operand in the 32-byte swizzle: 16-element atoms `lbo` bytes
// apart, 8-row groups 256 bytes apart, layout type 6.
__device__ __forceinline__ uint64_t sdesc_sw32_mn(uint32_t addr, uint32_t lbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)(256u >> 4) << 32) | (1ull << 46) | (6ull << 61);
}

// Instruction descriptor, kind::f16: FP32 accumulator, BF16 A and B, both MN-major
// (transpose bits 15 and 16), N >> 3 at bit 17, M >> 4 at bit 24.
__device__ __forceinline__ uint32_t idesc_bf16_mn(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(m >> 4) << 24);
}

struct WgradArgs {
    int m;        // MMA rows: 128, or 64 when the output channels (cpad) fit
    int cpad, cout, cin, N, H, W;
    int strips;   // N * ceil(H / kWgRows) * ceil(W / kWgStrip)
    float* part;  // [gridDim.x slices][9][cpad][cin]
    const bf16* coarse;  // decoder layers: input channels [0, coarse_ch) at half resolution
    int coarse_cs, coarse_ch;
    int* status;
};

__global__ void __launch_bounds__(kWgCoarseThreads, 1)
k_wgrad_tc(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_dy, const WgradArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);  // [kWgStages]
    uint64_t* empty = full + kWgStages;                  // [kWgStages]
    uint64_t* acc = empty + kWgStages;                   // [1]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + 128);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + 132);
    unsigned char* stage0 = smem + kWgHeader;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    if (saddr(smem) & 1023u) {  // the swizzled boxes need 1 KB aligned destinations
        grid_turn();
        if (tid == 0) atomicOr(a.status, 2);
        return;
    }
    const int c0 = blockIdx.y * kWgChunk;                    // this group's input channels
    const int ch = min(kWgChunk, a.cin - c0);               // 16, 32 or 48
    const int ndy = a.cpad / 16, nx = ch / 16;
    const int ncx = min(max(a.coarse_ch - c0, 0), ch) / 16;  // boxes expanded from the coarse level, before the others
    const int sx = (a.W + kWgStrip - 1) / kWgStrip, sy = (a.H + kWgRows - 1) / kWgRows;
    const int first = blockIdx.x;
    const int count = first < a.strips ? (a.strips - 1 - first) / (int)gridDim.x + 1 : 0;

    if (tid == 0) {
        for (int k = 0; k < kWgStages; ++k) {
            mbar_init(saddr(full + k), ncx ? 1 + kWgCoarseWarps : 1);  // the TMA thread, and the expanding warps
            mbar_init(saddr(empty + k), 1);
        }
        mbar_init(saddr(acc), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" :: "r"(saddr(tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    grid_turn();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);

    bool ok = true;
    if (warp == 0 && lane == 0) {
        asm volatile("prefetch.tensormap [%0];" :: "l"(reinterpret_cast<uint64_t>(&tm_x)) : "memory");
        asm volatile("prefetch.tensormap [%0];" :: "l"(reinterpret_cast<uint64_t>(&tm_dy)) : "memory");
        const uint32_t tx = (uint32_t)ndy * kWgDyBox + (uint32_t)(nx - ncx) * ((kWgRows + 2) * kWgHaloW * 32);
        for (int it = 0; it < count; ++it) {
            const int b = it % kWgStages;
            if (!wait_or_abort(saddr(empty + b), ((uint32_t)(it / kWgStages) & 1u) ^ 1u, abort_flag, a.status)) {
                ok = false;
                break;
            }
            const int s = first + it * (int)gridDim.x;
            const int xs = s % sx, t = s / sx;
            const int y0 = (t % sy) * kWgRows, n = t / sy;
            const int x0 = xs * kWgStrip;
            const uint32_t bar = saddr(full + b);
            mbar_expect_tx(bar, tx);
            const uint32_t dyb = saddr(stage0 + b * kWgStage), xb = dyb + 8 * kWgDyBox;
            for (int k = 0; k < ndy; ++k) tma_load_4d(dyb + k * kWgDyBox, &tm_dy, k * 16, x0, y0, n, bar);
            for (int k = ncx; k < nx; ++k)
                tma_load_4d(xb + k * kWgXBox, &tm_x, c0 + k * 16 - a.coarse_ch, x0 - 1, y0 - 1, n, bar);
        }
    } else if (warp == 1) {  // converged, one elected lane issues (see k_conv3x3_tma)
        const uint32_t el = elect_lane();
        const uint32_t idesc = idesc_bf16_mn(a.m, 48);
        const uint64_t da = sdesc_sw32_mn(0, kWgDyBox), db = sdesc_sw32_mn(0, 32);
        const uint32_t alo = (uint32_t)da, blo = (uint32_t)db, dhi = (uint32_t)(da >> 32);  // the upper halves are equal
        for (int it = 0; it < count; ++it) {
            const int b = it % kWgStages;
            if (!warp_wait(saddr(full + b), (uint32_t)(it / kWgStages) & 1u, abort_flag, a.status)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t dyb = saddr(stage0 + b * kWgStage), xb = dyb + 8 * kWgDyBox;
            const uint32_t a0 = alo + (dyb >> 4), b0 = blo + (xb >> 4);
            for (int r = 0; r < kWgRows; ++r)
                for (int k = 0; k < kWgStrip / 16; ++k) {
                    const uint32_t ak = a0 + (uint32_t)(r * kWgStrip + 16 * k) * 2u;
                    const uint32_t bk = b0 + (uint32_t)(r * kWgHaloW + 16 * k) * 2u;
#pragma unroll
                    for (int ky = 0; ky < 3; ++ky)
                        for (int j = 0; j < nx; ++j)
                            umma_elect(tmem + (uint32_t)(ky * nx + j) * 48u, ak,
                                       bk + (uint32_t)(j * kWgXBox / 16 + ky * kWgHaloW * 2), dhi, idesc, el,
                                       (it > 0 || r > 0 || k > 0) ? 1u : 0u);
                }
            umma_commit_elect(saddr(empty + b), el);
        }
        if (ok && count > 0) umma_commit_elect(saddr(acc), el);
    } else if (warp >= 2 && ncx) {
        // the coarse level's boxes: each coarse pixel loaded once and stored to its up to four
        // places in the swizzled halo (as in k_conv3x3_tma), so no concatenation is written
        constexpr int kCx = kWgStrip / 2 + 2, kCy = kWgRows / 2 + 2, kBoxJobs = kCx * kCy * 2;
        constexpr int kT = 32 * kWgCoarseWarps, kJobs = (kBoxJobs * (kWgChunk / 16) + kT - 1) / kT;
        const int ct = tid - 64, Hc = a.H >> 1, Wc = a.W >> 1;
        for (int it = 0; it < count; ++it) {
            const int b = it % kWgStages;
            const int s = first + it * (int)gridDim.x;
            const int xs = s % sx, t = s / sx;
            const int y0 = (t % sy) * kWgRows, n = t / sy, x0 = xs * kWgStrip;
            const int cy0 = (y0 - 1) >> 1, cx0 = (x0 - 1) >> 1;
            uint4 v[kJobs];
#pragma unroll
            for (int u = 0; u < kJobs; ++u) {
                const int i = ct + u * kT, box = i / kBoxJobs, j = i % kBoxJobs, half = j & 1, p = j >> 1;
                const int cy = cy0 + p / kCx, cx = cx0 + p % kCx;
                v[u] = make_uint4(0, 0, 0, 0);
                if (box < ncx && cy >= 0 && cy < Hc && cx >= 0 && cx < Wc)
                    v[u] = *reinterpret_cast<const uint4*>(a.coarse + (((size_t)n * Hc + cy) * Wc + cx) * a.coarse_cs + c0 +
                                                           box * 16 + half * 8);
            }
            if (!warp_wait(saddr(empty + b), ((uint32_t)(it / kWgStages) & 1u) ^ 1u, abort_flag, a.status)) {
                ok = false;
                break;
            }
            unsigned char* xb = stage0 + b * kWgStage + 8 * kWgDyBox;
#pragma unroll
            for (int u = 0; u < kJobs; ++u) {
                const int i = ct + u * kT, box = i / kBoxJobs, j = i % kBoxJobs, half = j & 1, p = j >> 1;
                if (box >= ncx) continue;
                const int hy0 = 2 * (cy0 + p / kCx) - (y0 - 1), hx0 = 2 * (cx0 + p % kCx) - (x0 - 1);
#pragma unroll
                for (int d = 0; d < 4; ++d) {
                    const int hy = hy0 + (d >> 1), hx = hx0 + ((d ^ (p >> 1)) & 1);
                    if (hy < 0 || hy >= kWgRows + 2 || hx < 0 || hx >= kWgHaloW) continue;
                    const int px = hy * kWgHaloW + hx;
                    *reinterpret_cast<uint4*>(xb + box * kWgXBox + px * 32 + ((half ^ ((px >> 2) & 1)) << 4)) = v[u];
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // these stores -> tensor core reads
            __syncwarp();
            if (lane == 0) mbar_arrive(saddr(full + b));
        }
    }
    __syncwarp();
    // epilogue: TMEM lane (warp * 32 + lane) holds output channel co for every tap
    const bool got = count == 0 || wait_or_abort(saddr(acc), 0u, abort_flag, a.status);
    if (warp >= 4) {
        // an expanding warp: the four warps below move the accumulators
    } else if (__all_sync(0xffffffffu, got && !*abort_flag)) {  // warp-uniform: tcgen05.ld is .aligned
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // M = 128: row i in TMEM lane i.  M = 64: rows 16w..16w+15 in lanes 32w..32w+15 of
        // warp w's quarter (the upper 16 lanes of each quarter are unused)
        const int co = a.m == 128 ? warp * 32 + lane : (lane < 16 ? warp * 16 + lane : a.cpad);
        float* part = a.part + (size_t)blockIdx.x * 9 * a.cpad * a.cin;
        for (int tap = 0; tap < 9; ++tap)
            for (int j = 0; j < nx; ++j) {
                uint32_t v[16];
                tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (tap / 3 * nx + j) * 48 + tap % 3 * 16, v);
                if (co >= a.cout) continue;
                float4* dst = reinterpret_cast<float4*>(part + ((size_t)tap * a.cpad + co) * a.cin + c0 + j * 16);
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    dst[q] = count > 0 ? make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]),
                                                     __uint_as_float(v[4 * q + 2]), __uint_as_float(v[4 * q + 3]))
                                       : make_float4(0.f, 0.f, 0.f, 0.f);
            }
    } else if (lane == 0) {
        atomicOr(a.status, 1);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" :: "r"(tmem) : "memory");
}

// Adds every entry's partial slices to its destination: a block takes 32 groups of four
// neighbouring outputs of one entry; its 8 rows of threads add a strided share of the slices
// each, and the shares are added in row order.  One launch for a whole backward pass: one per
// layer (8 us each, latency) took 190 us of 1.73 ms at 16 x 256 x 256.
__global__ void __launch_bounds__(256) k_grad_reduce(const __grid_constant__ GradReduceTable T) {
    __shared__ float4 sm[8][32];
    grid_turn();
    int e = 0;
    while (e + 1 < T.n && (int)blockIdx.x >= T.e[e + 1].block0) ++e;
    const GradReduceTable::Entry E = T.e[e];
    const int col = threadIdx.x & 31, row = threadIdx.x >> 5;
    const int i = ((int)blockIdx.x - E.block0) * 32 + col;
    float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (i < E.groups) {
        // output group i = (r, j) of the destination's rows of E.row4 groups, E.rows rows per
        // tap; a slice has E.pad_rows rows per tap
        const int j = i % E.row4, r = i / E.row4;
        const float* p = E.part + ((size_t)(r / E.rows) * E.pad_rows + r % E.rows) * E.row4 * 4 + j * 4;
#pragma unroll 4
        for (int k = row; k < E.slices; k += 8) {
            const float4 v = *reinterpret_cast<const float4*>(p + (size_t)k * E.stride);
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
    }
    sm[row][col] = s;
    __syncthreads();
    if (row != 0 || i >= E.groups) return;
    for (int k = 1; k < 8; ++k) {
        const float4 v = sm[k][col];
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    float* d = E.dst + (size_t)i * 4;  // a layer's gradients start on any 4-byte boundary
    d[0] += s.x;
    d[1] += s.y;
    d[2] += s.z;
    d[3] += s.w;
}

}  // namespace

// Image rows per strip for an output width of npad channels: R x npad accumulator columns
// fit in the CTA's 256.
int conv_tc_rows(int cout) {
    const int npad = (cout + 15) / 16 * 16;
    int R = kTmemCols / npad;
    return R > 8 ? 8 : R;
}

salty_status conv3x3_tc(salty_ctx* ctx, const ConvSrc& in, int cin, const bf16* wt, int wrows, const float* bias,
                        bf16* out, int out_cs, int out_co, int cout, int N, int H, int W, int relu, int* d_status) {
    const int npad = (cout + 15) / 16 * 16;
    if (cin % 16 || cin <= 0 || npad > 256 || npad < 16 || cout % 8 || in.a_cs % 8 || in.a_ch % 16 ||
        (in.a_ch < cin && (!in.b || in.b_cs % 8)) || out_cs % 8 || out_co % 8 || wrows < 1)
        return ctx->err.fail(SALTY_ERR_INVALID_ARG, "conv3x3_tc: unsupported shape (cin %d, cout %d)", cin, cout);
    const int R = conv_tc_rows(cout);
    const size_t smem = (size_t)kBarBytes + 2 * (size_t)stage_bytes(R, npad);
    SALTY_TRY_CUDA(ctx->err, cudaFuncSetAttribute(k_conv3x3_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const long long tiles = (long long)N * ((H + R - 1) / R) * ((W + kStrip - 1) / kStrip);
    TcConvArgs a{in, cin, wt, wrows, bias, out, out_cs, out_co, cout, npad, R, N, H, W, relu, d_status};
    k_conv3x3_tc<<<(unsigned)tiles, kTcThreads, smem, ctx->stream>>>(a);
    SALTY_TRY_CUDA(ctx->err, cudaGetLastError());
    return SALTY_OK;
}

salty_status conv3x3_tma(salty_ctx* ctx, const ConvSrc& in, int cin, const bf16* wt, int wrows, const float* bias,
                         bf16* out, bf16* pool, int out_cs, int cout, int N, int H, int W, int relu, int* d_status) {
    const int npad = (cout + 15) / 16 * 16;
    const bool coarse = in.a_ch < cin;  // [up2(a) | b]
    const bf16* src = coarse ? in.b : in.a;
    const int src_cs = coarse ? in.b_cs : in.a_cs;
    auto unaligned = [](const void* p, int by) { return reinterpret_cast<uintptr_t>(p) % by != 0; };
    if (cin % 16 || cin <= 0 || cin > 16 * kTmaMaxChunks || npad > 256 || npad < 16 || cout % 8 || wrows < 1 || wrows > 256 ||
        (coarse ? in.a_shift != 1 || in.a_ch % 16 || in.a_cs % 8 || H % 2 || W % 2 || unaligned(in.a, 16)
                : in.a_shift != 0) ||
        src_cs % 8 || (cout >= 16 ? out_cs % 16 != 0 : out_cs % 8 != 0) || unaligned(src, 16) || unaligned(wt, 16) ||
        unaligned(out, 32) || (pool && (unaligned(pool, 32) || H % 2 || W % 2)))
        return ctx->err.fail(SALTY_ERR_INVALID_ARG, "conv3x3_tma: unsupported shape (cin %d, cout %d)", cin, cout);
    EncodeTiledFn enc = tensor_map_encoder();
    if (!enc) return ctx->err.fail(SALTY_ERR_CUDA, "conv3x3_tma: cuTensorMapEncodeTiled is not available");
    int R = conv_tc_rows(cout);
    if (pool && (R & 1)) --R;  // pooled rows are pairs within a strip
    // Levels of fewer strips than SMs: shorter strips where that shortens the longest block's work,
    // strips per block times (halo rows + 2 rows' worth of fixed cost).  An output's sum keeps its
    // order.  A 32 x 32 denoise 150 -> 125 us, a 256 x 256 training step 491 -> 462; chosen by the
    // same cost above one strip per SM, an eight-fold 1080p denoise took 0.5 % longer.
    auto strips = [&](int r) { return (long long)N * ((H + r - 1) / r) * ((W + kStrip - 1) / kStrip); };
    auto cost = [&](int r) { return (strips(r) + ctx->num_sms - 1) / ctx->num_sms * (r + 4); };
    if (strips(R) <= ctx->num_sms)
        for (int r = R - (pool ? 2 : 1); r >= 2; r -= pool ? 2 : 1)
            if (cost(r) < cost(R)) R = r;
    if (pool && R < 2) return ctx->err.fail(SALTY_ERR_INVALID_ARG, "conv3x3_tma: no pooled output for cout %d", cout);
    // the layer's weights stay in shared memory for the whole kernel when they are small
    const int wbytes = (cin / 16) * 9 * npad * 32;
    const bool resident = wbytes <= kResidentMaxBytes;
    const int wres = resident ? (wbytes + 1023) / 1024 * 1024 : 0;
    const int sbytes = resident ? tma_halo(R) : tma_stage(R, npad);
    int S = (int)((227 * 1024 - kTmaHeader - wres) / sbytes);
    if (S > kMaxStages) S = kMaxStages;
    if (S < 2) return ctx->err.fail(SALTY_ERR_INVALID_ARG, "conv3x3_tma: stage too large");
    size_t smem = (size_t)kTmaHeader + wres + (size_t)S * sbytes;
    if (smem < (size_t)kTmaMinSmem) smem = kTmaMinSmem;
    // input: 4-D (channels, x, y, image), boxes of 16 channels x 130 pixels x R + 2 rows
    CUtensorMap tm_in, tm_w;
    const cuuint64_t gdim[4] = {(cuuint64_t)src_cs, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)N};
    const cuuint64_t gstride[3] = {(cuuint64_t)src_cs * 2, (cuuint64_t)W * src_cs * 2, (cuuint64_t)H * W * src_cs * 2};
    const cuuint32_t box[4] = {16, (cuuint32_t)kHaloW, (cuuint32_t)(R + 2), 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    if (enc(&tm_in, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(src), gdim, gstride, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return ctx->err.fail(SALTY_ERR_CUDA, "conv3x3_tma: input tensor map");
    // weights: 4-D (input channel, row, kx, ky), boxes of 16 channels x npad rows x the three ky
    const cuuint64_t wdim[4] = {(cuuint64_t)cin, (cuuint64_t)wrows, 3, 3};
    const cuuint64_t wstride[3] = {(cuuint64_t)cin * 2, (cuuint64_t)wrows * cin * 2, (cuuint64_t)3 * wrows * cin * 2};
    const cuuint32_t wbox[4] = {16, (cuuint32_t)npad, 1, 3};
    if (enc(&tm_w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(wt), wdim, wstride, wbox, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return ctx->err.fail(SALTY_ERR_CUDA, "conv3x3_tma: weight tensor map");
    const long long tiles = strips(R);
    const int grid = (int)(tiles < ctx->num_sms ? tiles : ctx->num_sms);
    TmaConvArgs a{cin, npad, R, cout, relu, out_cs, N, H, W, (int)tiles, S, resident ? 1 : 0, wres, bias, out, pool,
                  coarse ? in.a : nullptr, coarse ? in.a_cs : 0, coarse ? in.a_ch : 0, d_status};
    auto kern = coarse ? k_conv3x3_tma<true> : k_conv3x3_tma<false>;
    SALTY_TRY_CUDA(ctx->err, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    SALTY_TRY_CUDA(ctx->err, launch_early(kern, grid, kTmaThreads + (coarse ? 32 * kTmaCoarseWarps : 0), smem, ctx->stream,
                                          tm_in, tm_w, a));
    return SALTY_OK;
}

// Input-channel groups and strip slices for a layer: about one CTA per SM in all.
static void wgrad_plan(int num_sms, int cin, int N, int H, int W, int* groups, int* slices, int* strips) {
    *groups = (cin + kWgChunk - 1) / kWgChunk;
    const long long st = (long long)N * ((H + kWgRows - 1) / kWgRows) * ((W + kWgStrip - 1) / kWgStrip);
    long long s = num_sms / *groups;
    if (s < 1) s = 1;
    if (s > st) s = st;
    *slices = (int)s;
    *strips = (int)st;
}

size_t conv_wgrad_tc_workspace(int num_sms, int cin, int cpad, int N, int H, int W) {
    int groups, slices, strips;
    wgrad_plan(num_sms, cin, N, H, W, &groups, &slices, &strips);
    return (size_t)slices * 9 * cpad * cin;
}

salty_status conv_wgrad_tc(salty_ctx* ctx, const bf16* dy, int cpad, int cout, const ConvSrc& x, int cin, float* dw,
                           int N, int H, int W, float* ws, size_t ws_floats, int* d_status, GradReduceTable& table) {
    const bool coarse = x.a_ch < cin;  // [up2(a) | b]
    const bf16* src = coarse ? x.b : x.a;
    const int src_cs = coarse ? x.b_cs : x.a_cs;
    if (cin % 16 || cin <= 0 || cpad % 16 || cpad < 16 || cpad > 128 || cout > cpad || cout < 1 || src_cs % 16 ||
        (coarse ? x.a_shift != 1 || x.a_ch % 16 || x.a_cs % 8 || H % 2 || W % 2 || reinterpret_cast<uintptr_t>(x.a) % 16
                : x.a_shift != 0) ||
        reinterpret_cast<uintptr_t>(src) % 16 || reinterpret_cast<uintptr_t>(dy) % 16 || reinterpret_cast<uintptr_t>(ws) % 16)
        return ctx->err.fail(SALTY_ERR_INVALID_ARG, "conv_wgrad_tc: unsupported shape (cin %d, cout %d)", cin, cout);
    EncodeTiledFn enc = tensor_map_encoder();
    if (!enc) return ctx->err.fail(SALTY_ERR_CUDA, "conv_wgrad_tc: cuTensorMapEncodeTiled is not available");
    int groups, slices, strips;
    wgrad_plan(ctx->num_sms, cin, N, H, W, &groups, &slices, &strips);
    if ((size_t)slices * 9 * cpad * cin > ws_floats)
        return ctx->err.fail(SALTY_ERR_CAPACITY, "conv_wgrad_tc: workspace too small");
    CUtensorMap tm_x, tm_dy;
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const cuuint32_t xbox[4] = {16, (cuuint32_t)kWgHaloW, (cuuint32_t)(kWgRows + 2), 1};
    const cuuint64_t xdim[4] = {(cuuint64_t)src_cs, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)N};
    const cuuint64_t xstr[3] = {(cuuint64_t)src_cs * 2, (cuuint64_t)W * src_cs * 2, (cuuint64_t)H * W * src_cs * 2};
    if (enc(&tm_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(src), xdim, xstr, xbox, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return ctx->err.fail(SALTY_ERR_CUDA, "conv_wgrad_tc: input tensor map");
    const cuuint32_t dbox[4] = {16, (cuuint32_t)kWgStrip, (cuuint32_t)kWgRows, 1};
    const cuuint64_t ddim[4] = {(cuuint64_t)cpad, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)N};
    const cuuint64_t dstr[3] = {(cuuint64_t)cpad * 2, (cuuint64_t)W * cpad * 2, (cuuint64_t)H * W * cpad * 2};
    if (enc(&tm_dy, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(dy), ddim, dstr, dbox, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return ctx->err.fail(SALTY_ERR_CUDA, "conv_wgrad_tc: gradient tensor map");
    const size_t smem = (size_t)kWgHeader + (size_t)kWgStages * kWgStage;
    SALTY_TRY_CUDA(ctx->err, cudaFuncSetAttribute(k_wgrad_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    WgradArgs a{cpad <= 64 ? 64 : 128, cpad, cout, cin, N, H, W, strips, ws, coarse ? x.a : nullptr,
                coarse ? x.a_cs : 0, coarse ? x.a_ch : 0, d_status};
    SALTY_TRY_CUDA(ctx->err, launch_early(k_wgrad_tc, dim3(slices, groups), coarse ? kWgCoarseThreads : kWgThreads, smem,
                                          ctx->stream, tm_x, tm_dy, a));
    return grad_reduce_add(ctx, table, {ws, dw, slices, 9 * cpad * cin, cin / 4, cout, cpad, 9 * cout * (cin / 4), 0});
}

salty_status grad_reduce_add(salty_ctx* ctx, GradReduceTable& table, GradReduceTable::Entry e) {
    if (table.n >= GradReduceTable::kMax) return ctx->err.fail(SALTY_ERR_CAPACITY, "gradient reduction table full");
    e.block0 = table.blocks;
    table.blocks += (e.groups + 31) / 32;
    table.e[table.n++] = e;
    return SALTY_OK;
}

salty_status grad_reduce_run(salty_ctx* ctx, const GradReduceTable& table) {
    if (table.blocks > 0)
        SALTY_TRY_CUDA(ctx->err, launch_early(k_grad_reduce, table.blocks, 256, 0, ctx->stream, table));
    SALTY_TRY_CUDA(ctx->err, cudaGetLastError());
    return SALTY_OK;
}

}  // namespace salty
