// tl_conv.cu -- BF16 tensor-core kernels of the learned warm start: a
// residual network of 3x3 convolutions (32 channels, GELU) that predicts
// u^{n+1} - u^n from (u^n, log density, Kx, Ky, dt).  No reference
// counterpart: the reference solve always starts from u^n.
//
// Activations are NHWC BF16 with a one-pixel zero halo: [B][H+2][W+2][C].
// A 3x3 convolution is an implicit GEMM: M = pixels, N = output channels,
// K = 9 taps x input channels.  A warp owns 16 consecutive pixels of one
// row and all output channels; each (tap, 16-channel) step feeds
// mma.sync.m16n8k16 (BF16 inputs, FP32 accumulate) with A fragments loaded
// straight from the NHWC input (two channels per 32-bit load) and B
// fragments from weights stored [tap][cout][cin].  The data gradient is the
// same kernel on the output gradient with the weights flipped and
// transposed ([8 - tap][cin][cout]); the weight gradient is a GEMM over
// pixels (M = cout, N = cin per tap, K = pixels) whose per-CTA partial sums
// are reduced in a fixed order.
#include <cuda_bf16.h>
#include <math.h>
#include <stdint.h>

#include "tl_internal.cuh"

namespace tl {
namespace {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                         uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t ld32(const bf16 *p) {
    return *reinterpret_cast<const uint32_t *>(p);
}

__device__ __forceinline__ uint32_t pack2(bf16 lo, bf16 hi) {
    return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

// GELU, tanh form: 0.5 x (1 + tanh(u)) = x / (1 + exp(-2 u)), u = sqrt(2/pi) (x + 0.044715 x^3).
// With e = exp(-2 |u|) in (0, 1]: x - x e / (1 + e) for x > 0, |x| e / (1 + e) below
// zero.  11 instructions with the hardware's exponential and reciprocal where
// tanhf takes some 50, which bound the convolutions; its largest error
// against FP64 over -20..20 is 2.4e-7 (with tanhf, whose 1 + tanh cancels
// for x < 0: 4.3e-7), the root mean square lower too.
__device__ __forceinline__ float exp2_hw(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rcp_hw(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
constexpr float kG0 = 0.7978845608028654f, kG1 = 0.044715f;
constexpr float kE0 = (float)(2.0 * 0.7978845608028654 * 1.4426950408889634);  // 2 sqrt(2/pi) log2(e)
constexpr float kE1 = (float)(2.0 * 0.7978845608028654 * 1.4426950408889634 * 0.044715);
__device__ __forceinline__ float gelu(float x) {
    float a;  // |x|, finite for x = inf (whose e is 0); NaN stays
    asm("min.NaN.f32 %0, %1, 0f7F7FFFFF;" : "=f"(a) : "f"(x));
    a = fabsf(a);
    const float e = exp2_hw(-a * fmaf(kE1, x * x, kE0));
    return fmaf(-a, e * rcp_hw(1.f + e), fmaxf(x, 0.f));
}
// s + 2 x s (1 - s) u' with s = 1 / (1 + exp(-2 u)), s (1 - s) = e / (1 + e)^2
__device__ __forceinline__ float gelu_grad(float x) {
    const float x2 = x * x, e = exp2_hw(-fabsf(x) * fmaf(kE1, x2, kE0));
    const float r = rcp_hw(1.f + e), er = e * r;
    return fmaf((x * er) * r, fmaf(6.f * kG0 * kG1, x2, 2.f * kG0), x < 0.f ? er : r);
}

enum ConvMode { kModeGelu = 0, kModeGeluRes = 1, kModeHead = 2, kModeLinear = 3 };

template <int CIN, int COUTP, int MODE>
__global__ void __launch_bounds__(128) k_conv(const bf16 *__restrict__ in, const bf16 *__restrict__ wt,
                                              const float *__restrict__ bias,
                                              const bf16 *__restrict__ res, bf16 *__restrict__ out,
                                              bf16 *__restrict__ pre, float *__restrict__ outf, int B,
                                              int H, int W) {
    const int lane = threadIdx.x & 31;
    const long long task = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
    const int wx = W / 16;
    if (task >= (long long)B * H * wx) return;
    const int b = (int)(task / ((long long)H * wx));
    const int rem = (int)(task % ((long long)H * wx));
    const int y = rem / wx, x0 = (rem % wx) * 16;
    const int g = lane >> 2, t = lane & 3;
    constexpr int NT = COUTP / 8;
    float acc[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
    const long long Wp = W + 2;
    const bf16 *img = in + (long long)b * (H + 2) * Wp * CIN;
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
        const int dy = tap / 3, dx = tap % 3;
        const bf16 *r0 = img + ((long long)(y + dy) * Wp + (x0 + dx + g)) * CIN;
        const bf16 *r1 = r0 + 8 * CIN;
#pragma unroll
        for (int kc = 0; kc < CIN / 16; ++kc) {
            const int ch = kc * 16 + 2 * t;
            const uint32_t a0 = ld32(r0 + ch), a1 = ld32(r1 + ch);
            const uint32_t a2 = ld32(r0 + ch + 8), a3 = ld32(r1 + ch + 8);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const bf16 *wr = wt + (long long)(tap * COUTP + nt * 8 + g) * CIN + ch;
                mma16816(acc[nt], a0, a1, a2, a3, ld32(wr), ld32(wr + 8));
            }
        }
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        const int co = nt * 8 + 2 * t;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int px = x0 + g + 8 * half;
            float v0 = acc[nt][2 * half], v1 = acc[nt][2 * half + 1];
            const long long o = ((long long)b * (H + 2) + y + 1) * Wp + px + 1;
            if (MODE == kModeHead) {
                if (co == 0) outf[((long long)b * H + y) * W + px] = v0 + bias[0];
                continue;
            }
            if (MODE == kModeGelu || MODE == kModeGeluRes) {
                v0 += bias[co];
                v1 += bias[co + 1];
                if (pre)
                    *reinterpret_cast<uint32_t *>(pre + o * COUTP + co) =
                        pack2(__float2bfloat16(v0), __float2bfloat16(v1));
                v0 = gelu(v0);
                v1 = gelu(v1);
            }
            if ((MODE == kModeGeluRes || MODE == kModeLinear) && res) {
                const __nv_bfloat162 rv = *reinterpret_cast<const __nv_bfloat162 *>(res + o * COUTP + co);
                v0 += __bfloat162float(rv.x);
                v1 += __bfloat162float(rv.y);
            }
            *reinterpret_cast<uint32_t *>(out + o * COUTP + co) =
                pack2(__float2bfloat16(v0), __float2bfloat16(v1));
        }
    }
}

// ---------------------------------------------------------------------------
// The same convolution on the 5th-generation tensor cores (tcgen05).  A tile is
// 128 columns (M = 128) of R output rows.  Columns are counted over the
// padded rows of a group of R rows and on into the next group, q = group
// (W + 2) + x, and a tile is any 128 consecutive q, so the two columns a row
// that are no output are all that is computed in vain (1.4 % at W = 144, where
// tiles of one row's pixels wasted 44 %).  W + 2 is even: an even q and the
// next are neighbours in memory.
//
// A CTA of 4 warps walks tiles: the weights stay in shared memory, and the next
// tile's input is on its way (cp.async) while this one's result is written.
// Shared memory holds, per input row k of R + 2, the 130 input pixels that
// the three taps dx = 0, 1, 2 read, in the K-major no-swizzle layout of the MMA
// operands: 16-byte core-matrix rows (one pixel, 8 channels), the pixels of
// an 8-channel chunk contiguous (16 bytes apart) and the chunks kChunkA bytes
// apart.  The A operand of input row k, dx and 16-channel step kk is that block
// shifted by dx pixels: start + dx * 16, core matrices 128 bytes apart along
// M (SBO) and kChunkA along K (LBO).  The weights sit in the same layout, per
// dx, with the couts of dy = 2, 1, 0 one after the other along N (16 bytes
// apart): input row k is the dy = 2, 1, 0 neighbour of the output rows k - 2,
// k - 1 and k, whose accumulators lie side by side in the same order, so that one
// MMA adds it to all three (N = 3 COUTP; fewer at the tile's first and last rows).
// One thread issues the MMAs (M 128, K 16, BF16 in, FP32 accumulate) and commits
// them to an mbarrier; each warp then reads its 32 TMEM lanes (one pixel a
// lane, one channel a column) row by row and runs the epilogue of k_conv.
// Lanes trade half of their chunks with their neighbours before a store, so
// that every store writes whole 32-byte sectors.
// What bounds it, at 4 rows: latency, with three CTAs (12 warps) a multiprocessor that wait
// for their loads between the MMAs and the epilogue; then L2, from which an
// input row is read (R + 2) / R times (tensor cores 11-15 % busy,
// HBM 29 %).  4096 x 4096 pixels, 32 to 32 channels with GELU and the input
// added: 947 us, HBM's 2.1 GB take 317.  One row a tile (three reads): two
// buffers and 3 CTAs 1250, one buffer and 5 CTAs 1090; two rows and 4 CTAs 930,
// but 605 for the head where four rows take 527; three rows 986.  32 x 144 x 144
// pixels with the pre-activation written: one row 64 and 58, two 53, four 53 us.
constexpr int kTcPix = 128;               // pixels of a tile (MMA M)
constexpr int kTcRow = kTcPix + 2;        // input pixels a kernel row of a tile reads
constexpr int kChunkA = kTcRow * 16;      // bytes between 8-channel chunks of A
// CTAs a multiprocessor (43, 52 and 68 KB of shared memory each at 1, 2 and 4 rows)
__host__ __device__ constexpr int tc_ctas(int r) { return r == 1 ? 5 : r == 2 ? 4 : 3; }
__host__ __device__ constexpr int tmem_cols(int r) { return 32 * r; }  // accumulator columns allocated (>= R COUTP)
constexpr long long kTcWaitCycles = 2000000000LL;  // ~1 s: the MMA wait gives up after this

// set by a tcgen05 conv whose MMA completion wait ran out (read and cleared
// by tl_nn_conv_status)
__device__ int g_conv_tc_error;

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// shared-memory matrix descriptor: no swizzle, version 1 (bits 46-47)
__device__ __forceinline__ uint64_t mma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// instruction descriptor of kind::f16: FP32 accumulator (bits 4-5 = 1), BF16
// A and B (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
__host__ __device__ constexpr uint32_t mma_idesc(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.b32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// bounded wait on phase `parity` of an mbarrier: false if it ran out
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity) {
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity))
        if (clock64() - t0 > kTcWaitCycles) return false;
    return true;
}

template <int N>
__device__ __forceinline__ void tmem_load(uint32_t taddr, float (&v)[N]);

template <>
__device__ __forceinline__ void tmem_load<32>(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
          "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
          "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
          "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = __uint_as_float(r[k]);
}

template <>
__device__ __forceinline__ void tmem_load<16>(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
        "[%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
          "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}

template <int CIN, int COUTP, int R>
constexpr int conv_tc_smem() {
    return (R + 2) * (CIN / 8) * kChunkA + 9 * (CIN / 8) * COUTP * 16;
}

// store 8 channels a lane of COUTP, `at` the lane's pixel: two chunks of the
// lane's own pixel become one chunk of each of the pair's pixels
template <int COUTP>
__device__ __forceinline__ void store_chunks(bf16 *dst, long long at, int chunk, const uint32_t (&c0)[4],
                                             const uint32_t (&c1)[4], bool mine, bool partner, int lane) {
    const bool odd = lane & 1;
    uint32_t even_px[4], odd_px[4];  // this lane's chunk of the pair's even and odd pixel
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? c0[e] : c1[e], 1);
        even_px[e] = odd ? got : c0[e];
        odd_px[e] = odd ? c1[e] : got;
    }
    const int c = chunk + (odd ? 1 : 0);
    const long long e0 = odd ? at - 1 : at;
    if (odd ? partner : mine)
        *reinterpret_cast<uint4 *>(dst + e0 * COUTP + 8 * c) = make_uint4(even_px[0], even_px[1], even_px[2], even_px[3]);
    if (odd ? mine : partner)
        *reinterpret_cast<uint4 *>(dst + (e0 + 1) * COUTP + 8 * c) = make_uint4(odd_px[0], odd_px[1], odd_px[2], odd_px[3]);
}

template <int CIN, int COUTP, int MODE, int R>
__global__ void __launch_bounds__(128, tc_ctas(R)) k_conv_tc(const bf16 *__restrict__ in, const bf16 *__restrict__ wt,
                                                 const float *__restrict__ bias,
                                                 const bf16 *__restrict__ res, bf16 *__restrict__ out,
                                                 bf16 *__restrict__ pre, float *__restrict__ outf, int B,
                                                 int H, int W) {
    static_assert(CIN % 16 == 0 && COUTP % 16 == 0 && R * COUTP <= tmem_cols(R), "conv shape");
    constexpr int CA = CIN / 8;                    // 8-channel chunks of a pixel
    constexpr int CHUNK_B = 3 * COUTP * 16;        // bytes between chunks of the weights
    constexpr int A_BYTES = (R + 2) * CA * kChunkA;
    extern __shared__ __align__(128) unsigned char conv_smem[];
    unsigned char *const sb = conv_smem + A_BYTES;
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(16) float sbias[COUTP];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int Wp = W + 2;
    const long long npix = (long long)((H + R - 1) / R) * Wp, in_pix = (long long)(H + 2) * Wp;  // q range, padded image
    // (tiles count in 32 bits: 2^32 of them would be 2^39 pixels)
    const unsigned int per_image = (unsigned int)((npix + kTcPix - 1) / kTcPix), tiles = per_image * (unsigned int)B;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_addr(&tmem_slot)),
                     "r"(tmem_cols(R)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&mbar)));
        // the tensor cores arrive on it: make the initialisation visible to them
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // row group and column of q
    auto place = [&](long long q, int &y, int &x) {
        const int gr = npix >> 31 ? (int)(q / Wp) : (int)((unsigned int)q / (unsigned int)Wp);
        x = (int)(q - (long long)gr * Wp);
        y = gr * R;
    };
    // A: pixels q0 + 0..129 of R + 2 input rows, 16 bytes a copy; those past
    // the image read as zero (last tiles)
    auto stage = [&](unsigned int t) {
        const unsigned int b = t / per_image;
        const long long q0 = (long long)(t - b * per_image) * kTcPix;
        const bf16 *img = in + (long long)b * in_pix * CIN;
        const uint32_t dst = smem_addr(conv_smem);
        // a thread copies chunk tid % CA of every 128 / CA-th pixel
        constexpr int PX = 128 / CA;
        const int c = tid % CA, j0 = tid / CA;
        int y, x;
        place(q0 + j0, y, x);
#pragma unroll
        for (int i = 0; i < (kTcRow + PX - 1) / PX; ++i) {
            if ((i + 1) * PX > kTcRow && j0 + i * PX >= kTcRow) break;
            const bf16 *src = img + ((long long)y * Wp + x) * CIN + 8 * c;
            const uint32_t d = dst + c * kChunkA + (j0 + i * PX) * 16;
#pragma unroll
            for (int k = 0; k < R + 2; ++k) {
                const bool ok = y + k < H + 2;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d + k * CA * kChunkA),
                             "l"(ok ? src + (long long)k * Wp * CIN : img), "r"(ok ? 16 : 0));
            }
            for (x += PX; x >= Wp; x -= Wp) y += R;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    unsigned int t = blockIdx.x;
    if (t < tiles) stage(t);
    if (MODE != kModeLinear && tid < (MODE == kModeHead ? 1 : COUTP)) sbias[tid] = bias[tid];
    // B: weights [tap][cout][cin]
    for (int k = tid; k < 9 * COUTP * CA; k += 128) {
        const int c = k % CA, co = (k / CA) % COUTP, tap = k / (CA * COUTP);
        const uint4 v = *reinterpret_cast<const uint4 *>(wt + ((long long)tap * COUTP + co) * CIN + 8 * c);
        *reinterpret_cast<uint4 *>(sb + ((tap % 3) * CA + c) * CHUNK_B + ((2 - tap / 3) * COUTP + co) * 16) = v;
    }
    const uint32_t bar = smem_addr(&mbar);
    uint32_t tmem = 0, phase = 0;
    bool ok = true;
    for (; t < tiles; t += gridDim.x, phase ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        // the MMAs read shared memory through the async proxy
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem = tmem_slot;
        if (tid == 0) {
            const uint32_t a0 = smem_addr(conv_smem), b0 = smem_addr(sb);
            // one MMA for the output rows lo..hi of an input row, dx and 16 channels
            auto mma = [&](int k, int dx, int kk, int lo, int hi, uint32_t acc) {
                const uint64_t ad = mma_desc(a0 + (k * CA + 2 * kk) * kChunkA + dx * 16, kChunkA, 128);
                const uint64_t bd = mma_desc(b0 + (dx * CA + 2 * kk) * CHUNK_B + (2 - k + lo) * COUTP * 16, CHUNK_B, 128);
                asm volatile(
                    "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem + lo * COUTP),
                    "l"(ad), "l"(bd), "r"(mma_idesc(kTcPix, (hi - lo + 1) * COUTP)), "r"(acc));
            };
#pragma unroll
            for (int k = 0; k < R + 2; ++k) {
                const int lo = k < 2 ? 0 : k - 2, hi = k < R ? k : R - 1;
#pragma unroll
                for (int q = 0; q < 3 * (CIN / 16); ++q) {
                    const int dx = q % 3, kk = q / 3;
                    if (q == 0 && k < R) {  // row k's first product; its accumulator is overwritten
                        mma(k, dx, kk, k, k, 0u);
                        if (lo < k) mma(k, dx, kk, lo, k - 1, 1u);
                    } else {
                        mma(k, dx, kk, lo, hi, 1u);
                    }
                }
            }
            asm volatile(
                "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                : "memory");
        }
        // this lane's pixels, while the tensor cores work
        const unsigned int b = t / per_image;
        int x, y;
        const long long q = (long long)(t - b * per_image) * kTcPix + 32 * warp + lane;
        place(q, y, x);
        const bool column = q < npix && x < W;
        const long long o0 = (long long)b * in_pix + (long long)(y + 1) * Wp + x + 1;
        uint4 rv[R][COUTP / 8];
        const bool add = (MODE == kModeGeluRes || MODE == kModeLinear) && res;
        // what is added: where it is the input itself, the staged centre tap's
        // pixels (below), else from memory
        const bool own = add && CIN == COUTP && res == in;
        if (add && !own) {
#pragma unroll
            for (int row = 0; row < R; ++row)
#pragma unroll
                for (int h = 0; h < COUTP / 8; ++h)
                    if (column && y + row < H)
                        rv[row][h] = *reinterpret_cast<const uint4 *>(res + (o0 + (long long)row * Wp) * COUTP + 8 * h);
        }
        // warp-uniform outcome: tcgen05.ld below is executed by whole warps
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(bar, phase));
        if (own) {
            const uint4 *centre = reinterpret_cast<const uint4 *>(conv_smem + CA * kChunkA);
#pragma unroll
            for (int row = 0; row < R; ++row)
#pragma unroll
                for (int h = 0; h < COUTP / 8; ++h)
                    rv[row][h] = centre[(row * CA + h) * (kChunkA / 16) + 32 * warp + lane + 1];
        }
        if (!__syncthreads_and(ok)) {
            // the accumulator never became ready: flag it, wait once more
            // (bounded) for the MMAs in flight, release the columns and leave
            if (lane == 0) atomicExch(&g_conv_tc_error, 1);
            mbar_wait_bounded(bar, phase);
            break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // the next tile's input is on its way while this one is written
        if (t + gridDim.x < tiles) stage(t + gridDim.x);
#pragma unroll
        for (int row = 0; row < R; ++row, ++y) {
            const bool valid = column && y < H;
            const bool pvalid = __shfl_xor_sync(0xffffffffu, (int)valid, 1) != 0;
            const long long o = o0 + (long long)row * Wp;
            // warp w holds TMEM lanes 32w..32w+31: pixel m = 32 w + lane
            float acc[COUTP];
            tmem_load<COUTP>(tmem + row * COUTP + ((uint32_t)(32 * warp) << 16), acc);
            if (MODE == kModeHead) {
                if (valid) outf[((long long)b * H + y) * W + x] = acc[0] + sbias[0];
            } else {
#pragma unroll
                for (int q2 = 0; q2 < COUTP / 8; q2 += 2) {
                    uint32_t pk[2][4];
                    if (MODE == kModeGelu || MODE == kModeGeluRes) {
#pragma unroll
                        for (int h = 0; h < 2; ++h)
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                float &v0 = acc[8 * (q2 + h) + 2 * e], &v1 = acc[8 * (q2 + h) + 2 * e + 1];
                                v0 += sbias[8 * (q2 + h) + 2 * e];
                                v1 += sbias[8 * (q2 + h) + 2 * e + 1];
                                pk[h][e] = pack2(__float2bfloat16(v0), __float2bfloat16(v1));
                                v0 = gelu(v0);
                                v1 = gelu(v1);
                            }
                        if (pre) store_chunks<COUTP>(pre, o, q2, pk[0], pk[1], valid, pvalid, lane);
                    }
                    if (add && valid) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const uint32_t rw[4] = {rv[row][q2 + h].x, rv[row][q2 + h].y, rv[row][q2 + h].z, rv[row][q2 + h].w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                acc[8 * (q2 + h) + 2 * e] += __uint_as_float(rw[e] << 16);
                                acc[8 * (q2 + h) + 2 * e + 1] += __uint_as_float(rw[e] & 0xFFFF0000u);
                            }
                        }
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            pk[h][e] = pack2(__float2bfloat16(acc[8 * (q2 + h) + 2 * e]),
                                             __float2bfloat16(acc[8 * (q2 + h) + 2 * e + 1]));
                    store_chunks<COUTP>(out, o, q2, pk[0], pk[1], valid, pvalid, lane);
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_slot), "r"(tmem_cols(R)));
}

// dpre = dh * gelu'(pre) over the interior (halo left at zero).  Bound by HBM
// (6 bytes a value); V values (16 bytes) a thread and step where the channels
// come in eights and the buffers are 16-byte aligned, V = 1 otherwise.
// (32 x 144 x 144 x 32 values: see tl_nn_wgrad for the pass's times.)
template <int V>
__global__ void k_gelu_back(const bf16 *__restrict__ dh, const bf16 *__restrict__ pre,
                            bf16 *__restrict__ dpre, int C, int B, int H, int W) {
    const int per_row = W * (C / V);
    const long long n = (long long)B * H * per_row;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        // (32-bit division where the count allows)
        const long long row = n >> 32 ? t / per_row : (long long)((unsigned int)t / (unsigned int)per_row);
        const int k = (int)(t - row * per_row);
        const int b = (int)(row / H), y = (int)(row - (long long)b * H);
        {
            const long long o0 = (((long long)b * (H + 2) + y + 1) * (W + 2) + 1) * C;
            const long long o = o0 + (long long)k * V;
            if constexpr (V == 8) {
                const uint4 d4 = *reinterpret_cast<const uint4 *>(dh + o);
                const uint4 p4 = *reinterpret_cast<const uint4 *>(pre + o);
                const uint32_t dw[4] = {d4.x, d4.y, d4.z, d4.w}, pw[4] = {p4.x, p4.y, p4.z, p4.w};
                uint32_t ow[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float d0 = __uint_as_float(dw[e] << 16), d1 = __uint_as_float(dw[e] & 0xFFFF0000u);
                    const float p0 = __uint_as_float(pw[e] << 16), p1 = __uint_as_float(pw[e] & 0xFFFF0000u);
                    ow[e] = pack2(__float2bfloat16(d0 * gelu_grad(p0)), __float2bfloat16(d1 * gelu_grad(p1)));
                }
                *reinterpret_cast<uint4 *>(dpre + o) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
            } else {
                dpre[o] = __float2bfloat16(__bfloat162float(dh[o]) * gelu_grad(__bfloat162float(pre[o])));
            }
        }
    }
}

// Weight and bias gradients:
//   dW[tap][co][ci] = sum_p dpre[p][co] * in[p + off(tap)][ci],  db[co] = sum_p dpre[p][co]
// A contraction over the pixels, on mma.sync (M = co, N = ci, K = 16 pixels), one
// warp a tap; warp 4 also multiplies dpre by a column of ones, which is db.  (A
// product for the tensor memory's units would stack the taps, dx and ci along M,
// dy and co along N, both operands channel by channel; not tried.)  A CTA walks segments of kWgSeg pixels counted over the
// padded rows as k_conv_tc counts them (a grid-stride loop over the segments
// of all images; dpre enters as 0 for the two columns a row that are no pixels):
// it stages the segment's dpre and the input that its taps read in shared memory (16-byte
// cp.async, two buffers: the next segment loads while this one multiplies),
// pixels kWgStride bytes apart so that ldmatrix reads eight pixels' 16 bytes
// without bank conflicts, and takes both operands transposed by
// ldmatrix.trans.  Each CTA writes one partial [9][COUTP][CIN] (and [COUTP]).
constexpr int kWgSeg = 64;
constexpr int kWgThreads = 288;
__host__ __device__ constexpr int wg_stride(int ch) { return ch * 2 + 16; }
__host__ __device__ constexpr int wg_buffer(int cin, int coutp) {
    return 3 * (kWgSeg + 2) * wg_stride(cin) + kWgSeg * wg_stride(coutp);
}

__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}

// eight channels to shared memory, or zeros; buffers that are not 16-byte
// aligned go through registers
__device__ __forceinline__ void stage16(uint32_t dst, const bf16 *src, bool ok, const bf16 *any, bool aligned) {
    if (aligned) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(ok ? src : any), "r"(ok ? 16 : 0));
    } else {
        uint32_t v[4] = {0u, 0u, 0u, 0u};
        if (ok) {
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = pack2(src[2 * e], src[2 * e + 1]);
        }
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3])
                     : "memory");
    }
}

template <int CIN, int COUTP>
__global__ void __launch_bounds__(kWgThreads) k_wgrad(const bf16 *__restrict__ dpre, const bf16 *__restrict__ in,
                                                      float *__restrict__ partial, float *__restrict__ dbpart,
                                                      int B, int H, int W) {
    constexpr int SI = wg_stride(CIN), SO = wg_stride(COUTP);
    constexpr int BUF = wg_buffer(CIN, COUTP);
    constexpr int MT = COUTP / 16, NT = CIN / 8;
    extern __shared__ __align__(16) unsigned char wsm[];
    const uint32_t sm0 = smem_addr(wsm);
    const int tid = threadIdx.x, lane = tid & 31, tap = tid >> 5;
    const int dy = tap / 3, dx = tap % 3;
    float acc[MT][NT][4], accb[MT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i) {
        accb[i][0] = accb[i][1] = accb[i][2] = accb[i][3] = 0.f;
#pragma unroll
        for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
    }
    const int Wp = W + 2;
    const long long npix = (long long)H * Wp, in_pix = (long long)(H + 2) * Wp;
    const long long segs = (npix + kWgSeg - 1) / kWgSeg, tasks = segs * B;
    const bool aligned = (((uintptr_t)dpre | (uintptr_t)in) & 15) == 0;
    auto stage = [&](long long t, int buf) {
        const int b = (int)(t / segs);
        const long long q0 = (t - b * segs) * kWgSeg;
        const uint32_t base = sm0 + buf * BUF;
        constexpr int CI8 = CIN / 8, CO8 = COUTP / 8;
        const bf16 *ip = in + (long long)b * in_pix * CIN;
        static_assert(kWgThreads / CI8 >= kWgSeg + 2 && kWgThreads / CO8 >= kWgSeg, "one copy a thread and row");
        {
            const int c = tid % CI8, j = tid / CI8;
            if (j < kWgSeg + 2) {
                const long long s = q0 + j;
                const bf16 *src = ip + s * CIN + 8 * c;
#pragma unroll
                for (int r = 0; r < 3; ++r)
                    stage16(base + (r * (kWgSeg + 2) + j) * SI + c * 16, src + (long long)r * Wp * CIN,
                            s + (long long)r * Wp < in_pix, ip, aligned);
            }
        }
        const bf16 *dp = dpre + (long long)b * in_pix * COUTP;
        {
            const int c = tid % CO8, j = tid / CO8;
            if (j < kWgSeg) {
                const long long q = q0 + j;
                stage16(base + 3 * (kWgSeg + 2) * SI + j * SO + c * 16, dp + (q + Wp + 1) * COUTP + 8 * c,
                        q < npix && (int)(q % Wp) < W, dp, aligned);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    long long q = blockIdx.x;
    int buf = 0;
    if (q < tasks) stage(q, 0);
    for (; q < tasks; q += gridDim.x, buf ^= 1) {
        if (q + gridDim.x < tasks) {
            stage(q + gridDim.x, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const uint32_t sin = sm0 + buf * BUF + (dy * (kWgSeg + 2) + dx) * SI;
        const uint32_t sdp = sm0 + buf * BUF + 3 * (kWgSeg + 2) * SI;
#pragma unroll 2
        for (int p0 = 0; p0 < kWgSeg; p0 += 16) {
            // 8 x 8 blocks [pixel][channel], transposed by the load: lane l
            // addresses pixel l % 8 (+8 by bit 3 or 4) of its block
            uint32_t a[MT][4], b[NT / 2][4];
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)  // (co, px): (0,0) (8,0) (0,8) (8,8)
                ldsm4t(a[mt], sdp + (p0 + (lane & 7) + ((lane >> 4) & 1) * 8) * SO + (mt * 16 + ((lane >> 3) & 1) * 8) * 2);
#pragma unroll
            for (int n2 = 0; n2 < NT / 2; ++n2)  // (px, ci): (0,0) (8,0) (0,8) (8,8)
                ldsm4t(b[n2], sin + (p0 + (lane & 7) + ((lane >> 3) & 1) * 8) * SI + (n2 * 16 + ((lane >> 4) & 1) * 8) * 2);
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
                    mma16816(acc[mt][nt], a[mt][0], a[mt][1], a[mt][2], a[mt][3], b[nt / 2][(nt & 1) * 2],
                             b[nt / 2][(nt & 1) * 2 + 1]);
                if (tap == 4) mma16816(accb[mt], a[mt][0], a[mt][1], a[mt][2], a[mt][3], 0x3F803F80u, 0x3F803F80u);
            }
        }
        __syncthreads();  // the buffer is loaded again in the next iteration
    }
    const int g = lane >> 2, t = lane & 3;
    float *pp = partial + ((long long)blockIdx.x * 9 + tap) * COUTP * CIN;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const int co = mt * 16 + g, ci = nt * 8 + 2 * t;
            pp[co * CIN + ci] = acc[mt][nt][0];
            pp[co * CIN + ci + 1] = acc[mt][nt][1];
            pp[(co + 8) * CIN + ci] = acc[mt][nt][2];
            pp[(co + 8) * CIN + ci + 1] = acc[mt][nt][3];
        }
        if (tap == 4 && t == 0 && dbpart) {
            dbpart[(long long)blockIdx.x * COUTP + mt * 16 + g] = accb[mt][0];
            dbpart[(long long)blockIdx.x * COUTP + mt * 16 + g + 8] = accb[mt][2];
        }
    }
}

// dW (and db) = sum over CTAs of the partials: a CTA takes 32 values, its 8
// warps every eighth partial each, then the warps' sums in order
__global__ void __launch_bounds__(256) k_wreduce(const float *__restrict__ partial, float *__restrict__ dw, int n,
                                                 const float *__restrict__ dbpart, float *__restrict__ db, int nb,
                                                 int nparts) {
    const int nblk = (n + 31) / 32;
    const bool bias = (int)blockIdx.x >= nblk;
    const int m = bias ? nb : n;
    const int k = (bias ? (int)blockIdx.x - nblk : (int)blockIdx.x) * 32 + (threadIdx.x & 31);
    const int w = threadIdx.x >> 5;
    const float *src = bias ? dbpart : partial;
    float s = 0.f;
    if (k < m)
        for (int p = w; p < nparts; p += 8) s += src[(long long)p * m + k];
    __shared__ float sh[8][32];
    sh[w][threadIdx.x & 31] = s;
    __syncthreads();
    if (w == 0 && k < m) {
        float t = sh[0][threadIdx.x];
#pragma unroll
        for (int v = 1; v < 8; ++v) t += sh[v][threadIdx.x];
        (bias ? db : dw)[k] = t;
    }
}

// db[c] = sum over interior pixels of dpre[p][c], one CTA per channel: where
// the partial buffer has no room for k_wgrad's (one CTA, a few pixels)
__global__ void k_dbias(const bf16 *__restrict__ dpre, float *__restrict__ db, int C, int B, int H, int W) {
    const int c = blockIdx.x;
    const long long n = (long long)B * H * W;
    float s = 0.f;
    for (long long p = threadIdx.x; p < n; p += blockDim.x) {
        const int x = (int)(p % W), y = (int)((p / W) % H), b = (int)(p / ((long long)W * H));
        s += __bfloat162float(dpre[(((long long)b * (H + 2) + y + 1) * (W + 2) + x + 1) * C + c]);
    }
    __shared__ float sh[256];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int off = 128; off > 0; off >>= 1) {
        if ((int)threadIdx.x < off) sh[threadIdx.x] += sh[threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x == 0) db[c] = sh[0];
}

// Adam on FP32 master parameters
__global__ void k_adam(float *__restrict__ p, const float *__restrict__ gr, float *__restrict__ m,
                       float *__restrict__ v, int n, float lr, float b1, float b2, float eps,
                       float c1, float c2) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const float g = gr[k];
    const float mk = b1 * m[k] + (1.f - b1) * g;
    const float vk = b2 * v[k] + (1.f - b2) * g * g;
    m[k] = mk;
    v[k] = vk;
    p[k] -= lr * (mk / c1) / (sqrtf(vk / c2) + eps);
}

// FP32 [9][COUTP][CIN] -> BF16 forward layout (same) and the data-gradient
// layout [8 - tap][CIN][COUTP]
__global__ void k_pack(const float *__restrict__ w, bf16 *__restrict__ wf, bf16 *__restrict__ wb,
                       int cin, int coutp) {
    const int n = 9 * cin * coutp;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int ci = k % cin, co = (k / cin) % coutp, tap = k / (cin * coutp);
    const bf16 v = __float2bfloat16(w[k]);
    wf[k] = v;
    if (wb) wb[((8 - tap) * cin + ci) * coutp + co] = v;
}

// MSE over the central region of each [H][W] image (margin cells excluded);
// dy[b][y][x][0] = 2 (y - t) / count there and 0 elsewhere (channel stride C);
// per-CTA partial sums of the squared error
__global__ void k_loss(const float *__restrict__ yv, const float *__restrict__ tv, bf16 *__restrict__ dy,
                       float *__restrict__ partial, int C, int B, int H, int W, int margin, float inv_count) {
    const long long n = (long long)B * H * W;
    float s = 0.f;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
         k += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(k % W), y = (int)((k / W) % H), b = (int)(k / ((long long)W * H));
        const bool in_region = x >= margin && x < W - margin && y >= margin && y < H - margin;
        const float e = in_region ? yv[k] - tv[k] : 0.f;
        s += e * e;
        dy[(((long long)b * (H + 2) + y + 1) * (W + 2) + x + 1) * C] = __float2bfloat16(2.f * e * inv_count);
    }
    __shared__ float sh[256];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int off = 128; off > 0; off >>= 1) {
        if ((int)threadIdx.x < off) sh[threadIdx.x] += sh[threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

// crops of a stored dataset into a training batch: fields [N][H][W][F]
// (F-1 features then the target), origins (n, y, x) per batch item; writes
// x [B][S+2][S+2][C] (halo and channels >= F-1 zero) and t [B][S][S]
__global__ void k_gather(const float *__restrict__ fields, const int *__restrict__ org, bf16 *__restrict__ x,
                         float *__restrict__ tgt, int F, int C, int Hs, int Ws, int B, int S) {
    const long long n = (long long)B * S * S;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
         k += (long long)gridDim.x * blockDim.x) {
        const int xx = (int)(k % S), yy = (int)((k / S) % S), b = (int)(k / ((long long)S * S));
        const int sn = org[3 * b], sy = org[3 * b + 1] + yy, sx = org[3 * b + 2] + xx;
        const float *src = fields + (((long long)sn * Hs + sy) * Ws + sx) * F;
        bf16 *dst = x + (((long long)b * (S + 2) + yy + 1) * (S + 2) + xx + 1) * C;
        for (int c = 0; c < C; ++c) dst[c] = __float2bfloat16(c < F - 1 ? src[c] : 0.f);
        tgt[k] = src[F - 1];
    }
}

// which kernel tl_nn_conv runs: the tcgen05 one (default) or mma.sync
bool g_conv_tcgen05 = true;

// tiles of r rows
long long conv_tiles(int r, int B, int H, int W) {
    return (((long long)((H + r - 1) / r) * (W + 2) + kTcPix - 1) / kTcPix) * B;
}
// Rows of a tile: four read an input row least often; one, or two, where the device
// is not full, whose blocks have less to do one after the other, and where taller
// tiles would be no fewer.  Microseconds with 1, 2 and 4 rows, 32 to 32 channels,
// GELU and residual, batch x height x width (one-row tiles in brackets): 8.4, 10.3,
// 12.5 at 1 x 64 x 64 (33), 10.3, 10.5, 12.6 at 1 x 200 x 192 (304), 12.5, 12.4, 12.5 at
// 1 x 256 x 256 (516), 14.5, 14.5, 16.5 at 8 x 100 x 96 (616; 312 of two rows), 16.6, 16.6,
// 16.5 at 12 x 100 x 96 (924; 468), 33, 29, 31 at 16 x 144 x 144, 60, 52, 51 at 32 x 144 x
// 144; the head 6.4, 7.8, 8.3, then 8.3, 8.3, 8.4, 10.3, 8.4, 8.4, 10.5, 10.4, 10.4, 12.5, 11.2,
// 10.5, 25, 21, 19 and 41, 35, 29; 512 x 1 x 32: 10.6, 14.5, 22.6.
int conv_rows(int B, int H, int W) {
    const long long t1 = conv_tiles(1, B, H, W), t2 = conv_tiles(2, B, H, W), t4 = conv_tiles(4, B, H, W);
    if (t1 <= 3 * kSms || t1 <= t2) return 1;
    return t2 <= 3 * kSms || t2 <= t4 ? 2 : 4;
}

template <int CIN, int COUTP, int MODE, int R>
int launch_conv_tc(const void *in, const void *w, const float *bias, const void *res, void *out, void *pre,
                   float *outf, int B, int H, int W, cudaStream_t s) {
    constexpr int bytes = conv_tc_smem<CIN, COUTP, R>();
    const cudaError_t e = cudaFuncSetAttribute(k_conv_tc<CIN, COUTP, MODE, R>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return cuda_fail(e, "conv shared memory");
    const long long tiles = conv_tiles(R, B, H, W), ctas = kSms * tc_ctas(R);
    k_conv_tc<CIN, COUTP, MODE, R><<<(unsigned)(tiles < ctas ? tiles : ctas), 128, bytes, s>>>(
        (const bf16 *)in, (const bf16 *)w, bias, (const bf16 *)res, (bf16 *)out, (bf16 *)pre, outf, B, H, W);
    return TL_OK;
}

template <int CIN, int COUTP, int MODE>
int launch_conv(const void *in, const void *w, const float *bias, const void *res, void *out, void *pre,
                float *outf, int B, int H, int W, cudaStream_t s) {
    if (g_conv_tcgen05) {
        int rc;
        switch (conv_rows(B, H, W)) {
        case 1: rc = launch_conv_tc<CIN, COUTP, MODE, 1>(in, w, bias, res, out, pre, outf, B, H, W, s); break;
        case 2: rc = launch_conv_tc<CIN, COUTP, MODE, 2>(in, w, bias, res, out, pre, outf, B, H, W, s); break;
        default: rc = launch_conv_tc<CIN, COUTP, MODE, 4>(in, w, bias, res, out, pre, outf, B, H, W, s); break;
        }
        if (rc) return rc;
    } else {
        const long long tasks = (long long)B * H * (W / 16);
        const unsigned grid = (unsigned)((tasks + 3) / 4);
        k_conv<CIN, COUTP, MODE><<<grid, 128, 0, s>>>((const bf16 *)in, (const bf16 *)w, bias,
                                                      (const bf16 *)res, (bf16 *)out, (bf16 *)pre, outf, B,
                                                      H, W);
    }
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TL_OK : cuda_fail(e, "conv launch");
}

}  // namespace
}  // namespace tl

using namespace tl;

extern "C" {

int tl_nn_conv(int mode, int cin, int coutp, const void *in, const void *w, const float *bias,
               const void *res, void *out, void *pre, float *outf, int B, int H, int W, void *stream) {
    if (W % 16 != 0 || B < 1 || H < 1) {
        set_error("tl_nn_conv: width must be a multiple of 16 (got %d)", W);
        return TL_ERR_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
#define TL_CONV_CASE(CI, CO, MD)                                                          \
    if (cin == CI && coutp == CO && mode == MD)                                           \
        return launch_conv<CI, CO, MD>(in, w, bias, res, out, pre, outf, B, H, W, s);
    TL_CONV_CASE(16, 32, kModeGelu)
    TL_CONV_CASE(32, 32, kModeGeluRes)
    TL_CONV_CASE(32, 32, kModeGelu)
    TL_CONV_CASE(32, 16, kModeHead)
    TL_CONV_CASE(32, 32, kModeLinear)
    TL_CONV_CASE(16, 32, kModeLinear)
#undef TL_CONV_CASE
    set_error("tl_nn_conv: unsupported shape cin=%d coutp=%d mode=%d", cin, coutp, mode);
    return TL_ERR_ARG;
}

int tl_nn_set_conv_kernel(int tcgen05) {
    g_conv_tcgen05 = tcgen05 != 0;
    return TL_OK;
}

int tl_nn_conv_status(void) {
    int flag = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&flag, g_conv_tc_error, sizeof flag);
    if (e != cudaSuccess) return cuda_fail(e, "tl_nn_conv_status");
    if (flag) {
        const int zero = 0;
        e = cudaMemcpyToSymbol(g_conv_tc_error, &zero, sizeof zero);
        if (e != cudaSuccess) return cuda_fail(e, "tl_nn_conv_status");
        set_error("tcgen05 conv: the wait for the tensor-core result ran out");
        return TL_ERR_CUDA;
    }
    return TL_OK;
}

int tl_nn_gelu_backward(const void *dh, const void *pre, void *dpre, int C, int B, int H, int W, void *stream) {
    const bool vec = C % 8 == 0 && (((uintptr_t)dh | (uintptr_t)pre | (uintptr_t)dpre) & 15) == 0;
    if (vec)
        k_gelu_back<8><<<1216, 256, 0, (cudaStream_t)stream>>>((const bf16 *)dh, (const bf16 *)pre, (bf16 *)dpre, C, B,
                                                              H, W);
    else
        k_gelu_back<1><<<1216, 256, 0, (cudaStream_t)stream>>>((const bf16 *)dh, (const bf16 *)pre, (bf16 *)dpre, C, B,
                                                              H, W);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TL_OK : cuda_fail(e, "gelu backward launch");
}

long long tl_nn_wgrad_partial_floats(int cin, int coutp, int B, int H, int W, int groups_per_cta) {
    const long long groups = (long long)B * H * (W / 16);
    const long long ctas = (groups + groups_per_cta - 1) / groups_per_cta;
    return ctas * 9LL * cin * coutp;
}

// The partial buffer holds one [9][coutp][cin] block per groups_per_cta
// 16-pixel groups (tl_nn_wgrad_partial_floats); the kernel needs far fewer:
// three CTAs a multiprocessor, and behind their blocks the CTAs' db partials
// (one block less than the buffer holds leaves them room).
int tl_nn_wgrad(const void *dpre, const void *in, int cin, int coutp, float *partial, float *dw, float *db,
                int B, int H, int W, int groups_per_cta, void *stream) {
    cudaStream_t s = (cudaStream_t)stream;
    if (W % 16 != 0 || groups_per_cta < 1) {
        set_error("tl_nn_wgrad: bad shape");
        return TL_ERR_ARG;
    }
    const long long groups = (long long)B * H * (W / 16);
    const long long blocks = (groups + groups_per_cta - 1) / groups_per_cta;  // room in `partial`
    const long long tasks = (((long long)H * (W + 2) + kWgSeg - 1) / kWgSeg) * B;
    const int n = 9 * cin * coutp;
    long long ctas = tasks < kSms * 3 ? tasks : kSms * 3;
    const bool bias_here = db && blocks >= 2;
    if (bias_here) {
        // ctas blocks and ctas * coutp floats: floor(blocks * n / (n + coutp))
        const long long fit = blocks * n / (n + coutp);
        if (ctas > fit) ctas = fit;
    } else if (ctas > blocks) {
        ctas = blocks;
    }
    float *dbpart = bias_here ? partial + ctas * n : nullptr;
#define TL_WGRAD_CASE(CI, CO)                                                                                  \
    if (cin == CI && coutp == CO) {                                                                            \
        constexpr int bytes = 2 * wg_buffer(CI, CO);                                                           \
        k_wgrad<CI, CO><<<(unsigned)ctas, kWgThreads, bytes, s>>>((const bf16 *)dpre, (const bf16 *)in, partial, \
                                                                  dbpart, B, H, W);                            \
    } else
    TL_WGRAD_CASE(16, 32)
    TL_WGRAD_CASE(32, 32)
    TL_WGRAD_CASE(32, 16) {
        set_error("tl_nn_wgrad: unsupported shape cin=%d coutp=%d", cin, coutp);
        return TL_ERR_ARG;
    }
#undef TL_WGRAD_CASE
    k_wreduce<<<(n + 31) / 32 + (bias_here ? 1 : 0), 256, 0, s>>>(partial, dw, n, dbpart, db, coutp, (int)ctas);
    if (db && !bias_here) k_dbias<<<coutp, 256, 0, s>>>((const bf16 *)dpre, db, coutp, B, H, W);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TL_OK : cuda_fail(e, "wgrad launch");
}

int tl_nn_adam(float *p, const float *g, float *m, float *v, int n, float lr, float b1, float b2, float eps,
               int step, void *stream) {
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    k_adam<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(p, g, m, v, n, lr, b1, b2, eps, c1, c2);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TL_OK : cuda_fail(e, "adam launch");
}

int tl_nn_pack(const float *w, void *wf, void *wb, int cin, int coutp, void *stream) {
    const int n = 9 * cin * coutp;
    k_pack<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(w, (bf16 *)wf, (bf16 *)wb, cin, coutp);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TL_OK : cuda_fail(e, "pack launch");
}

int tl_nn_loss(const float *y, const float *t, void *dy, float *partial, int C, int B, int H, int W,
               int margin, void *stream) {
    const long long cnt = (long long)B * (H - 2 * margin) * (W - 2 * margin);
    if (cnt <= 0) {
        set_error("tl_nn_loss: margin too large");
        return TL_ERR_ARG;
    }
    k_loss<<<1216, 256, 0, (cudaStream_t)stream>>>(y, t, (bf16 *)dy, partial, C, B, H, W, margin,
                                                   (float)(1.0 / (double)cnt));
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TL_OK : cuda_fail(e, "loss launch");
}

int tl_nn_gather(const float *fields, const int *org, void *x, float *t, int F, int C, int Hs, int Ws, int B,
                 int S, void *stream) {
    k_gather<<<1216, 256, 0, (cudaStream_t)stream>>>(fields, org, (bf16 *)x, t, F, C, Hs, Ws, B, S);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TL_OK : cuda_fail(e, "gather launch");
}

}  // extern "C"
