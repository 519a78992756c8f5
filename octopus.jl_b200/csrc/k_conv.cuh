// 3x3 / padding-1 convolution of an NHWC bf16 tensor on the fifth-generation tensor cores, one band of output rows of
// one image a CTA: the forward layers and the input gradients of the learned field correction's network.
//
// The band's input rows (with their halo, zero-padded to W + 2 columns) are brought into shared memory once, as one
// plane of 16-byte pixels per 8 channels.  Pixel p of a plane lies 16 p bytes after its start, which is the canonical
// no-swizzle K-major layout with 8-row groups 128 bytes apart, so the A operand of a tap is the same planes read from
// a start address 16 bytes x (dy (W + 2) + dx) further on: no im2col is written or loaded.  Row o = y (W + 2) + x of
// the product is output pixel (y, x); the two columns x >= W of each row are computed and dropped (4 % at W = 48).
// The weights of the CTA's NB output channels lie beside it in the same form.  A warp's first lane issues every
// tcgen05.mma (M = 128 pixels, N = NB, K = 16) of its share of the tiles' parts of K into TMEM and commits once; an
// instruction's operands are two additions away from the one before (rebuilt descriptors made the issuing lane the
// layer's longest part).
//   C = 8: the two K halves of an instruction are two taps, their distance in the plane the descriptor's leading
//   offset (16 bytes, or to the next row of taps); the ninth tap's partner is a block of zeros with zero weights, so no
//   pixel outside an output's nine taps enters its sum, were it infinite.
//   parts: where the im2col GEMM of a small layer splits K, a tile has an accumulator for each of its parts, issued by
//   warps of their own, and the epilogue adds them in order: a layer's fp32 sums are the GEMM's to the bit, whichever of
//   the two runs it.
//   pool: the input is read as the 2x2 average of a tensor of twice the height and width.
//   skip: the input is [nearest-upsampled in (Cu channels), skip] (a decoder level).
// Bound by latency: a layer is a few microseconds of loads, instructions and stores between two launches.  The im2col
// GEMM (k_umma.cuh) reads every input nine times in K chunks that wait for one another: a forward pass over 20 planes of
// 48 x 48 took 304 us with it (split-K folds and pools included) and takes 167 us (158 with each layer's sum in one part:
// the accumulators of the parts take TMEM, and the second 128-channel layer runs a second wave of CTAs).
//
// The mbarrier wait is bounded (about one second of the global timer); on expiry the kernel records OCTO_ERR_TIMEOUT
// in *error after a second such wait for the instructions in flight, frees its TMEM and returns.
#pragma once
#include <algorithm>

#include "k_cnn.cuh"
#include "k_umma.cuh"

namespace octo {
namespace nn {

constexpr int kConvThreads = 256;

struct ConvArgs {
    const bf16 *in, *skip;   // skip: null, or [b][H][W][C - Cu] beside the upsampled in [b][H/2][W/2][Cu]
    int Cu, pool;            // pool: in is [b][2H][2W][C]
    int H, W, C;             // C = 8 or a multiple of 16 with C / 8 a divisor of the block; Cu a multiple of 8
    const bf16 *w;           // [N][3][3][C]
    int N;                   // output channels (row length of the output)
    const float *bias;       // null: none
    int relu;
    bf16 *out_bf16;          // bf16 result, or null:
    float *out;              // fp32 result
    int parts, part_steps;   // parts of K (C = 8: one) and the 16-channel steps of each but the last
    int *error;
    // the split (conv_plan): rows a band, 128-row tiles a band, pixels of a plane (odd), TMEM columns
    int R, tiles, plane, cols;
};

// Shared memory of a CTA: weights (16-byte chunks, an even number), input planes, and for C = 8 the ninth tap's zeros.
constexpr int kConvZeros = 128 * 16;
__host__ __device__ inline int conv_chunks(int C) { return C == 8 ? 10 : 9 * (C / 8); }
inline size_t conv_smem(int C, int nb, int plane) {
    return (size_t)conv_chunks(C) * nb * 16 + (size_t)(C / 8) * plane * 16 + (C == 8 ? kConvZeros : 0);
}

// Rows a band for B images at nb channels a CTA: the least of a launch's fixed latency per wave, the bytes each SM brings
// in and the instructions it issues, over the bands that fit (TMEM, half of it for a sum in one part, and kConvSmem:
// 227 KB less the 1 KB of this kernel itself).  Returns that cost, in microseconds: the three weights are a least-squares
// fit to the 33 launches of forward passes over 1, 20 and 64 images of 48 x 48 (5.4 to 34 us each, cold caches under ncu),
// which it gives within 12 % rms; 1e30 when no band fits (very wide images: the im2col GEMM runs those).  While bands were
// held to 200 KB the widest decoder layer (256 to 64 channels, 12 x 12, 20 images) ran 240 CTAs in two waves, 31 us; now
// one band an image, 80 CTAs, 19 us.
constexpr size_t kConvSmem = 226 * 1024;
constexpr double kConvNone = 1e30;
inline double conv_plan(ConvArgs &g, int B, int nb, int sms) {
    if ((g.C % 16 && g.C != 8) || kConvThreads % (g.C / 8)) return kConvNone;
    const int wp = g.W + 2, nblk = (g.N + nb - 1) / nb, steps = conv_chunks(g.C) / 2;
    double best = kConvNone;
    for (int R = 1; R <= g.H; ++R) {
        const int tiles = (R * wp + 127) / 128;
        if (tiles * nb * g.parts > (g.parts == 1 ? 256 : 512)) break;
        const int plane = (tiles * 128 + 2 * wp + 4) | 1;
        const size_t smem = conv_smem(g.C, nb, plane);
        if (smem > kConvSmem) break;
        int cols = 32;
        while (cols < tiles * nb * g.parts) cols *= 2;
        const long long ctas = (long long)((g.H + R - 1) / R) * B * nblk;
        const int res = (int)std::min<long long>({(long long)(228 * 1024 / (smem + 2048)), 512 / cols, 8});
        const double per_sm = (double)((ctas + sms - 1) / sms), waves = (double)((ctas + (long long)sms * res - 1) / ((long long)sms * res));
        const double cost = 5.8 * waves + per_sm * (smem * 1.5e-5 + 0.026 * tiles * steps * (nb / 16));
        if (cost < best) {
            best = cost;
            g.R = R;
            g.tiles = tiles;
            g.plane = plane;
            g.cols = cols;
        }
    }
    return best;
}

// grid (bands of an image x images, ceil(N / NB)): the images lie on x, whose limit no batch reaches.
template <int NB>
__global__ void __launch_bounds__(kConvThreads) k_conv3(const __grid_constant__ ConvArgs g) {
    static_assert(NB == 16 || NB == 32, "NB");
    extern __shared__ __align__(1024) unsigned char g_umma_smem[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    __shared__ float sbias[NB];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int c8 = g.C / 8, n0 = blockIdx.y * NB, wp = g.W + 2;
    const int bands = (g.H + g.R - 1) / g.R, y0 = (int)(blockIdx.x % bands) * g.R, rows = min(g.R, g.H - y0);
    const int tiles = (rows * wp + 127) / 128, units = tiles * g.parts, issuers = min(units, kConvThreads / 32);
    const long long img = blockIdx.x / bands;
    const uint32_t sB = smem_u32(g_umma_smem), sA = sB + (uint32_t)(conv_chunks(g.C) * NB * 16),
                   sZ = sA + (uint32_t)(c8 * g.plane * 16);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&bar)), "r"(issuers));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        abort_flag = 0;
    }
    // weights and bias, before the wait on the previous kernel: they are written by k_cnn_weights and k_cnn_adam, which
    // lie at least one whole kernel before it in the stream.  Chunk (tap, 8 channels) of output channel n: [chunk][n] of
    // 16 bytes; for C = 8 a tenth chunk of zeros.  Two chunks of 16 channels a warp.
    if (tid < NB) sbias[tid] = g.bias && n0 + tid < g.N ? g.bias[n0 + tid] : 0.f;
    {
        const int k8 = 9 * c8, chunks = conv_chunks(g.C);
        // a thread keeps its channel and its parity of chunk: 2 NB divides the block
        const int r = tid % (2 * NB), n = r >> 1;
        constexpr int kStep = kConvThreads / NB;
        const bool row = n0 + n < g.N;
        const bf16 *src = g.w + (long long)(row ? n0 + n : 0) * k8 * 8;
        for (int k = 2 * (tid / (2 * NB)) + (r & 1); k < chunks; k += kStep) {
            const bool ok = row && k < k8;
            cp_async16(sB + (uint32_t)((k * NB + n) * 16), ok ? src + k * 8 : g.w, ok ? 16 : 0);
        }
        if (g.C == 8 && tid < kConvZeros / 16) cp_async16(sZ + (uint32_t)(tid * 16), g.w, 0);
    }
    pdl_wait();
    pdl_release();
    // TMEM only now: the previous kernel's CTAs have all ended and freed theirs, so none of them can be waiting for
    // columns that this kernel holds while it waits for them
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(g.cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    // input rows y0 - 1 .. y0 + rows, zero outside the image
    {
        // One 16-byte chunk of a pixel a step: the chunks of a pixel lie side by side in memory, so neighbouring
        // threads take them.  256 is a multiple of c8, so a thread keeps its chunk and walks the pixels by additions
        // alone (with a division or two a chunk this loop was the layer's longest part).
        const int Cs = g.C - g.Cu, pixels = (rows + 2) * wp;
        const int dp = kConvThreads / c8, dy = dp / wp, dx = dp - dy * wp;
        const int k = tid % c8;
        for (int p = tid / c8, y = y0 - 1 + p / wp, x = p % wp - 1; p < pixels; p += dp) {
            const int c = k * 8;
            const uint32_t dst = sA + (uint32_t)((k * g.plane + p) * 16);
            const bool in = y >= 0 && y < g.H && x >= 0 && x < g.W;
            if (g.pool) {
                float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                if (in) {
                    const long long ld = 2LL * g.W * g.C;
                    const bf16 *s = g.in + ((img * 2 * g.H + 2 * y) * 2 * g.W + 2 * x) * g.C + c;
                    const Bf8 q0 = load_bf8(s), q1 = load_bf8(s + g.C), q2 = load_bf8(s + ld), q3 = load_bf8(s + ld + g.C);
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] = 0.25f * (q0.v[e] + q1.v[e] + q2.v[e] + q3.v[e]);
                }
                store_bf8(reinterpret_cast<bf16 *>(g_umma_smem + (dst - sB)), v);
            } else {
                const bf16 *s = g.in;
                if (in) {
                    if (!g.skip) s = g.in + ((img * g.H + y) * g.W + x) * g.C + c;
                    else if (c < g.Cu) s = g.in + ((img * (g.H / 2) + y / 2) * (g.W / 2) + x / 2) * g.Cu + c;
                    else s = g.skip + ((img * g.H + y) * g.W + x) * Cs + (c - g.Cu);
                }
                cp_async16(dst, s, in ? 16 : 0);
            }
            y += dy;
            x += dx;
            if (x >= wp - 1) {
                x -= wp;
                ++y;
            }
        }
    }
    cp_async_commit();
    cp_async_wait<0>();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_slot;
    if (warp < issuers && lane == 0) {
        const uint32_t idesc = umma_idesc_bf16(NB);
        // both descriptors' upper words are constants; the lower words hold the address and, from bit 16 on, the distance
        // of the K halves, in 16-byte units
        const uint64_t da0 = umma_desc(sA, 0, 128), db0 = umma_desc(sB, NB * 16, 128);
        const uint32_t ha = (uint32_t)(da0 >> 32), hb = (uint32_t)(db0 >> 32);
        auto mma = [&](uint32_t d, uint32_t a, uint32_t b, uint32_t acc) {
            asm volatile(
                "{\n\t.reg .pred p;\n\t.reg .b64 x, y;\n\t"
                "setp.ne.b32 p, %6, 0;\n\t"
                "mov.b64 x, {%1, %2};\n\t"
                "mov.b64 y, {%3, %4};\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %5, p;\n\t}"
                :
                : "r"(d), "r"(a), "r"(ha), "r"(b), "r"(hb), "r"(idesc), "r"(acc));
        };
        const int per_tap = g.C / 16, steps = 9 * per_tap;
        for (int u = warp; u < units; u += kConvThreads / 32) {
            const int t = u / g.parts, s0 = (u - t * g.parts) * g.part_steps, s1 = min(steps, s0 + g.part_steps);
            const uint32_t d = tmem + (uint32_t)(u * NB);
            uint32_t b = (uint32_t)db0 + (uint32_t)(s0 * 2 * NB), acc = 0;
            if (g.C == 8) {
#pragma unroll
                for (int tap = 0; tap < 9; tap += 2) {
                    const uint32_t at = (uint32_t)(t * 128 + (tap / 3) * wp + tap % 3);
                    const uint32_t half = tap == 8 ? ((sZ - sA) >> 4) - at
                                                   : (uint32_t)(((tap + 1) / 3 - tap / 3) * wp + (tap + 1) % 3 - tap % 3);
                    mma(d, ((uint32_t)da0 + at) | half << 16, b, tap != 0);
                    b += 2 * NB;
                }
                continue;
            }
            int tap = s0 / per_tap, k = s0 - tap * per_tap;
            for (int s = s0; s < s1; ++tap, k = 0) {
                uint32_t a = ((uint32_t)da0 + (uint32_t)(t * 128 + (tap / 3) * wp + tap % 3 + 2 * k * g.plane)) |
                             (uint32_t)g.plane << 16;
                const int run = min(per_tap - k, s1 - s);
                s += run;
#pragma unroll 2
                for (int i = 0; i < run; ++i) {
                    mma(d, a, b, acc);
                    acc = 1;
                    a += 2u * (uint32_t)g.plane;
                    b += 2 * NB;
                }
            }
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&bar))
                     : "memory");
    }
    if (tid == 0 && !mbar_wait(smem_u32(&bar), 0)) {
        mbar_wait(smem_u32(&bar), 0);
        abort_flag = 1;
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (abort_flag) {
        if (tid == 0 && g.error) atomicExch(g.error, kTimeoutCode);
    } else {
        // warp w reads TMEM lanes 32 (w % 4) .. + 31 of every other tile; a lane holds one pixel, 16 channels at a time
        for (int t = warp >> 2; t < tiles; t += 2) {
            const int o = t * 128 + (warp & 3) * 32 + lane, y = o / wp, x = o - y * wp;
            const bool in = y < rows && x < g.W;
            const long long m = (img * g.H + y0 + y) * g.W + x;
            const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(t * g.parts * NB);
#pragma unroll
            for (int c = 0; c < NB; c += 16) {
                __syncwarp();
                float sum[16];
                for (int z = 0; z < g.parts; ++z) {
                    uint32_t r[16];
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                        "%14, %15}, [%16];"
                        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                          "=r"(r[15])
                        : "r"(taddr + (uint32_t)(z * NB + c)));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        asm volatile("" : "+r"(r[e]));  // the values exist from here on
                        sum[e] = z ? sum[e] + __uint_as_float(r[e]) : __uint_as_float(r[e]);
                    }
                }
#pragma unroll
                for (int h = 0; h < 16; h += 8) {
                    if (!in || n0 + c + h >= g.N) break;  // N is a multiple of 8
                    float v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        v[e] = sum[h + e] + sbias[c + h + e];
                        if (g.relu) v[e] = fmaxf(v[e], 0.f);
                    }
                    if (g.out_bf16) store_bf8(g.out_bf16 + m * g.N + n0 + c + h, v);
                    else store_f8(g.out + m * g.N + n0 + c + h, v);
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(g.cols));
}

}  // namespace nn
}  // namespace octo
