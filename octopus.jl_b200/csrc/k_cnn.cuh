// Element-wise and reduction kernels of the learned field correction's CNN (a 4-level U-Net of 3x3
// convolutions, 32 base channels).  The convolutions themselves run on the tensor cores (k_conv.cuh, k_umma.cuh); these
// kernels move activations between them: 2x2 average pooling, nearest upsampling with skip concatenation,
// the adjoints of both, ReLU masks, transposes and im2col for the weight gradients, the fixed-order
// reductions of the weight and bias gradients, the loss, and Adam.  Activations are NHWC bf16 with rows
// m = (b * H + y) * W + x; gradients are accumulated in fp32 and rounded to bf16 where a GEMM reads them.
// Every reduction folds in a fixed order, so a training step is deterministic.  Channel counts are multiples of 8, so
// the element-wise kernels move 8 channels (16 bytes of bf16) a thread.
#pragma once
#include <cuda_bf16.h>

#include "octo_internal.cuh"

namespace octo {
namespace nn {

using bf16 = __nv_bfloat16;

struct Bf8 {
    float v[8];
};
__device__ __forceinline__ Bf8 load_bf8(const bf16 *p) {
    const uint4 q = *reinterpret_cast<const uint4 *>(p);
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&q);
    Bf8 r;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        r.v[2 * e] = __low2float(h[e]);
        r.v[2 * e + 1] = __high2float(h[e]);
    }
    return r;
}
__device__ __forceinline__ void store_bf8(bf16 *p, const float (&v)[8]) {
    uint4 q;
    __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&q);
#pragma unroll
    for (int e = 0; e < 4; ++e) h[e] = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
    *reinterpret_cast<uint4 *>(p) = q;
}
__device__ __forceinline__ Bf8 load_f8(const float *p) {
    const float4 a = reinterpret_cast<const float4 *>(p)[0], b = reinterpret_cast<const float4 *>(p)[1];
    return Bf8{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
}
__device__ __forceinline__ void store_f8(float *p, const float (&v)[8]) {
    reinterpret_cast<float4 *>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4 *>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
}

// Element i of a tensor of C8 groups of 8 channels: its group, pixel column, row and image.
struct Pix {
    int c, x, y, b;
    __device__ __forceinline__ Pix(long long i, int C8, int W, int H) {
        c = (int)(i % C8) * 8;
        i /= C8;
        x = (int)(i % W);
        i /= W;
        y = (int)(i % H);
        b = (int)(i / H);
    }
};

// out[b][y][x][c] = mean of the 2x2 block of in (H, W even).
__global__ void k_cnn_pool(const bf16 *__restrict__ in, bf16 *__restrict__ out, int B, int H, int W, int C) {
    pdl_wait();
    pdl_release();
    const int Ho = H / 2, Wo = W / 2;
    const long long n = (long long)B * Ho * Wo * (C / 8);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const Pix p(i, C / 8, Wo, Ho);
        const bf16 *r = in + (((long long)p.b * H + 2 * p.y) * W + 2 * p.x) * C + p.c;
        const Bf8 q0 = load_bf8(r), q1 = load_bf8(r + C), q2 = load_bf8(r + (long long)W * C),
                  q3 = load_bf8(r + (long long)W * C + C);
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = 0.25f * (q0.v[e] + q1.v[e] + q2.v[e] + q3.v[e]);
        store_bf8(out + i * 8, v);
    }
}

// out[b][y][x][0..Cu) = coarse[b][y/2][x/2][..] (nearest upsampling), out[..][Cu..Cu+Cs) = skip[b][y][x][..].
__global__ void k_cnn_upcat(const bf16 *__restrict__ coarse, const bf16 *__restrict__ skip, bf16 *__restrict__ out, int B,
                            int H, int W, int Cu, int Cs) {
    pdl_wait();
    pdl_release();
    const int C = Cu + Cs;
    const long long n = (long long)B * H * W * (C / 8);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const Pix p(i, C / 8, W, H);
        const bf16 *src = p.c < Cu ? coarse + (((long long)p.b * (H / 2) + p.y / 2) * (W / 2) + p.x / 2) * Cu + p.c
                                   : skip + (((long long)p.b * H + p.y) * W + p.x) * Cs + (p.c - Cu);
        *reinterpret_cast<uint4 *>(out + i * 8) = *reinterpret_cast<const uint4 *>(src);
    }
}

// g = bf16(dy * (y > 0)): the gradient through a ReLU whose output y was stored (n a multiple of 8).
__global__ void k_cnn_relu_grad(const float *__restrict__ dy, const bf16 *__restrict__ y, bf16 *__restrict__ g, long long n) {
    pdl_wait();
    pdl_release();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n / 8; i += (long long)gridDim.x * blockDim.x) {
        const Bf8 d = load_f8(dy + i * 8), a = load_bf8(y + i * 8);
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = a.v[e] > 0.f ? d.v[e] : 0.f;
        store_bf8(g + i * 8, v);
    }
}

// Adjoint of k_cnn_upcat: dcoarse[b][y][x][c] = sum of the 2x2 fine children's du[..][c] (c < Cu), and
// dskip (fine) = du[..][Cu + c].
__global__ void k_cnn_upcat_adj(const float *__restrict__ du, float *__restrict__ dcoarse, float *__restrict__ dskip, int B,
                                int H, int W, int Cu, int Cs) {
    pdl_wait();
    pdl_release();
    const int C = Cu + Cs, Hc = H / 2, Wc = W / 2;
    const long long nc = (long long)B * Hc * Wc * (Cu / 8), nf = (long long)B * H * W * (Cs / 8);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nc + nf; i += (long long)gridDim.x * blockDim.x) {
        if (i < nc) {
            const Pix p(i, Cu / 8, Wc, Hc);
            const float *f = du + (((long long)p.b * H + 2 * p.y) * W + 2 * p.x) * C + p.c;
            const Bf8 q0 = load_f8(f), q1 = load_f8(f + C), q2 = load_f8(f + (long long)W * C),
                      q3 = load_f8(f + (long long)W * C + C);
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = (q0.v[e] + q1.v[e]) + (q2.v[e] + q3.v[e]);
            store_f8(dcoarse + i * 8, v);
        } else {
            const long long j = i - nc;
            const Pix p(j, Cs / 8, W, H);
            const Bf8 d = load_f8(du + (((long long)p.b * H + p.y) * W + p.x) * C + Cu + p.c);
            store_f8(dskip + j * 8, d.v);
        }
    }
}

// Adjoint of k_cnn_pool added into the fine gradient: ds[child] += dp[parent] / 4.
__global__ void k_cnn_pool_adj_add(const float *__restrict__ dp, float *__restrict__ ds, int B, int H, int W, int C) {
    pdl_wait();
    pdl_release();
    const long long n = (long long)B * H * W * (C / 8);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const Pix p(i, C / 8, W, H);
        Bf8 d = load_f8(ds + i * 8);
        const Bf8 q = load_f8(dp + (((long long)p.b * (H / 2) + p.y / 2) * (W / 2) + p.x / 2) * C + p.c);
#pragma unroll
        for (int e = 0; e < 8; ++e) d.v[e] += 0.25f * q.v[e];
        store_f8(ds + i * 8, d.v);
    }
}

// Transposed im2col of a 3x3 / pad-1 convolution's NHWC input: out[(tap * C + c)][m] = x[pixel m shifted by tap][c]
// (zero outside the image and for M <= m < ld); TAPS = 1: the plain transpose, out[c][m] = x[m][c]; TAPS = 3: the three
// column shifts alone, out[(dx * C + c)][m] = x[pixel m shifted by dx - 1 in its row][c].
// Bound by the write of out.  A block moves CG channels of 2048 / CG pixels for one tap through shared memory: one
// 16-byte load of 8 channels and one 16-byte store of 8 pixels a thread (one element a thread, with its own divisions
// and a load 2 C bytes from its neighbour's, took 1.79 ms of a batch-64 training step; this takes
// 0.23 ms, for all layers, and 0.12 ms with the column shifts alone where the weight gradient's GEMM can take them).
// grid (ceil(ld / pixels), C / CG, TAPS); out rows and ld are multiples of 8 elements.
constexpr int kIm2colThreads = 256;
template <int CG, int TAPS>
__global__ void __launch_bounds__(kIm2colThreads) k_cnn_im2col_t(const bf16 *__restrict__ x, bf16 *__restrict__ out,
                                                                 long long M, int H, int W, int C, long long ld) {
    pdl_wait();
    pdl_release();
    constexpr int Q = CG / 8, PT = kIm2colThreads / Q, ROW = PT + 2;  // ROW / 2 words, odd: rows fall in other banks
    __shared__ __align__(16) bf16 tile[CG * ROW];
    const long long m0 = (long long)blockIdx.x * PT;
    const int c0 = blockIdx.y * CG, tap = blockIdx.z;
    {
        const int q = threadIdx.x % Q, p = threadIdx.x / Q;
        const long long m = m0 + p;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (m < M) {
            if (TAPS == 1) {
                v = *reinterpret_cast<const uint4 *>(x + m * C + c0 + q * 8);
            } else {
                const long long row = m / W;
                const int xx = (int)(m - row * W) + tap % 3 - 1, dy = TAPS == 3 ? 0 : tap / 3 - 1, yy = (int)(row % H) + dy;
                if (yy >= 0 && yy < H && xx >= 0 && xx < W)
                    v = *reinterpret_cast<const uint4 *>(x + (m + (long long)dy * W + tap % 3 - 1) * C + c0 + q * 8);
            }
        }
        const bf16 *h = reinterpret_cast<const bf16 *>(&v);
#pragma unroll
        for (int e = 0; e < 8; ++e) tile[(q * 8 + e) * ROW + p] = h[e];
    }
    __syncthreads();
    const int r = threadIdx.x / (PT / 8), u = threadIdx.x % (PT / 8);
    const long long m = m0 + u * 8;
    if (m >= ld) return;
    const uint32_t *src = reinterpret_cast<const uint32_t *>(tile + r * ROW + u * 8);
    *reinterpret_cast<uint4 *>(out + ((long long)tap * C + c0 + r) * ld + m) = make_uint4(src[0], src[1], src[2], src[3]);
}

// Per-block sums of the output gradient's channels, bpart[block][c] = sum over the block's pixels of g[m][c]: each
// thread adds 8 channels of every (256 / (C / 8))th pixel, then the block folds its threads in order.  grid kBiasBlocks.
constexpr int kBiasBlocks = 148;
__global__ void __launch_bounds__(256) k_cnn_bias_part(const bf16 *__restrict__ g, long long M, int C,
                                                       float *__restrict__ bpart) {
    pdl_wait();
    pdl_release();
    __shared__ float red[256][9];
    const int c8 = C / 8, q = threadIdx.x % c8, rows = 256 / c8, r = threadIdx.x / c8;
    const long long per = (M + kBiasBlocks - 1) / kBiasBlocks, m1 = min(M, (blockIdx.x + 1) * per);
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (long long m = blockIdx.x * per + r; m < m1; m += rows) {
        const Bf8 v = load_bf8(g + m * C + q * 8);
#pragma unroll
        for (int e = 0; e < 8; ++e) s[e] += v.v[e];
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) red[threadIdx.x][e] = s[e];
    __syncthreads();
    if ((int)threadIdx.x >= C) return;
    float t = 0.f;
    for (int k = 0; k < rows; ++k) t += red[k * c8 + threadIdx.x / 8][threadIdx.x % 8];
    bpart[(long long)blockIdx.x * C + threadIdx.x] = t;
}

// dW[co][k] = sum over the splits s of part[s][k][co], the weight-gradient GEMM's split-K partials, transposed to the
// weights' [Cout][9 Cin] layout; and db[co], the sum of k_cnn_bias_part's blocks.  A block takes 32 outputs; its 8 warps
// sum every 8th term of them and are folded in order (a thread adding its output's up to 296 terms one after the other
// waits for memory some 20 us a layer).
__global__ void __launch_bounds__(256) k_cnn_wgrad_reduce(const float *__restrict__ part, int splits, int K9, int Cout,
                                                          float *__restrict__ dw, const float *__restrict__ bpart,
                                                          float *__restrict__ db) {
    pdl_wait();
    pdl_release();
    __shared__ float red[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long n = (long long)K9 * Cout, groups = (n + 31) / 32;  // whole groups of weights, then of biases
    for (long long g = blockIdx.x; g < groups + (Cout + 31) / 32; g += gridDim.x) {
        const bool bias = g >= groups;
        const long long i = (bias ? g - groups : g) * 32 + lane, count = bias ? Cout : n;
        const float *p = bias ? bpart : part;
        const int terms = bias ? kBiasBlocks : splits;
        float s = 0.f;
        if (i < count) {
#pragma unroll 8
            for (int z = warp; z < terms; z += 8) s += p[z * count + i];
        }
        red[warp][lane] = s;
        __syncthreads();
        if (warp == 0 && i < count) {
#pragma unroll
            for (int w = 1; w < 8; ++w) s += red[w][lane];
            if (bias) db[i] = s;
            else dw[(i % Cout) * K9 + i / Cout] = s;
        }
        __syncthreads();
    }
}

// Sums of the pixel weights by block, for the loss's normalisation.  grid kMaskBlocks.
constexpr int kMaskBlocks = 64;
__global__ void __launch_bounds__(256) k_cnn_mask_sum(const float *__restrict__ mask, long long M, double *__restrict__ wpart) {
    pdl_wait();
    pdl_release();
    __shared__ double red[8];
    double s = 0.0;
#pragma unroll 8
    for (long long m = (long long)blockIdx.x * 256 + threadIdx.x; m < M; m += (long long)kMaskBlocks * 256) s += (double)mask[m];
#pragma unroll
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x) return;
    for (int w = 1; w < 8; ++w) s += red[w];
    wpart[blockIdx.x] = s;
}

// Weights of one layer from the fp32 master copy: w[co][tap][ci] as bf16, and the flipped transpose the input
// gradient's convolution uses: wf[ci][tap'][co] = w[co][8 - tap'][ci].
__global__ void k_cnn_weights(const float *__restrict__ master, int Cout, int Cin, bf16 *__restrict__ w, bf16 *__restrict__ wf) {
    pdl_wait();
    pdl_release();
    const int n = Cout * 9 * Cin;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int ci = i % Cin, tap = (i / Cin) % 9, co = i / (9 * Cin);
        const bf16 v = __float2bfloat16_rn(master[i]);
        w[i] = v;
        if (wf) wf[((long long)ci * 9 + (8 - tap)) * Cout + co] = v;
    }
}

// Masked mean-square loss over output channels 0 and 1 of an 8-channel fp32 head: out[m][c] against
// target[m][c] (2 channels), weight mask[m] (null = 1), normalised by the total weight (k_cnn_mask_sum's wpart; M
// without a mask).  Writes the loss gradient 2 w (out - target) * scale as bf16 (channels 2..7 zero) and per-block
// partial sums of w (out - target)^2 and of w.
__global__ void __launch_bounds__(256) k_cnn_loss(const float *__restrict__ out, const float *__restrict__ target,
                                                   const float *__restrict__ mask, long long M,
                                                   const double *__restrict__ wpart, bf16 *__restrict__ dout,
                                                   double *__restrict__ partial) {
    pdl_wait();
    pdl_release();
    __shared__ float sscale;
    if (threadIdx.x == 0) {
        double wt = (double)M;
        if (mask) {
            wt = 0.0;
            for (int b = 0; b < kMaskBlocks; ++b) wt += wpart[b];
        }
        sscale = (float)(1.0 / (2.0 * fmax(wt, 1e-300)));  // mean over 2 channels
    }
    __syncthreads();
    const float scale = sscale;
    __shared__ double red[2][256];
    double se = 0.0, sw = 0.0;
    for (long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x; m < M; m += (long long)gridDim.x * blockDim.x) {
        const float w = mask ? mask[m] : 1.f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            float gv = 0.f;
            if (c < 2) {
                const float d = out[m * 8 + c] - target[m * 2 + c];
                se += (double)w * (double)d * (double)d;
                gv = 2.f * w * d * scale;
            }
            dout[m * 8 + c] = __float2bfloat16_rn(gv);
        }
        sw += (double)w;
    }
    red[0][threadIdx.x] = se;
    red[1][threadIdx.x] = sw;
    __syncthreads();
    for (int o = 128; o; o >>= 1) {
        if ((int)threadIdx.x < o) {
            red[0][threadIdx.x] += red[0][threadIdx.x + o];
            red[1][threadIdx.x] += red[1][threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        partial[2 * blockIdx.x] = red[0][0];
        partial[2 * blockIdx.x + 1] = red[1][0];
    }
}

// Adam (Kingma & Ba 2015) on the fp32 master parameters; bias corrections from the step count t.
__global__ void k_cnn_adam(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m1, float *__restrict__ m2,
                           long long n, float lr, float b1, float b2, float eps, float c1, float c2) {
    pdl_wait();
    pdl_release();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float a = b1 * m1[i] + (1.f - b1) * gi;
        const float b = b2 * m2[i] + (1.f - b2) * gi * gi;
        m1[i] = a;
        m2[i] = b;
        p[i] -= lr * (a / c1) / (sqrtf(b / c2) + eps);
    }
}

}  // namespace nn
}  // namespace octo
