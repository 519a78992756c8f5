// Beam moment rows as the moment observer records them (src/tasks/BeamObservers.jl:1000-1060, 1254-1271):
// the means of the six coordinates, then central moments mean(prod_d (c_d - <c_d>)^p_d) of the requested
// power rows, over the live particles (all six coordinates finite) when lost particles are masked, else
// over all particles (one non-finite particle then makes the row NaN).
//
// One pass over the beam: k_moment_pass sums the six deviations from a pivot near the beam's centre and their 21
// products, and k_moment_finish turns them into the means and the second central moments, m_ij = S_ij / n - d_i d_j
// with d = S / n the mean's offset from the pivot.  The definition takes the means first, in a pass of its own; one
// read of the beam instead of two, and three launches instead of six, took the rows of a 2.56M and a 1.024M-particle
// float64 beam from 128 to 65 us of kernel time together (26 us of reading at the measured copy bandwidth).  The pivot
// (k_moment_pivot) is zero for a centred coordinate, where d is the mean itself, and else the mean of 4096 particles
// spread over the beam (its live ones when lost particles are masked), about sigma / 64 from the mean and at most
// sqrt(n) / 4096 of the sigma that a stray particle makes; either way the
// subtraction loses nothing.  (Zero matters: a mean far smaller than sigma would be the sum of a pivot and its
// opposite, which costs it three digits.)  Rows of order 3 and more (k_moment_general) read the beam
// again, in chunks, with the means known.  Each pass writes per-block partials (a fixed block count) that are summed
// in a fixed order, so a row is deterministic for a given beam size; the row goes to device memory, so observing a
// turn never synchronises the host.
#pragma once
#include "octo_internal.cuh"

namespace octo {

constexpr int kMomentBlocks = 592;      // partial-sum blocks (a fixed count: fold order independent of the GPU)
constexpr int kMomentThreads = 256;
constexpr int kMomentWarps = kMomentThreads / 32;
constexpr int kMomentChunk = 8;         // rows of order >= 3 per generic pass (accumulators held in registers)
constexpr int kMomentPairs = 21;        // second-order rows: the products of deviations (i <= j)
constexpr int kMomentsMax = 256;
constexpr int kMomentSums1 = 6 + kMomentPairs + 1;  // k_moment_pass: deviations, their products, the live count
constexpr int kMeanBlocks = 592, kMeanSums = 7;      // k_moment_means: partial-sum blocks; deviations, the live count

// Rows of order >= 3 of one generic pass.
struct MomentPowers {
    int n;
    unsigned char p[kMomentChunk][6];
    unsigned char slot[kMomentChunk];   // each row's position among the row's moments
};
// Second-order rows: which of the 21 pair sums (pair index of (i, j), i <= j, row-major over the upper
// triangle) goes to which slot.
struct MomentPairRows {
    int n;
    unsigned char pair[kMomentPairs], slot[kMomentPairs];
};
// The order-1 entries of a row: row slot and coordinate of each mean.
struct MomentHead {
    int n;
    unsigned char slot[6], coord[6];
};

__device__ __forceinline__ bool live6(const double (&c)[6]) {
    return isfinite(c[0]) && isfinite(c[1]) && isfinite(c[2]) && isfinite(c[3]) && isfinite(c[4]) && isfinite(c[5]);
}

// Block sums of N per-thread values in a fixed order: a shuffle tree inside each warp, then the warps' sums
// in warp order by thread k < N; partial[blockIdx.x * N + k] receives sum k.
template <int N>
__device__ __forceinline__ void block_sums(double (&v)[N], double *red /* N * kMomentWarps */, double *partial) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        double t = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) red[k * kMomentWarps + warp] = t;
    }
    __syncthreads();
    if ((int)threadIdx.x < N) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < kMomentWarps; ++w) t += red[threadIdx.x * kMomentWarps + w];
        partial[blockIdx.x * N + threadIdx.x] = t;
    }
}

template <class R>
__device__ __forceinline__ void load6(double (&c)[6], const R *x, const R *px, const R *y, const R *py, const R *z,
                                      const R *pz, long long i) {
    c[0] = (double)x[i];
    c[1] = (double)px[i];
    c[2] = (double)y[i];
    c[3] = (double)py[i];
    c[4] = (double)z[i];
    c[5] = (double)pz[i];
}

// The beam's arrays of one moment pass.
template <class R>
struct MomentBeam {
    const R *c[6];
    long long n;
    int mask;
};

// Block d: coordinate d's pivot from 4096 particles spread over the beam, of them the live ones when lost particles are
// masked and else those with a finite value: their mean, or zero when there is none or the mean lies within an eighth of
// their rms spread.  (A lost particle's other coordinates can be anything: taken in, they would put the pivot far from
// the live beam, where the row's differences cancel.)  When every sample is lost, the next live particles of the
// whole beam take their place, which a beam with few of them or none pays for with up to one read of it.
constexpr int kPivotThreads = 1024, kPivotPer = 4;
template <class R>
__global__ void __launch_bounds__(kPivotThreads) k_moment_pivot(const __grid_constant__ MomentBeam<R> B, double *pivot) {
    pdl_wait();
    pdl_release();
    __shared__ double red[3][kPivotThreads / 32];
    __shared__ double total[3];
    const R *c = B.c[blockIdx.x];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr long long kSamples = kPivotThreads * kPivotPer;
    // the sum, the sum of squares and the count of kSamples particles' values, particle(q) the q-th one's index
    auto gather = [&](auto particle) {
        double v[kPivotPer], s[3] = {0.0, 0.0, 0.0};
        bool on[kPivotPer];
#pragma unroll
        for (int k = 0; k < kPivotPer; ++k) {
            const long long i = particle((long long)k * kPivotThreads + threadIdx.x);
            on[k] = i < B.n;
            v[k] = on[k] ? (double)c[i] : 0.0;
            if (B.mask && on[k]) {
                double p[6];
                load6(p, B.c[0], B.c[1], B.c[2], B.c[3], B.c[4], B.c[5], i);
                on[k] = live6(p);
            }
        }
#pragma unroll
        for (int k = 0; k < kPivotPer; ++k)
            if (on[k] && isfinite(v[k])) {
                s[0] += v[k];
                s[1] = fma(v[k], v[k], s[1]);
                s[2] += 1.0;
            }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
            if (lane == 0) red[k][warp] = s[k];
        }
        __syncthreads();
        if (warp == 0) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                s[k] = red[k][lane];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
                if (lane == 0) total[k] = s[k];
            }
        }
        __syncthreads();
    };
    // every particle of a small beam once, else 4096 of them (q n / 4096 without the product's overflow); with lost ones
    // masked, 128 runs of 32 neighbours, whose six loads a particle coalesce (one by one they took 12 us)
    constexpr long long kRuns = kSamples / 32;
    gather([&](long long q) {
        if (B.n <= kSamples) return q;
        const long long m = B.mask ? kRuns : kSamples, g = B.mask ? q / 32 : q;
        return B.n / m * g + B.n % m * g / m + (B.mask ? q % 32 : 0);
    });
    if (B.mask && B.n > kSamples)
        for (long long k = 0; k < B.n && total[2] == 0.0; k += kSamples) gather([&](long long q) { return k + q; });
    if (threadIdx.x != 0) return;
    const double mean = total[0] / total[2], square = total[1] / total[2];
    const bool centred = isfinite(square) && 65.0 * mean * mean <= square;  // mean^2 <= (square - mean^2) / 64
    pivot[blockIdx.x] = isfinite(mean) && !centred ? mean : 0.0;
}

// Bound by HBM with 56 of its registers holding sums: two blocks per SM, and the next two particles' twelve loads
// issued before the current two are summed.  Two particles' terms are added to each other before they go to the sum:
// half as many roundings of the running sums, which is what a covariance near zero shows.
template <class R>
__global__ void __launch_bounds__(kMomentThreads, 2) k_moment_pass(const __grid_constant__ MomentBeam<R> B,
                                                                   const double *pivots, double *partial) {
    pdl_wait();
    pdl_release();
    __shared__ double red[kMomentSums1 * kMomentWarps];
    double pivot[6];
#pragma unroll
    for (int d = 0; d < 6; ++d) pivot[d] = pivots[d];
    double s[kMomentSums1];
#pragma unroll
    for (int k = 0; k < kMomentSums1; ++k) s[k] = 0.0;
    int live = 0;
    auto deviations = [&](const R (&v)[6], bool there, double (&dv)[6]) {
        double c[6];
#pragma unroll
        for (int d = 0; d < 6; ++d) c[d] = (double)v[d];
        const bool on = there && (!B.mask || live6(c));
        live += on;
#pragma unroll
        for (int d = 0; d < 6; ++d) dv[d] = on ? c[d] - pivot[d] : 0.0;
    };
    auto load = [&](R (&v)[6], long long i) {
#pragma unroll
        for (int d = 0; d < 6; ++d) v[d] = B.c[d][i];
    };
    const long long step = (long long)gridDim.x * blockDim.x;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    R na[6], nb[6] = {};
    if (i < B.n) load(na, i);
    if (i + step < B.n) load(nb, i + step);
    while (i < B.n) {
        R a[6], b[6];
#pragma unroll
        for (int d = 0; d < 6; ++d) {
            a[d] = na[d];
            b[d] = nb[d];
        }
        const bool two = i + step < B.n;
        i += 2 * step;
        if (i < B.n) load(na, i);
        if (i + step < B.n) load(nb, i + step);
        double da[6], db[6];
        deviations(a, true, da);
        deviations(b, two, db);
#pragma unroll
        for (int d = 0; d < 6; ++d) s[d] += da[d] + db[d];
        int k = 6;
#pragma unroll
        for (int p = 0; p < 6; ++p)
#pragma unroll
            for (int q = p; q < 6; ++q, ++k) s[k] += fma(da[p], da[q], db[p] * db[q]);
    }
    s[kMomentSums1 - 1] = (double)live;
    block_sums<kMomentSums1>(s, red, partial);
}

// The pass of a row without second-order moments: the deviations alone.  Its pivot only has to lie within some sigma of
// the mean, so each block takes it from the beam's first 32 particles (their mean where that is more than four of their
// rms spreads from zero, else zero) and k_moment_pivot is not launched.  Bound by HBM; four blocks a
// SM with one particle in flight a thread (two, or five and six blocks within fewer registers, measured no better).
// 2.56M and 100,000 float64 particles, orders (1,): 36 and 13 us a row; 46 and 21 by k_moment_pass with its products.
template <class R>
__global__ void __launch_bounds__(kMomentThreads, 4) k_moment_means(const __grid_constant__ MomentBeam<R> B, double *pivots,
                                                                    double *partial) {
    pdl_wait();
    pdl_release();
    __shared__ double red[kMeanSums * kMomentWarps], pivot[6];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp < 6) {
        double c[6], t[3] = {0.0, 0.0, 0.0};
        if (lane < B.n) {
            load6(c, B.c[0], B.c[1], B.c[2], B.c[3], B.c[4], B.c[5], lane);
            const double v = (double)B.c[warp][lane];
            if (isfinite(v) && (!B.mask || live6(c))) {
                t[0] = v;
                t[1] = v * v;
                t[2] = 1.0;
            }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t[k] += __shfl_xor_sync(0xffffffffu, t[k], o);
        const double mean = t[0] / t[2];
        if (lane == 0) {
            pivot[warp] = isfinite(mean) && !(17.0 * mean * mean <= 16.0 * (t[1] / t[2])) ? mean : 0.0;
            if (blockIdx.x == 0) pivots[warp] = pivot[warp];
        }
    }
    __syncthreads();
    double s[kMeanSums] = {};
#pragma unroll 1
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < B.n; i += (long long)gridDim.x * blockDim.x) {
        double c[6];
        load6(c, B.c[0], B.c[1], B.c[2], B.c[3], B.c[4], B.c[5], i);
        if (B.mask && !live6(c)) continue;
#pragma unroll
        for (int d = 0; d < 6; ++d) s[d] += c[d] - pivot[d];
        s[6] += 1.0;
    }
    block_sums<kMeanSums>(s, red, partial);
}

// Fixed-order sum of partial[b * stride + k] over b < nb by one block of kMomentThreads threads: thread t
// takes b = t, t + kMomentThreads, ... in order, then the block's fixed shuffle/warp tree.
__device__ __forceinline__ double fold_partials(const double *partial, int nb, int stride, int k) {
    __shared__ double red[kMomentWarps];
    double t = 0.0;
    for (int b = threadIdx.x; b < nb; b += kMomentThreads) t += partial[(size_t)b * stride + k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
    __syncthreads();
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < kMomentWarps; ++w) s += red[w];
    return s;
}

// Block d < 6: the mean of coordinate d (0 / 0 = NaN for a beam without live particles, as the reference reports it),
// block 0 also the live count means[6] and the row's turn; block 6 + k: requested pair k, NaN where a mean it
// involves is not finite, as the deviations from such a mean are.  The four columns a pair takes are folded together.
__global__ void __launch_bounds__(kMomentThreads) k_moment_finish(const double *pivots, const double *partial, int nb,
                                                                  int sums, double turn, const __grid_constant__ MomentHead head,
                                                                  const __grid_constant__ MomentPairRows Q,
                                                                  double *means, double *row) {
    pdl_wait();
    pdl_release();
    __shared__ double red[4][kMomentWarps];
    const int q = (int)blockIdx.x - 6;
    int a = blockIdx.x, b = blockIdx.x, pair = 0;
    if (q >= 0) {
        pair = Q.pair[q];
        a = 0;
        int first = 0;
        while (pair >= first + 6 - a) first += 6 - a++;
        b = a + pair - first;
    }
    const int col[4] = {sums - 1, a, b, q >= 0 ? 6 + pair : a};
    double t[4] = {0.0, 0.0, 0.0, 0.0};
    for (int p = threadIdx.x; p < nb; p += kMomentThreads)
#pragma unroll
        for (int k = 0; k < 4; ++k) t[k] += partial[(size_t)p * sums + col[k]];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t[k] += __shfl_xor_sync(0xffffffffu, t[k], o);
        if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = t[k];
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        t[k] = 0.0;
#pragma unroll
        for (int w = 0; w < kMomentWarps; ++w) t[k] += red[k][w];
    }
    const double n = t[0], da = t[1] / n, db = t[2] / n;
    if (q >= 0) {
        row[1 + Q.slot[q]] = isfinite(da) && isfinite(db) ? fma(-da, db, t[3] / n) : (double)NAN;
        return;
    }
    const double mean = pivots[a] + da;
    means[8 + a] = mean;
    for (int k = 0; k < head.n; ++k)
        if (head.coord[k] == a) row[1 + head.slot[k]] = mean;
    if (a == 0) {
        means[6] = n;
        row[0] = turn;
    }
}

__device__ __noinline__ double ipow(double v, int p) {
    double r = v;
    for (int k = 1; k < p; ++k) r *= v;
    return r;
}

// Rows of order >= 3: term = 1.0 * prod_d (c_d - <c_d>)^p_d in coordinate order, the power by repeated
// products.
template <class R>
__global__ void __launch_bounds__(kMomentThreads, 2) k_moment_general(const R *__restrict__ x, const R *__restrict__ px,
                                                                     const R *__restrict__ y, const R *__restrict__ py,
                                                                     const R *__restrict__ z, const R *__restrict__ pz,
                                                                     long long n, int mask, const double *means,
                                                                     const __grid_constant__ MomentPowers P,
                                                                     double *partial) {
    pdl_wait();
    pdl_release();
    __shared__ double red[kMomentChunk * kMomentWarps];
    double mu[6];
#pragma unroll
    for (int d = 0; d < 6; ++d) mu[d] = means[8 + d];
    double acc[kMomentChunk];
#pragma unroll
    for (int k = 0; k < kMomentChunk; ++k) acc[k] = 0.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        double c[6];
        load6(c, x, px, y, py, z, pz, i);
        if (mask && !live6(c)) continue;
        double dv[6];
#pragma unroll
        for (int d = 0; d < 6; ++d) dv[d] = c[d] - mu[d];
#pragma unroll
        for (int k = 0; k < kMomentChunk; ++k) {
            double term = 1.0;
#pragma unroll
            for (int d = 0; d < 6; ++d) {
                const int p = P.p[k][d];
                if (p) term *= ipow(dv[d], p);
            }
            acc[k] += k < P.n ? term : 0.0;
        }
    }
    block_sums<kMomentChunk>(acc, red, partial);
}

// Folds of the block partials (fixed order), divided by the live count (0 / 0 = NaN for a beam without
// live particles, as the reference reports it).  Block k folds requested row k.
__global__ void __launch_bounds__(kMomentThreads) k_moment_fold(const double *partial, int nb, const double *means,
                                                                  MomentPowers P, double *row) {
    pdl_wait();
    pdl_release();
    const int k = blockIdx.x;
    const double s = fold_partials(partial, nb, kMomentChunk, k);
    if (threadIdx.x == 0) row[1 + P.slot[k]] = s / means[6];
}

}  // namespace octo
