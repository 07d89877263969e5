// equil.cu -- the round driver's equilibration test on the device.
//
// The reference decides that the walkers are equilibrated when the Spearman
// rank correlation between the energies at the latest checkpoint and those
// one and two checkpoints earlier is insignificant (scipy.stats.spearmanr,
// p > 0.02 for both; NewtonSteps.py:395-442).  spearmanr (scipy 1.18.1) is:
// average ranks of each vector (rankdata, ties get the mean of their
// positions), the Pearson correlation r of the two rank vectors, and the
// two-sided Student-t p-value of t = r sqrt((n-2) / ((1+r)(1-r))) with n-2
// degrees of freedom; a constant input gives r = NaN.  Since |t| grows with
// |r|, p > 0.02 is the same as |r| < r_crit with r_crit = t_c / sqrt(n - 2 +
// t_c^2), t_c the upper 1% point of that t distribution -- a number the host
// computes once per n.  Here:
//   mi3_rank_average   ranks of n floats (radix sort of (key, index) pairs,
//                      tie runs found by binary search, average rank
//                      scattered back to the input order);
//   mi3_rank_corr      Pearson r of two rank vectors in FP64 (fixed-order
//                      reduction, so the result is deterministic);
//   mi3_equil_decide   the verdict |r1| < r_crit and |r2| < r_crit as an
//                      int32 flag in device memory (NaN fails).
#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace mi3 {

// Order-preserving map float -> uint32 (finite inputs); -0 and +0 are one
// value, as for a float comparison.
__device__ __forceinline__ uint32_t float_key(float x) {
    const uint32_t u = __float_as_uint(x == 0.0f ? 0.0f : x);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Least-significant-digit radix sort, 8 bits a pass.  A pass is one kernel: each
// CTA sorts a tile of RK_TILE pairs stably by its digit and finds where each
// digit's run goes from all CTAs' digit counts, which the pass before it made
// (count[tile][digit], 1 KB per tile, read by every CTA from L2).  So a sort is
// six launches, tie handling included, whatever n; the bitonic network it
// replaces took 44 at n = 2^18, most of them 3 us long.  Call times, before and
// now: 103 and 68 us at n = 2^14, 235 and 84 us at 2^18, 514 and 172 us at 2^20,
// 3.5 and 2.7 ms at 2^23 - 1, where a pass reads 4 GB of counts from L2 (they grow
// with n^2).  Below that a pass is bound by its latencies: the reads of the counts,
// then 16 rounds of matching.
constexpr uint32_t RK_THREADS = 256, RK_WARPS = RK_THREADS / 32, RK_PER = 16;
constexpr uint32_t RK_TILE = RK_THREADS * RK_PER, RK_DIGITS = 256;

__global__ void __launch_bounds__(RK_THREADS) k_rank_count(const float *__restrict__ x, uint32_t n, uint32_t *count) {
    __shared__ uint32_t c[RK_DIGITS];
    c[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t base = blockIdx.x * RK_TILE;
#pragma unroll
    for (uint32_t e = 0; e < RK_PER; ++e) {
        const uint32_t i = base + e * RK_THREADS + threadIdx.x;
        if (i < n) atomicAdd(&c[float_key(x[i]) & 255u], 1u);
    }
    __syncthreads();
    count[blockIdx.x * RK_DIGITS + threadIdx.x] = c[threadIdx.x];
}

// One pass by bits [shift, shift + 8): the pairs of (x, index) if FIRST, else of
// (keys_in, vals_in), to keys_out / vals_out; counts the next digit of what it
// writes into next (nullable, zeroed).
template <bool FIRST>
__global__ void __launch_bounds__(RK_THREADS) k_rank_pass(const float *__restrict__ x,
                                                          const uint32_t *__restrict__ keys_in,
                                                          const uint32_t *__restrict__ vals_in, uint32_t n,
                                                          uint32_t shift, const uint32_t *__restrict__ count,
                                                          uint32_t *next, uint32_t *keys_out, uint32_t *vals_out) {
    __shared__ uint32_t cnt[RK_WARPS][RK_DIGITS], scan[RK_DIGITS];
    const uint32_t t = threadIdx.x, warp = t >> 5, lane = t & 31;
    for (uint32_t w = 0; w < RK_WARPS; ++w) cnt[w][t] = 0;
    // digit t: its total, and its count in the tiles before this one
    uint32_t total = 0, before = 0;
#pragma unroll 8
    for (uint32_t b = 0; b < gridDim.x; ++b) {
        const uint32_t v = __ldg(&count[b * RK_DIGITS + t]);
        total += v;
        before += b < blockIdx.x ? v : 0u;
    }
    __syncthreads();

    // stable rank of each pair among its warp's pairs of the same digit: the
    // warp takes RK_PER rounds of 32 neighbouring pairs
    const uint32_t seg = blockIdx.x * RK_TILE + warp * (RK_PER * 32);
    uint32_t key[RK_PER], val[RK_PER], rank[RK_PER];
#pragma unroll
    for (uint32_t e = 0; e < RK_PER; ++e) {
        const uint32_t i = seg + e * 32 + lane;
        key[e] = i < n ? (FIRST ? float_key(x[i]) : keys_in[i]) : 0u;
        val[e] = FIRST || i >= n ? i : vals_in[i];
    }
#pragma unroll
    for (uint32_t e = 0; e < RK_PER; ++e) {
        const bool in = seg + e * 32 + lane < n;
        const uint32_t live = __ballot_sync(0xffffffffu, in), d = (key[e] >> shift) & 255u;
        if (in) {
            const uint32_t same = __match_any_sync(live, d), mine = __popc(same & ((1u << lane) - 1u));
            rank[e] = cnt[warp][d] + mine;
            __syncwarp(live);
            if (mine == 0) cnt[warp][d] += __popc(same);
        }
        __syncwarp();
    }
    __syncthreads();
    // exclusive scan of the digit totals; each warp's share of its digits
    uint32_t inc = total;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) scan[warp] = inc;
    __syncthreads();
    uint32_t start = inc - total + before;
    for (uint32_t w = 0; w < warp; ++w) start += scan[w];
    for (uint32_t w = 0; w < RK_WARPS; ++w) {
        const uint32_t c = cnt[w][t];
        cnt[w][t] = start;
        start += c;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t e = 0; e < RK_PER; ++e) {
        if (seg + e * 32 + lane >= n) continue;
        const uint32_t at = cnt[warp][(key[e] >> shift) & 255u] + rank[e];
        keys_out[at] = key[e];
        vals_out[at] = val[e];
        if (next) atomicAdd(&next[at / RK_TILE * RK_DIGITS + ((key[e] >> (shift + 8)) & 255u)], 1u);
    }
}

// rank (1-based, average over the tie run [lo, hi]) scattered to the input
// order; a run's ends by binary search in the sorted keys
__global__ void k_rank_scatter(const uint32_t *__restrict__ keys, const uint32_t *__restrict__ vals, uint32_t n,
                               float *ranks) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const uint32_t k = keys[p];
    uint32_t lo = p, hi = p;
    if (p > 0 && keys[p - 1] == k) {
        uint32_t a = 0, b = p - 1;  // first index with this key is in [a, b]
        while (a < b) {
            const uint32_t m = (a + b) / 2;
            if (keys[m] < k)
                a = m + 1;
            else
                b = m;
        }
        lo = a;
    }
    if (p + 1 < n && keys[p + 1] == k) {
        uint32_t a = p + 1, b = n - 1;  // last index with this key is in [a, b]
        while (a < b) {
            const uint32_t m = (a + b + 1) / 2;
            if (keys[m] > k)
                b = m - 1;
            else
                a = m;
        }
        hi = a;
    }
    ranks[vals[p]] = 0.5f * (float)(lo + hi) + 1.0f;  // exact: lo + hi < 2^24
}

// Pearson correlation of two rank vectors: per-block FP64 partial sums of
// (a-m)^2, (b-m)^2, (a-m)(b-m), m = (n+1)/2, then one thread in fixed order.
constexpr uint32_t PC_THREADS = 256, PC_BLOCKS = 296;

__global__ void __launch_bounds__(PC_THREADS) k_rank_corr_partial(const float *__restrict__ ra,
                                                                  const float *__restrict__ rb, uint32_t n,
                                                                  double *part) {
    __shared__ double s[3][PC_THREADS];
    const double m = 0.5 * ((double)n + 1.0);
    double aa = 0.0, bb = 0.0, ab = 0.0;
    for (uint32_t p = blockIdx.x * PC_THREADS + threadIdx.x; p < n; p += PC_BLOCKS * PC_THREADS) {
        const double a = (double)ra[p] - m, b = (double)rb[p] - m;
        aa += a * a;
        bb += b * b;
        ab += a * b;
    }
    s[0][threadIdx.x] = aa;
    s[1][threadIdx.x] = bb;
    s[2][threadIdx.x] = ab;
    __syncthreads();
    for (uint32_t o = PC_THREADS / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o)
            for (int c = 0; c < 3; ++c) s[c][threadIdx.x] += s[c][threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int c = 0; c < 3; ++c) part[3 * blockIdx.x + c] = s[c][0];
}

__global__ void k_rank_corr_final(const double *__restrict__ part, double *r) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    double aa = 0.0, bb = 0.0, ab = 0.0;
    for (uint32_t b = 0; b < PC_BLOCKS; ++b) {
        aa += part[3 * b];
        bb += part[3 * b + 1];
        ab += part[3 * b + 2];
    }
    // a constant input has no correlation (scipy: NaN)
    *r = (aa > 0.0 && bb > 0.0) ? ab / sqrt(aa * bb) : __longlong_as_double(0x7ff8000000000000ll);
}

__global__ void k_equil_decide(const double *r1, const double *r2, double rcrit, int32_t *flag) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const double a = fabs(*r1), b = fabs(*r2);
    *flag = (a < rcrit && b < rcrit) ? 1 : 0;  // false for NaN
}

}  // namespace mi3

using namespace mi3;

extern "C" size_t mi3_rank_workspace(uint32_t n) {
    if (n == 0 || n >= (1u << 23)) return 0;
    // two key and two index arrays, one table of digit counts per pass
    const size_t nb = (n + RK_TILE - 1) / RK_TILE;
    return 4 * (size_t)n * 4 + 4 * nb * RK_DIGITS * 4;
}

extern "C" int mi3_rank_average(const float *x, uint32_t n, float *ranks, void *workspace, size_t ws_bytes,
                                void *stream) {
    if (!x || !ranks || !workspace) return fail(MI3_ERR_ARG, "mi3_rank_average: null pointer");
    if (n == 0 || n >= (1u << 23)) return fail(MI3_ERR_ARG, "mi3_rank_average: need 0 < n < 2^23");
    if (ws_bytes < mi3_rank_workspace(n)) return fail(MI3_ERR_WORKSPACE, "mi3_rank_average: workspace too small");
    if (!aligned(workspace, 16)) return fail(MI3_ERR_ALIGN, "mi3_rank_average: workspace must be 16B aligned");
    cudaStream_t st = as_stream(stream);
    const uint32_t nb = (n + RK_TILE - 1) / RK_TILE, table = nb * RK_DIGITS;
    uint32_t *count = reinterpret_cast<uint32_t *>(workspace);
    uint32_t *ka = count + 4 * table, *va = ka + n, *kb = va + n, *vb = kb + n;
    if (cudaMemsetAsync(count + table, 0, (size_t)3 * table * 4, st) != cudaSuccess)
        return check_launch("mi3_rank_average: memset");
    k_rank_count<<<nb, RK_THREADS, 0, st>>>(x, n, count);
    k_rank_pass<true><<<nb, RK_THREADS, 0, st>>>(x, nullptr, nullptr, n, 0, count, count + table, ka, va);
    k_rank_pass<false><<<nb, RK_THREADS, 0, st>>>(nullptr, ka, va, n, 8, count + table, count + 2 * table, kb, vb);
    k_rank_pass<false><<<nb, RK_THREADS, 0, st>>>(nullptr, kb, vb, n, 16, count + 2 * table, count + 3 * table, ka, va);
    k_rank_pass<false><<<nb, RK_THREADS, 0, st>>>(nullptr, ka, va, n, 24, count + 3 * table, nullptr, kb, vb);
    k_rank_scatter<<<(n + 255) / 256, 256, 0, st>>>(kb, vb, n, ranks);
    return check_launch("mi3_rank_average");
}

extern "C" size_t mi3_rank_corr_workspace(void) { return (size_t)PC_BLOCKS * 3 * 8; }

extern "C" int mi3_rank_corr(const float *ranks_a, const float *ranks_b, uint32_t n, double *r, void *workspace,
                             size_t ws_bytes, void *stream) {
    if (!ranks_a || !ranks_b || !r || !workspace) return fail(MI3_ERR_ARG, "mi3_rank_corr: null pointer");
    if (n < 2) return fail(MI3_ERR_ARG, "mi3_rank_corr: need n >= 2");
    if (ws_bytes < mi3_rank_corr_workspace()) return fail(MI3_ERR_WORKSPACE, "mi3_rank_corr: workspace too small");
    if (!aligned(workspace, 8)) return fail(MI3_ERR_ALIGN, "mi3_rank_corr: workspace must be 8B aligned");
    cudaStream_t st = as_stream(stream);
    double *part = reinterpret_cast<double *>(workspace);
    k_rank_corr_partial<<<PC_BLOCKS, PC_THREADS, 0, st>>>(ranks_a, ranks_b, n, part);
    k_rank_corr_final<<<1, 32, 0, st>>>(part, r);
    return check_launch("mi3_rank_corr");
}

extern "C" int mi3_equil_decide(const double *r1, const double *r2, double rcrit, int32_t *flag, void *stream) {
    if (!r1 || !r2 || !flag) return fail(MI3_ERR_ARG, "mi3_equil_decide: null pointer");
    k_equil_decide<<<1, 32, 0, as_stream(stream)>>>(r1, r2, rcrit, flag);
    return check_launch("mi3_equil_decide");
}
