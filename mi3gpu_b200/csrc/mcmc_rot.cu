// mcmc_rot.cu -- Metropolis sampler with rotated gathers and verdicts by
// error bound.
//
// The reference's DeltaEnergy (mcmc.cl:360-413) adds, in site order, the
// differences J[pos,m](mut, s_m) - J[pos,m](cur, s_m).  Keeping that order
// ties a kernel to one float add per term, one term per site and either bank
// conflicts (k_metropolis) or a skew between lanes (k_metropolis_skew).  Here
// the terms are summed as 32-bit integers, in whatever order is cheapest, and
// the acceptance test's two sides are compared with a proven bound on how far
// that sum can be from the reference's.  Nearly always the verdict is certain;
// where it is not, the warp sums that walker's terms again in site order with
// the reference's float operations.  Walkers, generator states and verdicts are
// therefore the same bits as with k_metropolis and the CPU oracle.
//
// Order.  The step's coupling row lies in shared memory as chunks
// [cell][32 columns]: a 128-byte line per cell.  Lane w visits column
// (t + w) mod 32 of a chunk at step t, so the 32 gathers of a warp use 32
// banks; chunks rotate independently of one another.  S = 1, 2 or 4 lanes share
// a walker: lane w holds walker w mod (32 / S) and takes steps t < 32 / S, which
// makes the S lanes' columns complementary.  S = 1 costs least per walker; S > 1
// puts a few walkers on more warps, and a long row in fewer registers per lane.
// With S = 1 a last chunk of at most 8 or 16 columns holds them repeated with
// that period (`tail`), so that it takes `tail` steps, still without conflicts;
// the table has such a chunk padded with zeros as well, for S > 1.
//
// Joint columns.  With the order free, neighbouring sites can share a gather:
//   PAIR1 (q 9..21)  column = site, cells (a, s): two gathers a site,
//                    J(mut, s) and J(cur, s)
//   PAIR2 (q 5..8)   column = two sites, cells (a, s + q s'): the sum over both
//                    sites, two gathers a column
//   DIFF2 (q 2..4)   column = two sites, cells (mut, cur, s + q s'): the whole
//                    difference, one gather a column
// PAIR1 also serves q <= 8 where a joint table would exceed ROT_JOINT_MAX (it
// should stay L2-resident).
//
// Sequences.  Each lane holds its columns' states in registers, in the order it
// visits them.  A field is the state + 1, or the state alone where t + w wraps
// past column 31: the line of cell s lies 128 bytes behind that of s - 1, so the
// wrap of the column address (-128 bytes) is part of the field, and the address
// is base + 128 * field + 4 t with 4 t in the load's immediate offset.  Fields of
// 8 bits give that address in one dp4a (the byte selected by the weight vector,
// 128 its weight): 5 instructions a PAIR term and 2.5 a DIFF term.  PAIR1 rows of
// more than 160 columns a lane take 5-bit fields, 6 to a register (6.7
// instructions): the registers saved hold more walkers, which share the fill.
//
// Couplings.  One bulk copy per chunk fills a ring of slots.  There is no
// producer warp: the last warp to finish with a slot starts its next copy, so
// all registers of the SM hold walkers -- up to 1024 lanes per CTA.
//
// Integers.  Row pos is quantised to multiples of delta(pos), a power of two
// with room for the largest sum in 31 bits; integer adds are exact, and one
// three-input add takes a term's two couplings (packed float adds: 22.6 against
// 21.3 ms per 232 steps at L=232, q=21, 2^20).
//
// Bound.  u = 2^-24, terms d_m = fl(a_m - b_m), M_m(x) = max_s |J[pos,m](x, s)|,
// |d_m| <= (1 + u) (M_m(mut) + M_m(cur)).  In site order each partial sum S_k is
// rounded once, |S_ref - S| <= u (sum_k |S_k| + sum_m |d_m|) up to second order.
// With h = L / 2, |S_k| <= sum_{m <= k} |d_m| for k <= h, and <= |S| + sum_{m > k}
// |d_m| beyond, so that
//   |S_ref - S| <= u (sum_m (|h - m| + 2) |d_m| + (L - h) |S|).
// Here each entry is rounded by at most delta / 2: |S' - S| <= columns * delta.
// k_unpack_rot stores 1.01 (u sum_m (|h - m| + 2) M_m(a) + (columns + 2) delta / 2)
// per (pos, a) (infinite where a coupling is not finite: then the exact sum
// decides); the values of mut and cur plus 1.01 u (L - h + 1) |S'| bound
// |S' - S_ref|.  With the benchmark's couplings (L=232, q=21) about 3 in 1000 of
// a warp's steps have a lane whose verdict is open.
//
// What bounds it (L=232, q=21): the shared-memory pipe (466 gathers per warp and
// step plus the fill: 60% busy) and issue (75%) together, at 7 warps per
// scheduler; 72 registers leave few loads in flight per warp.  Site-updates per
// second of calls of 1 to 16 sweeps after new couplings, before (the faster of the
// two older kernels) and now: L=48 q=4 2^14 2.9e10, 4.5e10; L=93 q=4 2^18 2.4e10,
// 6.1e10; L=187 q=8 50688 9.8e9, 1.9e10; L=232 q=21 2^20 8.6e9, 1.18e10; L=512
// q=21 2^18 3.2e9, 3.7e9 (the fill: 0.9 MB of couplings per step for 448 walkers).
//
// The couplings' size enters: the bound grows with them, and with a constant in
// them that no dE contains, and an open verdict holds up its CTA for about 32 L
// adds.  One sweep after new couplings N(0, s^2), in us (in brackets the older
// kernel, which does not depend on them):
//                      s=0.05   0.3     1      3    0.05 and 1 added  and 30 added
//   L=93  q=4  2^18     517     517    518    523     522               668  [1248]
//   L=187 q=8  50688    707     720    736    775     796              1629  [1459]
//   L=232 q=21 2^18    5663    5825   6249   6938    7544             15713  [8317]
//   L=400 q=21 2^16    6498    6628   7218   8223    9036             25681 [11718]
// Couplings with such a constant are better re-gauged first
// (mi3_gauge_fieldless_even leaves every dE as it is).
#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace mi3 {

constexpr uint32_t ROT_HEAD = 256;  // mbarriers, copy counts, abort flag
constexpr uint32_t ROT_MAX_SLOTS = 6;
constexpr uint64_t ROT_JOINT_MAX = 96ull << 20;  // bytes of a joint table

double metro_cycles(uint32_t L, uint32_t q, uint32_t nseqs);  // mcmc.cu

enum RotMode { ROT_PAIR1 = 0, ROT_PAIR2 = 1, ROT_DIFF2 = 2 };

struct RotShape {
    RotMode mode;
    uint32_t G;      // sites per column
    uint32_t Q;      // states of a column
    uint32_t cells;  // lines per chunk
    uint32_t cols;   // columns
    uint32_t nc;     // chunks of 32 columns
    uint32_t tail;   // period of the last chunk's columns; below 32, chunk nc is the padded form
    uint64_t row_words;  // one site's chunks
    uint64_t bound_at;   // word offset of the bounds and deltas, L x (q + 1)
    uint64_t j_at;       // word offset of the copy of J
    uint64_t words;      // all
};

static RotShape rot_shape_of(uint32_t L, uint32_t q, RotMode mode) {
    RotShape r;
    r.mode = mode;
    r.G = mode == ROT_PAIR1 ? 1 : 2;
    r.Q = r.G == 1 ? q : q * q;
    r.cells = (mode == ROT_DIFF2 ? q * q : q) * r.Q;
    r.cols = (L + r.G - 1) / r.G;
    r.nc = (r.cols + 31) / 32;
    const uint32_t last = r.cols - 32 * (r.nc - 1);
    r.tail = last <= 8 ? 8 : last <= 16 ? 16 : 32;
    r.row_words = (uint64_t)(r.nc + (r.tail < 32)) * r.cells * 32;
    r.bound_at = r.row_words * L;
    r.j_at = (r.bound_at + (uint64_t)L * (q + 1) + 3) & ~uint64_t(3);
    r.words = r.j_at + npairs_of(L) * q * q;
    return r;
}

static bool rot_shape(uint32_t L, uint32_t q, RotShape &r) {
    if (L < 2 || L > 576 || q < 2 || q > 21) return false;
    r = rot_shape_of(L, q, q <= 4 ? ROT_DIFF2 : q <= 8 ? ROT_PAIR2 : ROT_PAIR1);
    if (r.mode != ROT_PAIR1 && r.bound_at * 4 > ROT_JOINT_MAX) r = rot_shape_of(L, q, ROT_PAIR1);
    return true;
}

// J_{pos,m}(a, s) of the packed table, 0 for m == pos and m >= L.
__device__ __forceinline__ float j_at(const float *__restrict__ J, uint32_t L, uint32_t q, uint32_t pos, uint32_t m,
                                      uint32_t a, uint32_t s) {
    if (m >= L || m == pos) return 0.0f;
    if (pos < m) return __ldg(&J[((uint64_t)pos * (2 * L - pos - 1) / 2 + (m - pos - 1)) * q * q + a * q + s]);
    return __ldg(&J[((uint64_t)m * (2 * L - m - 1) / 2 + (pos - m - 1)) * q * q + s * q + a]);
}

// The tables of one site per CTA: its bounds and delta, its row of cells, and
// its share of the copy of J.  T[pos][chunk][cell][column] holds the cell's value
// in multiples of delta(pos).
__global__ void __launch_bounds__(1024) k_unpack_rot(const float *__restrict__ J, float *__restrict__ out, uint32_t L,
                                                     uint32_t q, RotShape sh) {
    __shared__ float part_w[32][32], part_r[32][32], scale;
    const uint32_t pos = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    float *bound = out + sh.bound_at + (uint64_t)pos * (q + 1);
    // lane a takes letter a
    float W = 0.0f, R = 0.0f;
    if (lane < q)
        for (uint32_t m = warp; m < L; m += nw) {
            float big = 0.0f;
            for (uint32_t s = 0; s < q; ++s) {
                const float v = fabsf(j_at(J, L, q, pos, m, lane, s));
                big = isnan(big) || v <= big ? big : v;  // a NaN stays, and makes the bound infinite
            }
            W += big;
            R += (fabsf((float)(L / 2) - (float)m) + 2.0f) * big;
        }
    part_w[warp][lane] = W;
    part_r[warp][lane] = R;
    __syncthreads();
    if (warp == 0) {
        W = R = 0.0f;
        for (uint32_t k = 0; k < nw; ++k) {
            W += part_w[k][lane];
            R += part_r[k][lane];
        }
        const bool finite = R <= 1e37f;
        float top = finite && lane < q ? W : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        int e = 0;
        frexpf(2.05f * top, &e);
        const float delta = ldexpf(1.0f, max(e, -60) - 31);  // sums of two letters stay below 2^31 delta
        if (lane < q)
            bound[lane] = finite ? 1.01f * (0x1p-24f * R + 0.5f * (float)(sh.cols + 2) * delta) : __int_as_float(0x7f800000);
        if (lane == 0) {
            bound[q] = delta;
            scale = delta;
        }
    }
    __syncthreads();
    const double inv = 1.0 / (double)scale;
    int32_t *row = reinterpret_cast<int32_t *>(out) + (uint64_t)pos * sh.row_words;
    const uint32_t lines = (sh.nc + (sh.tail < 32)) * sh.cells;
    for (uint32_t t = warp; t < lines; t += nw) {
        const uint32_t chunk = t / sh.cells, cell = t - chunk * sh.cells, hi = cell / sh.Q, S = cell - hi * sh.Q;
        const uint32_t col = chunk == sh.nc ? 32 * (chunk - 1) + lane
                             : 32 * chunk + (chunk == sh.nc - 1 ? lane & (sh.tail - 1) : lane);
        double v;
        if (sh.mode == ROT_PAIR1) {
            v = j_at(J, L, q, pos, col, hi, S);
        } else {
            const uint32_t s1 = S / q, s0 = S - q * s1, m = 2 * col;
            if (sh.mode == ROT_PAIR2) {
                v = (double)j_at(J, L, q, pos, m, hi, s0) + (double)j_at(J, L, q, pos, m + 1, hi, s1);
            } else {
                const uint32_t mut = hi / q, cur = hi - q * mut;
                v = ((double)j_at(J, L, q, pos, m, mut, s0) - (double)j_at(J, L, q, pos, m, cur, s0)) +
                    ((double)j_at(J, L, q, pos, m + 1, mut, s1) - (double)j_at(J, L, q, pos, m + 1, cur, s1));
            }
        }
        row[32 * t + lane] = __double2int_rn(v * inv);  // saturates
    }
    // pairs (pos, m > pos) are contiguous
    const uint64_t first = (uint64_t)pos * (2 * L - pos - 1) / 2 * q * q;
    const uint32_t n = (L - 1 - pos) * q * q;
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) out[sh.j_at + first + k] = J[first + k];
}

struct RotParams {
    const int32_t *T;
    const float *bound;
    const float *J;
    uint64_t row_words;
    uint4 *rng;
    const uint32_t *poslist;
    uint32_t pos_off, nsteps;
    const float *betas;
    float beta;
    uint32_t *seq;
    uint32_t nseqs, L, q;
    uint32_t Q, nc, tail, cells, slots;
    uint32_t last;     // chunk of the table that ends a row
    uint32_t line;     // 128
    uint32_t q_inv;    // ceil(2^16 / q): S / q for S < 64
    uint32_t q_magic;  // floor(2^32 / q)
    float half_u;      // 1.01 u (L - h + 1)
    int32_t *status;
};

// idx == k ? a : b kept as a select per register (as PTX, so that a chain of
// them is not turned into an indexed access of the register array).
__device__ __forceinline__ uint32_t rot_sel(uint32_t idx, uint32_t k, uint32_t a, uint32_t b) {
    uint32_t r;
    asm("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %1, %2;\n\tselp.b32 %0, %3, %4, p;\n\t}"
        : "=r"(r)
        : "r"(idx), "r"(k), "r"(a), "r"(b));
    return r;
}

template <uint32_t OFF>
__device__ __forceinline__ uint32_t rot_lds(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(addr), "n"(OFF));
    return v;
}

// Fields of BITS in NW words; S lanes per walker.
template <uint32_t BITS_, uint32_t NW_, uint32_t S_>
struct RotLay {
    static constexpr uint32_t BITS = BITS_, NW = NW_, S = S_, FPW = 32 / BITS, MASK = (1u << BITS) - 1;
    static constexpr uint32_t STEPS = 32 / S;                       // per chunk
    static constexpr uint32_t CAP = FPW * NW;                       // fields
    static constexpr uint32_t HC = (CAP + STEPS - 1) / STEPS;       // chunks
};

// base + 128 * (field of step T).
template <typename Y, uint32_t T>
__device__ __forceinline__ uint32_t rot_addr(const uint32_t (&sq)[Y::NW], uint32_t line, uint32_t base) {
    constexpr uint32_t F = T % Y::FPW;
    const uint32_t w = sq[T / Y::FPW];
    if constexpr (Y::BITS == 8) {
        return __dp4a(w, 128u << (8 * F), base);
    } else {
        uint32_t x;
        if constexpr (F == 0)
            x = w & Y::MASK;
        else if constexpr (F == Y::FPW - 1)
            x = w >> (Y::BITS * F);  // the word's spare top bits are zero
        else
            x = (w >> (Y::BITS * F)) & Y::MASK;
        // one multiply-add, off the pipe that extracts x (written out, the two
        // bases of a term share a product and pay an add each)
        uint32_t r;
        asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(x), "r"(line), "r"(base));
        return r;
    }
}

// Steps T and T + 1 of a lane's row.
template <int MODE, typename Y, uint32_t T>
__device__ __forceinline__ void rot_two(const uint32_t (&sq)[Y::NW], uint32_t bA, uint32_t bB, uint32_t line,
                                        uint32_t &sum) {
    if constexpr (T + 1 < Y::CAP) {
        constexpr uint32_t O0 = 4 * (T % Y::STEPS), O1 = O0 + 4;
        if constexpr (MODE == ROT_DIFF2) {
            sum = sum + rot_lds<O0>(rot_addr<Y, T>(sq, line, bA)) + rot_lds<O1>(rot_addr<Y, T + 1>(sq, line, bA));
        } else {
            sum = sum + rot_lds<O0>(rot_addr<Y, T>(sq, line, bA)) - rot_lds<O0>(rot_addr<Y, T>(sq, line, bB));
            sum = sum + rot_lds<O1>(rot_addr<Y, T + 1>(sq, line, bA)) - rot_lds<O1>(rot_addr<Y, T + 1>(sq, line, bB));
        }
    }
}

template <int MODE, typename Y, uint32_t T>
__device__ __forceinline__ void rot_eight(const uint32_t (&sq)[Y::NW], uint32_t bA, uint32_t bB, uint32_t line,
                                          uint32_t &sum) {
    rot_two<MODE, Y, T + 0>(sq, bA, bB, line, sum);
    rot_two<MODE, Y, T + 2>(sq, bA, bB, line, sum);
    rot_two<MODE, Y, T + 4>(sq, bA, bB, line, sum);
    rot_two<MODE, Y, T + 6>(sq, bA, bB, line, sum);
}

// Ring addresses are 32-bit shared-memory addresses.
struct RotRing {
    uint32_t full_s;   // mbarriers: the slot's chunk has landed
    uint32_t empty_s;  // mbarriers: every warp is done with the slot's chunk
    uint32_t ring_s, slot_bytes;
    uint32_t *issued;  // copies started into each slot
    volatile int *abort_flag;
    uint32_t lane;
    uint32_t s, phase;  // this warp's next slot and its phase
    uint32_t at;        // 4 lane - 128 + the slot's address
};

__device__ __forceinline__ bool rot_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Wait for a phase, at most WAIT_LIMIT_NS or until the CTA aborts.  A warp that
// runs ahead of the others waits here every chunk; it sleeps between tests, for
// the others need its issue slots (try_wait polls about every 100 cycles: 3.30
// against 3.23 ms at L=93, q=4, 2^18, 744 steps).
__device__ __noinline__ bool rot_wait_long(uint32_t bar, uint32_t parity, const volatile int *abort_flag) {
    const uint64_t t0 = globaltimer_ns();
    while (!rot_test(bar, parity)) {
        if (abort_flag && *abort_flag) return false;
        if (globaltimer_ns() - t0 > WAIT_LIMIT_NS) return false;
        __nanosleep(200);
    }
    return true;
}
__device__ __forceinline__ bool rot_wait(uint32_t bar, uint32_t parity, const volatile int *abort_flag) {
    if (rot_test(bar, parity)) return true;
#pragma unroll 1
    for (int i = 0; i < 256; ++i) {
        __nanosleep(200);
        if (rot_test(bar, parity)) return true;
    }
    return rot_wait_long(bar, parity, abort_flag);
}

// Start the copy of chunk k of step `step` into a slot (one thread).
__device__ __forceinline__ void rot_issue(const RotParams &p, const RotRing &r, uint32_t slot, uint32_t step,
                                          uint32_t k) {
    uint32_t pos = __ldg(&p.poslist[p.pos_off + step]);
    if (pos >= p.L) pos = 0;  // invalid site: the walkers' loop reports it
    const int32_t *src = p.T + (uint64_t)pos * p.row_words + (uint64_t)(k == p.nc - 1 ? p.last : k) * p.cells * 32;
    const uint32_t bar = r.full_s + 8 * slot;
    r.issued[slot] += 1;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(r.slot_bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     r.ring_s + slot * r.slot_bytes),
                 "l"(src), "r"(r.slot_bytes), "r"(bar)
                 : "memory");
}

// Chunk k (= B): wait for it, add its terms, hand its slot on.
template <int MODE, typename Y, uint32_t B>
__device__ __forceinline__ bool rot_chunk(const RotParams &p, RotRing &r, const uint32_t (&sq)[Y::NW], uint32_t offA,
                                          uint32_t offB, uint32_t step, uint32_t &sum) {
    const bool w = rot_wait(r.full_s + 8 * r.s, r.phase, r.abort_flag);
    if (!__all_sync(0xffffffffu, w)) {
        if (r.lane == 0) {
            if (!*r.abort_flag) report(p.status, ST_TIMEOUT_FULL);
            *r.abort_flag = 1;
        }
        return false;
    }
    const uint32_t bA = r.at + offA, bB = r.at + offB;
    constexpr uint32_t T = Y::STEPS * B;
    const uint32_t n = Y::S == 1 && B == p.nc - 1 ? p.tail : Y::STEPS;
    rot_eight<MODE, Y, T>(sq, bA, bB, p.line, sum);
    if constexpr (Y::STEPS > 8) {
        if (n > 8) {
            rot_eight<MODE, Y, T + 8>(sq, bA, bB, p.line, sum);
            if constexpr (Y::STEPS > 16) {
                if (n > 16) {
                    rot_eight<MODE, Y, T + 16>(sq, bA, bB, p.line, sum);
                    rot_eight<MODE, Y, T + 24>(sq, bA, bB, p.line, sum);
                }
            }
        }
    }
    __syncwarp();
    if (r.lane == 0) {
        uint32_t pending;
        const uint32_t bar = r.empty_s + 8 * r.s;
        asm volatile(
            "{\n\t.reg .b64 st;\n\t"
            "mbarrier.arrive.shared::cta.b64 st, [%1];\n\t"
            "mbarrier.pending_count.b64 %0, st;\n\t}"
            : "=r"(pending)
            : "r"(bar)
            : "memory");
        if (pending == 1) {
            // the last warp: the phase is complete, so every warp's loads
            // from this slot have returned (the wait acquires them)
            uint32_t k = B + p.slots, i = step;
            while (k >= p.nc) {
                k -= p.nc;
                ++i;
            }
            if (rot_wait(bar, r.phase, r.abort_flag) && i < p.nsteps) rot_issue(p, r, r.s, i, k);
        }
    }
    __syncwarp();
    r.at += r.slot_bytes;
    if (++r.s == p.slots) {
        r.s = 0;
        r.phase ^= 1;
        r.at -= p.slots * r.slot_bytes;
    }
    return true;
}

template <int MODE, typename Y, uint32_t B>
__device__ __forceinline__ bool rot_chunks(const RotParams &p, RotRing &r, const uint32_t (&sq)[Y::NW], uint32_t offA,
                                           uint32_t offB, uint32_t step, uint32_t &sum) {
    if constexpr (B < Y::HC) {
        if (B >= p.nc) return true;
        if (!rot_chunk<MODE, Y, B>(p, r, sq, offA, offB, step, sum)) return false;
        return rot_chunks<MODE, Y, B + 1>(p, r, sq, offA, offB, step, sum);
    } else {
        return true;
    }
}

// Word wi of the sequence registers, which lies in chunk k (warp-uniform).
template <typename Y, uint32_t B>
__device__ __forceinline__ uint32_t rot_word(const uint32_t (&sq)[Y::NW], uint32_t k, uint32_t wi) {
    if constexpr (B < Y::HC) {
        if (k == B) {
            uint32_t word = 0;
#pragma unroll
            for (uint32_t w = Y::STEPS * B / Y::FPW; w <= (Y::STEPS * B + Y::STEPS - 1) / Y::FPW && w < Y::NW; ++w)
                word = rot_sel(wi, w, sq[w], word);
            return word;
        }
        return rot_word<Y, B + 1>(sq, k, wi);
    } else {
        return 0;
    }
}

// Word wi takes (SET) or grows by (else) `word`.
template <typename Y, bool SET, uint32_t B>
__device__ __forceinline__ void rot_put(uint32_t (&sq)[Y::NW], uint32_t k, uint32_t wi, uint32_t word) {
    if constexpr (B < Y::HC) {
        if (k == B) {
#pragma unroll
            for (uint32_t w = Y::STEPS * B / Y::FPW; w <= (Y::STEPS * B + Y::STEPS - 1) / Y::FPW && w < Y::NW; ++w)
                sq[w] = SET ? rot_sel(wi, w, word, sq[w]) : sq[w] + rot_sel(wi, w, word, 0u);
        } else {
            rot_put<Y, SET, B + 1>(sq, k, wi, word);
        }
    }
}

// Where column `col` lies among the fields of the walker whose first lane is
// v = lane mod STEPS (S lanes v + j * STEPS): the lane that owns it, its word,
// shift, chunk, and the field's offset against the state.
struct RotPlace {
    uint32_t owner, wi, sh, k;
    uint32_t less;  // state = field - less
};

template <typename Y>
__device__ __forceinline__ RotPlace rot_place(uint32_t col, uint32_t v, uint32_t nc, uint32_t tail) {
    RotPlace o;
    o.k = col >> 5;
    uint32_t t = (col - v) & (Y::S == 1 && o.k == nc - 1 ? tail - 1 : 31u);
    o.owner = v + (t & ~(Y::STEPS - 1));
    t &= Y::STEPS - 1;
    const uint32_t pp = Y::STEPS * o.k + t;
    o.wi = pp / Y::FPW;
    o.sh = Y::BITS * (pp - Y::FPW * o.wi);
    o.less = 1u - ((t + o.owner) >> 5);
    return o;
}

template <int MODE, uint32_t BITS, uint32_t NW, uint32_t S, uint32_t MAXT>
__global__ void __launch_bounds__(MAXT, 1) k_metropolis_rot(const RotParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    using Y = RotLay<BITS, NW, S>;
    constexpr uint32_t G = MODE == ROT_PAIR1 ? 1 : 2;
    // the long rows' kernels have no register to keep the bound and the place
    // of the residue through the chunks: they read and work them out after
    // (L=512, 28 warps: 9.94 -> 9.47 ms per 128 steps of 2^18; the same costs
    // L=93, q=4 2.6%)
    constexpr bool LATE = NW > 40 && NW < 64;
    constexpr uint32_t STR = NW + 1;  // staging words per lane (odd: few bank conflicts)
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, v = lane & (Y::STEPS - 1);
    const uint32_t warps = blockDim.x >> 5;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem), *empty = full + ROT_MAX_SLOTS;
    uint32_t *scratch = reinterpret_cast<uint32_t *>(smem + ROT_HEAD) + warp * (S * NW);
    unsigned char *ring = smem + ROT_HEAD + ((warps * S * NW * 4 + 127) & ~127u);
    RotRing r;
    r.full_s = smem_addr(full);
    r.empty_s = smem_addr(empty);
    r.issued = reinterpret_cast<uint32_t *>(empty + ROT_MAX_SLOTS);
    r.abort_flag = reinterpret_cast<volatile int *>(r.issued + ROT_MAX_SLOTS);
    r.lane = lane;
    r.ring_s = smem_addr(ring);
    r.slot_bytes = p.cells * 128;
    r.s = r.phase = 0;
    r.at = r.ring_s + 4 * lane - 128;
    uint32_t *stage = reinterpret_cast<uint32_t *>(ring) + (tid - lane) * STR;  // this warp's, before and after the loop
    uint32_t *my = stage + lane * STR;
    const uint32_t g = (blockIdx.x * warps + warp) * Y::STEPS + v;
    // the last CTA may be partly filled, by whole warps: walkers past nseqs
    // run on a zero sequence and store nothing
    const bool valid = g < p.nseqs;

    if (tid == 0) {
        for (uint32_t s = 0; s < p.slots; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], warps);
            r.issued[s] = 0;
        }
        *r.abort_flag = 0;
        fence_mbar_init();
    }

    // ---- the walkers' sequences -> fields
    uint32_t sq[NW];
    for (uint32_t k = 0; k < NW; ++k) my[k] = 0;
    {
        uint32_t gw = 0, state = 0;
        const uint32_t cols = 32 * (p.nc - 1) + (S == 1 ? p.tail : 32);  // padded columns hold state 0
        for (uint32_t m = 0; m < cols * G; ++m) {
            if ((m & 3) == 0) gw = valid && m < p.L ? p.seq[(size_t)(m >> 2) * p.nseqs + g] : 0u;
            // residues >= q (invalid input) are clamped to q - 1 so that every
            // gather stays inside the ring
            const uint32_t s = m < p.L ? min(getbyte(gw, m & 3), p.q - 1) : 0u;
            state = G == 2 && (m & 1) ? state + p.q * s : s;
            if (G == 1 || (m & 1)) {
                const RotPlace o = rot_place<Y>(m / G, v, p.nc, p.tail);
                if (o.owner == lane) my[o.wi] |= (state + o.less) << o.sh;
            }
        }
    }
#pragma unroll
    for (uint32_t k = 0; k < NW; ++k) sq[k] = my[k];
    fence_proxy_async_smem();
    __syncthreads();
    if (tid == 0) {
        uint32_t i = 0, k = 0;
        for (uint32_t s = 0; s < p.slots && i < p.nsteps; ++s) {
            rot_issue(p, r, s, i, k);
            if (++k == p.nc) {
                k = 0;
                ++i;
            }
        }
    }
    __syncthreads();

    // the S lanes of a walker run the same generator and take the same verdict
    uint4 s4 = valid ? p.rng[g] : make_uint4(1, 1, 1, 1);
    Rng2 rng{s4.x, s4.y, s4.z, s4.w};
    const float Bta = (p.betas && valid) ? p.betas[g] : p.beta;
    uint32_t next_pos = __ldg(&p.poslist[p.pos_off]);
    for (uint32_t i = 0; i < p.nsteps; ++i) {
        uint32_t pos = next_pos;
        if (i + 1 < p.nsteps) next_pos = __ldg(&p.poslist[p.pos_off + i + 1]);
        if (pos >= p.L) {
            report(p.status, ST_BAD_INPUT);
            pos = 0;
        }
        uint32_t r0, r1;
        rng_next2(rng, r0, r1);
        // r0 mod q: the quotient by floor(2^32 / q) is at most one short
        uint32_t mut = r0 - __umulhi(r0, p.q_magic) * p.q;
        mut = mut >= p.q ? mut - p.q : mut;
        const RotPlace o = rot_place<Y>(pos / G, v, p.nc, p.tail);
        const uint32_t word = rot_word<Y, 0>(sq, o.k, o.wi);
        uint32_t state = ((word >> o.sh) & Y::MASK) - o.less;
        if constexpr (S > 1) {
            state = o.owner == lane ? state : 0u;
            state |= __shfl_xor_sync(0xffffffffu, state, 16);
            if constexpr (S > 2) state |= __shfl_xor_sync(0xffffffffu, state, 8);
        }
        uint32_t cur = state, unit = 1;
        if constexpr (G == 2) {
            const uint32_t s1 = (state * p.q_inv) >> 16;
            const bool second = pos & 1;
            cur = second ? s1 : state - p.q * s1;
            unit = second ? p.q : 1u;
        }
        const float *brow = p.bound + (size_t)pos * (p.q + 1);
        float bound = 0.0f, delta = 0.0f;
        if constexpr (!LATE) {
            bound = __ldg(&brow[mut]) + __ldg(&brow[cur]);
            delta = __ldg(&brow[p.q]);
        }
        uint32_t offA, offB = 0;
        if constexpr (MODE == ROT_DIFF2) {
            offA = (mut * p.q + cur) * p.Q * 128;
        } else {
            offA = mut * p.Q * 128;
            offB = cur * p.Q * 128;
        }
        uint32_t sum = 0;
        if (!rot_chunks<MODE, Y, 0>(p, r, sq, offA, offB, i, sum)) break;
        if constexpr (S > 1) sum += __shfl_xor_sync(0xffffffffu, sum, 16);
        if constexpr (S > 2) sum += __shfl_xor_sync(0xffffffffu, sum, 8);

        if constexpr (LATE) {
            bound = __ldg(&brow[mut]) + __ldg(&brow[cur]);
            delta = __ldg(&brow[p.q]);
        }
        const float dE = (float)(int32_t)sum * delta;
        const float u = uniform_map(r1);
        const float x = -Bta * dE;
        // |x - x_ref| <= xb (the products' roundings are below 2^-22 |x|); expf is
        // within 2 ulp = 2^-22 relative, |exp(+-xb) - 1| <= xb + xb^2
        const float xb = fabsf(Bta) * (bound + p.half_u * fabsf(dE)) * 1.0001f + fabsf(x) * 0x1p-22f;
        const float e = expf(x), tol = xb + xb * xb + 0x1p-20f;
        bool acc = e * (1.0f - tol) > fmaxf(u, 1e-30f);
        bool sure = xb <= 0.25f && (acc || e * (1.0f + tol) < u);
        // (an infinite x says nothing about dE: it may be within its bound of 0)
        if (x >= xb && xb < __int_as_float(0x7f800000)) acc = sure = true;
        uint32_t open = __ballot_sync(0xffffffffu, !sure && valid) & (0xffffffffu >> (32 - Y::STEPS));
        while (open) {
            // the warp sums walker vv's terms in site order
            const uint32_t vv = __ffs(open) - 1;
            open &= open - 1;
            if (v == vv) {
                uint32_t *mine = scratch + (lane / Y::STEPS) * NW;
#pragma unroll
                for (uint32_t k = 0; k < NW; ++k) mine[k] = sq[k];
            }
            __syncwarp();
            const uint32_t wmut = __shfl_sync(0xffffffffu, mut, vv), wcur = __shfl_sync(0xffffffffu, cur, vv);
            // 128 sites' loads in flight, then the sum: the other warps wait
            // for this one after a few chunks
            float ref = 0.0f;
#pragma unroll 1
            for (uint32_t m0 = 0; m0 < p.L; m0 += 128) {
                float d[4];
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) {
                    const uint32_t m = m0 + 32 * k + lane;
                    d[k] = 0.0f;
                    if (m < p.L) {
                        const RotPlace om = rot_place<Y>(m / G, vv, p.nc, p.tail);
                        uint32_t s = ((scratch[(om.owner / Y::STEPS) * NW + om.wi] >> om.sh) & Y::MASK) - om.less;
                        if constexpr (G == 2) {
                            const uint32_t s1 = (s * p.q_inv) >> 16;
                            s = (m & 1) ? s1 : s - p.q * s1;
                        }
                        d[k] = j_at(p.J, p.L, p.q, pos, m, wmut, s) - j_at(p.J, p.L, p.q, pos, m, wcur, s);
                    }
                }
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) {
                    if (m0 + 32 * k >= p.L) break;
#pragma unroll
                    for (uint32_t c = 0; c < 32; ++c) ref += __shfl_sync(0xffffffffu, d[k], c);
                }
            }
            if (v == vv) acc = accept_exp(-Bta * ref, u);
            __syncwarp();
        }
        if constexpr (LATE) {
            const RotPlace o2 = rot_place<Y>(pos / G, v, p.nc, p.tail);
            const uint32_t step = (mut - cur) * (G == 2 && (pos & 1) ? p.q : 1u) << o2.sh;
            rot_put<Y, false, 0>(sq, o2.k, acc && o2.owner == lane ? o2.wi : 0xffffffffu, step);
        } else {
            const uint32_t moved = word + ((mut - cur) * unit << o.sh);
            rot_put<Y, true, 0>(sq, o.k, acc && o.owner == lane ? o.wi : 0xffffffffu, moved);
        }
    }

    // ---- every copy started must land before the ring is reused
    __syncthreads();
    if (tid == 0)
        for (uint32_t s = 0; s < p.slots; ++s)
            if (r.issued[s]) rot_wait(r.full_s + 8 * s, (r.issued[s] - 1) & 1, nullptr);
    __syncthreads();

    // ---- fields -> sequences: the S lanes of a walker share its words
#pragma unroll
    for (uint32_t k = 0; k < NW; ++k) my[k] = sq[k];
    __syncwarp();
    if (valid) {
        if (lane < Y::STEPS) p.rng[g] = make_uint4(rng.x0, rng.x1, rng.c0, rng.c1);
        for (uint32_t w = lane / Y::STEPS; w < (p.L + 3) / 4; w += S) {
            uint32_t gw = 0;
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                const uint32_t m = 4 * w + k;
                if (m < p.L) {
                    const RotPlace o = rot_place<Y>(m / G, v, p.nc, p.tail);
                    uint32_t s = ((stage[o.owner * STR + o.wi] >> o.sh) & Y::MASK) - o.less;
                    if constexpr (G == 2) {
                        const uint32_t s1 = (s * p.q_inv) >> 16;
                        s = (m & 1) ? s1 : s - p.q * s1;
                    }
                    gw |= s << (8 * k);
                }
            }
            p.seq[(size_t)w * p.nseqs + g] = gw;
        }
    }
}

using RotKernel = void (*)(const RotParams);

struct RotPick {
    RotKernel kernel;
    uint32_t bits, nw, S, maxt;
};

// Threads per CTA by sequence words: 65536 registers shared by MAXT threads
// leave 64, 72, 80 or 128 each; the loop needs about 30 beside the words.
template <int MODE, uint32_t BITS, uint32_t NW, uint32_t S>
static RotPick rot_pick() {
    constexpr uint32_t MAXT = NW <= 28 ? 1024 : NW <= 43 ? 896 : NW <= 48 ? 768 : 512;
    return RotPick{k_metropolis_rot<MODE, BITS, NW, S, MAXT>, BITS, NW, S, MAXT};
}

// The kernel for a shape with S lanes per walker (nullptr: none).
static RotPick rot_kernel(const RotShape &r, uint32_t S) {
    const uint32_t f = S == 1 ? 32 * (r.nc - 1) + r.tail : 32 / S * r.nc;
    if (r.mode == ROT_DIFF2) {
        if (S == 1) {
            if (f <= 48) return rot_pick<ROT_DIFF2, 8, 12, 1>();
            if (f <= 96) return rot_pick<ROT_DIFF2, 8, 24, 1>();
            if (f <= 160) return rot_pick<ROT_DIFF2, 8, 40, 1>();
            return rot_pick<ROT_DIFF2, 8, 72, 1>();
        }
        if (S == 2) return f <= 48 ? rot_pick<ROT_DIFF2, 8, 12, 2>() : rot_pick<ROT_DIFF2, 8, 36, 2>();
        return f <= 32 ? rot_pick<ROT_DIFF2, 8, 8, 4>() : rot_pick<ROT_DIFF2, 8, 18, 4>();
    }
    if (r.mode == ROT_PAIR2) {
        if (S == 1) {
            if (f <= 96) return rot_pick<ROT_PAIR2, 8, 24, 1>();
            if (f <= 160) return rot_pick<ROT_PAIR2, 8, 40, 1>();
            return rot_pick<ROT_PAIR2, 8, 72, 1>();
        }
        if (S == 2) return f <= 96 ? rot_pick<ROT_PAIR2, 8, 24, 2>() : rot_pick<ROT_PAIR2, 8, 36, 2>();
        return f <= 48 ? rot_pick<ROT_PAIR2, 8, 12, 4>() : rot_pick<ROT_PAIR2, 8, 18, 4>();
    }
    if (S == 1) {
        if (f <= 64) return rot_pick<ROT_PAIR1, 8, 16, 1>();
        if (f <= 112) return rot_pick<ROT_PAIR1, 8, 28, 1>();
        if (f <= 160) return rot_pick<ROT_PAIR1, 8, 40, 1>();
        if (f <= 192) return rot_pick<ROT_PAIR1, 5, 32, 1>();
        if (f <= 234) return rot_pick<ROT_PAIR1, 5, 39, 1>();
        if (f <= 288) return rot_pick<ROT_PAIR1, 5, 48, 1>();
        return RotPick{nullptr, 0, 0, 0, 0};
    }
    if (S == 2) {
        if (f <= 64) return rot_pick<ROT_PAIR1, 8, 16, 2>();
        if (f <= 128) return rot_pick<ROT_PAIR1, 8, 32, 2>();
        if (f <= 192) return rot_pick<ROT_PAIR1, 5, 32, 2>();
        if (f <= 256) return rot_pick<ROT_PAIR1, 5, 43, 2>();
        return rot_pick<ROT_PAIR1, 5, 48, 2>();
    }
    return f <= 64 ? rot_pick<ROT_PAIR1, 8, 16, 4>() : rot_pick<ROT_PAIR1, 8, 36, 4>();
}

static size_t rot_smem(const RotShape &r, const RotPick &k, uint32_t warps, uint32_t slots) {
    const size_t ring = (size_t)slots * r.cells * 128, staging = (size_t)32 * warps * (k.nw + 1) * 4;
    return ROT_HEAD + (((size_t)warps * k.S * k.nw * 4 + 127) & ~size_t(127)) + std::max(ring, staging);
}

// Two steps' chunks ahead (at least 3 slots, at most 6) where they fit.  CTAs of
// few warps wait rather than compute and take two slots, so that CTAs of
// problems on other streams fit beside them: L=100, 8192 walkers, three problems
// in turn, q=4 243 -> 134 us each, q=21 526 -> 326, alone 358 -> 349 and 666 -> 651.
static uint32_t rot_slots(const RotShape &r, const RotPick &k, uint32_t warps) {
    const uint32_t most = warps <= 8 ? 2 : std::max(3u, std::min(2 * r.nc, ROT_MAX_SLOTS));
    for (uint32_t s = most; s >= 2; --s)
        if (rot_smem(r, k, warps, s) <= 227 * 1024) return s;
    return 0;
}

// SM cycles per step of all walkers with CTAs of w warps: as many CTAs share an
// SM as its memory and registers hold (8% more where they do, since small CTAs
// end raggedly), and a wave of them takes about the largest (the 3-norm) of their
// instructions (at 3 a cycle), their gathers plus half the fill through shared
// memory, and one warp's own chain (the waits of a chunk, and 20 to 25 cycles a
// term, 43 with 5-bit fields; more per chunk where lanes share a walker).  Fitted
// to 6000 timed (lanes, warps) of 140 shapes from L=48 to 570, of which the plan
// rot_plan picks is 1.8% slower alone than the fastest in the mean; the largest of
// the three with a chain half as long and one CTA per SM, taken before, was 6%
// slower in the mean and 45% at worst (L=256, q=21, 2^17 walkers: 1.57 ms per 64 steps, now 1.08;
// L=232, q=21, 65536: 0.71, now 0.54).
// work: the instructions' share of it, were all SMs full.
static double rot_cost(const RotShape &r, const RotPick &k, uint32_t w, uint32_t nseqs, double &work) {
    const bool diff = r.mode == ROT_DIFF2, late = k.nw > 40 && k.nw < 64;
    const double steps = k.S == 1 ? 32 * (r.nc - 1) + r.tail : 32.0 / k.S * r.nc;
    const double share = k.S == 1 ? 0 : k.S == 2 ? 1 : 2;
    const double instr = diff ? steps * 2.5 + 120.0 * r.nc + 228.0
                              : steps * (k.bits == 8 ? 5.0 : 6.7) + 95.0 * r.nc + 200.0;
    const double chain =
        steps * (diff ? 20.0 : k.bits == 8 ? 25.0 : 43.0) + r.nc * ((diff ? 600.0 : 780.0) + 110.0 * share) + 705.0;
    auto wave = [&](uint32_t ctas) {
        const double issue = ctas * w * instr / (diff ? 2.9 : 3.1);
        const double smem = ctas * (w * (diff ? 1 : 2) * steps + (double)r.nc * r.cells);
        return std::cbrt(issue * issue * issue + smem * smem * smem + chain * chain * chain) * (late ? 1.15 : 1.0);
    };
    const uint32_t regs = 65536 / k.maxt / 8 * 8, per_cta = w * 32 / k.S, ctas = (nseqs + per_cta - 1) / per_cta;
    const uint32_t fit = std::min((uint32_t)(228 * 1024 / (rot_smem(r, k, w, rot_slots(r, k, w)) + 1024)),
                                  std::min(65536 / (regs * 32 * w), 2048 / (32 * w)));
    const uint32_t per_sm = std::max(1u, fit), waves = ctas / (148 * per_sm), rest = ctas - waves * 148 * per_sm;
    const double t = waves * wave(per_sm) + (rest ? wave((rest + 147) / 148) : 0.0);
    work = (double)ctas * w * instr / (diff ? 2.9 : 3.1) / 148;
    return per_sm > 1 && ctas > 148 ? 1.08 * t : t;
}

// Lanes per walker and warps per CTA (fixed ones, or 0: the cheapest).  A plan is
// also charged 0.4 of its work: one problem that does not fill the device may have
// others beside it, and more lanes per walker are more instructions (three problems
// of L=48, q=4, 2^14 walkers in turn, 768 proposals: 339 us each at two lanes, 278
// at one, though two are 4% faster alone).
static RotPick rot_plan(const RotShape &r, uint32_t nseqs, uint32_t walkers, uint32_t lanes, uint32_t &warps) {
    RotPick pick{nullptr, 0, 0, 0, 0};
    double best = 1e300;
    for (uint32_t S = 1; S <= 4; S *= 2) {
        if (lanes && lanes != S) continue;
        const RotPick k = rot_kernel(r, S);
        if (!k.kernel) continue;
        for (uint32_t w = 1; w <= k.maxt / 32; ++w) {
            if (walkers && w * 32 != walkers * S) continue;
            if (!rot_slots(r, k, w)) continue;
            double work;
            const double t = rot_cost(r, k, w, nseqs, work), c = t + 0.4 * work;
            if (c < 0.999 * best) {
                best = c;
                pick = k;
                warps = w;
            }
        }
    }
    return pick;
}

}  // namespace mi3

using namespace mi3;

extern "C" uint64_t mi3_jrot_floats(uint32_t L, uint32_t q) {
    RotShape r;
    return rot_shape(L, q, r) ? r.words : 0;
}

// Both models' errors are about 5%; where one lane can hold a walker's row, rot_cost
// is the higher one by up to 20%, hence the tenth.  Beyond, q <= 4 never pays: the
// row kernel's gathers mostly broadcast there.  Of 150 shapes the rotated kernel was
// slower than the row kernel at ten before this test, taking up to 1.6 times as
// long (L=503, q=4, 23552 walkers).
extern "C" uint32_t mi3_metropolis_rot_pays(uint32_t L, uint32_t q, uint32_t nseqs) {
    RotShape r;
    if (!rot_shape(L, q, r) || nseqs == 0 || nseqs % 32) return 0;
    uint32_t warps = 0;
    const RotPick k = rot_plan(r, nseqs, 0, 0, warps);
    if (!k.kernel) return 0;
    const bool one_lane = rot_kernel(r, 1).kernel != nullptr;
    if (!one_lane && q <= 4) return 0;
    double work;
    return rot_cost(r, k, warps, nseqs, work) <= (one_lane ? 1.1 : 1.0) * metro_cycles(L, q, nseqs);
}

extern "C" int mi3_unpack_j_rot(const float *J, float *Jrot, uint32_t L, uint32_t q, void *stream) {
    if (!J || !Jrot) return fail(MI3_ERR_ARG, "mi3_unpack_j_rot: null pointer");
    RotShape r;
    if (!rot_shape(L, q, r)) return fail(MI3_ERR_ARG, "mi3_unpack_j_rot: needs 2 <= L <= 576 and 2 <= q <= 21");
    if (!aligned(Jrot, 16)) return fail(MI3_ERR_ALIGN, "mi3_unpack_j_rot: Jrot not 16B aligned");
    k_unpack_rot<<<L, 1024, 0, as_stream(stream)>>>(J, Jrot, L, q, r);
    return check_launch("mi3_unpack_j_rot");
}

extern "C" int mi3_metropolis_rot(const float *Jrot, uint32_t *rngstates, uint32_t position_offset,
                                  const uint32_t *position_list, uint32_t nsteps, const float *betas, float beta,
                                  uint32_t *seqmem, uint32_t nseqs, uint32_t L, uint32_t q, uint32_t walkers_per_cta,
                                  uint32_t lanes_per_walker, int32_t *status, void *stream) {
    if (!Jrot || !rngstates || !position_list || !seqmem || !status)
        return fail(MI3_ERR_ARG, "mi3_metropolis_rot: null pointer");
    RotShape r;
    if (!rot_shape(L, q, r)) return fail(MI3_ERR_ARG, "mi3_metropolis_rot: needs 2 <= L <= 576 and 2 <= q <= 21");
    if (nseqs == 0 || nseqs % 32)
        return fail(MI3_ERR_ARG, "mi3_metropolis_rot: nseqs must be a positive multiple of 32");
    if (!aligned(Jrot, 16) || !aligned(rngstates, 16))
        return fail(MI3_ERR_ALIGN, "mi3_metropolis_rot: Jrot/rngstates must be 16B aligned");
    // the plan of the thread's last call, while the call has the same sizes
    static thread_local struct {
        uint32_t L = 0, q, nseqs, walkers, lanes, warps;
        RotPick k;
    } last;
    if (last.L != L || last.q != q || last.nseqs != nseqs || last.walkers != walkers_per_cta ||
        last.lanes != lanes_per_walker) {
        last.warps = 0;
        last.k = rot_plan(r, nseqs, walkers_per_cta, lanes_per_walker, last.warps);
        last.L = L, last.q = q, last.nseqs = nseqs, last.walkers = walkers_per_cta, last.lanes = lanes_per_walker;
    }
    const uint32_t warps = last.warps;
    const RotPick k = last.k;
    if (!k.kernel)
        return fail(MI3_ERR_ARG, "mi3_metropolis_rot: no kernel with these walkers per CTA and lanes per walker");
    if (nsteps == 0) return MI3_OK;
    const uint32_t slots = rot_slots(r, k, warps);
    const size_t smem = rot_smem(r, k, warps, slots);
    cudaFuncSetAttribute(k.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    RotParams p;
    p.T = reinterpret_cast<const int32_t *>(Jrot);
    p.bound = Jrot + r.bound_at;
    p.J = Jrot + r.j_at;
    p.row_words = r.row_words;
    p.rng = reinterpret_cast<uint4 *>(rngstates);
    p.poslist = position_list;
    p.pos_off = position_offset;
    p.nsteps = nsteps;
    p.betas = betas;
    p.beta = beta;
    p.seq = seqmem;
    p.nseqs = nseqs;
    p.L = L;
    p.q = q;
    p.Q = r.Q;
    p.nc = r.nc;
    p.tail = r.tail;
    p.cells = r.cells;
    p.slots = slots;
    p.last = k.S > 1 && r.tail < 32 ? r.nc : r.nc - 1;
    p.line = 128;
    p.q_inv = (65536 + q - 1) / q;
    p.q_magic = (uint32_t)((1ull << 32) / q);
    p.half_u = 1.01f * 0x1p-24f * (float)(L - L / 2 + 1);
    p.status = status;
    const uint32_t per_cta = warps * 32 / k.S;
    k.kernel<<<(nseqs + per_cta - 1) / per_cta, 32 * warps, smem, as_stream(stream)>>>(p);
    return check_launch("mi3_metropolis_rot");
}
