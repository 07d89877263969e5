// joint.cuh -- slice tiling of the pair kernels over joint sites (q <= 21).
//
// The pair passes (energies, counts, weighted bimarginals) cost one shared-
// memory access per (sequence, pair of sites).  For small alphabets several
// site pairs fit one access: G neighbouring sites form a joint site whose
// state packs their residues (a0 + q*a1), and a table over pairs of joint
// sites holds the sum of the couplings of all GI*GJ site pairs in one cell
// (energies), or counts all of them in one bin, which the flush splits back
// into the site pairs' bins (exact integers).  GI joint sites are taken for
// the rows of a slice, GJ for its columns:
//
//   q       GI x GJ  joint sites per block B   table (4 q^(GI+GJ) B*B bytes)
//   1       1 x 1    16                        1 KB
//   2, 3    2 x 2    16                        16, 83 KB     4 pairs a gather
//   4, 5    2 x 2    8                         64, 160 KB    4 pairs a gather
//   6..8    2 x 1    8                         55..131 KB    2 pairs a gather
//   9, 10   1 x 1    16                        83, 102 KB
//   11..21  1 x 1    8                         31..113 KB
//
// The lines lie where the next larger table no longer fits shared memory
// (q=5 2x2 leaves 26 KB for staging; q=6 2x2 would need 332 KB).  Larger
// alphabets (22..42) keep the pair-major kernels of tiling.cuh.
//
// Tables are cell-major, [cell][P], P = B*B joint pairs, and each lane visits
// the pairs in its own order (tiling.cuh), so every access is one wavefront.
// Slices that cross the diagonal or the end of the sequence run the same
// code: their invalid site pairs add zero couplings, or are not flushed.
//
// Measured against the pair-major tiling with lanes over pairs in full slices
// only (Newton phases on one B200, l1z or l2z included):
//   L=93  q=4  2^18  8 steps   10.0 -> 2.15 ms (2.92 with the alphabet a
//                              run-time value in the packing and splitting)
//   L=151 q=8  66048 8 steps   5.55 -> 2.88 ms (3.58)
//   L=232 q=21 2^20  3 steps   38.6 -> 35.5 ms (edge slices, packed adds, one
//                              clamp test per word)
#pragma once
#include "tiling.cuh"

namespace mi3 {

struct JointGeom {
    uint32_t nbI, nbJ;  // row blocks of B*GI sites, column blocks of B*GJ sites
    uint32_t nslices;
    uint32_t chunk, nchunks;
};

// Row block bi pairs with the column blocks bj >= r*bi, r = GI / GJ.
template <int GI, int GJ>
__device__ __forceinline__ void joint_coords(uint32_t s, uint32_t nbJ, uint32_t &bi, uint32_t &bj) {
    constexpr uint32_t R = GI / GJ;
    uint32_t r = 0, base = 0;
    while (base + (nbJ - R * r) <= s) {
        base += nbJ - R * r;
        ++r;
    }
    bi = r;
    bj = R * r + (s - base);
}

inline void joint_slices(uint32_t L, uint32_t B, uint32_t GI, uint32_t GJ, JointGeom *g) {
    const uint32_t nbI = (L + B * GI - 1) / (B * GI), nbJ = (L + B * GJ - 1) / (B * GJ), R = GI / GJ;
    g->nbI = nbI;
    g->nbJ = nbJ;
    g->nslices = 0;
    for (uint32_t r = 0; r < nbI; ++r) g->nslices += nbJ - R * r;
}

__host__ __device__ constexpr uint32_t joint_states(uint32_t q, uint32_t G) { return G == 1 ? q : q * q; }

// Floats (bins) of a slice table, and of the staging area that holds the
// slice's site pairs [GI*B][GJ*B] of q*q entries while the joint table is
// built or taken apart (G > 1 only).  The staging strides -- S per pair
// (= 2 mod 16 for GJ = 2, 4 mod 32 for GJ = 1) and an odd row -- keep the 32
// pairs of a warp on different banks (two lanes a bank at most).
__host__ __device__ constexpr uint32_t joint_table(uint32_t q, uint32_t B, uint32_t GI, uint32_t GJ) {
    return joint_states(q, GI) * joint_states(q, GJ) * B * B;
}
__host__ __device__ constexpr uint32_t joint_stage_pair(uint32_t q, uint32_t GJ) {
    return GJ == 2 ? ((q * q + 13) / 16) * 16 + 2 : ((q * q + 27) / 32) * 32 + 4;
}
__host__ __device__ constexpr uint32_t joint_stage_row(uint32_t q, uint32_t B, uint32_t GJ) {
    return B * GJ * joint_stage_pair(q, GJ) + 1;
}
__host__ __device__ constexpr uint32_t joint_stage(uint32_t q, uint32_t B, uint32_t GI, uint32_t GJ) {
    return GI * GJ == 1 ? 0 : GI * B * joint_stage_row(q, B, GJ);
}
__host__ __device__ constexpr size_t joint_smem(uint32_t q, uint32_t B, uint32_t GI, uint32_t GJ) {
    return ((size_t)joint_table(q, B, GI, GJ) + joint_stage(q, B, GI, GJ)) * 4;
}

// The B joint states of a block as bytes (first joint site in byte 0 of
// word 0) from its G*B/4 sequence words.  Residues >= q (invalid input) are
// clamped to q - 1, so every state indexes its table.
template <int B, int G>
__device__ __forceinline__ void joint_words(const uint32_t (&w)[G * B / 4], uint32_t q, uint32_t (&o)[B / 4]) {
    // a byte >= q is rare (never in valid input): test all words at once
    const uint32_t lift = (128u - q) * 0x01010101u;
    uint32_t bad = 0;
#pragma unroll
    for (int k = 0; k < G * B / 4; ++k) bad |= (((w[k] & 0x7f7f7f7fu) + lift) | w[k]) & 0x80808080u;
    uint32_t v[G * B / 4];
#pragma unroll
    for (int k = 0; k < G * B / 4; ++k) v[k] = w[k];
    if (bad) {
#pragma unroll
        for (int k = 0; k < G * B / 4; ++k) v[k] = __vminu4(w[k], (q - 1) * 0x01010101u);
    }
    if constexpr (G == 1) {
#pragma unroll
        for (int k = 0; k < B / 4; ++k) o[k] = v[k];
    } else {
        // sites 0, 1 -> state a0 + q*a1 in the low half, sites 2, 3 in the high
#pragma unroll
        for (int k = 0; k < B / 4; ++k) {
            const uint32_t t0 = (v[2 * k] & 0x00ff00ffu) + q * ((v[2 * k] >> 8) & 0x00ff00ffu);
            const uint32_t t1 = (v[2 * k + 1] & 0x00ff00ffu) + q * ((v[2 * k + 1] >> 8) & 0x00ff00ffu);
            o[k] = __byte_perm(t0, t1, 0x6420);
        }
    }
}

// Per-lane constants of the lane's order: shared-memory address of the table
// (at `base`) plus row position k ^ w, and byte offset of column position
// k ^ w.  Hoisted out of the sequence loop.
template <int B>
struct LaneConst {
    uint32_t row[B], col[B], wh, wl;
    __device__ __forceinline__ LaneConst(uint32_t lane, uint32_t base) : wh(lane / B), wl(lane % B) {
#pragma unroll
        for (int k = 0; k < B; ++k) {
            row[k] = base + 4 * B * (k ^ wh);
            col[k] = 4 * (k ^ wl);
        }
    }
};

// Addresses in the [cell][P] table of the lane's row terms (joint row state A:
// A*QJ cells) and byte offsets of its column terms, in the lane's order.
template <int B>
__device__ __forceinline__ void joint_offsets(const uint32_t (&sI)[B / 4], const uint32_t (&sJ)[B / 4],
                                              uint32_t row_scale, const LaneConst<B> &lc, uint32_t (&row)[B],
                                              uint32_t (&col)[B]) {
    uint32_t rI[B / 4], rJ[B / 4];
    permute_block<B>(sI, lc.wh, rI);
    permute_block<B>(sJ, lc.wl, rJ);
#pragma unroll
    for (int k = 0; k < B; ++k) {
        row[k] = __byte_perm(rI[k >> 2], 0, 0x4440 + (k & 3)) * row_scale + lc.row[k];
        col[k] = __byte_perm(rJ[k >> 2], 0, 0x4440 + (k & 3)) * (4 * B * B) + lc.col[k];
    }
}

template <int W>
__device__ __forceinline__ void load_words(const uint32_t *__restrict__ seq, uint32_t buflen, uint32_t n,
                                           uint32_t w0, uint32_t swords, uint32_t (&w)[W]) {
#pragma unroll
    for (int k = 0; k < W; ++k) w[k] = (w0 + k < swords) ? __ldg(&seq[(size_t)(w0 + k) * buflen + n]) : 0u;
}

// fn(row addresses, column offsets, n) for every sequence of [nbeg, nend) that
// this thread takes; the next sequence's words load while one is processed.
template <int B, int GI, int GJ, typename F>
__device__ __forceinline__ void joint_sequences(const uint32_t *__restrict__ seq, uint32_t buflen, uint32_t nbeg,
                                                uint32_t nend, uint32_t L, uint32_t q, uint32_t bi, uint32_t bj,
                                                uint32_t base, F &&fn) {
    constexpr int WI = GI * B / 4, WJ = GJ * B / 4;
    const uint32_t swords = (L - 1) / 4 + 1;
    const LaneConst<B> lc(threadIdx.x & 31, base);
    const uint32_t row_scale = 4 * B * B * joint_states(q, GJ);
    uint32_t n = nbeg + threadIdx.x;
    if (n >= nend) return;
    uint32_t wI[WI], wJ[WJ];
    load_words<WI>(seq, buflen, n, bi * WI, swords, wI);
    load_words<WJ>(seq, buflen, n, bj * WJ, swords, wJ);
    while (true) {
        uint32_t sI[B / 4], sJ[B / 4], row[B], col[B];
        joint_words<B, GI>(wI, q, sI);
        joint_words<B, GJ>(wJ, q, sJ);
        const uint32_t next = n + blockDim.x;
        if (next < nend) {
            load_words<WI>(seq, buflen, next, bi * WI, swords, wI);
            load_words<WJ>(seq, buflen, next, bj * WJ, swords, wJ);
        }
        joint_offsets<B>(sI, sJ, row_scale, lc, row, col);
        fn(row, col, n);
        if (next >= nend) return;
        n = next;
    }
}

// o[k] = v[(k + r) mod 8], r < 8 a run-time value: three conditional swaps.
template <typename V>
__device__ __forceinline__ void rotate8(V (&v)[8], uint32_t r) {
#pragma unroll
    for (uint32_t s = 1; s < 8; s <<= 1) {
        V o[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) o[k] = (r & s) ? v[(k + s) & 7] : v[k];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) v[k] = o[k];
    }
}

// Moves a 1 x 1 slice between its [cell][P] table in shared memory and the
// packed [pair][cell] arrays.  A warp takes 8 cells of 32 pairs: lane l holds
// cell c0 + l % 8 of the pairs p0 + 4 j + l / 8, j = 0..7, which is 8 consecutive
// cells of 4 pairs per global access.  In the table those lanes would share a
// bank per pair, eight to one; in step k lane l instead moves pair group
// (k + l) mod 8, all 32 banks.  fn(cell, pair) gives the element to store, or
// fn(cell, pair, v) takes the one read.
template <uint32_t P, uint32_t T, bool TO_TABLE, typename V, typename F>
__device__ __forceinline__ void slice_transpose(V *table, uint32_t qq, F &&fn) {
    const uint32_t lane = threadIdx.x & 31, cl = lane & 7, pl = lane >> 3;
    const uint32_t cgroups = (qq + 7) / 8;
    for (uint32_t t = threadIdx.x >> 5; t < cgroups * (P / 32); t += T / 32) {
        const uint32_t c = (t % cgroups) * 8 + cl, p0 = (t / cgroups) * 32;
        V v[8];
        if constexpr (TO_TABLE) {
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j) v[j] = c < qq ? fn(c, p0 + 4 * j + pl) : V(0);
            rotate8(v, cl);
            if (c < qq) {
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k) table[c * P + p0 + 4 * ((k + cl) & 7) + pl] = v[k];
            }
        } else {
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) v[k] = c < qq ? table[c * P + p0 + 4 * ((k + cl) & 7) + pl] : V(0);
            rotate8(v, (8 - cl) & 7);
            if (c < qq) {
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) fn(c, p0 + 4 * j + pl, v[j]);
            }
        }
    }
}

// fn(row, column, entry) for all entries of a slice's GI*B x GJ*B site pairs, in
// the order of the packed arrays: a warp takes a site pair at a time, or, where
// that would leave half its lanes idle (q <= 4), the CTA takes consecutive entries
// (L=64, 4096 sequences, energies: q=2 36 -> 23 us, q=3 37 -> 25; counts at q=5 and
// 7 took 6 to 15% longer that way).
template <int B, int GI, int GJ, int T, int QC, typename F>
__device__ __forceinline__ void joint_pairs(F &&fn) {
    constexpr uint32_t qq = QC * QC, row = GJ * B * qq;
    if constexpr (qq <= 16) {
#pragma unroll 4
        for (uint32_t t = threadIdx.x; t < GI * B * row; t += T) fn(t / row, t % row / qq, t % qq);
    } else {
#pragma unroll 4
        for (uint32_t t = threadIdx.x >> 5; t < GI * B * GJ * B; t += T / 32)
            for (uint32_t e = threadIdx.x & 31; e < qq; e += 32) fn(t / (GJ * B), t % (GJ * B), e);
    }
}

// Tile configuration of an alphabet: B joint sites per block, GI x GJ sites
// per joint pair, T threads (1024 resident threads per SM at 64 registers, so T =
// 1024 where table and staging of two CTAs exceed the SM: q=3, 2^16 sequences,
// L=187, energies 121 us with 512, 78 with 1024; q=7, L=128, 85 and 72), and the alphabet QC where joint
// states are packed and split, so that those divisions and sums unroll (0: any).
// OVERHEAD: what building or splitting a CTA's table costs, in sequences.
template <int B_, int GI_, int GJ_, int T_, int QC_>
struct JointCfg {
    static constexpr int B = B_, GI = GI_, GJ = GJ_, T = T_, QC = QC_;
    static constexpr uint32_t OVERHEAD = GI * GJ == 1 ? 2048 : 4096;
    // 1024 resident threads per SM, whose 228 KB hold their tables (and 1 KB a CTA)
    static_assert(GI * GJ == 1 || (1024 / T) * (joint_smem(QC, B, GI, GJ) + 1024) <= 228 * 1024, "threads per CTA");
};

// Calls fn(JointCfg) for the alphabet; returns false when it has none.
template <typename F>
static bool joint_dispatch(uint32_t q, F &&fn) {
    if (q == 1 || q == 9 || q == 10) fn(JointCfg<16, 1, 1, 512, 0>());
    else if (q == 2) fn(JointCfg<16, 2, 2, 512, 2>());
    else if (q == 3) fn(JointCfg<16, 2, 2, 1024, 3>());
    else if (q == 4) fn(JointCfg<8, 2, 2, 512, 4>());
    else if (q == 5) fn(JointCfg<8, 2, 2, 1024, 5>());
    else if (q == 6) fn(JointCfg<8, 2, 1, 512, 6>());
    else if (q == 7) fn(JointCfg<8, 2, 1, 1024, 7>());
    else if (q == 8) fn(JointCfg<8, 2, 1, 1024, 8>());
    else if (q >= 11 && q <= 21) fn(JointCfg<8, 1, 1, 512, 0>());
    else return false;
    return true;
}

// All CTAs of a pass do the same work, so one wave will do.
template <typename C>
static JointGeom joint_geom(uint32_t L, uint32_t nseq) {
    JointGeom g;
    joint_slices(L, C::B, C::GI, C::GJ, &g);
    g.chunk = pick_chunk(g.nslices, nseq, 148 * (1024 / C::T), C::OVERHEAD);
    g.nchunks = (nseq - 1) / g.chunk + 1;
    return g;
}

}  // namespace mi3
