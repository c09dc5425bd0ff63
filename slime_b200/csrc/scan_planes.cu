// scan_planes.cu -- band searches as bit planes: exact counts of every centre (low thresholds, all
// band modes) and bounded counts of independent bands.
//
// Behaviour: the same kept set as the general scan (SlimeCoreGPU.cu:501-610 semantics) for
// first-draw slime chunks; the rare Java redraws are added back by rare_fix.cu.
//
// B200 design (see band_math.cuh for the arithmetic). scan_band.cu packs 32 columns of one combo (an
// X phase and Z band copy of the base tile) into a word; here a word is one column of up to 32 combos:
//  * A thread evaluates 4 columns and shifts every first-draw test into its own words: an add whose
//    carry says "no hit", and the add-with-carry that shifts it in. No ballot, and one store a word.
//  * The counter needs no funnel shifts or shuffles: neighbouring columns are neighbouring words of
//    shared memory, and every full adder (two LOP3) adds a bit of 32 combos at once.
//  * Rows advance in batches through a 24-row ring in shared memory (96 KB), two CTAs an SM, so that
//    one CTA computes while the other waits at its barriers. Row terms arrive by TMA bulk copies two
//    batches ahead.
//  * Exact counting: each window slides down a row by adding its 17 entering cells and the complement
//    of its 17 leaving cells to the 8 count planes: 38 full adders for 32 centres.
//  * Bounded counting: 4x4 block sums leave the generator as 5 planes; five neighbours add up to a
//    20-column strip sum, five strips to the 20x20 box that bounds the 16 windows of a 4x4 centre
//    group. Where boxes reach the threshold, the 68 cells that no window reaches are taken off, and a
//    group that still reaches it is counted exactly.
// What bounds it (B200): integer issue. Independent bands, radius 100,000: the generator is 19 of the
// 28.7 ms at threshold 42 (15.9 cycles a warp test in a probe of it alone; its one wide multiply costs
// about five of them) and the exact counter 9.5; packing columns took 42.4 ms. At threshold 60
// (bounded) 22.2 ms against 29.2. Grouped bands, radius 300,000, threshold 44: 211 against 276 ms.
// Bounded counts of shared and grouped bands stay with columns in words (1,134 against 1,408 ms at
// radius 1,250,000, 111 against 127 ms at radius 300,000, threshold 60): their five-instruction test
// gains too little here to pay for box sums over partly filled words.
#include "band_math.cuh"
#include "engine.h"

namespace slime {
namespace {

using namespace band;

constexpr int kTpb = 256;
constexpr int kCtasPerSm = 2;
constexpr int kMaxBands = 32;
// Band modes. Shared LCG: two X phases x up to 32 Z bands 2^17 apart, all sharing the low 17 bits
// of the row term. Independent bands: one X phase x up to 32 bands at any row spacing. Grouped
// bands: two X phases x up to 16 bands, in G groups at their own base rows, each group holding P
// copies 2^17 apart that share its low bits (band m = group * P + copy).
constexpr int kModeShared = 0, kModeIndep = 1, kModeGrouped = 2;
constexpr int kGrpBands = 16;
constexpr unsigned kFull = 0xFFFFFFFFu;

constexpr int kRingRows = 24;
constexpr int kRingWords = kRingRows * 1024;
constexpr int kMostBatchRows = 8;

// Row-term record of one base row (written by row_terms_kernel): [m] and [32 + m] the two parts of
// the row term in band m, or with the shared LCG [32] the low part of all bands; then the mask of
// the bands that hold the row. The rows of a batch are one contiguous bulk copy.
constexpr int kRowWordsS = 36, kRowWordsI = 72;
constexpr int kRowLo = 32;
template <int kMode>
constexpr int row_words() { return kMode == kModeShared ? kRowWordsS : kRowWordsI; }
template <int kMode>
constexpr int row_valid() { return kMode == kModeShared ? 33 : 64; }

// Independent bands split a term at bit 18, the low part shifted up by 14: the product's high word
// is then state1 >> 18 and the top bit of its low word the parity of the first draw.
constexpr int kIndepBits = 18;
__host__ __device__ __forceinline__ uint32_t indep_lo(uint64_t t) { return (uint32_t)t << (32 - kIndepBits); }
__host__ __device__ __forceinline__ uint32_t indep_hi(uint64_t t) { return (uint32_t)(t >> kIndepBits); }

// Tile shape of a mode: kNW words a column (one a phase with the shared LCG), kTW input columns.
// kNW * kTW = 1,024 words a row in every mode, so that ring and thread layout agree. Rows advance in
// batches with a barrier after generating and one after counting: 8 rows where counting looks back
// four strips from the first strip of the batch (24 rows with it), 6 where a window's slide looks
// back 17 rows from the first row of the batch (23 rows with it).
template <int kMode, bool kExact>
struct Shape {
    static constexpr int kNW = kMode == kModeShared ? 2 : 1;
    static constexpr int kTW = 1024 / kNW;
    static constexpr int kBlocks = kTW / 4;      // 4-column blocks: thread = (block, word)
    static constexpr int kOutW = kTW - 16;
    static constexpr int kBatchRows = kExact ? 6 : 8;
    static constexpr int kRingBatches = kRingRows / kBatchRows;
    static constexpr int kRowsPerThread = kBatchRows / kNW;  // generator: thread = (block, row part)
};

struct __align__(16) PlaneSmem {
    uint32_t ring[kRingWords];                // [row % 24][word][column]
    uint32_t sums[2][5][256];                 // block sums [strip of the batch][plane][word, block]
    uint32_t rows[2][kMostBatchRows * kRowWordsI];  // row terms of 2 batches, filled by bulk copies
    unsigned long long rows_bar[2];           // mbarriers of the two row-term buffers
    BandArgs args;                            // batched kernel: the current tile's search
    long long next_tile;                      // batched kernel: tile taken from the queue
    int search;                               // batched kernel: its search
    int failed;  // a bounded wait gave up: the CTA stops
    unsigned int hist[kHistBins];             // counts of this CTA's centres in range (if args.hist)
};
static_assert(sizeof(PlaneSmem) <= (233472 - 2048) / kCtasPerSm, "two CTAs an SM");

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Bulk copy (TMA engine, no multicast) of `bytes` from global memory into shared memory,
// completing on an mbarrier. Addresses and size are multiples of 16 bytes.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes,
                                          unsigned long long* bar) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                 :: "r"(smem_u32(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// Waits for the mbarrier phase with the given parity; gives up after `polls` polls and returns
// false (the caller flags an error instead of hanging the GPU).
__device__ __forceinline__ bool bar_wait(unsigned long long* bar, uint32_t parity, uint32_t polls) {
    for (uint32_t i = 0; i < polls; ++i) {
        uint32_t done;
        asm volatile("{ .reg .pred p;\n"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                     "selp.u32 %0, 1, 0, p; }"
                     : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}

struct Tile {
    int u0, v0, i0, out_h;
    int bands;      // bands tested: those with a centre of the area in this tile (grouped: copies)
    int copies;     // grouped bands: copies of a group
    uint32_t mask;  // their bits in a row's valid mask
};

// First area row (band axis) of band m, before the tile's base row is added.
template <int kMode>
__device__ __forceinline__ int64_t band_row0(const BandArgs& a, int m) {
    if (kMode != kModeGrouped) return (int64_t)(a.j0 + m) * a.row_stride;
    const int copies = a.nb / a.groups;
    return (int64_t)(m % copies) * kPeriod + (int64_t)(m / copies) * a.row_stride;
}

// ---- bit-sliced adders: bit j of every word belongs to combo j ----------------------------------

__device__ __forceinline__ void bs_fa(uint32_t a, uint32_t b, uint32_t c, uint32_t& s, uint32_t& cy) {
    const uint32_t x = a, y = b, z = c;
    s = x ^ y ^ z;
    cy = (x & y) | (z & (x | y));
}

// out = a + b over NO planes (a: NA planes, b: NB <= NA planes; the caller knows the sum fits).
template <int NA, int NB, int NO>
__device__ __forceinline__ void bs_add(const uint32_t (&a)[NA], const uint32_t (&b)[NB], uint32_t (&out)[NO]) {
    static_assert(NB <= NA && NO >= NA && NO <= NA + 1, "plane counts");
    uint32_t c = 0;
#pragma unroll
    for (int i = 0; i < NA; ++i) {
        if (i < NB) {
            bs_fa(a[i], b[i], c, out[i], c);
        } else {
            const uint32_t x = a[i];
            out[i] = x ^ c;
            c = x & c;
        }
    }
    if constexpr (NO > NA) out[NA] = c;
}

// Carry-save accumulator: planes p[0..], and per weight at most one waiting carry. add(k, a, b) is
// the k-th pair of single-bit inputs (k a compile-time constant after unrolling).
struct BitSum {
    uint32_t p[9], wait[9];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < 9; ++i) p[i] = 0;
    }
    __device__ __forceinline__ void add(int k, uint32_t a, uint32_t b) {
        uint32_t c;
        bs_fa(p[0], a, b, p[0], c);
#pragma unroll
        for (int w = 1; w < 8; ++w, k >>= 1) {
            if (!(k & 1)) {
                wait[w] = c;
                return;
            }
            bs_fa(p[w], wait[w], c, p[w], c);
        }
    }
    // Adds what still waits after `pairs` pairs; the planes are then the sum.
    __device__ __forceinline__ void finish(int pairs) {
        uint32_t c = 0;
#pragma unroll
        for (int w = 1; w < 9; ++w, pairs >>= 1) bs_fa(p[w], (w < 8 && (pairs & 1)) ? wait[w] : 0u, c, p[w], c);
    }
};

// Bits where the N-plane number x is at least t (0 <= t <= 2^N): the carry out of x + (2^N - t),
// whose bits are all-ones or zero words, so each plane is one majority LOP3.
template <int N>
__device__ __forceinline__ uint32_t bs_at_least(const uint32_t* x, int t) {
    const uint32_t k = (1u << N) - (uint32_t)t;
    uint32_t c = 0;
#pragma unroll
    for (int b = 0; b < N; ++b) {
        const uint32_t kb = 0u - ((k >> b) & 1u);
        c = (x[b] & c) | (kb & (x[b] | c));
    }
    return (k >> N) ? ~0u : c;
}

__device__ __forceinline__ int bs_value(const uint32_t (&cnt)[8], int j) {
    int v = 0;
#pragma unroll
    for (int b = 0; b < 8; ++b) v |= (int)((cnt[b] >> j) & 1u) << b;
    return v;
}

// Window-relative vertical half-extent of the column at horizontal offset k = |dx| from the centre
// (-1 outside the window).
__host__ __device__ constexpr int column_half_height(int k) {
    return k <= 2 ? 8 : k <= 4 ? 7 : k == 5 ? 6 : k == 6 ? 5 : k == 7 ? 4 : k == 8 ? 2 : -1;
}

// ---- generator ---------------------------------------------------------------------------------

// w = 2 w + (y >= kHitBelow): the carry of y + (2^32 - kHitBelow) shifted in.
__device__ __forceinline__ void shift_miss(uint32_t& w, uint32_t y, uint32_t below) {
    asm("{ .reg .u32 t;\n add.cc.u32 t, %1, %2;\n addc.u32 %0, %0, %0; }" : "+r"(w) : "r"(y), "r"(0u - below));
}

// First-draw test with the shared part of the low bits (x, d from shared_part).
__device__ __forceinline__ void shift_test(uint32_t& w, uint32_t x, uint32_t z, uint32_t d) {
    shift_miss(w, ((x + z) ^ kXorHi) * kMulH + d, kHitBelow);
}

// First-draw test of one chunk from split terms (independent bands: nothing is shared). With the
// seed mix M = H * 2^18 + l and lo = l * 2^14, the product (M ^ S) * A + 11, taken times 2^14, has
// u = state1 >> 18 in its high word and bit 17 of state1 (the parity of the first draw) in the top
// bit of its low word. An even draw is 2 u (u mod 2^30), and it is a multiple of 10 below the
// rejection bound iff 4 u inv5 (mod 2^32) < kHitBelow; kHitBelow < 2^31, so the parity bit is OR-ed
// in. Eleven instructions.
__device__ __forceinline__ void shift_indep(uint32_t& w, uint32_t xl, uint32_t xh, uint32_t zl, uint32_t zh) {
    uint32_t lo, hi;
    asm("{ add.cc.u32 %0, %2, %3;\n addc.u32 %1, %4, %5; }" : "=r"(lo), "=r"(hi) : "r"(xl), "r"(zl), "r"(xh), "r"(zh));
    lo ^= indep_lo(band::kSeedXor);
    hi ^= indep_hi(band::kSeedXor);
    const uint64_t prod = (uint64_t)lo * kA32 + (11ull << (32 - kIndepBits));
    // u = (high word) + 5 lo + A hi, and 20 inv5 = 4 (mod 2^32).
    const uint32_t y = (uint32_t)(prod >> 32) * (4u * kInv5) + (hi * (4u * kInv5 * kA32) + (lo << 2));
    shift_miss(w, y | ((uint32_t)prod & 0x80000000u), kHitBelow);
}

// Column terms of a generator thread's four columns, and which do not exist (bit k: column k of
// the first phase, bit 4 + k: of the second). Absent columns hold no hits, so that they reach no bound.
struct Columns {
    uint32_t lo[4], h0[4], h1[4], absent;
};

// The words of four columns of one row, into w[word][column]: zr is the row's record.
template <int kMode>
__device__ __forceinline__ void generate_row(const BandArgs& a, const Tile& T, const Columns& C, const uint32_t* zr,
                                             uint32_t (&w)[kMode == kModeShared ? 2 : 1][4]) {
    const uint32_t valid = zr[row_valid<kMode>()] & T.mask;
    const int bands = T.bands;
    uint32_t miss[4] = {0u, 0u, 0u, 0u};
    if constexpr (kMode == kModeIndep) {
#pragma unroll 1
        for (int m = (bands - 1) & ~3; m >= 0; m -= 4) {
            const uint4 zl = *reinterpret_cast<const uint4*>(zr + kRowLo + m);
            const uint4 zh = *reinterpret_cast<const uint4*>(zr + m);
#pragma unroll
            for (int k = 0; k < 4; ++k) shift_indep(miss[k], C.lo[k], C.h0[k], zl.w, zh.w);
#pragma unroll
            for (int k = 0; k < 4; ++k) shift_indep(miss[k], C.lo[k], C.h0[k], zl.z, zh.z);
#pragma unroll
            for (int k = 0; k < 4; ++k) shift_indep(miss[k], C.lo[k], C.h0[k], zl.y, zh.y);
#pragma unroll
            for (int k = 0; k < 4; ++k) shift_indep(miss[k], C.lo[k], C.h0[k], zl.x, zh.x);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) w[0][k] = ~miss[k] & valid;
        if (C.absent) {
#pragma unroll
            for (int k = 0; k < 4; ++k) w[0][k] = (C.absent >> k) & 1u ? 0u : w[0][k];
        }
    } else if constexpr (kMode == kModeShared) {
        const uint32_t zlo = zr[kRowLo], zpar = (zr[0] ^ kXorHi) & 1u;
        uint32_t xa[4], xb[4], dd[4], even[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            bool odd;
            shared_part(C.lo[k], C.h0[k], C.h1[k], zlo, zpar, xa[k], xb[k], dd[k], odd);
            even[k] = odd ? 0xAAAAAAAAu : 0x55555555u;  // bands whose hit belongs to phase 0
        }
#pragma unroll 2
        for (int m = (bands - 1) & ~3; m >= 0; m -= 4) {
            const uint4 z = *reinterpret_cast<const uint4*>(zr + m);
#pragma unroll
            for (int k = 0; k < 4; ++k) shift_test(miss[k], xb[k], z.w, dd[k]);
#pragma unroll
            for (int k = 0; k < 4; ++k) shift_test(miss[k], xa[k], z.z, dd[k]);
#pragma unroll
            for (int k = 0; k < 4; ++k) shift_test(miss[k], xb[k], z.y, dd[k]);
#pragma unroll
            for (int k = 0; k < 4; ++k) shift_test(miss[k], xa[k], z.x, dd[k]);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t hit = ~miss[k] & valid;
            w[0][k] = hit & even[k];
            w[1][k] = hit & ~even[k];
        }
        if (C.absent) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                w[0][k] = (C.absent >> k) & 1u ? 0u : w[0][k];
                w[1][k] = (C.absent >> (4 + k)) & 1u ? 0u : w[1][k];
            }
        }
    } else {
        const int G = a.groups, copies = T.copies;
        const uint32_t even_copies = 0x5555u & ((1u << copies) - 1u), odd_copies = 0xAAAAu & ((1u << copies) - 1u);
        uint32_t first[4] = {0u, 0u, 0u, 0u};  // per band: the hit belongs to phase 0
#pragma unroll 1
        for (int g = G - 1; g >= 0; --g) {
            const uint32_t* z = zr + g * copies;
            const uint32_t zlo = z[kRowLo], zpar = (z[0] ^ kXorHi) & 1u;
            uint32_t xa[4], xb[4], dd[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                bool odd;
                shared_part(C.lo[k], C.h0[k], C.h1[k], zlo, zpar, xa[k], xb[k], dd[k], odd);
                first[k] = (first[k] << copies) | (odd ? odd_copies : even_copies);
                miss[k] <<= copies - bands;  // copies without a centre in the tile: not valid
            }
            int c = bands;
            if (c & 1) {
                const uint32_t z0 = z[--c];
#pragma unroll
                for (int k = 0; k < 4; ++k) shift_test(miss[k], xa[k], z0, dd[k]);
            }
#pragma unroll 2
            while (c > 0) {
                const uint32_t z1 = z[c - 1], z0 = z[c - 2];
                c -= 2;
#pragma unroll
                for (int k = 0; k < 4; ++k) shift_test(miss[k], xb[k], z1, dd[k]);
#pragma unroll
                for (int k = 0; k < 4; ++k) shift_test(miss[k], xa[k], z0, dd[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t hit = ~miss[k] & valid;
            w[0][k] = (hit & first[k]) | ((hit & ~first[k]) << kGrpBands);
        }
        if (C.absent) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                w[0][k] &= ((C.absent >> k) & 1u ? 0u : 0xFFFFu) | ((C.absent >> (4 + k)) & 1u ? 0u : 0xFFFF0000u);
        }
    }
}

// ---- counters ----------------------------------------------------------------------------------

// A centre whose exact count lies in [min_size, max_size]: combo bit `bit` of word `word`, tile input
// column `col` and output row `rr`. Dropped when it lies outside the area or inside the rd_min disc;
// else it is added to the histogram and, from the emission gate on, appended to the hit list. Called
// by any subset of a warp.
template <int kMode>
__device__ __forceinline__ void keep_centre(PlaneSmem& S, const BandArgs& a, const Tile& T, int word, int bit, int col,
                                            int rr, int count) {
    const int ph = kMode == kModeShared ? word : kMode == kModeGrouped ? bit >> 4 : 0;
    const int m = kMode == kModeGrouped ? bit & 15 : bit;
    const int c = col - 8;
    if (m >= a.nb || c < 0 || c >= Shape<kMode, false>::kOutW || rr < 0 || rr >= T.out_h) return;
    const int64_t u = (int64_t)T.u0 + c;
    const int64_t cu = u + (int64_t)(T.i0 + ph) * kPeriod;
    const int64_t cv = (int64_t)T.v0 + rr + band_row0<kMode>(a, m);
    // Grouped bands: rows of the last group past the period belong to the next copy's first group.
    if (kMode == kModeGrouped && T.copies > 1 && T.v0 + rr + (m / T.copies) * a.row_stride >= kPeriod) return;
    if (u >= a.ubase || cu >= a.width_u || cv >= a.height_v) return;
    const int32_t cx = (int32_t)(a.transposed ? a.area_x0 + cv : a.area_x0 + cu);
    const int32_t cz = (int32_t)(a.transposed ? a.area_z0 + cu : a.area_z0 + cv);
    if (a.rd_min_sq) {
        const int64_t ddx = (int64_t)cx - a.center_x, ddz = (int64_t)cz - a.center_z;
        if (ddx * ddx + ddz * ddz < a.rd_min_sq) return;
    }
    if (a.hist) atomicAdd(&S.hist[count], 1u);
    if (count < a.emit_min) return;
    const unsigned mk = __activemask();
    const int lane = threadIdx.x & 31, leader = __ffs(mk) - 1;
    unsigned long long base = 0;
    if (lane == leader) base = atomicAdd(a.emitted, (unsigned long long)__popc(mk));
    base = __shfl_sync(mk, base, leader) + __popc(mk & ((1u << lane) - 1u));
    if (base < a.cap) a.out[base] = Hit{count, cx, cz};
}

// Word `word` of column `col` in ring row `row` (0 .. kRingRows - 1).
template <int kMode>
__device__ __forceinline__ const uint32_t* ring_at(const PlaneSmem& S, int row, int word, int col) {
    using Sh = Shape<kMode, false>;
    return &S.ring[(row * Sh::kNW + word) * Sh::kTW + col];
}

// The corner cells of the 20x20 box that no window of the group reaches (17 a corner), per box row
// 0..5 (or column: the shape is symmetric): columns 0 .. corner_cells(row) - 1 and their mirror images.
__host__ __device__ constexpr int corner_cells(int r) {
    return r == 0 ? 6 : r == 1 ? 4 : r == 2 ? 3 : r == 3 ? 2 : r <= 5 ? 1 : 0;
}

// Exact counts of the 16 windows of a 4x4 group (block `blk`, strip st, whose box starts at ring row
// row0) of one combo, by the whole warp: lane l < 20 collects the 20 rows of window column l as a bit
// column (box row r at bit 19 - r). First the 332 cells of the group's windows are counted: most
// groups whose box reaches the threshold end here. Then each lane's share of a window is one popcount.
template <int kMode>
__device__ __forceinline__ void count_group(PlaneSmem& S, const BandArgs& a, const Tile& T, int row0, int word, int bit,
                                            int blk, int st, int lane) {
    uint32_t v = 0;
    const int col = 4 * blk - 8 + min(lane, 19), up = 31 - bit;
#pragma unroll
    for (int r = 0; r < 20; ++r) {
        const int row = row0 + r < kRingRows ? row0 + r : row0 + r - kRingRows;
        v = __funnelshift_l(*ring_at<kMode>(S, row, word, col) << up, v, 1);
    }
    const int out = corner_cells(min(lane, 19 - min(lane, 19)));  // rows off the union at either end
    const uint32_t in_union = lane < 20 ? (0xFFFFFu >> (2 * out)) << out : 0u;
    if ((int)__reduce_add_sync(kFull, (unsigned)__popc(v & in_union)) < a.min_size) return;
    int mine = 0;
#pragma unroll
    for (int dx = 0; dx < 4; ++dx) {
        const int k = abs(lane - dx - 8), h = column_half_height(k);
        const uint32_t mask = h < 0 ? 0u : ((1u << (2 * h + 1)) - 1u) << (8 - h);
#pragma unroll
        for (int dz = 0; dz < 4; ++dz) {
            const int n = (int)__reduce_add_sync(kFull, (unsigned)__popc((v >> (3 - dz)) & mask));
            if (lane == 4 * dz + dx) mine = n;
        }
    }
    if (lane < 16 && mine >= a.min_size && mine <= a.max_size)
        keep_centre<kMode>(S, a, T, word, bit, 4 * blk + (lane & 3), 4 * (st - 4) + (lane >> 2), mine);
}

// Bounded counter of one thread (block, word): the strip sums of the last 5 strips (7 planes each,
// newest first) and the rolling 20x20 box (9 planes).
struct Bounded {
    uint32_t strip[5][7], box[9];
};

// Flagged groups of a warp from which the corner test of all lanes together is cheaper than
// counting each group's union (about 300 against 90 instructions a group).
constexpr int kCornerTestFrom = 4;

// Counts strip st, the `part`-th of the batch, for block `blk` of word `word`: row0 is the ring row of
// box row 0 (strip st - 4). Called by whole warps.
template <int kMode>
__device__ __forceinline__ void count_strip(PlaneSmem& S, const BandArgs& a, const Tile& T, Bounded& B, int part,
                                            int row0, int st, int word, int blk, int lane) {
    using Sh = Shape<kMode, false>;
    // Block sums of the five blocks blk - 2 .. blk + 2 (edge blocks read clamped neighbours and are
    // never flagged), added up to the 20-column strip sum.
    uint32_t s[7];
    {
        uint32_t b[5][5];
#pragma unroll
        for (int d = 0; d < 5; ++d) {
            const int n = min(max(blk + d - 2, 0), Sh::kBlocks - 1);
#pragma unroll
            for (int p = 0; p < 5; ++p) b[d][p] = S.sums[part][p][word * Sh::kBlocks + n];
        }
        uint32_t x[6], y[6], z[7];
        bs_add<5, 5, 6>(b[0], b[1], x);
        bs_add<5, 5, 6>(b[2], b[3], y);
        bs_add<6, 6, 7>(x, y, z);
        bs_add<7, 5, 7>(z, b[4], s);
    }
    // box += s - strip[4], as s + ~old + 1 over 9 planes.
    {
        uint32_t sv[9], cv[9];
#pragma unroll
        for (int i = 0; i < 9; ++i)
            bs_fa(B.box[i], i < 7 ? s[i] : 0u, i < 7 ? ~B.strip[4][i] : ~0u, sv[i], cv[i]);
        uint32_t c = ~0u;
#pragma unroll
        for (int i = 0; i < 9; ++i) bs_fa(sv[i], i ? cv[i - 1] : 0u, c, B.box[i], c);
    }
#pragma unroll
    for (int k = 4; k > 0; --k)
#pragma unroll
        for (int i = 0; i < 7; ++i) B.strip[k][i] = B.strip[k - 1][i];
#pragma unroll
    for (int i = 0; i < 7; ++i) B.strip[0][i] = s[i];

    if (st < 4) return;
    uint32_t flag = blk >= 2 && blk < Sh::kBlocks - 2 ? bs_at_least<9>(B.box, a.min_size) : 0u;
    if (!__any_sync(kFull, flag != 0)) return;
    if ((int)__reduce_add_sync(kFull, (unsigned)__popc(flag)) >= kCornerTestFrom && flag) {
        // The corners' cells taken off: what is left are the 332 cells of the group's 16 windows.
        BitSum sum;
        sum.clear();
        int k = 0;
        uint32_t odd = 0;
        bool have = false;
#pragma unroll
        for (int r = 0; r < 6; ++r)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int rr = q ? 19 - r : r, n = corner_cells(r);
                const int row = row0 + rr < kRingRows ? row0 + rr : row0 + rr - kRingRows;
                const uint32_t* left = ring_at<kMode>(S, row, word, 4 * blk - 8);
                const uint32_t* right = left + 16;
                uint32_t cell[12];
                if (n == 1) {
                    cell[0] = left[0];
                    cell[1] = right[3];
                } else {
                    const uint4 l = *reinterpret_cast<const uint4*>(left), g = *reinterpret_cast<const uint4*>(right);
                    cell[0] = l.x; cell[1] = g.w; cell[2] = l.y; cell[3] = g.z;
                    cell[4] = l.z; cell[5] = g.y; cell[6] = l.w; cell[7] = g.x;
                    if (n == 6) {
                        const uint2 l2 = *reinterpret_cast<const uint2*>(left + 4);
                        const uint2 g2 = *reinterpret_cast<const uint2*>(right - 2);
                        cell[8] = l2.x; cell[9] = l2.y; cell[10] = g2.x; cell[11] = g2.y;
                    }
                }
#pragma unroll
                for (int c = 0; c < 2 * n; ++c) {
                    if (have) sum.add(k++, odd, cell[c]);
                    odd = cell[c];
                    have = !have;
                }
            }
        sum.finish(34);
        // box >= corners + min_size
        uint32_t c = 0, ge = ~0u;
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            const uint32_t tb = 0u - (((uint32_t)a.min_size >> i) & 1u);
            uint32_t x;
            bs_fa(sum.p[i], tb, c, x, c);
            ge = (B.box[i] & ~x) | (ge & (B.box[i] | ~x));
        }
        flag &= ge;
    }
    for (unsigned todo = __ballot_sync(kFull, flag != 0); todo; todo &= todo - 1) {
        const int l = __ffs(todo) - 1;
        for (uint32_t f = __shfl_sync(kFull, flag, l); f; f &= f - 1)
            count_group<kMode>(S, a, T, row0, word, __ffs(f) - 1, blk - lane + l, st, lane);
    }
}

// Exact counter of one thread: the count planes of its four columns.
struct Exact {
    uint32_t cnt[4][8];
};

// Slides the windows of the thread's four columns down to row q of batch b (their last row; slot[j] is
// the first ring row of the batch j back) and keeps the centres in range. At |dx| columns from the centre, with half height h, the row 8 - h
// above the window's last row enters and the one 9 + h above it leaves.
template <int kMode, int q>
__device__ __forceinline__ void exact_row(PlaneSmem& S, const BandArgs& a, const Tile& T, Exact& E,
                                          const int (&slot)[4], int b, int word, int blk) {
    constexpr int kRows = Shape<kMode, true>::kBatchRows;
    static_assert((q - 17 + 3 * kRows) >= 0, "a slide reaches at most three batches back");
    auto at = [&](int back, int col) {  // word of the row `back` above the last one, column 4 blk + col
        const int d = q - back, j = d >= 0 ? 0 : (kRows - 1 - d) / kRows;
        return ring_at<kMode>(S, slot[j] + d + kRows * j, word, 4 * blk + col);
    };
    auto v4 = [&](int back, int col, uint32_t* o) {
        const uint4 v = *reinterpret_cast<const uint4*>(at(back, col));
        o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
    };
    auto v2 = [&](int back, int col, uint32_t* o) {
        const uint2 v = *reinterpret_cast<const uint2*>(at(back, col));
        o[0] = v.x; o[1] = v.y;
    };
    BitSum sum[4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < 8; ++i) sum[c].p[i] = E.cnt[c][i];
    {   // |dx| <= 2: columns -2 .. 5
        uint32_t in[8], out[8];
        v2(0, -2, in); v4(0, 0, in + 2); v2(0, 4, in + 6);
        v2(17, -2, out); v4(17, 0, out + 2); v2(17, 4, out + 6);
#pragma unroll
        for (int i = 0; i < 5; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) sum[c].add(i, in[c + i], ~out[c + i]);
    }
    {   // |dx| = 3, 4: columns -4 .. 0 and 3 .. 7
        uint32_t in[10], out[10];
        v4(1, -4, in); in[4] = *at(1, 0); in[5] = *at(1, 3); v4(1, 4, in + 6);
        v4(16, -4, out); out[4] = *at(16, 0); out[5] = *at(16, 3); v4(16, 4, out + 6);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            sum[c].add(5, in[c], ~out[c]);
            sum[c].add(6, in[c + 1], ~out[c + 1]);
            sum[c].add(7, in[c + 5], ~out[c + 5]);
            sum[c].add(8, in[c + 6], ~out[c + 6]);
        }
    }
    {   // |dx| = 5: columns -5 .. -2 and 5 .. 8
        uint32_t in[8], out[8], t[4];
        in[0] = *at(2, -5); v4(2, -4, t); in[1] = t[0]; in[2] = t[1]; in[3] = t[2];
        v4(2, 4, t); in[4] = t[1]; in[5] = t[2]; in[6] = t[3]; in[7] = *at(2, 8);
        out[0] = *at(15, -5); v4(15, -4, t); out[1] = t[0]; out[2] = t[1]; out[3] = t[2];
        v4(15, 4, t); out[4] = t[1]; out[5] = t[2]; out[6] = t[3]; out[7] = *at(15, 8);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            sum[c].add(9, in[c], ~out[c]);
            sum[c].add(10, in[c + 4], ~out[c + 4]);
        }
    }
    {   // |dx| = 6: columns -6 .. -3 and 6 .. 9
        uint32_t in[8], out[8];
        v2(3, -6, in); v2(3, -4, in + 2); v2(3, 6, in + 4); v2(3, 8, in + 6);
        v2(14, -6, out); v2(14, -4, out + 2); v2(14, 6, out + 4); v2(14, 8, out + 6);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            sum[c].add(11, in[c], ~out[c]);
            sum[c].add(12, in[c + 4], ~out[c + 4]);
        }
    }
    {   // |dx| = 7: columns -7 .. -4 and 7 .. 10
        uint32_t in[8], out[8], t[4];
        v4(4, -8, t); in[0] = t[1]; in[1] = t[2]; in[2] = t[3]; in[3] = *at(4, -4);
        in[4] = *at(4, 7); v4(4, 8, t); in[5] = t[0]; in[6] = t[1]; in[7] = t[2];
        v4(13, -8, t); out[0] = t[1]; out[1] = t[2]; out[2] = t[3]; out[3] = *at(13, -4);
        out[4] = *at(13, 7); v4(13, 8, t); out[5] = t[0]; out[6] = t[1]; out[7] = t[2];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            sum[c].add(13, in[c], ~out[c]);
            sum[c].add(14, in[c + 4], ~out[c + 4]);
        }
    }
    {   // |dx| = 8: columns -8 .. -5 and 8 .. 11
        uint32_t in[8], out[8];
        v4(6, -8, in); v4(6, 8, in + 4);
        v4(11, -8, out); v4(11, 8, out + 4);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            sum[c].add(15, in[c], ~out[c]);
            sum[c].add(16, in[c + 4], ~out[c + 4]);
        }
    }
    const int rr = kRows * b + q - 16;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        // 17 complements make the sum 17 too large: minus 17 is plus 239 = 0b11101111 (mod 256). A
        // one added to a plane with nothing else left leaves its complement and carries the plane.
        BitSum& s = sum[c];
        uint32_t t, k = s.p[0];
        s.p[0] = ~k;
        bs_fa(s.p[1], s.wait[1], k, s.p[1], t);
        k = s.p[1]; s.p[1] = ~k;
        bs_fa(s.p[2], t, k, s.p[2], t);
        k = s.p[2]; s.p[2] = ~k;
        bs_fa(s.p[3], t, k, s.p[3], t);
        k = s.p[3]; s.p[3] = ~k;
        bs_fa(s.p[4], t, k, s.p[4], t);
        bs_fa(s.p[5], s.wait[5], t, s.p[5], t);
        k = s.p[5]; s.p[5] = ~k;
        bs_fa(s.p[6], t, k, s.p[6], t);
        k = s.p[6]; s.p[6] = ~k;
        s.p[7] = ~(s.p[7] ^ t ^ k);
#pragma unroll
        for (int i = 0; i < 8; ++i) E.cnt[c][i] = s.p[i];
    }
    if (rr < 0) return;
    uint32_t pass[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) pass[c] = bs_at_least<8>(E.cnt[c], a.min_size);
    if (a.max_size < 221) {
#pragma unroll
        for (int c = 0; c < 4; ++c) pass[c] &= ~bs_at_least<8>(E.cnt[c], a.max_size + 1);
    }
    if (pass[0] | pass[1] | pass[2] | pass[3]) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
            for (uint32_t p = pass[c]; p; p &= p - 1) {
                const int bit = __ffs(p) - 1;
                keep_centre<kMode>(S, a, T, word, bit, 4 * blk + c, rr, bs_value(E.cnt[c], bit));
            }
    }
}

// ---- one tile ----------------------------------------------------------------------------------

// CTA set-up shared by the kernels: mbarriers and an empty histogram.
__device__ __forceinline__ void cta_init(PlaneSmem& S, int tid) {
    if (tid == 0) {
        S.failed = 0;
        for (int r = 0; r < 2; ++r)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&S.rows_bar[r])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < kHistBins; i += kTpb) S.hist[i] = 0;
    __syncthreads();
}

// One tile of one search (block-uniform arguments; all threads). Returns false when a bounded
// wait gave up (the search's overflow word gets bit 4 and the CTA must stop).
template <int kMode, bool kExact>
__device__ __forceinline__ bool plane_tile(PlaneSmem& S, const BandArgs& a, int64_t tile, int tid, uint32_t& bar_phase) {
    using Sh = Shape<kMode, kExact>;
    constexpr int kBatchRows = Sh::kBatchRows;
    const int lane = tid & 31;
    Tile T;
    const int ut = (int)(tile % a.u_tiles);
    const int64_t rest = tile / a.u_tiles;
    const int vt = (int)(rest % a.v_tiles);
    T.i0 = kMode == kModeIndep ? 0 : 2 * (int)(rest / a.v_tiles);
    T.u0 = ut * Sh::kOutW;
    T.v0 = vt * a.band_h;
    // Tiles with no centre of the area in any of their combos are skipped (block-uniform).
    if ((int64_t)T.u0 + (int64_t)T.i0 * kPeriod >= a.width_u || (int64_t)T.v0 + (int64_t)a.j0 * a.row_stride >= a.height_v)
        return true;
    T.out_h = min(a.band_h, a.vbase - T.v0);
    // Bands (grouped: copies) whose first row of this tile is still a centre row of the area.
    {
        const int64_t left = a.height_v - T.v0;
        const int64_t step = kMode == kModeGrouped ? kPeriod : a.row_stride;
        const int most = kMode == kModeGrouped ? a.nb / a.groups : a.nb;
        const int64_t held = (left + step - 1) / step - (kMode == kModeGrouped ? 0 : a.j0);
        T.bands = (int)min((int64_t)most, held);
        T.copies = most;
        T.mask = T.bands >= 32 ? ~0u : (1u << T.bands) - 1u;
        if (kMode == kModeGrouped)
            for (int g = 1; g < a.groups; ++g) T.mask |= (T.mask & ((1u << most) - 1u)) << (g * most);
    }
    const int batches = (T.out_h + 16 + kBatchRows - 1) / kBatchRows;
    constexpr int kRW = row_words<kMode>();
    constexpr uint32_t kBatchBytes = kBatchRows * kRW * 4;

    const int blk = tid % Sh::kBlocks, word = tid / Sh::kBlocks;  // word: also the generator's row part
    Columns C;
    C.absent = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int64_t idx0 = (int64_t)T.u0 + 4 * blk + k + (int64_t)T.i0 * kPeriod;
        const uint64_t x0 = idx0 < a.ncols ? a.ct[idx0] : 0;
        C.absent |= (idx0 < a.ncols ? 0u : 1u) << k;
        if (kMode == kModeIndep) {
            C.lo[k] = indep_lo(x0);
            C.h0[k] = indep_hi(x0);
            C.h1[k] = 0;
        } else {
            const uint64_t x1 = idx0 + kPeriod < a.ncols ? a.ct[idx0 + kPeriod] : 0;
            C.absent |= (idx0 + kPeriod < a.ncols ? 0u : 1u) << (4 + k);
            C.lo[k] = low_bits(x0);
            C.h0[k] = (uint32_t)(x0 >> kPeriodBits);
            C.h1[k] = (uint32_t)(x1 >> kPeriodBits);
        }
    }
    // Shared LCG: the word of a phase without centre columns in this tile is not counted.
    const bool counts = kMode != kModeShared || (int64_t)T.u0 + (int64_t)(T.i0 + word) * kPeriod < a.width_u;
    Bounded B;
    Exact E;
    if constexpr (kExact) {
        // The windows slide in from an empty ring.
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 8; ++i) E.cnt[c][i] = 0;
        for (int i = tid; i < kRingWords / 4; i += kTpb) reinterpret_cast<uint4*>(S.ring)[i] = make_uint4(0u, 0u, 0u, 0u);
    } else {
#pragma unroll
        for (int k = 0; k < 5; ++k)
#pragma unroll
            for (int i = 0; i < 7; ++i) B.strip[k][i] = 0;
#pragma unroll
        for (int i = 0; i < 9; ++i) B.box[i] = 0;
    }
    // Row terms of batches 0 and 1 (batch b lives in rows[b % 2]).
    if (tid == 0) {
        bulk_load(&S.rows[0][0], a.rt + (int64_t)T.v0 * kRW, kBatchBytes, &S.rows_bar[0]);
        if (batches > 1)
            bulk_load(&S.rows[1][0], a.rt + (int64_t)(T.v0 + kBatchRows) * kRW, kBatchBytes, &S.rows_bar[1]);
    }
    __syncthreads();

    int rb = 0, rs = 0;  // row-term buffer of b, ring row of its first row
    for (int b = 0; b < batches; ++b) {
        // ---- generator: batch b into its ring slot -----------------------------------------------
        if (!bar_wait(&S.rows_bar[rb], (bar_phase >> rb) & 1u, a.poll_limit)) {
            S.failed = 1;
            if (lane == 0) atomicOr(a.overflow, 4u);
        }
        bar_phase ^= 1u << rb;
        // Thread (block, part): rows part * kRowsPerThread .. of the batch, in all words. In the bounded
        // modes these are whole strips, whose block sums the thread adds up as it goes.
        uint32_t sum[Sh::kNW][5];
#pragma unroll 1
        for (int r = 0; r < Sh::kRowsPerThread; ++r) {
            const int row = word * Sh::kRowsPerThread + r;
            uint32_t w[Sh::kNW][4];
            generate_row<kMode>(a, T, C, &S.rows[rb][row * kRW], w);
            if (!kExact && (r & 3) == 0) {
#pragma unroll
                for (int n = 0; n < Sh::kNW; ++n)
#pragma unroll
                    for (int p = 0; p < 5; ++p) sum[n][p] = 0;
            }
#pragma unroll
            for (int n = 0; n < Sh::kNW; ++n) {
                *reinterpret_cast<uint4*>(&S.ring[((rs + row) * Sh::kNW + n) * Sh::kTW + 4 * blk]) =
                    make_uint4(w[n][0], w[n][1], w[n][2], w[n][3]);
                if constexpr (!kExact) {
                    uint32_t t0, t1, f;
                    bs_fa(sum[n][0], w[n][0], w[n][1], sum[n][0], t0);
                    bs_fa(sum[n][0], w[n][2], w[n][3], sum[n][0], t1);
                    bs_fa(sum[n][1], t0, t1, sum[n][1], f);
                    const uint32_t e = sum[n][2] & f, x = sum[n][3] & e;
                    sum[n][2] ^= f;
                    sum[n][3] ^= e;
                    sum[n][4] ^= x;
                }
            }
            if (!kExact && (r & 3) == 3) {
#pragma unroll
                for (int n = 0; n < Sh::kNW; ++n)
#pragma unroll
                    for (int p = 0; p < 5; ++p) S.sums[row >> 2][p][n * Sh::kBlocks + blk] = sum[n][p];
            }
        }
        __syncthreads();
        if (S.failed) {  // block-uniform after the barrier
            // Before the CTA leaves, wait (bounded) for its row-term copies still in flight:
            // batch b's (the wait that gave up) and batch b + 1's.
            if (tid == 0) {
                constexpr uint32_t kDrainPolls = 1u << 22;
                bar_wait(&S.rows_bar[rb], ((bar_phase >> rb) & 1u) ^ 1u, kDrainPolls);
                if (b + 1 < batches) {
                    const int rn = rb ^ 1;
                    bar_wait(&S.rows_bar[rn], (bar_phase >> rn) & 1u, kDrainPolls);
                }
            }
            __syncthreads();
            return false;
        }
        // Row terms of batch b + 2 (its buffer was last read before this batch's barrier).
        if (tid == kTpb - 32 && b + 2 < batches)
            bulk_load(&S.rows[rb][0], a.rt + (int64_t)(T.v0 + kBatchRows * (b + 2)) * kRW, kBatchBytes, &S.rows_bar[rb]);

        // ---- counter -----------------------------------------------------------------------------
        if (counts) {
            if constexpr (kExact) {
                int slot[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    slot[j] = rs - j * kBatchRows;
                    if (slot[j] < 0) slot[j] += kRingRows;
                }
                if (blk >= 2 && blk < Sh::kBlocks - 2) {
                    exact_row<kMode, 0>(S, a, T, E, slot, b, word, blk);
                    exact_row<kMode, 1>(S, a, T, E, slot, b, word, blk);
                    exact_row<kMode, 2>(S, a, T, E, slot, b, word, blk);
                    exact_row<kMode, 3>(S, a, T, E, slot, b, word, blk);
                    exact_row<kMode, 4>(S, a, T, E, slot, b, word, blk);
                    exact_row<kMode, 5>(S, a, T, E, slot, b, word, blk);
                }
            } else {
#pragma unroll 1
                for (int t = 0; t < 2; ++t) {
                    int row0 = rs + 4 * t - 16;  // ring row of strip 2 b + t - 4
                    if (row0 < 0) row0 += kRingRows;
                    count_strip<kMode>(S, a, T, B, t, row0, 2 * b + t, word, blk, lane);
                }
            }
        }
        __syncthreads();  // the next batch reuses the sums, and ring rows read above
        rb ^= 1;
        rs = rs == kRingRows - kBatchRows ? 0 : rs + kBatchRows;
    }
    return true;
}

template <int kMode, bool kExact>
__global__ void __launch_bounds__(kTpb, kCtasPerSm) plane_scan_kernel(const BandArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PlaneSmem& S = *reinterpret_cast<PlaneSmem*>(smem_raw);
    const int tid = threadIdx.x;
    uint32_t bar_phase = 0;  // bit r: parity of the next completion of rows_bar[r]
    cta_init(S, tid);
    for (int64_t tile = a.tile_begin + blockIdx.x; tile < a.tile_end; tile += gridDim.x)
        if (!plane_tile<kMode, kExact>(S, a, tile, tid, bar_phase)) return;
    if (a.hist) {
        __syncthreads();
        for (int i = tid; i < kHistBins; i += kTpb)
            if (S.hist[i]) atomicAdd(&a.hist[i], S.hist[i]);
    }
}

// Many searches of one launch class (band mode, bounded or exact counts) in one persistent launch:
// each CTA takes the next tile of the launch from a device counter, finds its search in the tile
// prefix sums and copies that search's arguments into shared memory. Work item i covers tiles
// args[i].tile_begin .. + (prefix[i+1] - prefix[i]) of its search; prefix[0] need not be 0. One
// class per launch keeps the kernel as lean as the single-search one.
template <int kMode, bool kExact>
__global__ void __launch_bounds__(kTpb, kCtasPerSm) plane_batch_kernel(const BandArgs* args, const int64_t* prefix,
                                                                     int32_t nsearch, unsigned long long* head) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PlaneSmem& S = *reinterpret_cast<PlaneSmem*>(smem_raw);
    const int tid = threadIdx.x;
    uint32_t bar_phase = 0;
    cta_init(S, tid);
    const int64_t first = prefix[0], total = prefix[nsearch];
    for (;;) {
        if (tid == 0) {
            const long long t = first + (long long)atomicAdd(head, 1ull);
            int lo = 0, hi = nsearch - 1;  // last search whose first tile is <= t
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (prefix[mid] <= t) lo = mid; else hi = mid - 1;
            }
            S.next_tile = t;
            S.search = lo;
        }
        __syncthreads();
        const int64_t t = S.next_tile;
        if (t >= total) return;  // block-uniform
        const int s = S.search;
        constexpr int kArgWords = (int)(sizeof(BandArgs) / 4);
        for (int i = tid; i < kArgWords; i += kTpb)
            reinterpret_cast<uint32_t*>(&S.args)[i] = reinterpret_cast<const uint32_t*>(&args[s])[i];
        __syncthreads();
        if (!plane_tile<kMode, kExact>(S, S.args, S.args.tile_begin + t - prefix[s], tid, bar_phase)) {
            if (tid == 0) atomicOr(S.args.overflow, 4u);
            return;
        }
        // The tile's search keeps a count histogram: add this tile's counts to it (plane_tile ended
        // with a barrier) and clear them before the next tile, which may be another search's.
        if (S.args.hist) {
            for (int i = tid; i < kHistBins; i += kTpb)
                if (S.hist[i]) {
                    atomicAdd(&S.args.hist[i], S.hist[i]);
                    S.hist[i] = 0;
                }
        }
    }
}

// Row-term table, one record per (band group g, base row v), records of a group contiguous; band j =
// 32 g + m holds base row v at input row v + offset(j), where offset(j) = j * stride, or, with grouped
// bands, (j % P) * 2^17 + (j / P) * stride (P copies a group). Record words (0 where the row lies
// outside the area plus halo):
//   shared LCG   [m] high part (>> 17) of the row term in band m, [32] its low_bits, [33] bands
//   independent  [m] and [32 + m]: indep_hi and indep_lo of the row term in band m, [64] bands
//   grouped      [m] high part and [32 + m] low_bits of the row term in band m, [64] bands
// "bands" is the mask of the bands that hold the row. Rows v >= vrows (padding) are zero.
template <int kMode>
__global__ void row_terms_kernel(uint32_t* rt, int32_t vrows_alloc, int32_t vrows, int32_t nj,
                                 int32_t first, int64_t limit, int64_t stride, int64_t seed,
                                 int32_t use_x_term, int32_t copies) {
    constexpr int kRW = row_words<kMode>();
    const int32_t groups = (nj + kMaxBands - 1) / kMaxBands;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (int64_t)groups * vrows_alloc * kRW) return;
    const int32_t w = (int32_t)(e % kRW);
    const int64_t rec = e / kRW;
    const int32_t v = (int32_t)(rec % vrows_alloc), g = (int32_t)(rec / vrows_alloc);
    auto input_row = [&](int32_t j) -> int64_t {
        return v + (kMode == kModeGrouped ? (int64_t)(j % copies) * kPeriod + (int64_t)(j / copies) * stride
                                          : (int64_t)j * stride);
    };
    uint32_t out = 0;
    if (v < vrows) {
        if (w == row_valid<kMode>()) {
            for (int32_t m = 0; m < kMaxBands && g * kMaxBands + m < nj; ++m)
                if (input_row(g * kMaxBands + m) < limit) out |= 1u << m;
        } else if (w < kMaxBands || (kMode == kModeShared ? w == kRowLo : w < 2 * kMaxBands)) {
            const bool hi = w < kMaxBands;
            const int32_t j = kMode == kModeShared && !hi ? 0 : g * kMaxBands + (w & (kMaxBands - 1));
            const int64_t row = input_row(j);
            if (j < nj && row < limit) {
                const int32_t c = (int32_t)((int64_t)first + row);
                const uint64_t t = (use_x_term ? x_term(c) : z_term(c)) + (uint64_t)seed;
                if (kMode == kModeIndep) out = hi ? indep_hi(t) : indep_lo(t);
                else out = hi ? (uint32_t)(t >> kPeriodBits) : low_bits(t);
            }
        }
    }
    rt[e] = out;
}

template <int kMode, bool kExact>
cudaError_t prepare_one() {
    cudaError_t e = cudaFuncSetAttribute(plane_scan_kernel<kMode, kExact>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(PlaneSmem));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(plane_batch_kernel<kMode, kExact>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(PlaneSmem));
    return e;
}

}  // namespace

int plane_tile_out_w(int mode) {
    return mode == kBandShared ? Shape<kModeShared, true>::kOutW : Shape<kModeIndep, true>::kOutW;
}
int plane_ctas_per_sm() { return kCtasPerSm; }
int plane_row_words(int mode) { return mode == kBandShared ? kRowWordsS : kRowWordsI; }

cudaError_t plane_prepare() {
    cudaError_t e;
    if ((e = prepare_one<kModeShared, true>()) != cudaSuccess || (e = prepare_one<kModeIndep, true>()) != cudaSuccess ||
        (e = prepare_one<kModeGrouped, true>()) != cudaSuccess || (e = prepare_one<kModeIndep, false>()) != cudaSuccess)
        return e;
    return cudaSuccess;
}

cudaError_t launch_plane_batch(const BandArgs* args, const int64_t* prefix, int32_t nsearch, unsigned long long* head,
                               int mode, bool exact, int grid, cudaStream_t s) {
    constexpr size_t bytes = sizeof(PlaneSmem);
    if (mode == kBandIndep && !exact)
        plane_batch_kernel<kModeIndep, false><<<grid, kTpb, bytes, s>>>(args, prefix, nsearch, head);
    else if (mode == kBandIndep)
        plane_batch_kernel<kModeIndep, true><<<grid, kTpb, bytes, s>>>(args, prefix, nsearch, head);
    else if (mode == kBandGrouped)
        plane_batch_kernel<kModeGrouped, true><<<grid, kTpb, bytes, s>>>(args, prefix, nsearch, head);
    else
        plane_batch_kernel<kModeShared, true><<<grid, kTpb, bytes, s>>>(args, prefix, nsearch, head);
    return cudaGetLastError();
}

cudaError_t launch_plane_scan(const BandArgs& a, int grid, cudaStream_t s) {
    constexpr size_t bytes = sizeof(PlaneSmem);
    if (a.indep && !a.exact) plane_scan_kernel<kModeIndep, false><<<grid, kTpb, bytes, s>>>(a);
    else if (a.indep) plane_scan_kernel<kModeIndep, true><<<grid, kTpb, bytes, s>>>(a);
    else if (a.groups) plane_scan_kernel<kModeGrouped, true><<<grid, kTpb, bytes, s>>>(a);
    else plane_scan_kernel<kModeShared, true><<<grid, kTpb, bytes, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_plane_row_terms(uint32_t* rt, int32_t vrows_alloc, int32_t vrows, int32_t nj, int32_t row_first,
                                   int64_t row_limit, int64_t row_stride, int64_t seed, bool transposed, bool indep,
                                   int32_t groups, cudaStream_t s) {
    const int64_t ngroups = (nj + kMaxBands - 1) / kMaxBands;
    const int64_t n = ngroups * vrows_alloc * (indep || groups > 0 ? kRowWordsI : kRowWordsS);
    const unsigned blocks = (unsigned)((n + 255) / 256);
    const int32_t x = transposed ? 1 : 0;
    if (groups > 0)
        row_terms_kernel<kModeGrouped><<<blocks, 256, 0, s>>>(rt, vrows_alloc, vrows, nj, row_first, row_limit, row_stride,
                                                              seed, x, nj / groups);
    else if (indep)
        row_terms_kernel<kModeIndep><<<blocks, 256, 0, s>>>(rt, vrows_alloc, vrows, nj, row_first, row_limit, row_stride,
                                                            seed, x, 1);
    else
        row_terms_kernel<kModeShared><<<blocks, 256, 0, s>>>(rt, vrows_alloc, vrows, nj, row_first, row_limit, row_stride,
                                                             seed, x, 1);
    return cudaGetLastError();
}

}  // namespace slime
