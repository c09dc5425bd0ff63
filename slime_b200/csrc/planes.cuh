// planes.cuh -- band searches as bit planes: low and middle thresholds in all band modes, and every
// threshold of independent bands.
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
//  * A window slides down a row by adding its entering cells and the complement of its leaving cells
//    to bit-sliced counts. A thread counts the union of the windows of 1, 2 or 4 adjacent centres (221,
//    238 or 272 cells, 17, 18 or 20 of which enter and leave a row), the wider the higher the threshold:
//    one count then stands for 1, 2 or 4 columns. A union that reaches the threshold is looked at by
//    the whole warp, which counts its windows one by one.
// What bounds it (B200): integer issue. Independent bands, radius 100,000: the generator is about 18 ms
// (13.9 cycles a warp test in a probe of it alone); with the counter 25.5 ms at threshold 42, 23.3 at 44 and
// 20.8 at 60. Packing columns took 42.4 ms at threshold 42 and 29.3 at 60. Grouped bands, radius 300,000,
// threshold 44: 160 against 276 ms, threshold 50 (there bounded): 133 against 183 ms.
// Shared and grouped bands at high thresholds stay with columns in words (radius 1,250,000, threshold 60:
// 1,012 ms; radius 300,000: 106 against 130 ms): their five-instruction test gains too little here to
// pay for counting partly filled words.
#pragma once

#include <type_traits>

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

// Row-term record of one base row (written by row_terms_kernel): [m] and [32 + m] the two parts of
// the row term in band m, or with the shared LCG [32] the low part of all bands; then the mask of
// the bands that hold the row. The rows of a batch are one contiguous bulk copy.
constexpr int kRowWordsS = 36, kRowWordsI = 72;
constexpr int kRowLo = 32;
template <int kMode>
constexpr int row_words() { return kMode == kModeShared ? kRowWordsS : kRowWordsI; }
template <int kMode>
constexpr int row_valid() { return kMode == kModeShared ? 33 : 64; }

// Independent bands split a term at bit 18. The low parts sit at bits 2..19 (where a double's high word
// wants them); a row's carries the bits above, so that the sum's carry leaves the word.
constexpr int kIndepBits = 18;
__host__ __device__ __forceinline__ uint32_t indep_lo(uint64_t t) { return ((uint32_t)t & 0x3FFFFu) << 2; }
__host__ __device__ __forceinline__ uint32_t indep_row_lo(uint64_t t) { return indep_lo(t) + 0xFFF00000u; }
__host__ __device__ __forceinline__ uint32_t indep_hi(uint64_t t) { return (uint32_t)(t >> kIndepBits); }

// Tile shape of a mode: kNW words a column (one a phase with the shared LCG), kTW input columns.
// kNW * kTW = 1,024 words a row in every mode, so that ring and thread layout agree. Rows advance in
// batches of 6 with a barrier after generating and one after counting; a slide looks back 17 rows
// from the first row of the batch (23 rows with it).
constexpr int kBatchRows = 6;
template <int kMode>
struct Shape {
    static constexpr int kNW = kMode == kModeShared ? 2 : 1;
    static constexpr int kTW = 1024 / kNW;
    static constexpr int kBlocks = kTW / 4;      // 4-column blocks: thread = (block, word)
    static constexpr int kOutW = kTW - 16;
    static constexpr int kRowsPerThread = kBatchRows / kNW;  // generator: thread = (block, row part)
};

constexpr int kListCap = 1024;  // what does not fit is counted at once

struct __align__(16) PlaneSmem {
    uint32_t ring[kRingWords];                // [row % 24][word][column]
    uint32_t rows[2][kBatchRows * kRowWordsI];  // row terms of 2 batches, filled by bulk copies
    unsigned long long rows_bar[2];           // mbarriers of the two row-term buffers
    BandArgs args;                            // batched kernel: the current tile's search
    long long next_tile;                      // batched kernel: tile taken from the queue
    int search;                               // batched kernel: its search
    int failed;  // a bounded wait gave up: the CTA stops
    uint32_t list[kListCap];                  // unions waiting for their windows' counts
    unsigned int listed;
    unsigned int hist[kHistBins];             // counts of this CTA's centres in range (if args.hist)
    // Grouped bands, of the current tile's search, by band: first area row (before the tile's base row), and
    // the base row from which its rows belong to the next copy's first group.
    int32_t row0[kGrpBands], row_end[kGrpBands];
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
    int groups, min_size, max_size;
};

// ---- bit-sliced adders: bit j of every word belongs to combo j ----------------------------------

__device__ __forceinline__ void bs_fa(uint32_t a, uint32_t b, uint32_t c, uint32_t& s, uint32_t& cy) {
    const uint32_t x = a, y = b, z = c;
    s = x ^ y ^ z;
    cy = (x & y) | (z & (x | y));
}

// Carry-save accumulator: planes p[0..], and per weight at most one waiting carry. add(k, a, b) is
// the k-th pair of single-bit inputs (k a compile-time constant after unrolling).
constexpr int kPlanes = 9;  // unions of four windows hold 272 cells
struct BitSum {
    uint32_t p[kPlanes], wait[kPlanes];
    __device__ __forceinline__ void add(int k, uint32_t a, uint32_t b) {
        uint32_t c;
        bs_fa(p[0], a, b, p[0], c);
#pragma unroll
        for (int w = 1; w < kPlanes; ++w, k >>= 1) {
            if (!(k & 1)) {
                wait[w] = c;
                return;
            }
            bs_fa(p[w], wait[w], c, p[w], c);
        }
    }
    // Adds what waits after N pairs and takes N off (a pair of an entering cell and the complement of a
    // leaving one counts one too many), as 2^P - N over P planes. A constant one added to a plane with
    // nothing else left leaves its complement and carries the plane.
    template <int N, int P>
    __device__ __forceinline__ void finish() {
        constexpr uint32_t kMinus = (1u << P) - (uint32_t)N;
        uint32_t carry[3];
        int n = 0;  // carries into plane w (compile-time after unrolling)
#pragma unroll
        for (int w = 0; w < P; ++w) {
            uint32_t item[4], next[3];
            int m = 0, out = 0;
#pragma unroll
            for (int i = 0; i < n; ++i) item[m++] = carry[i];
            if (w > 0 && ((N >> (w - 1)) & 1)) item[m++] = wait[w];
            if (m >= 2) {
                bs_fa(p[w], item[m - 1], item[m - 2], p[w], next[out++]);
                m -= 2;
            }
            const uint32_t x = p[w];
            if (m == 1 && ((kMinus >> w) & 1u)) {
                p[w] = ~(x ^ item[0]);
                next[out++] = x | item[0];
            } else if (m == 1) {
                p[w] = x ^ item[0];
                next[out++] = x & item[0];
            } else if ((kMinus >> w) & 1u) {
                p[w] = ~x;
                next[out++] = x;
            }
#pragma unroll
            for (int i = 0; i < out; ++i) carry[i] = next[i];
            n = out;
        }
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

// First-draw test of one chunk from split terms (independent bands: nothing is shared). With state0 =
// H * 2^18 + l, bits = v + H * 2 A (mod 2^31) with v = (l * A + 11) >> 17, a 53-bit product that one FP64
// multiply-add gives exactly: d = 2^18 + l + 2^-31 stands in the words of a double, d * A / 2^17 plus
// (3 * 2^51 - 2 A) is 3 * 2^51 + (l * A + 11.74) / 2^17, and rounding to zero leaves v in the low word (the
// .74 never reaches the next integer). y = 2 bits inv5 is below kHitBelow and a multiple of 4 iff the
// draw is an even multiple of 10 below the bound; rotated by 2 that is one comparison. The integer form
// (a 32 x 32 -> 64 multiply) ran 15.8 cycles a warp test, this one 13.9.
__device__ __forceinline__ void shift_indep(uint32_t& w, uint32_t xl, uint32_t xh, uint32_t zl, uint32_t zh) {
    constexpr double kA = 25214903917.0;  // 0x5DEECE66D
    static_assert(0x5DEECE66DLL == 25214903917LL, "LCG multiplier");
    uint32_t lo, hi;
    asm("{ add.cc.u32 %0, %2, %3;\n addc.u32 %1, %4, %5; }" : "=r"(lo), "=r"(hi) : "r"(xl), "r"(zl), "r"(xh), "r"(zh));
    const uint32_t high = (lo & 0xFFFFCu) ^ (0x41100000u ^ indep_lo(band::kSeedXor));  // 2^18 + l
    const double v = __fma_rz(__hiloint2double((int)high, 8), kA / 131072.0, 6755399441055744.0 - 2.0 * kA);
    hi ^= indep_hi(band::kSeedXor);
    const uint32_t y = (uint32_t)__double2loint(v) * kTwoInv5 + hi * (2u * kTwoInv5 * kA32);
    shift_miss(w, __funnelshift_r(y, y, 2), kHitBelow / 4u);
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
        const int G = T.groups, copies = T.copies;
        const uint32_t even_copies = 0x5555u & ((1u << copies) - 1u), odd_copies = 0xAAAAu & ((1u << copies) - 1u);
        // Shifts by a group's copies as multiplies: the integer ALU is the busy pipe.
        const uint32_t step = 1u << copies, skip = 1u << (copies - bands);
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
                first[k] = first[k] * step + (odd ? odd_copies : even_copies);
                miss[k] *= skip;  // copies without a centre in the tile: not valid
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
    if (m >= a.nb || c < 0 || c >= Shape<kMode>::kOutW || rr < 0 || rr >= T.out_h) return;
    const int64_t u = (int64_t)T.u0 + c;
    const int64_t cu = u + (int64_t)(T.i0 + ph) * kPeriod;
    const int64_t cv = (int64_t)T.v0 + rr + (kMode == kModeGrouped ? (int64_t)S.row0[m] : (a.j0 + m) * a.row_stride);
    if (kMode == kModeGrouped && T.v0 + rr >= S.row_end[m]) return;
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
    using Sh = Shape<kMode>;
    return &S.ring[(row * Sh::kNW + word) * Sh::kTW + col];
}

// Windows of `kUnion` adjacent centres, counted as one: a thread's four columns are 4 / kUnion unions.
// Half height of the union's column c, its first centre in column 0.
template <int kUnion>
__host__ __device__ constexpr int union_half_height(int c) {
    return column_half_height(c < 0 ? -c : c >= kUnion ? c - kUnion + 1 : 0);
}
// Whether any union of the thread's four columns needs column c (-8 .. 11) at half height H.
template <int kUnion>
__host__ __device__ constexpr bool needs_column(int c, int H) {
    for (int s = 0; s < 4; s += kUnion)
        if (union_half_height<kUnion>(c - s) == H) return true;
    return false;
}

// Counter of one thread: the count planes of its unions.
template <int kUnion>
struct Counter {
    static constexpr int kUnions = 4 / kUnion;
    static constexpr int kCells = 16 + kUnion;               // entering (and leaving) cells of a slide
    static constexpr int kP = kUnion == 4 ? 9 : 8;           // planes of a count
    uint32_t cnt[kUnions][kP];
};

// A union that reached the threshold: its combo bit, its first centre's column, its last window row (row
// `last` of the batch) and its word: 5 + 10 + 3 + 1 bits.
__device__ __forceinline__ uint32_t pack_union(int bit, int column, int last, int word) {
    return (uint32_t)bit | (uint32_t)column << 5 | (uint32_t)last << 15 | (uint32_t)word << 18;
}

// Exact counts of the windows of one union, by the whole warp: lane l collects the 17 rows of the
// union's column l - 8 as a bit column, whose share of each window is one popcount; the windows' counts
// (at most 221) add up in the bytes of one word. rs is the ring row of the batch's first row, row0 its
// tile row. Not inlined: it runs rarely, and its code would push the hot loops out of the instruction cache.
template <int kMode, int kUnion>
__device__ __noinline__ void count_union(const BandArgs& a, const Tile& T, uint32_t e, int rs, int row0) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PlaneSmem& S = *reinterpret_cast<PlaneSmem*>(smem_raw);
    const int lane = threadIdx.x & 31, l = min(lane, 15 + kUnion);
    const int up = 31 - (int)(e & 31), col = (int)(e >> 5 & 1023), last = (int)(e >> 15 & 7), word = (int)(e >> 18);
    uint32_t v = 0;
#pragma unroll
    for (int r = 0; r < 17; ++r) {
        const int row = rs + last - 16 + r;
        v = __funnelshift_l(*ring_at<kMode>(S, row < 0 ? row + kRingRows : row, word, col - 8 + l) << up, v, 1);
    }
    uint32_t sum = 0;
#pragma unroll
    for (int dx = 0; dx < kUnion; ++dx) {
        const int h = column_half_height(abs(l - dx - 8));
        const uint32_t mask = h < 0 || lane != l ? 0u : ((1u << (2 * h + 1)) - 1u) << (8 - h);
        sum |= (uint32_t)__popc(v & mask) << (8 * dx);
    }
    sum = __reduce_add_sync(kFull, sum);
    const int mine = (int)(sum >> (8 * (lane & 3)) & 255);
    if (lane < kUnion && mine >= T.min_size && mine <= T.max_size)
        keep_centre<kMode>(S, a, T, word, (int)(e & 31), col + lane, row0 + last - 16, mine);
    __syncwarp();
}

// A batch is counted in parts of kPartRows rows, whose code is laid out once.
constexpr int kPartRows = 3, kParts = kBatchRows / kPartRows;
constexpr int kPartsBack = (17 + kPartRows - 1) / kPartRows + 1;  // parts that a part's slides reach, itself included

// Slides the unions of the thread's four columns (block blk) down to row q of a part (their last row;
// slot[j] is the first ring row of the part j back): the row 8 - H above the last one enters and the one
// 9 + H above it leaves, H the half height of the column.
template <int kMode, int kUnion, int q>
__device__ __forceinline__ void slide(const PlaneSmem& S, Counter<kUnion>& E, const int (&slot)[kPartsBack], int word,
                                      int blk) {
    using C = Counter<kUnion>;
    auto at = [&](int back, int col) {  // word of the row `back` above the last one, column 4 blk + col
        const int d = q - back, j = d >= 0 ? 0 : (kPartRows - 1 - d) / kPartRows;
        return ring_at<kMode>(S, slot[j] + d + kPartRows * j, word, 4 * blk + col);
    };
    // The needed words of one row, columns -8 .. 11, in the widest loads that hold two or more of them.
    auto load = [&](int back, int H, uint32_t (&o)[20]) {
#pragma unroll
        for (int c = -8; c < 12; c += 4) {
            bool n[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) n[i] = needs_column<kUnion>(c + i, H);
            if ((n[0] || n[1]) && (n[2] || n[3]) && n[0] + n[1] + n[2] + n[3] >= 3) {
                const uint4 v = *reinterpret_cast<const uint4*>(at(back, c));
                o[c + 8] = v.x; o[c + 9] = v.y; o[c + 10] = v.z; o[c + 11] = v.w;
                continue;
            }
#pragma unroll
            for (int i = 0; i < 4; i += 2) {
                if (n[i] && n[i + 1]) {
                    const uint2 v = *reinterpret_cast<const uint2*>(at(back, c + i));
                    o[c + i + 8] = v.x; o[c + i + 9] = v.y;
                } else if (n[i]) {
                    o[c + i + 8] = *at(back, c + i);
                } else if (n[i + 1]) {
                    o[c + i + 9] = *at(back, c + i + 1);
                }
            }
        }
    };
    BitSum sum[C::kUnions];
#pragma unroll
    for (int u = 0; u < C::kUnions; ++u)
#pragma unroll
        for (int i = 0; i < C::kP; ++i) sum[u].p[i] = E.cnt[u][i];
    int k[C::kUnions] = {};
#pragma unroll
    for (int H = 8; H >= 2; --H) {
        if (H == 3) continue;  // no column of the window has half height 3
        uint32_t in[20], out[20];
        load(8 - H, H, in);
        load(9 + H, H, out);
#pragma unroll
        for (int c = -8; c < 12; ++c)
#pragma unroll
            for (int u = 0; u < C::kUnions; ++u)
                if (union_half_height<kUnion>(c - u * kUnion) == H) sum[u].add(k[u]++, in[c + 8], ~out[c + 8]);
    }
#pragma unroll
    for (int u = 0; u < C::kUnions; ++u) {
        sum[u].template finish<C::kCells, C::kP>();
#pragma unroll
        for (int i = 0; i < C::kP; ++i) E.cnt[u][i] = sum[u].p[i];
    }
}

// Counts part `part` of a batch (rs: ring row of the batch's first row, row0: its tile row); called by
// whole warps. Edge blocks (whose windows leave the tile) repeat an inner block's work and keep nothing.
// Unions that reach the threshold go to the list.
template <int kMode, int kUnion>
__device__ __forceinline__ void count_part(PlaneSmem& S, const BandArgs& a, const Tile& T, Counter<kUnion>& E, int rs,
                                           int row0, int part, int word, int blk, int lane) {
    using C = Counter<kUnion>;
    constexpr int kLastBlock = Shape<kMode>::kBlocks - 3;
    const bool inner = blk >= 2 && blk <= kLastBlock;
    const int at = min(max(blk, 2), kLastBlock);
    int slot[kPartsBack];
#pragma unroll
    for (int j = 0; j < kPartsBack; ++j) {
        slot[j] = rs + (part - j) * kPartRows;
        if (slot[j] < 0) slot[j] += kRingRows;
    }
    uint32_t flag[kPartRows][C::kUnions];
    uint32_t any = 0;
    auto row = [&](auto qc) {
        constexpr int q = decltype(qc)::value;
        slide<kMode, kUnion, q>(S, E, slot, word, at);
        const bool live = inner && row0 + part * kPartRows + q >= 16;  // the window's rows are complete
#pragma unroll
        for (int u = 0; u < C::kUnions; ++u) {
            uint32_t f = live ? bs_at_least<C::kP>(E.cnt[u], T.min_size) : 0u;
            if constexpr (kUnion == 1) {
                if (T.max_size < 221) f &= ~bs_at_least<C::kP>(E.cnt[u], T.max_size + 1);
                for (; f; f &= f - 1) {
                    const int bit = __ffs(f) - 1;
                    keep_centre<kMode>(S, a, T, word, bit, 4 * blk + u, row0 + part * kPartRows + q - 16, bs_value(E.cnt[u], bit));
                }
            } else {
                flag[q][u] = f;
                any |= f;
            }
        }
    };
    row(std::integral_constant<int, 0>{});
    row(std::integral_constant<int, 1>{});
    row(std::integral_constant<int, 2>{});
    if constexpr (kUnion > 1) {
        if (any) {
            any = 0;
#pragma unroll
            for (int q = 0; q < kPartRows; ++q)
#pragma unroll
                for (int u = 0; u < C::kUnions; ++u) {
                    for (; flag[q][u]; flag[q][u] &= flag[q][u] - 1) {
                        const unsigned n = atomicAdd(&S.listed, 1u);
                        if (n >= (unsigned)kListCap) break;
                        S.list[n] = pack_union(__ffs(flag[q][u]) - 1, 4 * blk + u * kUnion, part * kPartRows + q, word);
                    }
                    any |= flag[q][u];
                }
        }
        if (__any_sync(kFull, any != 0)) {  // the list is full: the warp counts what is left
#pragma unroll
            for (int q = 0; q < kPartRows; ++q)
#pragma unroll
                for (int u = 0; u < C::kUnions; ++u)
                    for (unsigned todo = __ballot_sync(kFull, flag[q][u] != 0); todo; todo &= todo - 1) {
                        const int l = __ffs(todo) - 1;
                        for (uint32_t f = __shfl_sync(kFull, flag[q][u], l); f; f &= f - 1)
                            count_union<kMode, kUnion>(a, T, pack_union(__ffs(f) - 1, 4 * (blk - lane + l) + u * kUnion,
                                                                        part * kPartRows + q, word), rs, row0);
                    }
        }
    }
}

// ---- one tile ----------------------------------------------------------------------------------

// CTA set-up shared by the kernels: mbarriers and an empty histogram.
__device__ __forceinline__ void cta_init(PlaneSmem& S, int tid) {
    if (tid == 0) {
        S.failed = 0;
        S.listed = 0;
        for (int r = 0; r < 2; ++r)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&S.rows_bar[r])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < kHistBins; i += kTpb) S.hist[i] = 0;
    __syncthreads();
}

// One tile of one search (block-uniform arguments; all threads). Returns false when a bounded
// wait gave up (the search's overflow word gets bit 4 and the CTA must stop).
template <int kMode, int kUnion>
__device__ __forceinline__ bool plane_tile(PlaneSmem& S, const BandArgs& a, int64_t tile, int tid, uint32_t& bar_phase) {
    using Sh = Shape<kMode>;
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
    // The broadcasts tell the compiler that these are warp-uniform: loop bounds, and the threshold whose
    // bits the comparisons take as masks.
    auto uniform = [](int v) { return __shfl_sync(kFull, v, 0); };
    T.bands = uniform(T.bands);
    T.copies = uniform(T.copies);
    T.mask = (uint32_t)uniform((int)T.mask);
    T.groups = uniform(a.groups);
    T.min_size = uniform(a.min_size);
    T.max_size = uniform(a.max_size);
    const int batches = uniform((T.out_h + 16 + kBatchRows - 1) / kBatchRows);
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
    // The windows slide in from an empty ring.
    Counter<kUnion> E;
#pragma unroll
    for (int u = 0; u < Counter<kUnion>::kUnions; ++u)
#pragma unroll
        for (int i = 0; i < Counter<kUnion>::kP; ++i) E.cnt[u][i] = 0;
    for (int i = tid; i < kRingWords / 4; i += kTpb) reinterpret_cast<uint4*>(S.ring)[i] = make_uint4(0u, 0u, 0u, 0u);
    // Worked out a kept centre at a time, the bands' rows cost five divisions each: grouped bands at thresholds
    // below 40 took up to twice as long (radius 180,000, threshold 37: 252 ms).
    if (kMode == kModeGrouped && tid < kGrpBands) {
        const int copy = tid % T.copies, group = tid / T.copies;
        S.row0[tid] = copy * (int32_t)kPeriod + group * (int32_t)a.row_stride;
        S.row_end[tid] = T.copies > 1 ? max(0, (int32_t)kPeriod - group * (int32_t)a.row_stride) : INT32_MAX;
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
        // Thread (block, part): rows part * kRowsPerThread .. of the batch, in all words.
#pragma unroll 1
        for (int r = 0; r < Sh::kRowsPerThread; ++r) {
            const int row = word * Sh::kRowsPerThread + r;
            uint32_t w[Sh::kNW][4];
            generate_row<kMode>(a, T, C, &S.rows[rb][row * kRW], w);
#pragma unroll
            for (int n = 0; n < Sh::kNW; ++n)
                *reinterpret_cast<uint4*>(&S.ring[((rs + row) * Sh::kNW + n) * Sh::kTW + 4 * blk]) =
                    make_uint4(w[n][0], w[n][1], w[n][2], w[n][3]);
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
        if (counts)
#pragma unroll 1
            for (int i = 0; i < kParts; ++i)
                count_part<kMode, kUnion>(S, a, T, E, rs, b * kBatchRows, i, word, blk, lane);
        if constexpr (kUnion > 1) {
            // The listed unions, shared out over the warps: left to the warp that found them, the others
            // waited at the barrier for the one with the most.
            __syncthreads();
            const int listed = min((int)S.listed, kListCap);
            for (int i = tid >> 5; i < listed; i += kTpb / 32)
                count_union<kMode, kUnion>(a, T, S.list[i], rs, b * kBatchRows);
        }
        __syncthreads();  // the next batch reuses ring rows read above
        if (kUnion > 1 && tid == 0) S.listed = 0;  // before the next batch's first barrier
        rb ^= 1;
        rs = rs == kRingRows - kBatchRows ? 0 : rs + kBatchRows;
    }
    return true;
}

// Tiles of one search (`args` null: tiles one.tile_begin + blockIdx.x, + gridDim.x, ... of `one`), or of
// many searches in one persistent launch: each CTA takes the next tile of the launch from a device counter,
// finds its search in the tile prefix sums and copies that search's arguments into shared memory. Work
// item i covers tiles args[i].tile_begin .. + (prefix[i+1] - prefix[i]) of its search; prefix[0] need
// not be 0. One kernel for both halves the build.
template <int kMode, int kUnion>
__global__ void __launch_bounds__(kTpb, kCtasPerSm) plane_kernel(const BandArgs one, const BandArgs* args,
                                                                 const int64_t* prefix, int32_t nsearch,
                                                                 unsigned long long* head) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PlaneSmem& S = *reinterpret_cast<PlaneSmem*>(smem_raw);
    const int tid = threadIdx.x;
    uint32_t bar_phase = 0;  // bit r: parity of the next completion of rows_bar[r]
    cta_init(S, tid);
    const int64_t first = args ? prefix[0] : one.tile_begin, total = args ? prefix[nsearch] : one.tile_end;
    if (!args && tid == 0) S.args = one;
    int64_t next = first + blockIdx.x;
    for (;;) {
        int64_t tile = next;
        if (args) {
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
            tile = t - prefix[s];
        } else if (tile >= total) {
            break;
        }
        __syncthreads();
        if (args) tile += S.args.tile_begin;
        if (!plane_tile<kMode, kUnion>(S, S.args, tile, tid, bar_phase)) {
            if (tid == 0) atomicOr(S.args.overflow, 4u);
            return;
        }
        next += gridDim.x;
        // Many searches: the tile's counts go to its search (plane_tile ended with a barrier) and are
        // cleared before the next tile, which may be another search's.
        if (args && S.args.hist) {
            for (int i = tid; i < kHistBins; i += kTpb)
                if (S.hist[i]) {
                    atomicAdd(&S.args.hist[i], S.hist[i]);
                    S.hist[i] = 0;
                }
        }
    }
    if (one.hist) {
        __syncthreads();
        for (int i = tid; i < kHistBins; i += kTpb)
            if (S.hist[i]) atomicAdd(&one.hist[i], S.hist[i]);
    }
}

template <int kMode, int kUnion>
cudaError_t run_union(const BandArgs& one, const BandArgs* args, const int64_t* prefix, int32_t nsearch,
                      unsigned long long* head, int grid, cudaStream_t s) {
    if (grid == 0)
        return cudaFuncSetAttribute(plane_kernel<kMode, kUnion>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sizeof(PlaneSmem));
    plane_kernel<kMode, kUnion><<<grid, kTpb, sizeof(PlaneSmem), s>>>(one, args, prefix, nsearch, head);
    return cudaGetLastError();
}

// The kernel of a mode and number of windows counted as one over `grid` CTAs; with grid == 0 it is only
// given its shared-memory size. Each mode is built in a file of its own (planes_*.cu).
template <int kMode>
cudaError_t run_mode(int joined, const BandArgs& one, const BandArgs* args, const int64_t* prefix, int32_t nsearch,
                     unsigned long long* head, int grid, cudaStream_t s) {
    return joined == 1   ? run_union<kMode, 1>(one, args, prefix, nsearch, head, grid, s)
           : joined == 2 ? run_union<kMode, 2>(one, args, prefix, nsearch, head, grid, s)
                         : run_union<kMode, 4>(one, args, prefix, nsearch, head, grid, s);
}

}  // namespace
}  // namespace slime
