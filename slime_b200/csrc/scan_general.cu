// scan_general.cu -- the general scan: any area, any threshold, exact predicate.
//
// Behaviour follows the reference GPU search (SlimeCoreGPU.cu:501-610, 3164-3851): every centre of
// the area whose exact 221-cell count lies in [min_size, max_size] (outside the rd_min disc) is kept.
//
// B200 design: a CTA owns a patch of 256 x (h + 16) chunks, the centres of 240 x h of them. Its warps
// first evaluate the patch, a lane a column and a ballot a word, into shared memory: no rolling state,
// so no barrier a row. Then every thread counts one word of centre rows with bit-sliced adders (a full
// adder of two LOP3 adds 32 centres' bits): the first of its rows in full, the others by sliding down a
// row (17 cells enter, 17 leave). Term tables are not needed: a patch computes its own.
// The scan is latency-bound on small areas and issue-bound on large ones; it replaces a rolling-square
// scan that ran 80 barriers a tile. B200, kernel time: radius 100 63 -> 9 us, radius 2,000
// (threshold 40) 131 -> 35 us, radius 9,001 (threshold 44, annulus) 1,150 -> 440 us.
#include <cmath>

#include "engine.h"

namespace slime {
namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr int kTpb = 256;
constexpr int kWarps = kTpb / 32;
constexpr int kWords = 8;               // words of a patch row
constexpr int kOutW = kWords * 32 - 16;
constexpr int kStride = kWords + 1;     // and a zero word: counting reads the next word
constexpr int kMaxRows = 128;           // centre rows of a patch
constexpr int kListCap = 1024;          // hits a CTA collects; more go out one by one

// ---- bit-sliced counts: bit j of every word belongs to centre (or column) j ----------------------

__device__ __forceinline__ void bs_fa(uint32_t a, uint32_t b, uint32_t c, uint32_t& s, uint32_t& cy) {
    s = a ^ b ^ c;
    cy = (a & b) | (c & (a | b));
}

// out = a + b over NO planes (a: NA planes, b: NB <= NA planes; the caller knows the sum fits).
template <int NA, int NB, int NO>
__device__ __forceinline__ void bs_add(const uint32_t (&a)[NA], const uint32_t (&b)[NB], uint32_t (&out)[NO]) {
    static_assert(NB <= NA && NO >= NA && NO <= NA + 1, "plane counts");
    uint32_t c = 0;
#pragma unroll
    for (int i = 0; i < NA; ++i) {
        if (i == 0) {
            out[0] = a[0] ^ b[0];
            c = a[0] & b[0];
        } else if (i < NB) {
            bs_fa(a[i], b[i], c, out[i], c);
        } else {
            out[i] = a[i] ^ c;
            c = a[i] & c;
        }
    }
    if constexpr (NO > NA) out[NA] = c;
}

// Copy of the N planes of v shifted right by dx within the 64-bit pair (own word, next word).
template <int N>
__device__ __forceinline__ void bs_shift(const uint32_t (&v)[N], const uint32_t (&vn)[N], int dx, uint32_t (&out)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) out[i] = __funnelshift_r(v[i], vn[i], dx);
}

// Sum of the shifted copies at dx and 16 - dx of one vertical level.
template <int N>
__device__ __forceinline__ void bs_pair(const uint32_t (&v)[N], const uint32_t (&vn)[N], int dx, uint32_t (&out)[N + 1]) {
    uint32_t a[N], b[N];
    bs_shift<N>(v, vn, dx, a);
    bs_shift<N>(v, vn, 16 - dx, b);
    bs_add<N, N, N + 1>(a, b, out);
}

// Vertical sums of one word's 32 columns over the runs of window rows that each column offset needs:
// nested, V5 = rows 6..10, V9 = 4..12, V11 = 3..13, V13 = 2..14, V15 = 1..15, V17 = 0..16.
struct Runs {
    uint32_t v5[3], v9[4], v11[4], v13[4], v15[4], v17[5];
};
__device__ __forceinline__ void bs_runs(const uint32_t* R, Runs& o) {
    uint32_t (&v5)[3] = o.v5;
    uint32_t (&v9)[4] = o.v9, (&v11)[4] = o.v11, (&v13)[4] = o.v13, (&v15)[4] = o.v15;
    uint32_t (&v17)[5] = o.v17;
    {
        uint32_t s1, c1, c2;
        bs_fa(R[6], R[7], R[8], s1, c1);
        bs_fa(R[9], R[10], s1, v5[0], c2);
        v5[1] = c1 ^ c2;
        v5[2] = c1 & c2;
    }
    {
        uint32_t s, c, cc, c4;
        bs_fa(R[4], R[5], R[11], s, c);
        bs_fa(R[12], s, v5[0], v9[0], cc);
        bs_fa(c, cc, v5[1], v9[1], c4);
        v9[2] = c4 ^ v5[2];
        v9[3] = c4 & v5[2];
    }
    auto add2 = [](const uint32_t (&v)[4], uint32_t x, uint32_t y, uint32_t (&o)[4]) {
        uint32_t c;
        bs_fa(x, y, v[0], o[0], c);
        o[1] = v[1] ^ c; c &= v[1];
        o[2] = v[2] ^ c; c &= v[2];
        o[3] = v[3] ^ c;  // the sum stays below 16
    };
    add2(v9, R[3], R[13], v11);
    add2(v11, R[2], R[14], v13);
    add2(v13, R[1], R[15], v15);
    {
        uint32_t c;
        bs_fa(R[0], R[16], v15[0], v17[0], c);
        v17[1] = v15[1] ^ c; c &= v15[1];
        v17[2] = v15[2] ^ c; c &= v15[2];
        v17[3] = v15[3] ^ c; c &= v15[3];
        v17[4] = c;
    }
}

// Exact window counts (8 planes) of the 32 centres of a word whose windows start at row R[0], from the
// rows of the word and of the next one.
__device__ __forceinline__ void bs_window_counts(const uint32_t* R, const uint32_t* Rn, uint32_t (&cnt)[8]) {
    Runs o, n;
    bs_runs(R, o);
    bs_runs(Rn, n);
    // Horizontal: offsets dx = 0..16 from the window's first column; level by |dx - 8|.
    uint32_t a1[4], a2[5], a3[5], a4[5], a5[5], a6[5], a7[6], a8[6], a9[5];
    bs_pair<3>(o.v5, n.v5, 0, a1);      // dx 0, 16: max 10
    bs_pair<4>(o.v9, n.v9, 1, a2);      // dx 1, 15: 18
    bs_pair<4>(o.v11, n.v11, 2, a3);    // dx 2, 14: 22
    bs_pair<4>(o.v13, n.v13, 3, a4);    // dx 3, 13: 26
    bs_pair<4>(o.v15, n.v15, 4, a5);    // dx 4, 12: 30
    bs_pair<4>(o.v15, n.v15, 5, a6);    // dx 5, 11: 30
    bs_pair<5>(o.v17, n.v17, 6, a7);    // dx 6, 10: 34
    bs_pair<5>(o.v17, n.v17, 7, a8);    // dx 7, 9: 34
    bs_shift<5>(o.v17, n.v17, 8, a9);   // dx 8: 17
    uint32_t b1[5], b2[6], b3[6], b4[7], c1[7], c2[8], d[8];
    bs_add<5, 4, 5>(a2, a1, b1);    // 28
    bs_add<5, 5, 6>(a3, a4, b2);    // 48
    bs_add<5, 5, 6>(a5, a6, b3);    // 60
    bs_add<6, 6, 7>(a7, a8, b4);    // 68
    bs_add<6, 5, 7>(b2, b1, c1);    // 76
    bs_add<7, 6, 8>(b4, b3, c2);    // 128
    bs_add<8, 7, 8>(c2, c1, d);     // 204
    bs_add<8, 5, 8>(d, a9, cnt);    // 221
}

// Number of set bits among 17 single-bit vectors (per bit position), as 5 planes: a carry-save
// tree of 12 full adders and 3 half adders.
__device__ __forceinline__ void bs_popcount17(const uint32_t (&b)[17], uint32_t (&o)[5]) {
    uint32_t s1[5], c2[8];
#pragma unroll
    for (int i = 0; i < 5; ++i) bs_fa(b[3 * i], b[3 * i + 1], b[3 * i + 2], s1[i], c2[i]);
    // weight 1: s1[0..4], b[15], b[16]
    uint32_t t0, t1, u0;
    bs_fa(s1[0], s1[1], s1[2], t0, c2[5]);
    bs_fa(s1[3], s1[4], b[15], t1, c2[6]);
    bs_fa(t0, t1, b[16], o[0], c2[7]);
    // weight 2: c2[0..7]
    uint32_t w2a, w2b, w4[4];
    bs_fa(c2[0], c2[1], c2[2], w2a, w4[0]);
    bs_fa(c2[3], c2[4], c2[5], w2b, w4[1]);
    bs_fa(c2[6], c2[7], w2a, u0, w4[2]);
    o[1] = u0 ^ w2b;
    w4[3] = u0 & w2b;
    // weight 4: w4[0..3]
    uint32_t w4a, w8[2];
    bs_fa(w4[0], w4[1], w4[2], w4a, w8[0]);
    o[2] = w4a ^ w4[3];
    w8[1] = w4a & w4[3];
    o[3] = w8[0] ^ w8[1];
    o[4] = w8[0] & w8[1];
}

// Window-relative vertical half-extent of column offset dx (0..16 from the window's first column):
// the column holds window rows 8 - H .. 8 + H.
__host__ __device__ constexpr int column_half_height(int dx) {
    return dx == 0 || dx == 16 ? 2 : dx == 1 || dx == 15 ? 4 : dx == 2 || dx == 14 ? 5
         : dx == 3 || dx == 13 ? 6 : dx <= 5 || dx >= 11 ? 7 : 8;
}

// Counts of the windows starting one row lower than `cnt` (window start DZ - 1 -> DZ among the
// rows R / next-word rows Rn): per column one cell enters (row DZ + 8 + H) and one leaves (row
// DZ + 7 - H), so count' = count + entering - leaving (mod 256, exact since counts are 0..221).
template <int DZ>
__device__ __forceinline__ void bs_slide(const uint32_t* R, const uint32_t* Rn, uint32_t (&cnt)[8]) {
    uint32_t in[17], out[17];
#pragma unroll
    for (int dx = 0; dx < 17; ++dx) {
        const int h = column_half_height(dx);
        in[dx] = __funnelshift_r(R[DZ + 8 + h], Rn[DZ + 8 + h], dx);
        out[dx] = __funnelshift_r(R[DZ + 7 - h], Rn[DZ + 7 - h], dx);
    }
    uint32_t a[5], b[5];
    bs_popcount17(in, a);
    bs_popcount17(out, b);
    // count + a + ~b + 1 over 8 planes: carry-save, then a ripple add with carry-in 1.
    uint32_t sv[8], cv[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t y = i < 5 ? a[i] : 0u, z = i < 5 ? ~b[i] : ~0u;
        bs_fa(cnt[i], y, z, sv[i], cv[i]);
    }
    uint32_t c = ~0u;  // the +1 of the two's complement
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t y = i == 0 ? 0u : cv[i - 1];
        uint32_t o;
        bs_fa(sv[i], y, c, o, c);
        cnt[i] = o;
    }
}

// Centres whose count is at least t (t in 0..256): the carry out of count + (256 - t), with
// the constant's bits known (one LOP3 per plane).
__device__ __forceinline__ uint32_t bs_at_least(const uint32_t (&cnt)[8], int t) {
    const uint32_t k = 256u - (uint32_t)t;
    uint32_t c = 0;
#pragma unroll
    for (int b = 0; b < 8; ++b) c = ((k >> b) & 1u) ? (cnt[b] | c) : (cnt[b] & c);
    return (k & 256u) ? ~0u : c;
}

__device__ __forceinline__ int bs_value(const uint32_t (&cnt)[8], int j) {
    int v = 0;
#pragma unroll
    for (int b = 0; b < 8; ++b) v |= (int)((cnt[b] >> j) & 1u) << b;
    return v;
}


// ---- predicate ---------------------------------------------------------------------------------

// Terms split at bit 18, the low part shifted up by 14: with lo = l * 2^14 the product
// (mix ^ kSeedXor) * A + 11, taken times 2^14, has u = state1 >> 18 in its high word and the parity of
// the first draw in the top bit of its low word.
constexpr int kSplit = 18;
__device__ __forceinline__ uint32_t lo_part(uint64_t t) { return (uint32_t)t << (32 - kSplit); }
__device__ __forceinline__ uint32_t hi_part(uint64_t t) { return (uint32_t)(t >> kSplit); }

// Java's first draw: an even draw 2 u is a multiple of 10 below the bound iff 4 u / 5 (mod 2^32) is
// below 858993456. `top` collects 4 u: draws from 2^31 - 8 on, which Java may draw again, have
// 4 u >= 2^32 - 16.
constexpr uint32_t kRedrawFrom = 0xFFFFFFF0u;
__device__ __forceinline__ bool first_draw(uint32_t xl, uint32_t xh, uint32_t zl, uint32_t zh, uint32_t& top) {
    uint32_t lo, hi;
    asm("{ add.cc.u32 %0, %2, %3;\n addc.u32 %1, %4, %5; }" : "=r"(lo), "=r"(hi) : "r"(xl), "r"(zl), "r"(xh), "r"(zh));
    lo ^= (uint32_t)kSeedXor << (32 - kSplit);
    hi ^= (uint32_t)(kSeedXor >> kSplit);
    constexpr uint32_t kMulLo = (uint32_t)kLcgMult, kMulHi = (uint32_t)(kLcgMult >> 32);
    const uint64_t prod = (uint64_t)lo * kMulLo + (kLcgAdd << (32 - kSplit));
    uint32_t u = (uint32_t)(prod >> 32) + lo * kMulHi;
    u += hi * kMulLo;
    const uint32_t u4 = u << 2;
    top = max(top, u4);
    return ((u4 * 0xCCCCCCCDu) | ((uint32_t)prod & 0x80000000u)) < 858993456u;
}

__global__ void __launch_bounds__(kTpb, 2) general_scan_kernel(const ScanArgs a) {
    __shared__ uint32_t rows[(kMaxRows + 16) * kStride];
    __shared__ unsigned int hist_s[kHistBins];
    __shared__ Hit list[kListCap];
    __shared__ unsigned int listed;
    __shared__ unsigned long long list_at;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < kHistBins; i += kTpb) hist_s[i] = 0;
    if (tid == 0) listed = 0;
    __syncthreads();
    // The CTA's hits go out together: reserving room for each cost its warp a round trip to L2.
    auto flush = [&] {
        const unsigned n = min(listed, (unsigned)kListCap);
        __syncthreads();
        if (tid == 0) {
            list_at = atomicAdd(a.emitted, (unsigned long long)n);
            listed = 0;
        }
        __syncthreads();
        for (unsigned i = tid; i < n; i += kTpb)
            if (list_at + i < a.cap) a.out[list_at + i] = list[i];
        __syncthreads();
    };

    const int64_t tiles = (int64_t)a.tiles_x * a.tiles_z;
    for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int x_base = (int)(t % a.tiles_x) * kOutW;
        const int z_base = a.slab_z0 + (int)(t / a.tiles_x) * a.band_h;
        const int out_w = min(kOutW, a.width - x_base);
        const int out_h = min(a.band_h, a.slab_z0 + a.slab_h - z_base);
        // Annulus searches: a patch whose centres all lie inside the rd_min disc keeps nothing
        // (block-uniform; the farthest corner decides).
        if (a.rd_min_sq && rect_inside_disc(a.area_x0 + (int64_t)x_base, a.area_x0 + (int64_t)x_base + out_w - 1,
                                            a.area_z0 + (int64_t)z_base, a.area_z0 + (int64_t)z_base + out_h - 1,
                                            a.center_x, a.center_z, a.rd_min_sq))
            continue;

        // Bitmap of the patch: warp w evaluates rows w, w + 8, ...
        uint32_t xl[kWords], xh[kWords];
#pragma unroll
        for (int k = 0; k < kWords; ++k) {
            const uint64_t xt = x_term((int32_t)((int64_t)a.area_x0 + x_base - 8 + 32 * k + lane));
            xl[k] = lo_part(xt);
            xh[k] = hi_part(xt);
        }
        __syncthreads();  // the previous patch's rows are no longer read
        if (listed > (unsigned)kListCap / 2) flush();
        for (int r = warp; r < out_h + 16; r += kWarps) {
            const uint64_t zt = z_term((int32_t)((int64_t)a.area_z0 + z_base - 8 + r)) + (uint64_t)a.seed;
            const uint32_t zl = lo_part(zt), zh = hi_part(zt);
            uint32_t word = 0, top = 0;
#pragma unroll
            for (int k = 0; k < kWords; ++k) {
                const uint32_t b = __ballot_sync(kFull, first_draw(xl[k], xh[k], zl, zh, top));
                word = lane == k ? b : word;
            }
            if (__any_sync(kFull, top >= kRedrawFrom)) {  // a draw of this row may be drawn again
#pragma unroll 1
                for (int k = 0; k < kWords; ++k) {
                    const uint64_t xt = x_term((int32_t)((int64_t)a.area_x0 + x_base - 8 + 32 * k + lane));
                    const uint32_t b = __ballot_sync(kFull, slime_from_terms(xt, zt));
                    word = lane == k ? b : word;
                }
            }
            if (lane < kStride) rows[r * kStride + lane] = word;  // lane 8: the zero word
        }
        __syncthreads();

        // Counts: a thread takes `step` centre rows of one word (at most four).
        const int step = (out_h * kWords + kTpb - 1) / kTpb;
        const int word = tid % kWords, j0 = tid / kWords * step;
        if (j0 < out_h && 32 * word < out_w) {
            uint32_t R[20], Rn[20];
#pragma unroll
            for (int i = 0; i < 20; ++i) {
                const int r = min(j0 + i, out_h + 15);
                R[i] = rows[r * kStride + word];
                Rn[i] = rows[r * kStride + word + 1];
            }
            const int cols = min(32, out_w - 32 * word);
            const uint32_t live = cols >= 32 ? ~0u : (1u << cols) - 1u;
            uint32_t cnt[8];
            auto keep = [&](int dz) {
                uint32_t pass = live & bs_at_least(cnt, a.min_size);
                if (a.max_size < 221) pass &= ~bs_at_least(cnt, a.max_size + 1);
                for (; pass; pass &= pass - 1) {
                    const int bit = __ffs(pass) - 1, count = bs_value(cnt, bit);
                    const int32_t cx = a.area_x0 + x_base + 32 * word + bit, cz = a.area_z0 + z_base + j0 + dz;
                    if (a.rd_min_sq) {
                        const int64_t dx = (int64_t)cx - a.center_x, dzz = (int64_t)cz - a.center_z;
                        if (dx * dx + dzz * dzz < a.rd_min_sq) continue;
                    }
                    atomicAdd(&hist_s[count], 1u);
                    if (count < a.emit_min) continue;
                    const Hit hit{count, cx, cz};
                    const unsigned n = atomicAdd(&listed, 1u);
                    if (n < (unsigned)kListCap) {
                        list[n] = hit;
                    } else {
                        const unsigned long long pos = atomicAdd(a.emitted, 1ull);
                        if (pos < a.cap) a.out[pos] = hit;
                    }
                }
            };
            bs_window_counts(R, Rn, cnt);
            keep(0);
            if (step > 1 && j0 + 1 < out_h) {
                bs_slide<1>(R, Rn, cnt);
                keep(1);
                if (step > 2 && j0 + 2 < out_h) {
                    bs_slide<2>(R, Rn, cnt);
                    keep(2);
                    if (step > 3 && j0 + 3 < out_h) {
                        bs_slide<3>(R, Rn, cnt);
                        keep(3);
                    }
                }
            }
        }
    }
    __syncthreads();
    if (listed) flush();
    for (int i = tid; i < kHistBins; i += kTpb)
        if (hist_s[i]) atomicAdd(&a.hist[i], hist_s[i]);
}

__global__ void predicate_kernel(int64_t seed, const int64_t* x, const int64_t* z, uint8_t* out,
                                 int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = is_slime(seed, x[i], z[i]) ? 1 : 0;
}

}  // namespace

int general_out_width() { return kOutW; }

// Centre rows of a patch: patches run in waves of one CTA an SM (two share an SM at half the speed
// each), a patch costs its rows, 16 halo rows and about 12 rows of fixed work (terms, counting); the
// height with the fewest rows in all waves wins. Radius 100: 8 rows on 26 CTAs; radius 2,000: 120 rows,
// 578 patches in 4 waves.
int general_band_rows(int64_t width, int64_t height, int sm_count) {
    const int64_t tx = (width + kOutW - 1) / kOutW;
    int best = 8;
    double best_cost = 0;
    for (int h = 8; h <= kMaxRows; h += 8) {
        const double tiles = (double)tx * (double)((height + h - 1) / h);
        const double waves = tiles > 16.0 * sm_count ? tiles / sm_count + 0.5 : std::ceil(tiles / sm_count);
        const double cost = waves * (h + 16 + 12);
        if (best_cost == 0 || cost < best_cost) {
            best = h;
            best_cost = cost;
        }
    }
    return best;
}

int general_max_grid() {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, general_scan_kernel, kTpb, 0);
    return (sms > 0 ? sms : 148) * (per_sm > 0 ? per_sm : 1);
}

cudaError_t launch_general_scan(const ScanArgs& a, int grid, cudaStream_t s) {
    general_scan_kernel<<<grid, kTpb, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_predicate(int64_t seed, const int64_t* x, const int64_t* z, uint8_t* out,
                             int64_t n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    predicate_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(seed, x, z, out, n);
    return cudaGetLastError();
}

}  // namespace slime
