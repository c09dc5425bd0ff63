// scan_planes.cu -- row-term tables and launches of the bit-plane band kernels (planes.cuh).
#include "planes.cuh"

namespace slime {
namespace {

// Row-term table, one record per (band group g, base row v), records of a group contiguous; band j =
// 32 g + m holds base row v at input row v + offset(j), where offset(j) = j * stride, or, with grouped
// bands, (j % P) * 2^17 + (j / P) * stride (P copies a group). Record words (0 where the row lies
// outside the area plus halo):
//   shared LCG   [m] high part (>> 17) of the row term in band m, [32] its low_bits, [33] bands
//   independent  [m] and [32 + m]: indep_hi and indep_row_lo of the row term in band m, [64] bands
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
                if (kMode == kModeIndep) out = hi ? indep_hi(t) : indep_row_lo(t);
                else out = hi ? (uint32_t)(t >> kPeriodBits) : low_bits(t);
            }
        }
    }
    rt[e] = out;
}

}  // namespace

int plane_tile_out_w(int mode) {
    return mode == kBandShared ? Shape<kModeShared>::kOutW : Shape<kModeIndep>::kOutW;
}
int plane_ctas_per_sm() { return kCtasPerSm; }
int plane_row_words(int mode) { return mode == kBandShared ? kRowWordsS : kRowWordsI; }

// Per four columns and row a warp issues about 336, 170 or 90 adders for unions of 1, 2 or 4 windows and
// 90 instructions for each union of its 1,024 x (4 / kUnion) that reaches the threshold (binomial tails of
// 238 and 272 cells: 8e-4 and 9e-3 at 40, 5e-5 and 1e-3 at 44). Measured, radius 100,000, independent
// bands, with 1 / 2 / 4: threshold 39 33.6 / 40.1 ms, 40 31.3 / 32.4 / 85.5, 42 28.4 / 25.5 / 44.6, 46 27.7 /
// 22.5 / 23.6, 47 27.6 / 22.4 / 22.5, 60 27.6 / 22.2 / 20.8; radius 300,000, grouped bands: 38 311 / 434, 40 265 /
// 241 / 726, 46 216 / 153 / 155, 47 216 / 152 / 145; radius 1,250,000, shared LCG: 46 3,355 / 2,061 / 2,086, 48
// 3,345 / 2,026 / 1,785.
constexpr int kUnionTwoFrom = 40, kUnionFourFrom = 47;
int plane_union(int min_size) { return min_size >= kUnionFourFrom ? 4 : min_size >= kUnionTwoFrom ? 2 : 1; }

namespace {
cudaError_t run_planes(int mode, int joined, const BandArgs& one, const BandArgs* args, const int64_t* prefix,
                       int32_t nsearch, unsigned long long* head, int grid, cudaStream_t s) {
    return mode == kBandIndep     ? run_planes_indep(joined, one, args, prefix, nsearch, head, grid, s)
           : mode == kBandGrouped ? run_planes_grouped(joined, one, args, prefix, nsearch, head, grid, s)
                                  : run_planes_shared(joined, one, args, prefix, nsearch, head, grid, s);
}
}  // namespace

cudaError_t plane_prepare() {
    for (int mode : {kBandShared, kBandIndep, kBandGrouped})
        for (int joined : {1, 2, 4}) {
            const cudaError_t e = run_planes(mode, joined, BandArgs{}, nullptr, nullptr, 0, nullptr, 0, nullptr);
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

cudaError_t launch_plane_batch(const BandArgs* args, const int64_t* prefix, int32_t nsearch, unsigned long long* head,
                               int mode, int joined, int grid, cudaStream_t s) {
    return run_planes(mode, joined, BandArgs{}, args, prefix, nsearch, head, grid, s);
}

cudaError_t launch_plane_scan(const BandArgs& a, int grid, cudaStream_t s) {
    return run_planes(band_mode(a), a.joined, a, nullptr, nullptr, 0, nullptr, grid, s);
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
