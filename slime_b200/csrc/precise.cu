// precise.cu -- precise AFK scoring of ranked sites.
//
// Semantics of score_candidates_precise (SlimeCore.cpp:654-726): for each site and each offset
// (dx, dz) in {-16..16 step 4}^2 (or only (0,0) without the XZ scan) and each Y level, count the
// block columns of slime chunks inside the annulus 24^2 < dx^2 + dy^2 + dz^2 <= 128^2 around the
// offset position (count_spawnable_cached_table, SlimeCore.cpp:291-331); keep the strict maximum,
// first in (dx, dz, Y) order, starting from 0 at the site centre.
//
// B200 design: a precomputed table gives each slime chunk's block-column count for the window
// alignment (o mod 16 on each axis), the chunk's place in the 21 x 21 window and the Y level, so a
// score is a sum of table entries over the window's slime chunks.
//  * One Y level (precise_one_kernel): the offsets of a site meet only 4 x 4 alignments, so a CTA keeps
//    those slices of the table in shared memory, padded to 25 x 25 chunks with zeros, and a warp takes a
//    site: it lists the slime chunks of the 23 x 23 that any offset reaches, and each lane adds up
//    the entries of its three offsets. Per chunk that is one broadcast and three lookups a warp; a CTA
//    per site with the table in global memory spent its time on 44 dependent steps of bit scanning a
//    lane and eight block barriers a site. 20,000 sites: 243 -> 69 us (issue slots 65 % busy).
//  * Several Y levels (precise_kernel): one CTA per site builds the 23 x 23 bitmap once; threads split the
//    (offset, Y) pairs, neighbours in Y, so the table reads coalesce; a block reduction picks (max obs,
//    first order).
#include "engine.h"

namespace slime {
namespace {

constexpr int kPreciseTpb = 128;
constexpr int kDxMin = -128, kDxCount = 257;

__device__ __forceinline__ int64_t floor_div16(int64_t v) { return v >> 4; }

__device__ __forceinline__ int interval_len(int a, int b) { return b >= a ? b - a + 1 : 0; }

// One Y level: weights[(ax * 16 + az) * kSlice + (i + 2) * kPad + j + 2], zero outside the window (a chunk
// that only other offsets reach has index -2 .. 22) and up to the slice's 16-byte multiple.
constexpr int kPad = 25;
constexpr int kSlice = (kPad * kPad + 7) / 8 * 8;
// Several: weights[(((ax * 16 + az) * 21 + i) * 21 + j) * y_count + yi].
__global__ void weight_table_kernel(uint16_t* weights, const int16_t* outer, const int16_t* inner,
                                    int32_t y_count) {
    const int64_t total = (int64_t)precise_weights(y_count);
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        int yi = 0, i, j, ax, az;
        if (y_count == 1) {
            const int slice = (int)(e / kSlice), at = (int)(e % kSlice);
            i = at / kPad - 2;
            j = at % kPad - 2;
            ax = slice / 16;
            az = slice % 16;
            if (i < 0 || i > 20 || j < 0 || j > 20) {
                weights[e] = 0;
                continue;
            }
        } else {
            yi = (int)(e % y_count);
            int64_t rest = e / y_count;
            j = (int)(rest % 21); rest /= 21;
            i = (int)(rest % 21); rest /= 21;
            az = (int)(rest % 16);
            ax = (int)(rest / 16);
        }
        // Block offsets of the chunk relative to the scored position.
        const int rx0 = (i - 10) * 16 - ax, rz0 = (j - 10) * 16 - az;
        const int x0 = max(-128, rx0), x1 = min(128, rx0 + 15);
        const int z0 = max(-128, rz0), z1 = min(128, rz0 + 15);
        const int16_t* o = outer + (int64_t)yi * kDxCount;
        const int16_t* n = inner + (int64_t)yi * kDxCount;
        int total_cols = 0;
        if (z0 <= z1) {
            for (int dx = x0; dx <= x1; ++dx) {
                const int ro = o[dx - kDxMin];
                if (ro < 0) continue;
                const int zl = max(z0, -ro), zr = min(z1, ro);
                int add = interval_len(zl, zr);
                if (!add) continue;
                const int ri = n[dx - kDxMin];
                if (ri >= 0) add -= interval_len(max(zl, -ri), min(zr, ri));
                total_cols += add;
            }
        }
        weights[e] = (uint16_t)total_cols;
    }
}

__global__ void __launch_bounds__(kPreciseTpb) precise_kernel(const PreciseArgs a) {
    __shared__ uint32_t bits[24];
    __shared__ int s_obs[kPreciseTpb];
    __shared__ int s_ord[kPreciseTpb];
    const int tid = threadIdx.x;
    const int lo = a.scan_xz ? -16 : 0, hi = a.scan_xz ? 16 : 0;
    const int side = a.scan_xz ? 9 : 1;
    const int pairs = side * side * a.y_count;

    for (int64_t site = blockIdx.x; site < a.n; site += gridDim.x) {
        const int64_t bx = a.sites[site].center_x, bz = a.sites[site].center_z;
        const int64_t ux0 = floor_div16(bx + lo) - 10, uz0 = floor_div16(bz + lo) - 10;
        const int nx = (int)(floor_div16(bx + hi) + 10 - ux0 + 1);
        const int nz = (int)(floor_div16(bz + hi) + 10 - uz0 + 1);
        if (tid < 24) bits[tid] = 0;
        __syncthreads();
        for (int e = tid; e < nx * nz; e += kPreciseTpb) {
            const int i = e / nz, j = e % nz;
            if (is_slime(a.seed, ux0 + i, uz0 + j)) atomicOr(&bits[i], 1u << j);
        }
        __syncthreads();

        int best = -1, best_ord = 0x7FFFFFFF;
        for (int p = tid; p < pairs; p += kPreciseTpb) {
            const int off = p / a.y_count, yi = p % a.y_count;
            const int64_t ox = bx + lo + (off / side) * 4, oz = bz + lo + (off % side) * 4;
            const int wx = (int)(floor_div16(ox) - 10 - ux0), wz = (int)(floor_div16(oz) - 10 - uz0);
            const uint16_t* w = a.weights +
                (int64_t)(((int)(ox & 15) * 16 + (int)(oz & 15)) * 441) * a.y_count + yi;
            int obs = 0;
            for (int i = 0; i < 21; ++i) {
                uint32_t row = (bits[wx + i] >> wz) & 0x1FFFFFu;
                while (row) {
                    const int j = __ffs(row) - 1;
                    row &= row - 1;
                    obs += w[(int64_t)(i * 21 + j) * a.y_count];
                }
            }
            if (obs > best) { best = obs; best_ord = p; }  // p ascends: first maximum wins
        }
        s_obs[tid] = best;
        s_ord[tid] = best_ord;
        __syncthreads();
        for (int stride = kPreciseTpb / 2; stride > 0; stride >>= 1) {
            if (tid < stride) {
                const int ob = s_obs[tid + stride], od = s_ord[tid + stride];
                if (ob > s_obs[tid] || (ob == s_obs[tid] && od < s_ord[tid])) {
                    s_obs[tid] = ob;
                    s_ord[tid] = od;
                }
            }
            __syncthreads();
        }
        if (tid == 0) {
            int obs = s_obs[0];
            int64_t ax = bx, az = bz;
            int y = a.platform_y;
            if (obs > 0) {
                const int off = s_ord[0] / a.y_count, yi = s_ord[0] % a.y_count;
                ax = bx + lo + (off / side) * 4;
                az = bz + lo + (off % side) * 4;
                y = a.y_values[yi];
            } else {
                obs = 0;
            }
            ExtChunkResult& r = a.sites[site];
            r.obs_count = a.pack_y ? (int32_t)((uint32_t)obs | ((uint32_t)(y + 1024) << 20)) : obs;
            r.afk_x = (int32_t)ax;
            r.afk_z = (int32_t)az;
        }
        __syncthreads();
    }
}

// ---- one Y level ---------------------------------------------------------------------------------

constexpr int kOneTpb = 256, kOneWarps = kOneTpb / 32;
constexpr int kSide = 23;               // chunks per axis that some offset's window reaches

__global__ void __launch_bounds__(kOneTpb) precise_one_kernel(const PreciseArgs a, int chunk) {
    __shared__ __align__(16) uint16_t table[16 * kSlice];  // [x alignment / 4][z alignment / 4][i + 2][j + 2]
    __shared__ uint16_t list[kOneWarps][kSide * kSide];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int lo = a.scan_xz ? -16 : 0, hi = a.scan_xz ? 16 : 0;
    const int side = a.scan_xz ? 9 : 1, pairs = side * side;
    int loaded = -1;  // alignment class (both centres mod 4) of the table
    auto class_of = [&](int64_t s) { return (int)(a.sites[s].center_x & 3) * 4 + (int)(a.sites[s].center_z & 3); };

    for (int64_t first = (int64_t)blockIdx.x * chunk; first < a.n; first += (int64_t)gridDim.x * chunk) {
        const int64_t last = min(first + chunk, (int64_t)a.n);
        // The offsets of a site meet 16 alignments, the same for all sites of a class. Search results are all of
        // class 0 (centres at 8 mod 16); a chunk of sites of several classes looks its entries up in global
        // memory. (A table for each class of a chunk in turn: 5,000 sites of random alignment 224 us a call
        // against 182 with a CTA a site.)
        const int cls = class_of(first);
        bool same = true;
        for (int64_t s = first + 1 + lane; s < last; s += 32) same &= class_of(s) == cls;
        const bool shared = __all_sync(0xFFFFFFFFu, same);  // the same in every warp
        if (shared && cls != loaded) {
            __syncthreads();  // the previous table is no longer read
            for (int e = tid; e < 16 * kSlice / 8; e += kOneTpb) {
                const int s = e / (kSlice / 8), ax = (s >> 2) * 4 + (cls >> 2), az = (s & 3) * 4 + (cls & 3);
                reinterpret_cast<uint4*>(table)[e] =
                    reinterpret_cast<const uint4*>(a.weights + (ax * 16 + az) * kSlice)[e % (kSlice / 8)];
            }
            __syncthreads();
            loaded = cls;
        }
        for (int64_t s = first + warp; s < last; s += kOneWarps) {
            const int64_t bx = a.sites[s].center_x, bz = a.sites[s].center_z;
            const int64_t ux0 = floor_div16(bx + lo) - 10, uz0 = floor_div16(bz + lo) - 10;
            const int nx = (int)(floor_div16(bx + hi) + 10 - ux0 + 1);
            const int nz = (int)(floor_div16(bz + hi) + 10 - uz0 + 1);
            // Slime chunks (i, j) as i * kPad + j: lane = j, one i at a time.
            const uint64_t xs = x_term((int32_t)(ux0 + lane)), zs = z_term((int32_t)(uz0 + lane)) + (uint64_t)a.seed;
            int n = 0;
            __syncwarp();
            for (int i = 0; i < nx; ++i) {
                const bool hit = slime_from_terms(__shfl_sync(0xFFFFFFFFu, xs, i), zs) && lane < nz;
                const unsigned m = __ballot_sync(0xFFFFFFFFu, hit);
                if (hit) list[warp][n + __popc(m & ((1u << lane) - 1u))] = (uint16_t)(i * kPad + lane);
                n += __popc(m);
            }
            __syncwarp();
            // This lane's offsets p = lane, lane + 32, lane + 64: first table entry of chunk (0, 0).
            int base[3], obs[3] = {0, 0, 0};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int p = min(lane + 32 * k, pairs - 1);
                const int64_t ox = bx + lo + (p / side) * 4, oz = bz + lo + (p % side) * 4;
                const int wx = (int)(floor_div16(ox) - 10 - ux0), wz = (int)(floor_div16(oz) - 10 - uz0);
                const int ax = (int)(ox & 15), az = (int)(oz & 15);
                base[k] = (shared ? (ax >> 2) * 4 + (az >> 2) : ax * 16 + az) * kSlice + (2 - wx) * kPad + 2 - wz;
            }
            if (shared) {
#pragma unroll 4
                for (int c = 0; c < n; ++c) {
                    const int at = list[warp][c];
#pragma unroll
                    for (int k = 0; k < 3; ++k) obs[k] += table[base[k] + at];
                }
            } else {
#pragma unroll 4
                for (int c = 0; c < n; ++c) {
                    const int at = list[warp][c];
#pragma unroll
                    for (int k = 0; k < 3; ++k) obs[k] += a.weights[base[k] + at];
                }
            }
            int best = -1, order = 0x7FFFFFFF;
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (lane + 32 * k < pairs && obs[k] > best) {  // offsets ascend: the first maximum wins
                    best = obs[k];
                    order = lane + 32 * k;
                }
            const int top = __reduce_max_sync(0xFFFFFFFFu, best);
            const int off = __reduce_min_sync(0xFFFFFFFFu, best == top ? order : 0x7FFFFFFF);
            if (lane == 0) {
                ExtChunkResult& r = a.sites[s];
                const int y = top > 0 ? a.y_values[0] : a.platform_y;
                r.obs_count = a.pack_y ? (int32_t)((uint32_t)top | ((uint32_t)(y + 1024) << 20)) : top;
                r.afk_x = (int32_t)(top > 0 ? bx + lo + (off / side) * 4 : bx);
                r.afk_z = (int32_t)(top > 0 ? bz + lo + (off % side) * 4 : bz);
            }
        }
    }
}

}  // namespace

__host__ __device__ size_t precise_weights(int32_t y_count) {
    return 16 * 16 * (size_t)(y_count == 1 ? kSlice : 21 * 21 * (size_t)y_count);
}

cudaError_t launch_weight_table(uint16_t* weights, const int16_t* outer, const int16_t* inner,
                                int32_t y_count, cudaStream_t s) {
    const int64_t total = (int64_t)precise_weights(y_count);
    const int blocks = (int)((total + 255) / 256 < 4096 ? (total + 255) / 256 : 4096);
    weight_table_kernel<<<blocks, 256, 0, s>>>(weights, outer, inner, y_count);
    return cudaGetLastError();
}

cudaError_t launch_precise(const PreciseArgs& a, cudaStream_t s) {
    if (a.n <= 0) return cudaSuccess;
    if (a.y_count == 1) {
        // Sites per CTA and round: an even share of one wave, whole rounds of the CTA's warps from one
        // round on, and at most 256 (each thread looks at all of a chunk's alignments).
        constexpr int kCtas = 148 * 4;
        int64_t chunk = ((int64_t)a.n + kCtas - 1) / kCtas;
        if (chunk > kOneWarps) chunk = (chunk + kOneWarps - 1) / kOneWarps * kOneWarps;
        if (chunk > 256) chunk = 256;
        const int64_t grid = ((int64_t)a.n + chunk - 1) / chunk;
        precise_one_kernel<<<(int)(grid < kCtas ? grid : kCtas), kOneTpb, 0, s>>>(a, (int)chunk);
        return cudaGetLastError();
    }
    const int grid = a.n < 148 * 16 ? a.n : 148 * 16;
    precise_kernel<<<grid, kPreciseTpb, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace slime
