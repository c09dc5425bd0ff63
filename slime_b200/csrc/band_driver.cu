// band_driver.cu -- host side of the band engine (scan_band.cu) and its redraw correction.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <thread>
#include <vector>

#include "band_math.cuh"
#include "driver.h"
#include "engine.h"

namespace slime {

namespace {
constexpr int64_t kP = band::kPeriod;
constexpr uint32_t kRareCap = 1u << 20;
}  // namespace

bool Context::ensure_band() {
    if (band_ready) return true;
    cudaError_t e = column_prepare();
    if (e == cudaSuccess) e = plane_prepare();
    if (e != cudaSuccess) { set_error("band smem", e); return false; }
    std::vector<uint64_t> t;
    std::vector<uint32_t> o;
    rare_target_table(t, o);
    if ((e = rare_targets.reserve(t.size())) != cudaSuccess || (e = rare_offsets.reserve(o.size())) != cudaSuccess ||
        (e = flags.reserve(4)) != cudaSuccess || (e = rare.reserve(kRareCap)) != cudaSuccess ||
        (e = cudaMemcpyAsync(rare_targets.ptr, t.data(), t.size() * 8, cudaMemcpyHostToDevice, stream)) != cudaSuccess ||
        (e = cudaMemcpyAsync(rare_offsets.ptr, o.data(), o.size() * 4, cudaMemcpyHostToDevice, stream)) != cudaSuccess ||
        (e = cudaStreamSynchronize(stream)) != cudaSuccess) {
        set_error("rare table", e);
        return false;
    }
    band_ready = true;
    return true;
}

// Engine choice. The automatic rule uses the band engines from threshold 28 on (the byte-lane bound test of
// the columns in words needs that). The shared LCG wants an area of many periods; the independent bands want
// enough centres to fill the GPU. The general scan takes the rest.
int32_t Context::engine_for(const SearchSpec& q) const {
    const int64_t w = 2 * q.rd_max + 1;
    // The band engines count a whole search into 32-bit bins; beyond that the general scan, which counts each
    // of its launches by itself (radius 1,250,000 with all sites in bins: threshold 40 3.6 s against 8.9).
    constexpr double kBandMaxSites = 4e9;
    if ((double)w * (double)w * tail_share(q.min_size) > kBandMaxSites) return kAlgoGeneral;
    if (engine_override == 4) return kAlgoBandExact;
    if (engine_override == 5) return kAlgoIndepExact;
    const bool groups_fit = w <= kGroupedMaxPeriods * kP;  // 16 copies at most
    if (engine_override == 7) return groups_fit ? kAlgoGroupedExact : kAlgoBandExact;
    if (engine_override == 1 || q.min_size < 28) return kAlgoGeneral;
    if (engine_override == 2) return kAlgoBand;
    if (engine_override == 3) return kAlgoIndep;
    if (engine_override == 6) return groups_fit ? kAlgoGrouped : kAlgoBand;
    // The rule's numbers are measured crossovers (slime_b200/autotune.py writes them; the defaults are
    // the B200 values).
    const bool wide = w >= kGroupedExactMinWidth;
    // Columns in words (bounded counts): shared LCG and grouped bands at high thresholds. Their
    // generator is cheaper than the bit planes', and few groups of windows pass its bounds there.
    const bool shared = (q.min_size >= band_min_threshold && w >= (int64_t)band_min_periods * kP) ||
                        (q.min_size >= band_fast_threshold && w >= (int64_t)band_fast_periods * kP);
    // Past grouped_max_width the shared LCG goes first; where its branches leave off, grouped bands go on
    // (radius 510,000, threshold 60: grouped 212 ms, shared 231 at 524,288, independent bands 513).
    const bool grouped = q.min_size >= grouped_min_threshold && w >= grouped_min_width && groups_fit &&
                         (w <= grouped_max_width || !shared);
    // Bit planes (exact counts) below that. The generator's sharing and how full the words are decide the
    // mode. B200, T centres/s at threshold 44: independent bands 1.60-1.68 at any width; grouped bands 1.26 /
    // 1.64 / 1.74 / 2.22 / 3.41 at 1.5 / 2.3 / 3.1 / 4.6 / 15.3 periods; the shared LCG 1.54 / 2.43 / 2.86 at
    // 9.2 / 15.3 / 19.1.
    if (!shared && !grouped && q.min_size < (wide ? exact_wide_below_threshold : exact_below_threshold) &&
        w * w >= exact_min_centres) {
        const bool single = plane_union(q.min_size) == 1;  // every window counted by itself: thresholds below 40
        // Bit planes count all combos of a column at once, those inside the rd_min disc too; the general scan
        // skips the patches there. From these shares of the area outside the disc on down it is the faster one
        // at low thresholds. B200, inner radius 0.8 / 0.9 / 0.99 of the outer: radius 400,000, threshold 39 480 /
        // 357 / 234 ms against 495 / 490 / 486; 900,000 at 40 2,382 / 1,772 / 1,161 against 1,694 / 1,692 / 1,690.
        // Where more centres are kept, those inside the disc cost more: radius 300,000, threshold 35, 0.79 327
        // against 380; 80,000 at 28, 0.7 45 against 57.
        const double outside = 1.0 - 3.14159265358979 * (double)q.rd_min * (double)q.rd_min / ((double)w * (double)w);
        const int t = q.min_size;
        if (outside < (t < 30 ? 0.78 : t < 36 ? 0.6 : t < 40 ? 0.5 : t == 40 ? 0.36 : 0.0)) return kAlgoGeneral;
        // An upper bound can stop the emission gate at a count that many centres share, and a site sent costs
        // more here (its filter against the redrawn chunks, launches cut to the hit buffer) than in the general
        // scan: by the share of the centres sent, 1.2e-3 (radius 100,000, counts 30 to 36) 582 ms against 310,
        // 1.8e-4 (1,000,000, 39) 10.9 s against 9.3, 8.9e-5 (1,250,000, 40) 9.3 against 12.1.
        if (q.max_size < kHistBins - 1 &&
            tail_share(emission_gate(q, q.max_results)) - tail_share(q.max_size + 1) > 1.3e-4)
            return kAlgoGeneral;
        // Single windows cost more to count than to generate, and grouped bands leave bits of a word empty:
        // they start at 4 periods there (radius 200,000, threshold 39 160 ms against 129 with independent
        // bands; 262,144: 218 against 221). Independent bands run the same kernels either way; counted by
        // unions of windows they are reported as bounded.
        if (!wide || (single && w < kGroupedSingleMinWidth)) return single ? kAlgoIndepExact : kAlgoIndep;
        return groups_fit ? kAlgoGroupedExact : kAlgoBandExact;
    }
    if (grouped) return kAlgoGrouped;
    if (shared) return kAlgoBand;
    if (w * w >= indep_min_centres && q.min_size >= indep_min_threshold) return kAlgoIndep;
    return kAlgoGeneral;
}

BandGeom band_geometry(int64_t W, int64_t H, int mode, bool planes, int sm_count) {
    BandGeom g{};
    const bool indep = mode == kBandIndep, grouped = mode == kBandGrouped;
    g.indep = indep;
    g.planes = planes;
    g.transposed = mode == kBandShared && W < 2 * kP && H >= 2 * kP;
    g.width_u = g.transposed ? H : W;
    g.height_v = g.transposed ? W : H;
    const int out_w = planes ? plane_tile_out_w(mode) : column_tile_out_w();
    const int nb_max = band_max_bands();
    // Shared LCG: X phases and Z bands 2^17 apart. Independent bands: one phase, 32 bands (one a bit;
    // fewer only below 8 rows a band) of `stride` rows each. Grouped bands: X phase pairs and G groups
    // of `copies` bands 2^17 apart (G * copies <= 16), group g starting at row g * stride, where
    // G * stride covers 2^17 (or the whole height in one copy). The plane kernels take as many groups
    // as fit (each fills bits of a word); the column kernels want G a power of two.
    g.nI = indep ? 1 : (g.width_u + kP - 1) / kP;
    if (grouped) {
        const int64_t copies = std::max<int64_t>(1, (g.height_v + kP - 1) / kP);
        int64_t G = std::max<int64_t>(1, kGroupedMaxBands / copies);
        if (!planes)
            while (G & (G - 1)) --G;
        g.groups = (int32_t)G;
        g.nJ = G * copies;
        g.stride = ((copies > 1 ? kP : g.height_v) + G - 1) / G;
    } else {
        g.nJ = indep ? std::max<int64_t>(1, std::min<int64_t>(nb_max, g.height_v / 8)) : (g.height_v + kP - 1) / kP;
        g.stride = indep ? (g.height_v + g.nJ - 1) / g.nJ : kP;
    }
    g.ubase = (int32_t)(indep ? g.width_u : std::min(kP, g.width_u));
    g.vbase = (int32_t)std::min(g.stride, g.height_v);
    g.vrows = g.vbase + 16;
    g.vrows_alloc = g.vbase + 32;  // zero rows: the bulk copies of a batch never run past the end
    g.ngroups = (g.nJ + nb_max - 1) / nb_max;
    g.u_tiles = (g.ubase + out_w - 1) / out_w;
    g.pairs = (g.nI + 1) / 2;
    // Tile height: the tiles of a launch run in waves of `slots` CTAs, each tile 16 halo rows taller
    // than its centres. The height (at most 2,048 rows) whose waves take the fewest rows wins; with
    // many waves the last one hardly counts. (Radius 20,011, 40 columns of tiles of the bit planes: 8 tiles
    // high would be 320 tiles on 296 CTAs, 2 waves of 173 rows where 7 make one of 195.)
    const int64_t slots = band_grid(planes, sm_count), columns = g.u_tiles * g.pairs;
    int64_t best_vt = 0;
    double best_rows = 0;
    for (int64_t vt = (g.vbase + 2047) / 2048; vt <= std::max<int64_t>(1, (g.vbase + 7) / 8); ++vt) {
        const int64_t h = (g.vbase + vt - 1) / vt, tiles = columns * ((g.vbase + h - 1) / h);
        const double waves = tiles > 16 * slots ? (double)tiles / (double)slots + 0.5
                                                : (double)((tiles + slots - 1) / slots);
        const double rows = waves * (double)(h + 16 + 8);  // and a batch's worth of set-up
        if (!best_vt || rows < best_rows) {
            best_vt = vt;
            best_rows = rows;
        }
        if (tiles > 24 * slots) break;
    }
    g.band_h = (int32_t)((g.vbase + best_vt - 1) / best_vt);
    g.v_tiles = (g.vbase + g.band_h - 1) / g.band_h;
    g.tiles = g.u_tiles * g.v_tiles * g.pairs;
    return g;
}

int band_grid(bool planes, int sm_count) { return sm_count * (planes ? plane_ctas_per_sm() : 1); }

size_t band_row_table_words(const BandGeom& g) {
    const int mode = g.indep ? kBandIndep : g.groups > 0 ? kBandGrouped : kBandShared;
    return (size_t)g.ngroups * g.vrows_alloc * (g.planes ? plane_row_words(mode) : column_row_words(mode));
}

cudaError_t launch_band_terms(uint64_t* ct, uint32_t* rt, const BandGeom& g, int64_t seed, int32_t area_x0,
                              int32_t area_z0, cudaStream_t s) {
    // Columns carry no seed; rows carry it. Transposed searches swap which axis is x.
    const int32_t col_first = (g.transposed ? area_z0 : area_x0) - 8;
    const int32_t row_first = (g.transposed ? area_x0 : area_z0) - 8;
    const cudaError_t e = launch_column_terms(ct, col_first, (int32_t)(g.width_u + 16), g.transposed, s);
    if (e != cudaSuccess) return e;
    return g.planes ? launch_plane_row_terms(rt, g.vrows_alloc, g.vrows, (int32_t)g.nJ, row_first, g.height_v + 16, g.stride,
                                             seed, g.transposed, g.indep, g.groups, s)
                    : launch_column_row_terms(rt, g.vrows_alloc, g.vrows, (int32_t)g.nJ, row_first, g.height_v + 16,
                                              g.stride, seed, g.transposed, g.groups, s);
}

cudaError_t launch_band_scan(const BandArgs& a, int grid, cudaStream_t s) {
    return band_planes(band_mode(a), a.exact != 0) ? launch_plane_scan(a, grid, s) : launch_column_scan(a, grid, s);
}

// 0..3: columns in words, by mode (shared, grouped) and survivor lists; 4..12: bit planes, by mode and
// windows counted as one.
int band_class(const BandArgs& a) {
    const int mode = band_mode(a);
    if (!band_planes(mode, a.exact != 0)) return (mode == kBandGrouped ? 2 : 0) + (band_keeps_candidates(a.min_size) ? 1 : 0);
    return 4 + 3 * mode + (a.joined == 4 ? 2 : a.joined - 1);
}

bool Context::scan_band(const SearchSpec& q, std::vector<Hit>& best, Counts& h,
                        bool& cancelled, int mode, bool exact) {
    if (!ensure_band()) return false;
    const int64_t W = 2 * q.rd_max + 1, H = W;
    const int32_t area_x0 = (int32_t)((int64_t)q.center_x - q.rd_max);
    const int32_t area_z0 = (int32_t)((int64_t)q.center_z - q.rd_max);
    const BandGeom G = band_geometry(W, H, mode, band_planes(mode, exact), sm_count);
    const bool indep = G.indep;
    const bool transposed = G.transposed;
    const int64_t width_u = G.width_u, height_v = G.height_v;
    const int nb_max = band_max_bands();
    const int64_t nJ = G.nJ, stride = G.stride;
    const int32_t ubase = G.ubase, vbase = G.vbase, vrows = G.vrows;
    const int64_t ngroups = G.ngroups;
    cudaError_t e;
    if ((e = xt.reserve((size_t)width_u + 16)) != cudaSuccess ||
        (e = rt.reserve(band_row_table_words(G))) != cudaSuccess ||
        (e = counters.reserve(4)) != cudaSuccess ||
        (e = hits.reserve(hit_capacity(q.max_results))) != cudaSuccess ||
        (e = fixed.reserve(1u << 20)) != cudaSuccess) {
        set_error("alloc", e);
        return false;
    }
    if ((e = launch_band_terms(xt.ptr, rt.ptr, G, q.seed, area_x0, area_z0, stream)) != cudaSuccess) {
        set_error("band terms", e);
        return false;
    }
    last_launches += 2;

    // Rare redraw chunks of the area and its 8-chunk halo, found before the scan so that the
    // scan's hits can be filtered on the device.
    if ((e = cudaMemsetAsync(flags.ptr, 0, 16, stream)) != cudaSuccess ||
        (e = launch_rare_scan(rare_targets.ptr, rare_offsets.ptr, q.seed, area_z0 - 8, (int32_t)(H + 16),
                              area_x0 - 8, (int32_t)(W + 16), rare.ptr, kRareCap, flags.ptr + 2, stream)) != cudaSuccess ||
        (e = cudaMemcpyAsync(pinned, flags.ptr + 2, 4, cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
        (e = cudaStreamSynchronize(stream)) != cudaSuccess) {
        set_error("rare scan", e);
        return false;
    }
    ++last_launches;
    const uint32_t nrare = *(uint32_t*)pinned;
    if (nrare > kRareCap) { set_error("too many rare chunks", cudaErrorMemoryAllocation); return false; }
    last_rare = nrare;
    // The rare list sorted by x: the hit filter then binary-searches it.
    if (nrare > 1) {
        std::vector<int2> rl(nrare);
        if ((e = cudaMemcpyAsync(rl.data(), rare.ptr, (size_t)nrare * sizeof(int2), cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
            (e = cudaStreamSynchronize(stream)) != cudaSuccess) {
            set_error("rare list", e);
            return false;
        }
        std::sort(rl.begin(), rl.end(), [](const int2& a, const int2& b) { return a.x != b.x ? a.x < b.x : a.y < b.y; });
        if ((e = cudaMemcpyAsync(rare.ptr, rl.data(), (size_t)nrare * sizeof(int2), cudaMemcpyHostToDevice, stream)) != cudaSuccess ||
            (e = cudaStreamSynchronize(stream)) != cudaSuccess) {
            set_error("rare list", e);
            return false;
        }
    }

    const int64_t u_tiles = G.u_tiles, v_tiles = G.v_tiles;
    const int32_t band_h = G.band_h;
    const int grid = band_grid(G.planes, sm_count);
    const uint64_t cap = hits.count;
    // Count histogram on the device (first-draw counts of every centre in range, corrected for
    // rare chunks by the fix-up) and an emission gate (emission_gate); if it falls short, the scan runs
    // again with the exact gate the histogram gives.
    if ((e = hist.reserve(2 * kHistBins)) != cudaSuccess) { set_error("alloc", e); return false; }
    unsigned int* dhist = hist.ptr;
    int* ddelta = reinterpret_cast<int*>(hist.ptr + kHistBins);
    int32_t emit_min = emission_gate(q, q.max_results);

    for (int pass = 0; pass < 3; ++pass) {
        best.clear();
        std::fill(h.begin(), h.end(), 0u);
        if ((e = cudaMemsetAsync(dhist, 0, 2 * kHistBins * sizeof(unsigned int), stream)) != cudaSuccess) {
            set_error("band histogram", e);
            return false;
        }
        for (int64_t g = 0; g < ngroups; ++g) {
            const int32_t j0 = (int32_t)(g * nb_max);
            const int32_t nb = (int32_t)std::min<int64_t>(nb_max, nJ - j0);
            if (nb <= 0) break;
            const int64_t tiles = G.tiles;
            // At most 24 waves a launch. More sites expected than the hit buffer holds (an upper bound can stop the
            // gate where many share a count): as many even launches as it takes at four fifths of the buffer each. A
            // launch that overflows is run again in halves (radius 450,000, counts 38 to 40 2,273 ms, now 1,489);
            // one more than needed costs a wave (109,888, 41 to 46, 33 ms of kernel and 11 more).
            int64_t chunk = std::max<int64_t>(grid, std::min<int64_t>(tiles, (int64_t)grid * 24));
            const double sent = ((double)W * (double)H - 3.14159265358979 * (double)q.rd_min * (double)q.rd_min) *
                                (tail_share(emit_min) - tail_share(q.max_size + 1)) / (double)ngroups;
            if (sent > 0.95 * (double)cap) {
                const int64_t launches = (int64_t)std::ceil(sent / (0.8 * (double)cap));
                chunk = std::max<int64_t>(1, std::min<int64_t>(chunk, (tiles + launches - 1) / launches));
            }
            for (int64_t t0 = 0; t0 < tiles;) {
                while (paused.load() && !cancel.load()) std::this_thread::sleep_for(std::chrono::milliseconds(20));
                if (cancel.load()) { cancelled = true; return true; }
                const int64_t t1 = std::min(tiles, t0 + chunk);
                BandArgs a{};
                a.ct = xt.ptr;
                a.ncols = width_u + 16;
                a.rt = rt.ptr + (size_t)g * (band_row_table_words(G) / (size_t)ngroups);
                a.vrows = vrows;
                a.vbase = vbase;
                a.ubase = ubase;
                a.width_u = width_u;
                a.height_v = height_v;
                a.j0 = j0;
                a.nb = nb;
                a.u_tiles = (int32_t)u_tiles;
                a.v_tiles = (int32_t)v_tiles;
                a.band_h = band_h;
                a.tile_begin = t0;
                a.tile_end = t1;
                a.min_size = q.min_size;
                a.max_size = q.max_size;
                a.rd_min_sq = q.rd_min * q.rd_min;
                a.area_x0 = area_x0;
                a.area_z0 = area_z0;
                a.center_x = q.center_x;
                a.center_z = q.center_z;
                a.transposed = transposed ? 1 : 0;
                a.out = hits.ptr;
                a.cap = cap;
                a.emitted = counters.ptr;
                a.overflow = flags.ptr;
                a.indep = indep ? 1 : 0;
                a.groups = G.groups;
                a.exact = exact ? 1 : 0;
                a.joined = joined_windows(q.min_size);
                a.one = 1u;
                a.poll_limit = wait_polls;
                a.hist = dhist;
                a.emit_min = emit_min;
                a.row_stride = stride;
                const auto c0 = std::chrono::steady_clock::now();
                // A launch whose hits overflow the buffer is redone in halves: its histogram
                // counts are taken back first (snapshot before, restore after).
                if ((e = cudaMemcpyAsync(ddelta, dhist, kHistBins * sizeof(unsigned int), cudaMemcpyDeviceToDevice,
                                         stream)) != cudaSuccess ||
                    (e = cudaMemsetAsync(counters.ptr, 0, 8, stream)) != cudaSuccess ||
                    (e = cudaEventRecord(ev_a, stream)) != cudaSuccess ||
                    (e = launch_band_scan(a, (int)std::min<int64_t>(grid, t1 - t0), stream)) != cudaSuccess ||
                    (e = cudaEventRecord(ev_b, stream)) != cudaSuccess ||
                    (e = cudaMemcpyAsync(pinned, counters.ptr, 8, cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
                    (e = cudaStreamSynchronize(stream)) != cudaSuccess) {
                    set_error("band scan", e);
                    return false;
                }
                const auto c1 = std::chrono::steady_clock::now();
                float kms = 0.f;
                cudaEventElapsedTime(&kms, ev_a, ev_b);
                last_kernel_ms += kms;
                ++last_launches;
                const uint64_t emitted = *(unsigned long long*)pinned;
                if (emitted > cap) {
                    if (t1 - t0 <= 1) { set_error("band hit buffer overflow", cudaErrorMemoryAllocation); return false; }
                    if ((e = cudaMemcpyAsync(dhist, ddelta, kHistBins * sizeof(unsigned int), cudaMemcpyDeviceToDevice,
                                             stream)) != cudaSuccess) {
                        set_error("band histogram", e);
                        return false;
                    }
                    chunk = std::max<int64_t>(1, (t1 - t0) / 2);
                    continue;
                }
                work_ns.fetch_add(std::max<int64_t>(1, std::chrono::duration_cast<std::chrono::nanoseconds>(c1 - c0).count()));
                if (emitted) {
                    if ((e = launch_filter_hits(hits.ptr, (int64_t)emitted, rare.ptr, (int32_t)nrare, true, stream)) != cudaSuccess) {
                        set_error("filter", e);
                        return false;
                    }
                    if (nrare) ++last_launches;
                    const size_t old = best.size();
                    best.resize(old + emitted);
                    if ((e = cudaMemcpyAsync(best.data() + old, hits.ptr, emitted * sizeof(Hit), cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
                        (e = cudaStreamSynchronize(stream)) != cudaSuccess) {
                        set_error("copy", e);
                        return false;
                    }
                    size_t w = old;
                    for (size_t i = old; i < best.size(); ++i)
                        if (best[i].count >= 0) best[w++] = best[i];  // window holds a rare chunk: fixed below
                    best.resize(w);
                    if (best.size() > 2 * (size_t)q.max_results + 1000000) {
                        std::nth_element(best.begin(), best.begin() + q.max_results, best.end(),
                                         [](const Hit& x, const Hit& y) { return hit_order(x, y); });
                        best.resize(q.max_results);
                    }
                }
                const double done = ((double)g * tiles + (double)t1) / ((double)ngroups * tiles);
                processed.store((int64_t)(done * (double)W * (double)H));
                progress.store(1 + (int32_t)(done * 78));
                t0 = t1;
            }
        }

        // Exact counts of every centre whose window holds a rare redraw chunk, and the matching
        // correction of the histogram (first-draw count out, exact count in).
        if ((e = cudaMemsetAsync(ddelta, 0, kHistBins * sizeof(int), stream)) != cudaSuccess) {
            set_error("band histogram", e);
            return false;
        }
        if (nrare) {
            FixArgs f{};
            f.area_x0 = area_x0;
            f.area_z0 = area_z0;
            f.width = W;
            f.height = H;
            f.rd_min_sq = q.rd_min * q.rd_min;
            f.center_x = q.center_x;
            f.center_z = q.center_z;
            f.min_size = q.min_size;
            f.max_size = q.max_size;
            f.fixed = fixed.ptr;
            f.fixed_count = counters.ptr + 1;
            f.cap = fixed.count;
            f.error = flags.ptr + 1;
            f.hist_delta = ddelta;
            if ((e = cudaMemsetAsync(counters.ptr + 1, 0, 8, stream)) != cudaSuccess ||
                (e = launch_fixup(rare.ptr, (int32_t)nrare, q.seed, f, stream)) != cudaSuccess ||
                (e = cudaMemcpyAsync(pinned, counters.ptr + 1, 8, cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
                (e = cudaMemcpyAsync((char*)pinned + 8, flags.ptr, 8, cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
                (e = cudaStreamSynchronize(stream)) != cudaSuccess) {
                set_error("fixup", e);
                return false;
            }
            ++last_launches;
            const uint64_t nf = *(unsigned long long*)pinned;
            const uint32_t* fl = (const uint32_t*)((char*)pinned + 8);
            if (nf > fixed.count || fl[1]) { set_error("fixup overflow", cudaErrorUnknown); return false; }
            if (nf) {
                const size_t old = best.size();
                best.resize(old + nf);
                if ((e = cudaMemcpyAsync(best.data() + old, fixed.ptr, nf * sizeof(Hit), cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
                    (e = cudaStreamSynchronize(stream)) != cudaSuccess) {
                    set_error("copy", e);
                    return false;
                }
            }
        }
        if ((e = cudaMemcpyAsync(pinned, flags.ptr, 4, cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
            (e = cudaMemcpyAsync((char*)pinned + 64, dhist, 2 * kHistBins * sizeof(unsigned int), cudaMemcpyDeviceToHost,
                                 stream)) != cudaSuccess ||
            (e = cudaStreamSynchronize(stream)) != cudaSuccess) {
            set_error("flags", e);
            return false;
        }
        if (*(uint32_t*)pinned & 4u) { set_error("band engine: row-term copy timed out", cudaErrorLaunchTimeout); return false; }
        if (*(uint32_t*)pinned & 1u) {
            // A 4-row strip too dense for the byte-lane box: redo the search with the general scan.
            std::fill(h.begin(), h.end(), 0u);
            best.clear();
            return scan_general(q, best, h, cancelled);
        }
        const uint32_t* hs = (const uint32_t*)((const char*)pinned + 64);
        const int32_t* hd = (const int32_t*)(hs + kHistBins);
        for (int i = 0; i < kHistBins; ++i) h[i] = (uint64_t)((int64_t)hs[i] + hd[i]);
        uint64_t total = 0, have = 0;
        for (int c = q.min_size; c <= q.max_size; ++c) {
            total += h[c];
            if (c >= emit_min) have += h[c];
        }
        const uint64_t need = std::min<uint64_t>(total, (uint64_t)q.max_results);
        if (have >= need || emit_min <= q.min_size) {
            drop_below_gate(best, emit_min);
            return true;
        }
        // Too few sites sent: the exact gate (highest count whose cumulative number covers need).
        uint64_t acc = 0;
        int32_t gate = q.max_size;
        for (int c = q.max_size; c >= q.min_size; --c) {
            acc += h[c];
            gate = c;
            if (acc >= need) break;
        }
        emit_min = gate;
    }
    set_error("band gate did not converge", cudaErrorUnknown);
    return false;
}

}  // namespace slime
