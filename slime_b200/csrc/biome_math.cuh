// biome_math.cuh -- FP64 climate noise, depth spline and biome-tree search of the biome filter.
//
// Bit-exact restatement of the reference's biome module (gpu_noise/MinecraftGPUNoise.cu) with its
// floating-point operations in source order and no contraction: the file that includes this
// header is compiled with --fmad=false, so every double/float operation is one IEEE operation, as
// in the reference's source text (and as Minecraft's Java code computes them).
//
//   Xoroshiro128++ seeding and draws ........ MinecraftGPUNoise.cu:15-73
//   improved Perlin noise .................... :75-190
//   octave sets and double-Perlin climate .... :196-422
//   depth spline ............................. spline_generated.cuh (control points in biome_data.h)
//   parameter-tree nearest leaf .............. :650-809
//   quart climate and biome .................. :868-913
#pragma once

#include <cstdint>

#include "biome_data.h"

namespace slime {
namespace biome {

// ---- Xoroshiro128++ -------------------------------------------------------------------------

struct Xr {
    uint64_t lo, hi;
};

__host__ __device__ inline uint64_t rotl64(uint64_t x, unsigned b) { return (x << b) | (x >> (64u - b)); }

__host__ __device__ inline uint64_t mix13(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

// 64-bit seed to the 128-bit state (Java RandomSupport.upgradeSeedTo128bit).
__host__ __device__ inline Xr xr_seed(uint64_t seed) {
    const uint64_t lo = seed ^ 0x6a09e667f3bcc909ull;
    return Xr{mix13(lo), mix13(lo + 0x9e3779b97f4a7c15ull)};
}

__host__ __device__ inline uint64_t xr_next(Xr& s) {
    const uint64_t l = s.lo;
    uint64_t h = s.hi;
    const uint64_t out = rotl64(l + h, 17) + l;
    h ^= l;
    s.lo = rotl64(l, 49) ^ h ^ (h << 21);
    s.hi = rotl64(h, 28);
    return out;
}

// Java nextInt(bound): multiply-high of the low word, rejecting the biased low products.
__host__ __device__ inline uint32_t xr_next_int(Xr& s, uint32_t n) {
    uint64_t r = (xr_next(s) & 0xffffffffull) * (uint64_t)n;
    if ((uint32_t)r < n) {
        const uint32_t bound = (0u - n) % n;
        while ((uint32_t)r < bound) r = (xr_next(s) & 0xffffffffull) * (uint64_t)n;
    }
    return (uint32_t)(r >> 32);
}

__host__ __device__ inline double xr_next_double(Xr& s) { return (double)(xr_next(s) >> 11) * 0x1.0p-53; }

// ---- improved Perlin noise --------------------------------------------------------------------

// One octave of a noise: offsets, permutation, the y cell/fraction/fade for samples at y = 0,
// amplitude and lacunarity. 320 bytes; the 46 octaves of the six climate noises stay in shared
// memory during sampling.
struct Octave {
    double ox, oy, oz;
    double y_frac, y_fade;
    double amp, lac;
    uint8_t perm[257];
    uint8_t y_cell;
    uint8_t pad[6];
};

struct Noise {
    int32_t first, na, nb, pad;
    double amp;
};

// The six climate noises of a world seed (shift, temperature, humidity, continentalness,
// erosion, weirdness): 14.8 KB.
struct Climate {
    Noise noise[6];
    Octave oct[46];
};

enum { kShift = 0, kTemp = 1, kHumid = 2, kCont = 3, kEros = 4, kWeird = 5 };

__host__ __device__ inline double fade(double t) { return t * t * t * (t * (t * 6.0 - 15.0) + 10.0); }
__host__ __device__ inline double lerp(double t, double a, double b) { return a + t * (b - a); }

// Gradient dot product of improved noise for hash h: the 12 cube edges, 4 of them repeated, as u + v
// with u, v two of x, y, z and a sign each (u = x below 8, else y; v = y below 4, x at 12 and 14, else
// z; bit 0 negates u and bit 1 v). Selects and sign flips instead of a 12-way branch, which a warp ran
// nearly all of.
__device__ __forceinline__ double with_sign(double v, uint32_t flip) {
    return __hiloint2double(__double2hiint(v) ^ (int)flip, __double2loint(v));
}
__device__ __forceinline__ double grad(uint32_t h, double x, double y, double z) {
    const double u = h & 8u ? y : x;
    const double v = (h & 13u) == 12u ? x : h & 12u ? z : y;
    return with_sign(u, h << 31) + with_sign(v, (h << 30) & 0x80000000u);
}

// Octave set initialisation on the host (the permutation shuffle is serial): two seeds from the
// parent, then per non-zero amplitude an octave seeded with the hash of "octave_<k>".
void octave_set_init(Octave* out, Xr& parent, const double* amp, int first, int n, int* count);

__device__ __forceinline__ double perlin_sample(const Octave& p, double x, double y, double z) {
    uint32_t hy;
    double ty;
    if (y == 0.0) {
        y = p.y_frac;
        hy = p.y_cell;
        ty = p.y_fade;
    } else {
        y += p.oy;
        const double cy = floor(y);
        y -= cy;
        hy = (uint8_t)(int)cy;
        ty = fade(y);
    }
    x += p.ox;
    z += p.oz;
    const double cx = floor(x), cz = floor(z);
    x -= cx;
    z -= cz;
    const uint32_t hx = (uint8_t)(int)cx, hz = (uint8_t)(int)cz;
    const double tx = fade(x), tz = fade(z);
    const uint8_t* d = p.perm;
    const uint32_t a1 = (uint8_t)(d[hx] + hy), b1 = (uint8_t)(d[hx + 1] + hy);
    const uint32_t a2 = (uint8_t)(d[a1] + hz), b2 = (uint8_t)(d[b1] + hz);
    const uint32_t a3 = (uint8_t)(d[a1 + 1] + hz), b3 = (uint8_t)(d[b1 + 1] + hz);
    const double x1 = x - 1.0, y1 = y - 1.0, z1 = z - 1.0;
    double l1 = grad(d[a2], x, y, z), l2 = grad(d[b2], x1, y, z);
    double l3 = grad(d[a3], x, y1, z), l4 = grad(d[b3], x1, y1, z);
    double l5 = grad(d[a2 + 1], x, y, z1), l6 = grad(d[b2 + 1], x1, y, z1);
    double l7 = grad(d[a3 + 1], x, y1, z1), l8 = grad(d[b3 + 1], x1, y1, z1);
    l1 = lerp(tx, l1, l2);
    l3 = lerp(tx, l3, l4);
    l5 = lerp(tx, l5, l6);
    l7 = lerp(tx, l7, l8);
    l1 = lerp(ty, l1, l3);
    l5 = lerp(ty, l5, l7);
    return lerp(tz, l1, l5);
}

// The two octave sets of a noise, the second at 337/331 of the position. One loop body for both: the
// seven samples of a quart column would otherwise inline it fourteen times.
__device__ __forceinline__ double noise_sample(const Climate& c, int s, double x, double y, double z) {
    const Noise& n = c.noise[s];
    const double f = 337.0 / 331.0;
    double v = 0.0;
#pragma unroll 1
    for (int set = 0; set < 2; ++set) {
        const Octave* o = c.oct + n.first + (set ? n.na : 0);
        const int count = set ? n.nb : n.na;
        double acc = 0.0;
#pragma unroll 1
        for (int i = 0; i < count; ++i) {
            const double l = o[i].lac;
            const double p = perlin_sample(o[i], x * l, y * l, z * l);
            acc += o[i].amp * p;
        }
        v = set ? v + acc : acc;
        x *= f;
        y *= f;
        z *= f;
    }
    return v * n.amp;
}

// ---- depth spline ---------------------------------------------------------------------------

struct SplinePt {
    float loc, der, val;
    int32_t child;  // -1: constant value
};

struct SplineHead {
    int32_t coord, first, count, pad;
};

// Cubic Hermite segments between control points, linear outside (cubiomes getSpline); values of
// points may be child splines, evaluated to depth LEVEL.
template <int LEVEL>
__device__ __forceinline__ float spline_eval(const SplineHead* heads, const SplinePt* pts, int s, const float* v);

template <int LEVEL>
__device__ __forceinline__ float spline_value(const SplineHead* heads, const SplinePt* pts, const SplinePt& p,
                                              const float* v) {
    if constexpr (LEVEL <= 0) {
        return p.val;
    } else {
        return p.child < 0 ? p.val : spline_eval<LEVEL - 1>(heads, pts, p.child, v);
    }
}

template <int LEVEL>
__device__ __forceinline__ float spline_eval(const SplineHead* heads, const SplinePt* pts, int s, const float* v) {
    const SplineHead hd = heads[s];
    const SplinePt* p = pts + hd.first;
    const float f = v[hd.coord];
    if (f <= p[0].loc) return spline_value<LEVEL>(heads, pts, p[0], v) + p[0].der * (f - p[0].loc);
    for (int i = 1; i < hd.count; ++i) {
        const float h = p[i].loc;
        if (f > h) continue;
        const float g = p[i - 1].loc;
        const float k = (f - g) / (h - g);
        const float l = p[i - 1].der, m = p[i].der;
        const float v0 = spline_value<LEVEL>(heads, pts, p[i - 1], v);
        const float v1 = spline_value<LEVEL>(heads, pts, p[i], v);
        const float pp = l * (h - g) - (v1 - v0);
        const float q = -m * (h - g) + (v1 - v0);
        const double a = lerp((double)k, (double)v0, (double)v1);
        const float kk = k * (1.0f - k);
        const double b = lerp((double)k, (double)pp, (double)q);
        return (float)(a + (double)kk * b);
    }
    const SplinePt& last = p[hd.count - 1];
    return spline_value<LEVEL>(heads, pts, last, v) + last.der * (f - last.loc);
}

__device__ __forceinline__ float peaks_valleys(float w) {
    return -(fabsf(fabsf(w) - 0.6666667f) - 0.33333334f) * 3.0f;
}

// Climate of quart column (x, z): the quantised {T, H, C, E, W} (x 1e4, truncated) and the float
// depth offset of the spline; the depth parameter of quart Y y is depth_at(offset, y).
struct Column {
    int32_t t, h, c, e, w;
    float off;
};

template <int SPLINE_LEVELS>
__device__ __forceinline__ Column column_climate(const Climate& cl, const SplineHead* heads, const SplinePt* pts,
                                                 int32_t xi, int32_t zi) {
    const double x = (double)xi, z = (double)zi;
    double at[2];  // shifted position
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
        const double d = noise_sample(cl, kShift, k ? z : x, k ? x : 0.0, k ? 0.0 : z) * 4.0;
        at[0] = k ? at[0] : x + d;
        at[1] = z + d;
    }
    float v[6];  // by noise, kTemp .. kWeird
#pragma unroll 1
    for (int s = kTemp; s <= kWeird; ++s) {
        const float d = (float)noise_sample(cl, s, at[0], 0.0, at[1]);
#pragma unroll
        for (int k = kTemp; k <= kWeird; ++k) v[k] = s == k ? d : v[k];
    }
    const float c = v[kCont], e = v[kEros], w = v[kWeird], t = v[kTemp], h = v[kHumid];
    const float in[4] = {c, e, peaks_valleys(w), w};
    Column col;
    col.off = spline_eval<SPLINE_LEVELS>(heads, pts, 0, in) + 0.015f;
    col.t = (int32_t)(10000.0f * t);
    col.h = (int32_t)(10000.0f * h);
    col.c = (int32_t)(10000.0f * c);
    col.e = (int32_t)(10000.0f * e);
    col.w = (int32_t)(10000.0f * w);
    return col;
}

__device__ __forceinline__ int32_t depth_at(float off, int32_t y) {
    const double d0 = 1.0 - ((double)(y * 4)) / 128.0 - 83.0 / 160.0 + (double)off;
    const float d = (float)d0;
    return (int32_t)(10000.0f * d);
}

// ---- biome parameter tree -------------------------------------------------------------------

// Tree geometry (device copy of a BdTree's scalars); nodes and parameter ranges live in device
// memory / shared memory.
struct TreeGeom {
    int32_t order, depth, nnodes, nparams;
    int32_t steps[8];
};

// Distance of v to the range r along one axis. kWide: exact for every int32 v (64-bit
// differences); otherwise 32-bit differences, exact while |v| <= 2^30 (range bounds are within
// +-12,000, so no difference overflows).
template <bool kWide>
__device__ __forceinline__ uint32_t axis_gap(int32_t v, int2 r) {
    if constexpr (kWide) {
        return (uint32_t)(v > r.y ? (int64_t)v - r.y : v < r.x ? (int64_t)r.x - v : 0);
    } else {
        return (uint32_t)max(max(r.x - v, v - r.y), 0);
    }
}

// The squared distance sum of one node's box plus g^2 (squares of 32-bit gaps, summed in 64 bits,
// as the reference's int64 / uint64 arithmetic gives for these magnitudes).
__device__ __forceinline__ uint64_t add_sq(uint64_t acc, uint32_t g) { return acc + (uint64_t)g * g; }

// A node word: parameter indices of the six axes in bytes 0..5 (depth in byte 4), then the first
// child's node index, or a leaf's biome id. `order` children lie steps[d] apart below a node at tree
// depth d; a node whose subtree would run past the end descends in place.
template <bool kWide>
__device__ __forceinline__ uint64_t node_d2(uint64_t node, const int2* __restrict__ param, const int32_t (&p)[6]) {
    uint64_t d = 0;
#pragma unroll
    for (int a = 0; a < 6; ++a) d = add_sq(d, axis_gap<kWide>(p[a], param[(node >> (8 * a)) & 0xff]));
    return d;
}
__host__ __device__ __forceinline__ int node_depth(const TreeGeom& g, int32_t node, int d) {
    while (d < g.depth && node + g.steps[d] >= g.nnodes) ++d;
    return d;
}

// Index of the nearest leaf of parameters p (temperature, humidity, continentalness, erosion, depth,
// weirdness): the reference's branch and bound (MinecraftGPUNoise.cu:686-809). A child is entered
// when its box is strictly closer than the best leaf, and a leaf replaces the best only when strictly
// closer, so with boxes that enclose their leaves the answer is the first of the nearest leaves.
template <bool kWide>
__device__ __forceinline__ int32_t tree_nearest_impl(const uint64_t* __restrict__ nodes, const int2* __restrict__ param,
                                                     const TreeGeom& g, const int32_t (&p)[6]) {
    constexpr int kMaxDepth = 8;
    uint64_t ds = ~0ull;
    int32_t best = 0;
    // Stack level: next child (bits 0-15), children left (16-23), tree depth (24-31).
    uint32_t st_node[kMaxDepth];
    int sp = 0;
    st_node[0] = (uint32_t)((nodes[0] >> 48) & 0xffff) | ((uint32_t)g.order << 16) | ((uint32_t)node_depth(g, 0, 0) << 24);
    while (sp >= 0) {
        const uint32_t top = st_node[sp];
        const int32_t child = (int32_t)(top & 0xffff);
        const int left = (int)((top >> 16) & 0xff), d = (int)(top >> 24);
        if (left <= 0 || child >= g.nnodes) {
            --sp;
            continue;
        }
        st_node[sp] = (uint32_t)(child + g.steps[d]) | ((uint32_t)(left - 1) << 16) | ((uint32_t)d << 24);
        const uint64_t node = nodes[child];
        const uint64_t dist = node_d2<kWide>(node, param, p);
        if (dist >= ds) continue;
        const int cd = node_depth(g, child, d + 1);
        if (cd >= g.depth) {
            ds = dist;
            best = child;
            continue;
        }
        st_node[++sp] = (uint32_t)((node >> 48) & 0xffff) | ((uint32_t)g.order << 16) | ((uint32_t)cd << 24);
    }
    return best;
}

// The 32-bit-gap traversal when every coordinate is within +-2^30 (always, for climate values and
// the depths of quart Y within the world), else the 64-bit one; both give the same leaves.
__device__ __forceinline__ bool wide_params(const int32_t (&p)[6]) {
    constexpr int32_t kLim = 1 << 30;
    bool wide = false;
#pragma unroll
    for (int i = 0; i < 6; ++i) wide |= p[i] > kLim || p[i] < -kLim;
    return wide;
}
__device__ __forceinline__ int32_t tree_biome(const uint64_t* __restrict__ nodes, const int2* __restrict__ param,
                                              const TreeGeom& g, const int32_t (&p)[6]) {
    const int32_t leaf = wide_params(p) ? tree_nearest_impl<true>(nodes, param, g, p)
                                        : tree_nearest_impl<false>(nodes, param, g, p);
    return (int32_t)((nodes[leaf] >> 48) & 0xff);
}

// Leaves of one biome (at most kTargetMax of them), for a verdict "is the nearest leaf one of these".
constexpr int kTargetMax = 4;
struct Targets {
    int32_t n;
    int32_t leaf[kTargetMax];
};

// Whether the nearest leaf of parameters p is a leaf of `t`. The nearest of t's own leaves sets a
// bound, and the search only asks whether any other leaf is nearer (or as near and earlier in leaf
// order, which is the order the reference visits them in): it ends at the first one. At each node all
// children are measured and the nearest is followed first, so that a column far from the biome's
// climate ends after one descent (about 30 node distances; the full search for the nearest leaf of
// 18 depths took 168,000 instructions a warp, noise included). `killer`: a leaf to try first, and the
// leaf that ended the search.
template <bool kWide>
__device__ __forceinline__ bool tree_wins_impl(const uint64_t* __restrict__ nodes, const int2* __restrict__ param,
                                               const TreeGeom& g, const int32_t (&p)[6], const Targets& t, int32_t& killer) {
    constexpr int kMaxDepth = 8;
    uint64_t bound = ~0ull;
    int32_t first = 0;  // the target leaf at `bound`
    for (int i = 0; i < t.n; ++i) {  // ascending leaves: the first of the nearest
        const uint64_t dist = node_d2<kWide>(nodes[t.leaf[i]], param, p);
        if (dist < bound) {
            bound = dist;
            first = t.leaf[i];
        }
    }
    // Nearer than the bound, or as near and earlier (a subtree's leaves come after its own index).
    auto beats = [&](uint64_t dist, int32_t node) { return dist < bound || (dist == bound && node < first); };
    if (killer >= 0 && beats(node_d2<kWide>(nodes[killer], param, p), killer)) return false;
    // Stack level: first child (bits 0-15), tree depth (16-23); the children still to enter.
    uint32_t st_node[kMaxDepth], st_todo[kMaxDepth];
    int sp = -1;
    int32_t inner = (int32_t)((nodes[0] >> 48) & 0xffff);
    int d = node_depth(g, 0, 0);
    bool measure = true;
    uint32_t todo = 0;
    int pick = 0;
    for (;;) {
        if (measure) {  // children that can hold a leaf that beats the bound, and the nearest of them
            todo = 0;
            uint64_t nearest = ~0ull;
#pragma unroll 2
            for (int k = 0; k < g.order; ++k) {
                const int32_t child = inner + k * g.steps[d];
                if (child >= g.nnodes) break;
                const uint64_t dist = node_d2<kWide>(nodes[child], param, p);
                if (!beats(dist, child)) continue;
                todo |= 1u << k;
                if (dist < nearest) {
                    nearest = dist;
                    pick = k;
                }
            }
            measure = false;
        }
        if (!todo) {
            if (sp < 0) return true;
            inner = (int32_t)(st_node[sp] & 0xffff);
            d = (int)(st_node[sp] >> 16);
            todo = st_todo[sp--];
            pick = __ffs(todo) - 1;
        }
        const int32_t child = inner + pick * g.steps[d];
        todo &= ~(1u << pick);
        const int cd = node_depth(g, child, d + 1);
        if (cd >= g.depth) {
            bool own = false;
            for (int i = 0; i < t.n; ++i) own |= t.leaf[i] == child;
            if (!own) {
                killer = child;
                return false;
            }
            pick = __ffs(todo) - 1;
            continue;
        }
        if (todo) {
            st_node[++sp] = (uint32_t)inner | ((uint32_t)d << 16);
            st_todo[sp] = todo;
        }
        inner = (int32_t)((nodes[child] >> 48) & 0xffff);
        d = cd;
        measure = true;
    }
}
__device__ __forceinline__ bool tree_wins(const uint64_t* __restrict__ nodes, const int2* __restrict__ param,
                                          const TreeGeom& g, const int32_t (&p)[6], const Targets& t, int32_t& killer) {
    return wide_params(p) ? tree_wins_impl<true>(nodes, param, g, p, t, killer)
                          : tree_wins_impl<false>(nodes, param, g, p, t, killer);
}

}  // namespace biome
}  // namespace slime
