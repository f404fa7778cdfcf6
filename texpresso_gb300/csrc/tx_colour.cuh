// tx_colour.cuh -- per-block device code for BC1/BC2/BC3 colour endpoints and
// the BC2/BC3 alpha halves, shared by the single-texture kernels (tx_colour.cu)
// and the persistent batch kernel (tx_batch.cu).
//
// Two execution shapes (and a third, for large ClusterFit launches of BC2 and BC3,
// in tx_cluster_lanes.cuh):
//   thread-per-block  ColourSet, SingleColourFit and RangeFit are short and
//                     branch-light; a thread owns a block and 32 neighbouring
//                     blocks load as four coalesced 512-byte rows.
//   team-per-block    ClusterFit: a team of TEAM lanes (16 or 32) owns a block.
//                     Lane p owns pixel p for ColourSet; the candidates (967
//                     least-squares fits at 16 colours) are spread over the
//                     team: each gets a bound of its error, only those
//                     the bound cannot exclude get the reference's exact error
//                     (see sweep4 and, for compress3, cand_bound), and the lexicographic minimum on (error,
//                     position in the reference's loop order) selects exactly
//                     the candidate the sequential "first strictly smaller
//                     error" loop selects.
// Both reproduce the reference's f32 operation order (see tx_device.cuh).
// The constant tables are TU-local: every translation unit that includes this
// header uploads its own copy with upload_tables_this_tu().
#pragma once
#include "tx_device.cuh"

namespace tx {

// Single-colour tables (lib/src/colourfit/single_lut.rs): [table][target], x and
// y for the two indices, packed start | end << 8 | error << 16.  Tables: 0 = 5_3,
// 1 = 6_3, 2 = 5_4, 3 = 6_4.  (Neighbouring blocks look up different colours, which
// constant memory would serve one after another.)
static __device__ uint2 g_lut[4][256];

// compress3's candidate list.  Entry bits: 0-3 i (offset of S(0,i)),
// 4-11 offset of S(i,j), 20-29 rank of (i,j) in the reference's loop order at
// 16 colours, so comparing entries compares loop positions.
// Entries are sorted so that the first N[n] are exactly the candidates of an
// n-colour set (those with max(i+1, j) <= n).
constexpr int kCand4 = 967, kCand3 = 151;
static __device__ uint32_t g_cand[kCand3 + 1];
static __constant__ uint32_t c_ncand3[17];
// Position, in the list an n-colour set uses, of its candidate with every
// point in one cluster, (0,n).
static __constant__ uint16_t c_one3[17];
// The same candidates in the reference's loop order (i, j nested), used for
// 16-colour sets: a round of consecutive candidates then mostly shares S(0,i)
// and reads S(i,j) at consecutive addresses.
static __device__ uint32_t g_cand16[kCand3 + 1];
// Lower-bound terms (F1, r, C, S offsets) of the g_cand16 candidates of a
// 16-colour set whose weights are all exactly 1 (the w lanes of the partial
// sums are then the counts i, j-i), from the reference's f32 alpha2,
// beta2, alphabeta (see unit_terms and unit_bound).  The w lane holds the
// bits i | S(i,j) << 8 (table offsets, one byte each).
static __device__ float4 g_ub3[kCand3 + 1];
// The pairs (j, k), 0 <= j <= k <= n, k > 0, of compress4's candidates (i, j, k)
// of an n-colour set, j | k << 5, j ascending: neighbouring pairs then take the
// same i (0 .. min(j, n - 1)).
constexpr int kPairs = 152;
static __device__ uint16_t g_pairs[17][kPairs];
// unorm8(v) for every byte v and sqrt(n) for n <= 16 (filled by k_unorm_tables
// with the same correctly rounded division and square root as the kernels).
static __device__ float g_unorm8[256];
static __device__ float g_sqrt_count[17];

// Partial-sum table S(a,b), 0 <= a <= b <= 16, stored as the upper triangle
// row by row: S(a,b) at tri_idx(a,b) (153 entries).
__host__ __device__ constexpr int tri_idx(int a, int b) { return a * (33 - a) / 2 + b; }
constexpr int kTri = tri_idx(16, 16) + 1;

// ===========================================================================
// Shared pieces

// Bit i of a 16-bit mask at bits 2 i and 2 i + 1.
__device__ __forceinline__ uint32_t both_bits(uint32_t m) {
    m = (m | m << 8) & 0x00FF00FFu;
    m = (m | m << 4) & 0x0F0F0F0Fu;
    m = (m | m << 2) & 0x33333333u;
    m = (m | m << 1) & 0x55555555u;
    return m * 3u;
}

// SingleColourFit::compute_endpoints (single.rs:58-106) for the RGB bytes of rgb.
// Its endpoints v / 31 and v / 63 are packed again as round(31 x) and round(63 x),
// which is v, so they stay integers: start and end as 5:6:5, error, and index (0 or
// 2).  The first index of the smaller error is taken.
struct Single {
    uint32_t err, start, end, index;
};
__device__ __forceinline__ Single single_endpoints(uint32_t rgb, int t5, int t6) {
    const uint2 r = __ldg(&g_lut[t5][rgb & 0xFFu]), g = __ldg(&g_lut[t6][(rgb >> 8) & 0xFFu]),
                b = __ldg(&g_lut[t5][(rgb >> 16) & 0xFFu]);
    auto error = [](uint32_t x, uint32_t y, uint32_t z) {
        x = (x >> 16) & 0xFFu; y = (y >> 16) & 0xFFu; z = (z >> 16) & 0xFFu;
        return x * x + y * y + z * z;
    };
    const uint32_t e0 = error(r.x, g.x, b.x), e1 = error(r.y, g.y, b.y);
    const bool second = e1 < e0;
    const uint32_t x = second ? r.y : r.x, y = second ? g.y : g.x, z = second ? b.y : b.x;
    return Single{second ? e1 : e0, (x & 0xFFu) << 11 | (y & 0xFFu) << 5 | (z & 0xFFu),
                  ((x >> 8) & 0xFFu) << 11 | ((y >> 8) & 0xFFu) << 5 | ((z >> 8) & 0xFFu), second ? 2u : 0u};
}

// SingleColourFit + ColourFit::compress (colourfit.rs:44-60) given the colour.
// One block in ten of a textured image has a single colour, so nearly every warp
// of the thread-per-block kernels comes here: with divisions and float packing it
// took a third of RangeFit's time (2048x2048, noisy ramps: BC3 RangeFit 49.4 -> 40.6
// us, BC1 62.0 -> 43.6; BC1 IterativeClusterFit 1,336 -> 1,242).
template <int FMT>
__device__ __forceinline__ uint2 single_fit(uint32_t rgb, uint32_t valid16, bool transparent) {
    const uint32_t out3 = both_bits(~valid16 & 0xFFFFu);  // 3 for pixels that take no part
    auto indices = [&](uint32_t index) { return out3 | (index ? 0xAAAAAAAAu : 0u); };
    uint32_t best_err = 0xFFFFFFFFu;
    uint2 best = make_uint2(0u, 0u);
    if (FMT == BC1) {
        const Single f = single_endpoints(rgb, 0, 1);  // LOOKUP_5_3, 6_3, 5_3
        best = write3(f.start, f.end, indices(f.index));
        best_err = f.err;
    }
    if (FMT != BC1 || !transparent) {
        const Single f = single_endpoints(rgb, 2, 3);  // LOOKUP_5_4, 6_4, 5_4
        if (f.err < best_err) best = write4(f.start, f.end, indices(f.index));
    }
    return best;
}

// Sym3x3::principle_component (math.rs:75-97); only lanes x,y,z matter.
__device__ __forceinline__ void principle_component(const float (&m)[6], float (&v)[3]) {
    float vx = 1.0f, vy = 1.0f, vz = 1.0f;
#pragma unroll 1
    for (int it = 0; it < 8; ++it) {
        float wx = m[0] * vx, wy = m[1] * vx, wz = m[2] * vx;
        wx = m[1] * vy + wx; wy = m[3] * vy + wy; wz = m[4] * vy + wz;
        wx = m[2] * vz + wx; wy = m[4] * vz + wy; wz = m[5] * vz + wz;
        const float a = fmaxf(wx, fmaxf(wy, wz));
        const float r = rcp_rn(a);
        vx = wx * r; vy = wy * r; vz = wz * r;
    }
    v[0] = vx; v[1] = vy; v[2] = vz;
}

// Clamp to [0,1] and snap to the 5:6:5 grid (range.rs:87-98, cluster.rs:206-210).
__device__ __forceinline__ float snap(float x, float grid, float gridrcp) {
    x = fminf(1.0f, fmaxf(0.0f, x));
    return truncf(grid * x + 0.5f) * gridrcp;
}

__device__ __forceinline__ uint32_t u8_of(uint32_t px, int c) { return (px >> (8 * c)) & 0xFFu; }

// ===========================================================================
// k_range: one thread per block

// Per-thread point store for the thread-per-block path: pixel i of thread t
// lives at pts[i * stride + t] as (x, y, z, weight), so a warp's loads of one
// pixel are 512 contiguous bytes (no bank conflicts) and the fit keeps only
// accumulators in registers.
struct PointCol {
    float4 *base;
    int stride;
    __device__ __forceinline__ float4 &operator[](int i) const { return base[i * stride]; }
};

// The duplicate search of ColourSet::new (colourset.rs:82-102) for one block:
// each pixel's point is the first pixel with its key, and a point's pixel
// count is one plus the later pixels that join it.  res (4 words) receives
// byte p = pixel p's point index | (count - 1) << 4 (the count half is kept
// for points only).  Keys: the RGB of a valid pixel, or 0x01000000 | p for a
// pixel that is not (so it matches nothing).
__device__ __forceinline__ void colour_dedup(const uint32_t (&key)[16], uint32_t (&res)[4]) {
    // One comparison per pair j < i: it moves i's point down to j (the last
    // assignment, at the smallest j, wins) and counts i as a later pixel of
    // j's colour in the high nibble of byte j.  Every shift is a constant.
    uint32_t cnt[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int w = 0; w < 4; ++w) res[w] = 0u;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        uint32_t r = (uint32_t)i;
#pragma unroll
        for (int j = i - 1; j >= 0; --j) {
            const bool e = key[j] == key[i];
            r = e ? (uint32_t)j : r;
            cnt[j >> 2] += e ? (0x10u << (8 * (j & 3))) : 0u;
        }
        res[i >> 2] |= r << (8 * (i & 3));
    }
#pragma unroll
    for (int w = 0; w < 4; ++w) res[w] |= cnt[w];
}

// Point index and (pixel count - 1) of pixel i from colour_dedup's bytes.
__device__ __forceinline__ uint32_t dd_rep(const uint32_t (&res)[4], int i) { return (res[i >> 2] >> (8 * (i & 3))) & 0xFu; }
__device__ __forceinline__ uint32_t dd_dup(const uint32_t (&res)[4], int i) {
    return (res[i >> 2] >> (8 * (i & 3) + 4)) & 0xFu;
}

// One thread's colour set (colourset.rs:35-141), pixel-indexed: a "point" is
// the first pixel of its colour, and pixel order is point order.
struct ColourSet {
    uint32_t valid;    // pixels taking part
    uint32_t newbits;  // pixels that are points
    uint32_t dd[4];    // byte p: pixel p's point | (its colour's pixel count - 1) << 4
    int count;         // points
    bool transparent;
};

// px is overwritten with the colour-set keys (the RGB bytes of every valid
// pixel are kept; alpha is not needed after the packed copy a4), so the pixels
// and the keys never occupy registers at the same time.
template <int FMT>
__device__ __forceinline__ void colour_set_thread(uint32_t (&px)[16], uint32_t inb, bool alpha_weighted,
                                                  uint32_t (&a4)[4], ColourSet &cs) {
    uint32_t tbits = 0;
    if (FMT == BC1) {
#pragma unroll
        for (int i = 0; i < 16; ++i) tbits |= ((px[i] >> 31) ^ 1u) << i;
        tbits &= inb;
    }
    const uint32_t valid = inb & ~tbits;
    cs.valid = valid;
    cs.transparent = tbits != 0;
    if (alpha_weighted) channel_words(px, 3, a4);
#pragma unroll
    for (int i = 0; i < 16; ++i) px[i] = ((valid >> i) & 1u) ? (px[i] & 0xFFFFFFu) : (0x01000000u | (uint32_t)i);
    colour_dedup(px, cs.dd);
    // a valid pixel that is its own point starts a new point (excluded pixels
    // match nothing, so they are their own "point" too and are masked out)
    uint32_t newbits = 0;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const uint32_t eq = bytes_eq(cs.dd[w] & 0x0F0F0F0Fu, 0x03020100u + 0x04040404u * (uint32_t)w);
        newbits |= (((eq & 0x08040201u) * 0x01010101u) >> 24) << (4 * w);
    }
    cs.newbits = newbits & valid;
    cs.count = __popc(cs.newbits);
}

// The block of a one-colour set (px as colour_set_thread leaves it).
template <int FMT>
__device__ __forceinline__ uint2 single_thread(const uint32_t (&px)[16], const ColourSet &cs) {
    uint32_t rgb = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) rgb |= ((cs.valid >> i) & 1u) ? px[i] : 0u;
    return single_fit<FMT>(rgb, cs.valid, cs.transparent);
}

// Points and weights.  Pixels that are not points get weight exactly 0,
// which makes their terms +-0 in every ordered sum below.  Those sums start
// at +0 and add non-negative values (total, centroid) or can only reach
// zero as +0 (round-to-nearest x + (-x) = +0), so they are never -0 and
// adding +-0 leaves them unchanged: the sums equal the reference's sums
// over points.
__device__ __forceinline__ void colour_points_thread(const uint32_t (&px)[16], const uint32_t (&a4)[4],
                                                     const ColourSet &cs, bool alpha_weighted, const float *s_unorm,
                                                     const float *s_sqrt, const PointCol &pt) {
    if (!alpha_weighted) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float w = ((cs.newbits >> i) & 1u) ? s_sqrt[1 + (int)dd_dup(cs.dd, i)] : 0.0f;
            pt[i] = make_float4(s_unorm[u8_of(px[i], 0)], s_unorm[u8_of(px[i], 1)], s_unorm[u8_of(px[i], 2)], w);
        }
    } else {
        // alpha weights (colourset.rs:69-74, :94-97): every valid pixel adds
        // (a + 1) / 256 to its point's weight in pixel order, the point's own
        // pixel first (0 + w = w); an excluded pixel adds +0 to its own slot,
        // which stays +0.  Then sqrt for the points.
#pragma unroll
        for (int j = 0; j < 16; ++j)
            pt[j] = make_float4(s_unorm[u8_of(px[j], 0)], s_unorm[u8_of(px[j], 1)], s_unorm[u8_of(px[j], 2)], 0.0f);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float wa = ((cs.valid >> i) & 1u)
                                 ? (float)(((a4[i >> 2] >> (8 * (i & 3))) & 0xFFu) + 1u) * (1.0f / 256.0f)
                                 : 0.0f;
            float &w = pt[(int)dd_rep(cs.dd, i)].w;
            w = w + wa;
        }
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if ((cs.newbits >> j) & 1u) pt[j].w = sqrt_rn(pt[j].w);
    }
}

// Sym3x3::weighted_covariance (math.rs:44-73) of a thread's points.
__device__ __forceinline__ void covariance_thread(const PointCol &pt, float (&m)[6]) {
    float total = 0.0f, cx = 0.0f, cy = 0.0f, cz = 0.0f;
#pragma unroll 4
    for (int i = 0; i < 16; ++i) {
        const float4 q = pt[i];
        total = total + q.w;
        cx = cx + q.x * q.w; cy = cy + q.y * q.w; cz = cz + q.z * q.w;
    }
    if (total > FLT_EPSILON) { cx = div_rn(cx, total); cy = div_rn(cy, total); cz = div_rn(cz, total); }
#pragma unroll
    for (int c = 0; c < 6; ++c) m[c] = 0.0f;
#pragma unroll 4
    for (int i = 0; i < 16; ++i) {
        const float4 q = pt[i];
        const float ax = q.x - cx, ay = q.y - cy, az = q.z - cz;
        const float bx = ax * q.w, by = ay * q.w, bz = az * q.w;
        m[0] += ax * bx; m[1] += ax * by; m[2] += ax * bz;
        m[3] += ay * by; m[4] += ay * bz; m[5] += az * bz;
    }
}

// remap_indices (colourset.rs:130-141): 2-bit code of every point's pixel ->
// code of every pixel, 3 for the excluded ones.  With 16 distinct valid
// pixels every pixel is its own point and the map is the identity.
__device__ __forceinline__ uint32_t remap_thread(const ColourSet &cs, uint32_t closest) {
    if (cs.newbits == 0xFFFFu) return closest;
    uint32_t out = 0;
#pragma unroll
    for (int p = 0; p < 16; ++p) {
        const uint32_t r = dd_rep(cs.dd, p);
        const uint32_t v = ((cs.valid >> p) & 1u) ? ((closest >> (2 * r)) & 3u) : 3u;
        out |= v << (2 * p);
    }
    return out;
}

// Colour set, points and weights of RangeFit (colourset.rs:35-141).  A pixel with
// the colour of its point gets the point's index by itself, so only the first
// pixel of every colour (a point) and the number of its pixels are needed.
//
// The 120 comparisons are arithmetic: ISETP, SEL and IADD share a pipe of half the
// rate of FADD and FFMA.  A pixel's RGB under the exponent of 2^23 or 2^24 is a
// float of its own (pixels that take no part have others above them), so the
// difference of two is 0, or at least 1 in size, and 1 - d^2 saturates to 1 or 0.
// t counts the later pixels of the colour, and 32 for every earlier one.  (BC3
// 4096x4096 128 -> 123 us, BC1 2048x2048 43.6 -> 41.6.)
template <int FMT>
__device__ __forceinline__ void range_points_thread(uint32_t (&px)[16], uint32_t inb, bool alpha_weighted,
                                                    const float *s_unorm, const float *s_sqrt, const PointCol &pt,
                                                    uint32_t &valid, uint32_t &newbits) {
    uint32_t tbits = 0;
    if (FMT == BC1) {
#pragma unroll
        for (int i = 0; i < 16; ++i) tbits |= ((px[i] >> 31) ^ 1u) << i;
    }
    valid = inb & ~tbits;
    uint32_t a4[4];  // alpha of pixel 4r + c at byte c of a4[r] (alpha weighting only)
    if (alpha_weighted) channel_words(px, 3, a4);
    float t[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const bool in = (valid >> i) & 1u;
        px[i] = in ? (px[i] & 0xFFFFFFu) | 0x4B000000u : 0x4C000000u | (uint32_t)i;
        t[i] = in ? 0.0f : 32.0f;
    }
    auto same = [&](int i, int j) {  // 1 or 0
        const float d = __uint_as_float(px[i]) - __uint_as_float(px[j]);
        float e;
        asm("fma.rn.sat.f32 %0, %1, %2, 0f3F800000;" : "=f"(e) : "f"(-d), "f"(d));
        return e;
    };
    if (!alpha_weighted) {
#pragma unroll
        for (int i = 1; i < 16; ++i)
#pragma unroll
            for (int j = 0; j < i; ++j) {
                const float e = same(i, j);
                t[j] += e;
                t[i] = __fmaf_rn(e, 32.0f, t[i]);
            }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            // at most 15 later pixels; entry 17 is 0, for pixels that are no points
            const float w = s_sqrt[1 + (int)(__float_as_uint(fminf(t[i], 16.0f) + 8388608.0f) & 31u)];
            pt[i] = make_float4(s_unorm[u8_of(px[i], 0)], s_unorm[u8_of(px[i], 1)], s_unorm[u8_of(px[i], 2)], w);
        }
    } else {
        // (a + 1) / 256 of the colour's pixels, added in pixel order, and the root
        // (colourset.rs:69-74, :94-97); 0 of another colour's leaves the sum as it is
        float w[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            w[i] = ((valid >> i) & 1u) ? (float)(((a4[i >> 2] >> (8 * (i & 3))) & 0xFFu) + 1u) * (1.0f / 256.0f) : 0.0f;
#pragma unroll
            for (int j = 0; j < i; ++j) {
                const float e = same(i, j);
                w[j] = __fmaf_rn(e, w[i], w[j]);
                t[i] = __fmaf_rn(e, 32.0f, t[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < 16; ++i)
            pt[i] = make_float4(s_unorm[u8_of(px[i], 0)], s_unorm[u8_of(px[i], 1)], s_unorm[u8_of(px[i], 2)],
                                t[i] < 32.0f ? sqrt_rn(w[i]) : 0.0f);
    }
    newbits = 0;
#pragma unroll
    for (int i = 15; i >= 0; --i) newbits = __funnelshift_l(__float_as_uint(t[i] - 32.0f), newbits, 1);
}

template <int FMT>
__device__ __forceinline__ uint2 colour_range_thread(uint32_t (&px)[16], uint32_t inb,
                                                     const DevParams &prm, const float *s_unorm,
                                                     const float *s_sqrt, const PointCol &pt) {
    uint32_t valid, newbits;
    range_points_thread<FMT>(px, inb, prm.alpha_weighted, s_unorm, s_sqrt, pt, valid, newbits);
    const int count = __popc(newbits);
    const bool transparent = FMT == BC1 && valid != inb;
    if (count == 1) {
        uint32_t rgb = 0;
#pragma unroll
        for (int i = 0; i < 16; ++i) rgb |= ((newbits >> i) & 1u) ? px[i] : 0u;
        return single_fit<FMT>(rgb, valid, transparent);
    }
    float m[6];
    covariance_thread(pt, m);
    float axis[3];
    principle_component(m, axis);

    // RangeFit::new (range.rs:44-101): the first point starts both ends; a later
    // point moves start on a strictly smaller dot, else end on a strictly larger one
    float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, e0 = 0.0f, e1 = 0.0f, e2 = 0.0f;
    if (count > 0) {
        bool seen = false;
        float mn = 0.0f, mx = 0.0f;
        int si = 0, ei = 0;
#pragma unroll 4
        for (int i = 0; i < 16; ++i) {
            const float4 q = pt[i];
            const bool p = (newbits >> i) & 1u;
            const float d = q.x * axis[0] + q.y * axis[1] + q.z * axis[2];
            const bool first = p && !seen;
            const bool lo = first || (p && d < mn);
            const bool hi = first || (p && !(d < mn) && d > mx);
            si = lo ? i : si; mn = lo ? d : mn;
            ei = hi ? i : ei; mx = hi ? d : mx;
            seen = seen || p;
        }
        const float4 qs = pt[si], qe = pt[ei];
        s0 = qs.x; s1 = qs.y; s2 = qs.z;
        e0 = qe.x; e1 = qe.y; e2 = qe.z;
    }
    s0 = snap(s0, 31.0f, 1.0f / 31.0f); s1 = snap(s1, 63.0f, 1.0f / 63.0f); s2 = snap(s2, 31.0f, 1.0f / 31.0f);
    e0 = snap(e0, 31.0f, 1.0f / 31.0f); e1 = snap(e1, 63.0f, 1.0f / 63.0f); e2 = snap(e2, 31.0f, 1.0f / 31.0f);

    const float w0 = prm.w[0], w1 = prm.w[1], w2 = prm.w[2];
    const uint32_t out3 = valid == 0xFFFFu ? 0u : both_bits(~valid & 0xFFFFu);  // 3 for pixels that take no part
    const uint32_t a565 = pack_565(s0, s1, s2), b565 = pack_565(e0, e1, e2);
    const float c23 = 2.0f / 3.0f, c13 = 1.0f / 3.0f;
    const float cr4[4] = {s0, e0, s0 * c23 + e0 * c13, s0 * c13 + e0 * c23};
    const float cg4[4] = {s1, e1, s1 * c23 + e1 * c13, s1 * c13 + e1 * c23};
    const float cb4[4] = {s2, e2, s2 * c23 + e2 * c13, s2 * c13 + e2 * c23};

    // BC2 and BC3 need the nearest codes only (BC1 compares the errors of two
    // codebooks).  The codes lie on a line, so the nearest one follows from a
    // point's position q = g . (x - s) on it (0 at s, 1 at e): from 3 q rounded,
    // unless that is within `near` of a rounding boundary, where the reference's own
    // rounding decides and the point is measured.
    //
    // Rounding (R = 2^-24): a distance D to a code is off by 7.1 R D, and by 8 R Om
    // sqrt(D), Om^2 = sum w^2, because codes are rounded (4 R); all D <= G^2 = sum
    // of w_c^2 (8 var_c / wmin + 2 / 62^2) + L^2 (L the length of the line; points
    // are within sqrt(var_c / wmin) of the mean, endpoints within half a grid step
    // of points).  Between neighbouring codes D changes by 2 L^2 / 3 over a step, so
    // 3 q decides but for 9 (7.1 R G^2 + 8 R Om G) / L^2, and is itself off by 3 (8
    // R Om / L + 6 R): near = R ((64 G^2 + 100 Om G) / L^2 + 60).
    //
    // 9 instructions a point where measuring four codes takes 60 (BC3 2048x2048 of
    // noisy ramps 40.6 -> 37.4 us, of smooth fields 40.6 -> 38.3).  With BC1, whose
    // sums of distances would have to be told apart too, ramps gained as much, but
    // smooth fields lost 20 %: there the two codebooks are often that close.
    if (FMT != BC1) {
        auto ordinary = [](float w) { w = fabsf(w); return w == 0.0f || (w >= 0x1p-20f && w <= 0x1p20f); };
        const bool usual = ordinary(w0) && ordinary(w1) && ordinary(w2);
        if (usual && a565 == b565) return write4(a565, b565, 0u);  // (which sets the indices to 0)
        const float dr = e0 - s0, dg = e1 - s1, db = e2 - s2;
        const float ww0 = w0 * w0, ww1 = w1 * w1, ww2 = w2 * w2;
        const float L2 = __fmaf_rn(ww0 * dr, dr, __fmaf_rn(ww1 * dg, dg, (ww2 * db) * db));
        const float wv = prm.alpha_weighted ? 8.1f * 16.0f : 8.1f;  // a weight is at least 1, or sqrt(1 / 256)
        const float G2 = __fmaf_rn(ww0, __fmaf_rn(wv, m[0], 5.3e-4f), __fmaf_rn(ww1, __fmaf_rn(wv, m[3], 5.3e-4f),
                                   __fmaf_rn(ww2, __fmaf_rn(wv, m[5], 5.3e-4f), L2)));
        float omG, iL2;
        asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(omG) : "f"((ww0 + ww1 + ww2) * G2));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(iL2) : "f"(L2));
        const float near = 5.9604645e-8f * __fmaf_rn(__fmaf_rn(64.0f, G2, 100.0f * omG), iL2, 60.0f);
        if (usual && L2 > 0.0f && near < 0.25f) {
            const float gx = ww0 * dr * iL2, gy = ww1 * dg * iL2, gz = ww2 * db * iL2;
            const float q0 = -__fmaf_rn(gx, s0, __fmaf_rn(gy, s1, gz * s2));
            const float M = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer
            float pos[2] = {0.f, 0.f};    // positions in base 4
            uint32_t todo = 0;            // bit i: point i is in doubt
#pragma unroll
            for (int h = 1; h >= 0; --h)
#pragma unroll 4
                for (int i = 8 * h + 7; i >= 8 * h; --i) {
                    const float4 q = pt[i];
                    const float t = __saturatef(__fmaf_rn(gx, q.x, __fmaf_rn(gy, q.y, __fmaf_rn(gz, q.z, q0))));
                    const float k = __fmaf_rn(t, 3.0f, M) - M;
                    pos[h] = __fmaf_rn(pos[h], 4.0f, k);
                    todo = __funnelshift_l(__float_as_uint(0.5f - near - fabsf(__fmaf_rn(t, 3.0f, -k))), todo, 1);
                }
            const uint32_t p = (uint32_t)pos[0] | (uint32_t)pos[1] << 16;
            const uint32_t hi = (p >> 1) & 0x55555555u, lo = p & 0x55555555u;
            uint32_t closest = ((hi ^ lo) << 1) | hi;  // positions 0 .. 3 are codes 0 2 3 1
            todo &= valid;
#pragma unroll 1
            while (todo) {
                const int i = __ffs((int)todo) - 1;
                todo &= todo - 1u;
                const float4 q = pt[i];
                float dist = FLT_MAX;
                uint32_t idx = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float dx = w0 * (q.x - cr4[j]), dy = w1 * (q.y - cg4[j]), dz = w2 * (q.z - cb4[j]);
                    const float d = dx * dx + dy * dy + dz * dz;
                    idx = d < dist ? (uint32_t)j : idx;
                    dist = d < dist ? d : dist;
                }
                closest = (closest & ~(3u << (2 * i))) | idx << (2 * i);
            }
            return write4(a565, b565, closest | out3);
        }
    }

    float best_err = FLT_MAX;
    uint2 best = make_uint2(0u, 0u);

    // compression_helper (range.rs:103-143) over a codebook of nc codes.  The
    // error sum adds +0 for pixels that are not points (it starts at +0 and
    // its terms are non-negative).
    // The weighted differences w (x - c) of codes (0,1) and (2,3) are formed
    // in pairs by the paired f32 operations add2_rn / mul2_rn (each lane the
    // IEEE operation of the scalar form, x - c being x + (-c); an add followed
    // by a multiply leaves nothing to fuse).  The squares and their sum stay
    // scalar: a paired multiply followed by a paired add was contracted into
    // a fused multiply-add even when written with .rn, which changes the
    // rounding.  So every distance is the reference's
    // ((w0 (x - cr))^2 + (w1 (y - cg))^2) + (w2 (z - cb))^2.
    const float2 W0 = make_float2(w0, w0), W1 = make_float2(w1, w1), W2 = make_float2(w2, w2);
    auto helper = [&](const float (&cr)[4], const float (&cg)[4], const float (&cb)[4], int nc,
                      uint32_t &indices) -> bool {
        const float2 nr01 = make_float2(-cr[0], -cr[1]), nr23 = make_float2(-cr[2], -cr[3]);
        const float2 ng01 = make_float2(-cg[0], -cg[1]), ng23 = make_float2(-cg[2], -cg[3]);
        const float2 nb01 = make_float2(-cb[0], -cb[1]), nb23 = make_float2(-cb[2], -cb[3]);
        uint32_t closest = 0;
        float err = 0.0f;
#pragma unroll 4
        for (int i = 0; i < 16; ++i) {
            const float4 q = pt[i];
            const float2 X = make_float2(q.x, q.x), Y = make_float2(q.y, q.y), Z = make_float2(q.z, q.z);
            const float2 dx01 = mul2_rn(W0, add2_rn(X, nr01)), dx23 = mul2_rn(W0, add2_rn(X, nr23));
            const float2 dy01 = mul2_rn(W1, add2_rn(Y, ng01)), dy23 = mul2_rn(W1, add2_rn(Y, ng23));
            const float2 dz01 = mul2_rn(W2, add2_rn(Z, nb01)), dz23 = mul2_rn(W2, add2_rn(Z, nb23));
            const float dx[4] = {dx01.x, dx01.y, dx23.x, dx23.y}, dy[4] = {dy01.x, dy01.y, dy23.x, dy23.y};
            const float dz[4] = {dz01.x, dz01.y, dz23.x, dz23.y};
            float d[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) d[j] = dx[j] * dx[j] + dy[j] * dy[j] + dz[j] * dz[j];
            float dist = FLT_MAX;
            uint32_t idx = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (j < nc) {
                    idx = d[j] < dist ? (uint32_t)j : idx;
                    dist = d[j] < dist ? d[j] : dist;
                }
            }
            closest |= idx << (2 * i);
            err = err + (((newbits >> i) & 1u) ? dist : 0.0f);
        }
        if (err < best_err) {
            indices = closest | out3;
            best_err = err;
            return true;
        }
        return false;
    };

    if (FMT == BC1) {
        const float cr[4] = {s0, e0, s0 * 0.5f + e0 * 0.5f, 0.0f};
        const float cg[4] = {s1, e1, s1 * 0.5f + e1 * 0.5f, 0.0f};
        const float cb[4] = {s2, e2, s2 * 0.5f + e2 * 0.5f, 0.0f};
        uint32_t idx;
        if (helper(cr, cg, cb, 3, idx)) best = write3(a565, b565, idx);
    }
    if (FMT != BC1 || !transparent) {
        uint32_t idx;
        if (helper(cr4, cg4, cb4, 4, idx)) best = write4(a565, b565, idx);
    }
    return best;
}

__device__ __forceinline__ void init_unorm_tables(float *s_unorm, float *s_sqrt) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) s_unorm[i] = unorm8((uint32_t)i);
    if (threadIdx.x < 18) s_sqrt[threadIdx.x] = threadIdx.x < 17 ? sqrt_rn((float)threadIdx.x) : 0.0f;
    __syncthreads();
}

// The same tables in global memory (one CTA of 256 threads).
static __global__ void k_unorm_tables() {
    g_unorm8[threadIdx.x] = unorm8(threadIdx.x);
    if (threadIdx.x < 17) g_sqrt_count[threadIdx.x] = sqrt_rn((float)threadIdx.x);
}

// ===========================================================================
// k_cluster: one team per block

template <int TEAM>
struct Team {
    unsigned mask;
    int lane;
    int base;
    __device__ __forceinline__ Team() {
        const int wl = threadIdx.x & 31;
        lane = wl & (TEAM - 1);
        base = wl & ~(TEAM - 1);
        mask = (TEAM == 32) ? 0xFFFFFFFFu : (0xFFFFu << base);
    }
    __device__ __forceinline__ unsigned ballot(bool p) const {
        const unsigned b = __ballot_sync(mask, p);
        return (TEAM == 32) ? b : ((b >> base) & 0xFFFFu);
    }
    __device__ __forceinline__ bool all(bool p) const { return __all_sync(mask, p); }
    template <class T> __device__ __forceinline__ T shfl(T v, int src) const { return __shfl_sync(mask, v, src, TEAM); }
    template <class T> __device__ __forceinline__ T shfl_up(T v, int d) const { return __shfl_up_sync(mask, v, d, TEAM); }
    __device__ __forceinline__ void sync() const { __syncwarp(mask); }
    __device__ __forceinline__ float least(float v) const {
        float r;
        asm volatile("redux.sync.min.f32 %0, %1, %2;" : "=f"(r) : "f"(v), "r"(mask));
        return r;
    }
    __device__ __forceinline__ unsigned match(uint32_t key) const {
        const unsigned m = __match_any_sync(mask, key);
        return (TEAM == 32) ? m : ((m >> base) & 0xFFFFu);
    }
};

struct __align__(16) TeamSmem {
    float4 S[kTri + 3];     // S(a,b) running sums at tri_idx(a,b) (+pad)
    float4 Q[17];           // compress4: centred prefix sums and prefix weights of the ordering
    float G[17];            // compress4: the bound's terms of i
    union {                 // lifetimes do not overlap within an iteration:
        float LB[kCand3 + 9];   // compress3: candidate lower bounds, then the survivor queue; scratch
        uint16_t queue[kCand4 + 1];  // compress4: the candidates to evaluate, i << 10 | j << 5 | k
        struct {
            float4 PW[16];      // points_weights in the current ordering
            uint32_t D[16];     // sort keys of the dot products
        };
    };
    float P[4][16];         // x, y, z, weight of each point, point order
    uint32_t hist[8][4];    // orderings of earlier iterations (16 bytes each)
};

// Sym3x3::principle_component (math.rs:75-97) for a team: lane c < 3 forms
// component c of each product M v in the reference's order (row 0 times vx,
// then row 1 times vy added, then row 2 times vz), and every lane takes the
// three components by shuffle for the max and the scaling.
template <int TEAM>
__device__ __forceinline__ void principle_component_team(const Team<TEAM> &tm, const float (&m)[6], float (&v)[3]) {
    const int c = tm.lane < 3 ? tm.lane : 0;
    const float a0 = c == 0 ? m[0] : (c == 1 ? m[1] : m[2]);
    const float a1 = c == 0 ? m[1] : (c == 1 ? m[3] : m[4]);
    const float a2 = c == 0 ? m[2] : (c == 1 ? m[4] : m[5]);
    float vx = 1.0f, vy = 1.0f, vz = 1.0f;
#pragma unroll 1
    for (int it = 0; it < 8; ++it) {
        float w = a0 * vx;
        w = a1 * vy + w;
        w = a2 * vz + w;
        const float wx = tm.shfl(w, 0), wy = tm.shfl(w, 1), wz = tm.shfl(w, 2);
        const float r = rcp_rn(fmaxf(wx, fmaxf(wy, wz)));
        vx = wx * r; vy = wy * r; vz = wz * r;
    }
    v[0] = vx; v[1] = vy; v[2] = vz;
}

// Sort key of cluster.rs:90-97 as an unsigned integer: finite values keep
// their order (-0 and +0 tie), every non-finite value ties after all finite
// ones.  Comparing keys is comparing with fcmp.
__device__ __forceinline__ uint32_t dps_key(float x) {
    if (!isfinite(x)) return 0xFFFFFFFFu;
    const uint32_t u = (uint32_t)__float_as_int(x + 0.0f);  // -0 -> +0
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// min(1, max(0, fl(a * b))) in one instruction: mul.rn with .sat clamps the
// rounded product to [0, 1] and turns NaN into +0, as f32::max/min do in
// cluster.rs:207-208 (max(0, NaN) = 0).
__device__ __forceinline__ float mul_sat(float a, float b) {
    float d;
    asm("mul.rn.sat.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}

// Snap a value already clamped to [0, 1] to the grid (cluster.rs:209-210).
__device__ __forceinline__ float snap01(float x, float grid, float gridrcp) {
    return truncf(grid * x + 0.5f) * gridrcp;
}

__device__ __forceinline__ uint8_t hist_get(const TeamSmem &sm, int it, int m) {
    return reinterpret_cast<const uint8_t *>(sm.hist[it])[m];
}

// Weight-lane terms of one compress4 candidate (cluster.rs:320-335).
__device__ __forceinline__ float4 wterms4(float p0w, float p1w, float p2w, float xsw) {
    const float c19 = 1.0f / 9.0f, c49 = 4.0f / 9.0f, c29 = 2.0f / 9.0f;
    const float p3w = xsw - p2w - p1w - p0w;
    const float alpha2 = p2w * c19 + (p1w * c49 + p0w);
    const float beta2 = p1w * c19 + (p2w * c49 + p3w);
    const float ab = c29 * (p1w + p2w);
    return make_float4(alpha2, beta2, ab, rcp_rn((alpha2 * beta2) - ab * ab));
}

// Weight-lane terms of one compress3 candidate (cluster.rs:189-202).  The
// products part1 * (.5, .25) are exact, so each sum is one fused op.
__device__ __forceinline__ float4 wterms3(float p0w, float p1w, float xsw) {
    const float p2w = xsw - p1w - p0w;
    const float alpha2 = __fmaf_rn(p1w, 0.25f, p0w);
    const float beta2 = __fmaf_rn(p1w, 0.25f, p2w);
    const float ab = p1w * 0.25f;
    return make_float4(alpha2, beta2, ab, rcp_rn((alpha2 * beta2) - ab * ab));
}

// Endpoint fit and error of one candidate given its x/y/z sums ax, bx and its
// weight-lane terms wt (cluster.rs:200-220, :333-353).
template <bool WANT_AB>
__device__ __forceinline__ float fit_error(const float (&ax)[3], const float (&bx)[3], const float4 wt,
                                           const float (&cw)[3], float (&ea)[3], float (&eb)[3]) {
    const float alpha2 = wt.x, beta2 = wt.y, ab = wt.z, factor = wt.w;
    const float grid[3] = {31.0f, 63.0f, 31.0f};
    const float gridrcp[3] = {1.0f / 31.0f, 1.0f / 63.0f, 1.0f / 31.0f};
    float e5[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float a = snap01(mul_sat((ax[c] * beta2) - bx[c] * ab, factor), grid[c], gridrcp[c]);
        const float b = snap01(mul_sat((bx[c] * alpha2) - ax[c] * ab, factor), grid[c], gridrcp[c]);
        const float e1 = (a * a) * alpha2 + (b * b * beta2);
        const float e2 = (a * b * ab) - a * ax[c];
        const float e3 = e2 - b * bx[c];
        const float e4 = __fmaf_rn(2.0f, e3, e1);  // 2*e3 is exact, so this equals fl(fl(2*e3) + e1)
        e5[c] = e4 * cw[c];
        if (WANT_AB) { ea[c] = a; eb[c] = b; }
    }
    return e5[0] + e5[1] + e5[2];
}

// One compress4 candidate (cluster.rs:320-353); wt = wterms4(...) of its w lanes.
template <bool WANT_AB>
__device__ __forceinline__ float eval4(const float4 p0, const float4 p1, const float4 p2, const float4 xs,
                                       const float4 wt, const float (&cw)[3], float (&ea)[3], float (&eb)[3]) {
    const float c13 = 1.0f / 3.0f, c23 = 2.0f / 3.0f;
    const float p3x = xs.x - p2.x - p1.x - p0.x;
    const float p3y = xs.y - p2.y - p1.y - p0.y;
    const float p3z = xs.z - p2.z - p1.z - p0.z;
    const float ax[3] = {p2.x * c13 + (p1.x * c23 + p0.x), p2.y * c13 + (p1.y * c23 + p0.y),
                         p2.z * c13 + (p1.z * c23 + p0.z)};
    const float bx[3] = {p1.x * c13 + (p2.x * c23 + p3x), p1.y * c13 + (p2.y * c23 + p3y),
                         p1.z * c13 + (p2.z * c23 + p3z)};
    return fit_error<WANT_AB>(ax, bx, wt, cw, ea, eb);
}

// One compress3 candidate (cluster.rs:189-220); wt = wterms3(...) of its w lanes.
template <bool WANT_AB>
__device__ __forceinline__ float eval3(const float4 p0, const float4 p1, const float4 xs, const float4 wt,
                                       const float (&cw)[3], float (&ea)[3], float (&eb)[3]) {
    const float p2x = xs.x - p1.x - p0.x, p2y = xs.y - p1.y - p0.y, p2z = xs.z - p1.z - p0.z;
    const float ax[3] = {__fmaf_rn(p1.x, 0.5f, p0.x), __fmaf_rn(p1.y, 0.5f, p0.y), __fmaf_rn(p1.z, 0.5f, p0.z)};
    const float bx[3] = {__fmaf_rn(p1.x, 0.5f, p2x), __fmaf_rn(p1.y, 0.5f, p2y), __fmaf_rn(p1.z, 0.5f, p2z)};
    return fit_error<WANT_AB>(ax, bx, wt, cw, ea, eb);
}

// Decode (i, j) from a candidate entry of compress3.
__host__ __device__ __forceinline__ void decode_entry(uint32_t e, int &i, int &j) {
    i = (int)(e & 0xFu);
    j = (int)((e >> 4) & 0xFFu) - tri_idx(i, 0);
}

// ---------------------------------------------------------------------------
// Candidate pruning of compress3.  For a candidate with weight-lane terms alpha, beta,
// gamma (> 0 definite) and per-channel sums ax, bx, the reference's error at
// any endpoints (a, b) is  sum_c w_c Q_c(a_c, b_c)  with
//     Q(a, b) = alpha a^2 + beta b^2 + 2 gamma a b - 2 a ax - 2 b bx
// (cluster.rs:345-353, evaluated in f32).  Q is minimised over all real (a, b)
// by the unclamped least-squares endpoints, where it equals
//     -q,  q = (beta ax^2 - 2 gamma ax bx + alpha bx^2) / det,
// so no clamping or grid snapping can bring the error below -sum_c w_c q_c.
// With bx = X - ax (X_c the channel sums) and A = alpha + beta + 2 gamma,
// B = alpha + gamma, the numerator summed over channels is
//     sum_c w_c q_c det = A sum_c w_c ax_c^2 - 2B sum_c w_c X_c ax_c + alpha Z,
// Z = sum_c w_c X_c^2 being the same for every candidate of the block.  The
// bound is evaluated in that form with cheaper arithmetic than the reference
// (FMA, an approximate reciprocal), and the difference to the reference's f32
// error is covered by a margin (weights w_c >= 0, all sums non-negative,
// W = weight sum, u = 2^-24):
//   * rounding of the reference's own error evaluation, and using f32
//     weight-lane terms that differ from its by a few ulps: <= 36 u W sum(w);
//   * our ax (and X - ax) within 16 u X of the reference's ax, bx, moving the
//     minimum by at most 32 u X (|A*| + |B*|) <= 32 u f W X^2, plus rounding of
//     the three sums, their combination and f: <= 26 u f W Z;
// so  E_ref >= -f (sum_c w_c q_c det + Kb) - eps1  with  Kb = 2^-17 W Z and
// eps1 = 2^-17 W sum w_c (128 u, about twice the derived terms) + 1e-30, for
// weights so small that products with them leave the normal range: each is then off
// by up to 2^-150, at most 2^30 times that in the bound.
// A candidate whose bound exceeds an error some candidate actually reaches
// can neither win nor tie, so the exact sweep only needs the others.  The
// result is the reference's choice bit for bit; only the work changes.

// Bound terms (A, -2B, alpha, 1/det) from the w lanes of the partial sums, for
// blocks whose weights are not all 1 (no table entry applies).
__device__ __forceinline__ float4 lb_terms(float p0w, float p1w, float xsw) {
    const float p2r = xsw - p0w - p1w;
    const float al = __fmaf_rn(p1w, 0.25f, p0w);
    const float be = __fmaf_rn(p1w, 0.25f, p2r);
    const float g2 = 0.5f * p1w;
    // det = al*be - g*g with the product g*g split exactly (its rounding error
    // recovered by an FMA), so det carries only the final roundings
    const float g = 0.5f * g2;
    const float gg = g * g;
    const float gerr = __fmaf_rn(g, g, -gg);
    const float det = __fmaf_rn(al, be, -gg) - gerr;
    float f;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"(det));
    return make_float4(al + be + g2, -(2.0f * al + g2), al, det > 0.0f ? f : __int_as_float(0x7fc00000));  // NaN: no bound
}

// Per-block constants of the bound: w_c X_c, Z = sum_c w_c X_c^2, Kb, eps1.
struct BoundBlock {
    float wx[3], z, kb, eps1;
};

__device__ __forceinline__ BoundBlock bound_block(const float4 xs, const float (&cw)[3]) {
    BoundBlock bb;
    bb.wx[0] = cw[0] * xs.x;
    bb.wx[1] = cw[1] * xs.y;
    bb.wx[2] = cw[2] * xs.z;
    float z = 0.0f;
    z = __fmaf_rn(cw[0], xs.x * xs.x, z);
    z = __fmaf_rn(cw[1], xs.y * xs.y, z);
    z = __fmaf_rn(cw[2], xs.z * xs.z, z);
    bb.z = z;
    bb.kb = 7.62939453125e-6f * xs.w * z;                          // 2^-17 W Z
    bb.eps1 = __fmaf_rn(7.62939453125e-6f * xs.w, cw[0] + cw[1] + cw[2], 1e-30f);  // 2^-17 W sum w, + 1e-30
    return bb;
}

// -f (A sum w ax^2 - 2B sum w X ax + alpha Z + Kb) - eps1 for one candidate;
// lt = (A, -2B, alpha, f).
__device__ __forceinline__ float cand_bound(const float4 p0, const float4 p1, const float4 lt,
                                            const float (&cw)[3], const BoundBlock &bb) {
    const float pa[3] = {p0.x, p0.y, p0.z}, pb[3] = {p1.x, p1.y, p1.z};
    float ax[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) ax[c] = __fmaf_rn(pb[c], 0.5f, pa[c]);
    float s1 = (cw[0] * ax[0]) * ax[0];
    s1 = __fmaf_rn(cw[1] * ax[1], ax[1], s1);
    s1 = __fmaf_rn(cw[2] * ax[2], ax[2], s1);
    float s2 = bb.wx[0] * ax[0];
    s2 = __fmaf_rn(bb.wx[1], ax[1], s2);
    s2 = __fmaf_rn(bb.wx[2], ax[2], s2);
    const float acc = __fmaf_rn(lt.x, s1, __fmaf_rn(lt.y, s2, __fmaf_rn(lt.z, bb.z, bb.kb)));
    return __fmaf_rn(-lt.w, acc, -bb.eps1);  // NaN when there is no bound: the candidate is kept
}

// The same bound for a 16-colour set of weight-1 points (W = 16), with the
// candidate's constants folded into q = (F1, r, C) = (-A f, 2B / A,
// -f (alpha + 2^-13)) (double, rounded once): since
//     -f (A s1 - 2B s2) = F1 sum_c w_c ax_c (ax_c - r X_c)
// and -f (alpha Z + Kb) = C Z (Kb = 2^-17 W Z = 2^-13 Z), the bound is
//     F1 sum_c w_c ax_c (ax_c - r X_c) + C Z - eps1.
// Rounding: A = W exactly, 0 <= r <= 2, so each of the three products is at
// most 2 w_c X_c^2 in size and the sum carries at most ~10 u Z; with the
// rounding of F1, r, C and the two final FMAs that is <= ~17 u f W Z, inside
// the 26 u f W Z budgeted for the general form above.
__device__ __forceinline__ float unit_bound(const float4 p0, const float4 p1, const float4 q, const float4 xs, const float (&cw)[3], const BoundBlock &bb) {
    const float pa[3] = {p0.x, p0.y, p0.z}, pb[3] = {p1.x, p1.y, p1.z};
    const float X[3] = {xs.x, xs.y, xs.z};
    float sum = 0.0f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float ax = __fmaf_rn(pb[c], 0.5f, pa[c]);
        const float d = __fmaf_rn(-q.y, X[c], ax);
        sum = c == 0 ? (cw[0] * ax) * d : __fmaf_rn(cw[c] * ax, d, sum);
    }
    return __fmaf_rn(q.x, sum, __fmaf_rn(q.z, bb.z, -bb.eps1));  // NaN when there is no bound
}

// Per-lane best of the candidates a lane evaluated exactly: error, entry and
// endpoints, compared lexicographically on (error, entry).
struct LaneBest {
    float err;
    uint32_t ent;
    float a[3], b[3];
};

// Exact error and endpoints of the compress3 candidate entry e (cluster.rs:189-220),
// folded into the lane's best.
__device__ __forceinline__ void eval_candidate(const TeamSmem &sm, uint32_t e, const float4 xs, const float (&cw)[3],
                                               LaneBest &lb) {
    float a[3], b[3];
    const float4 p0 = sm.S[e & 0xFu];
    const float4 p1 = sm.S[(e >> 4) & 0xFFu];
    const float err = eval3<true>(p0, p1, xs, wterms3(p0.w, p1.w, xs.w), cw, a, b);
    if (err < lb.err || (err == lb.err && e < lb.ent)) {
        lb.err = err;
        lb.ent = e;
#pragma unroll
        for (int c = 0; c < 3; ++c) { lb.a[c] = a[c]; lb.b[c] = b[c]; }
    }
}

// The same for compress4 candidate i << 10 | j << 5 | k (cluster.rs:315-372).
__device__ __forceinline__ void eval_key(const TeamSmem &sm, uint32_t e, const float4 xs, const float (&cw)[3],
                                         LaneBest &lb) {
    float a[3], b[3];
    const int i = (int)(e >> 10), j = (int)((e >> 5) & 31u), k = (int)(e & 31u);
    const float4 p0 = sm.S[i], p1 = sm.S[tri_idx(i, j)], p2 = sm.S[tri_idx(j, k)];
    const float err = eval4<true>(p0, p1, p2, xs, wterms4(p0.w, p1.w, p2.w, xs.w), cw, a, b);
    if (err < lb.err || (err == lb.err && e < lb.ent)) {
        lb.err = err;
        lb.ent = e;
#pragma unroll
        for (int c = 0; c < 3; ++c) { lb.a[c] = a[c]; lb.b[c] = b[c]; }
    }
}

// compress4's candidates of one ordering of n points (cluster.rs:315-372): folds
// them into the team's bests ob.  part: those that the bound excludes may be left
// out; var: weighted variances per channel; guess: i | j << 5 | k << 10.
//
// A lane takes a pair (j, k) and all its i.  With Q(t), w(t) the centred prefix
// sums and the prefix weights of the ordering, candidate (i, j, k) can only reach
// an error of thr if
//     s = |Q(i) + V|^2 / 2 + tol - c den >= 0,   V = Q(j) + Q(k)
// (bound, c, den and rounding terms: tx_cluster_lanes.cuh), which is one addition
// and four fused multiply-adds per candidate:
//     s = P + G(i) + V . Q(i) + 2 c a w(i),   a = w(j) + w(k),
//     P = |V|^2 / 2 + c (a (a - W) - 2 W w(j)) + tol,
//     G(i) = |Q(i)|^2 / 2 + c w(i) (w(i) - 5 W).
// Q is scaled by the square roots of the channel weights.  tol = 512 W T R covers
// the 75 for these sums, the 204 for the prefixes and 16 for the scaling; eps is
// the one for |a|, |b| <= 1 (121 W sum w_c R; 128 is taken).  Channel weights
// below 2^-60 count as zero in the bound: all of their error, at most 128 w_c, is
// in eps.  thr is the least error of the candidates around a guess.
//
// Bound by instruction issue and fetch, like all of the team form.  The bounds of
// a block take 350 warp instructions and their set-up 200, where bounds from the
// table S, a candidate per lane, with a division unless a table held the terms
// for weights of 1, took 1,020 (1,490).  BC1 256x256 28.6 -> 22.2 us, 2048x2048
// 969 -> 829, iterative 1,535 -> 1,338; BC3 900x900 of noisy ramps 155 -> 128,
// of smooth fields 362 -> 352 (there nearly all candidates have to be evaluated).
// A grid filter for such blocks (as in tx_cluster_lanes.cuh) cost the noisy ramps
// 15 % in place and 6 % as a function of its own, for 9 % on smooth fields.
template <int TEAM>
__device__ __forceinline__ void sweep4(const Team<TEAM> &tm, TeamSmem &sm, int n, const float4 xs, const float (&cw)[3],
                                       const float (&var)[3], bool part, uint32_t guess, LaneBest &ob) {
    const int lane = tm.lane;
    float c = 0.f, tol = 0.f;
    if (part) {
        const int gi = (int)(guess & 31u), gj = (int)((guess >> 5) & 31u), gk = (int)(guess >> 10);
#pragma unroll 1
        for (int t = lane; t < 32; t += TEAM) {
            const int t3 = t * 11 >> 5, t9 = t * 57 >> 9;  // t / 3, t / 9
            const int i = min(max(gi + (t - 3 * t3) - 1, 0), n - 1);
            const int j = min(max(gj + (t3 - 3 * t9) - 1, i), n);
            const int k = min(max(gk + t9 - 1, max(j, 1)), n);
            eval_key(sm, (uint32_t)(i << 10 | j << 5 | k), xs, cw, ob);
        }
        const float thr = tm.least(ob.err);
        float T = 0.f, z = 0.f, sum = 0.f, tiny = 0.f, sq[3];
        const float X[3] = {xs.x, xs.y, xs.z};
#pragma unroll
        for (int h = 0; h < 3; ++h) {
            const float w = cw[h] < 0x1p-60f ? 0.0f : cw[h];
            tiny += cw[h] - w;
            sum += w;
            z = __fmaf_rn(w * X[h], X[h], z);
            T = __fmaf_rn(w, var[h], T);
            asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(sq[h]) : "f"(w));
        }
        const float W = xs.w;
        float rw;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rw) : "f"(W));
        // the gain a candidate needs for thr, and c = gain / (2 W)
        const float g = -__fmaf_rn(z, rw, thr) - __fmaf_rn(0x1p-17f * W, sum, 128.0f * tiny);
        c = g > 0.0f ? g * (0.4999995f * rw) : 0.0f;
        tol = __fmaf_rn(0x1.03p-15f * W, T, 1e-30f);  // 512 R W T
        // centred weighted point of position `lane`, and the sums up to it
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        if (lane < n) q = sm.S[tri_idx(lane, 0) + lane + 1];
        q.x = __fmaf_rn(-X[0] * rw, q.w, q.x) * sq[0];
        q.y = __fmaf_rn(-X[1] * rw, q.w, q.y) * sq[1];
        q.z = __fmaf_rn(-X[2] * rw, q.w, q.z) * sq[2];
#pragma unroll
        for (int off = 1; off < 16; off <<= 1) {
            const float x = tm.shfl_up(q.x, off), y = tm.shfl_up(q.y, off), z1 = tm.shfl_up(q.z, off);
            if (lane >= off) { q.x += x; q.y += y; q.z += z1; }
        }
        if (lane < n) {
            q.w = sm.S[lane + 1].w;
            sm.Q[lane + 1] = q;
            const float h = __fmaf_rn(q.x, q.x, __fmaf_rn(q.y, q.y, q.z * q.z));
            sm.G[lane + 1] = __fmaf_rn(c * q.w, __fmaf_rn(-5.0f, W, q.w), 0.5f * h);
        }
        if (lane == 0) {
            sm.Q[0] = make_float4(0.f, 0.f, 0.f, 0.f);
            sm.G[0] = 0.0f;
        }
        tm.sync();
    }
    const int pairs = (n + 1) * (n + 2) / 2 - 1;
    // 0: no candidate can be left out (nearly flat blocks), so none is looked at.  As a
    // mask on the loop's bound: a branch around the bounds made what follows it
    // divergent code.  (1023x769 of cut-out fields 342 -> 329 us, BC1 1024x1024 of smooth
    // fields 518 -> 504, 64 textures 1,259 -> 1,238; BC1 iterative ramps 1,244 -> 1,253;
    // with the branch 331, 508, 1,278, 1,344.)
    const int some = c > 0.0f ? -1 : 0;
    const unsigned below = (1u << lane) - 1u;
    uint32_t nq = 0;
#pragma unroll 1
    for (int p0 = 0; p0 < pairs; p0 += TEAM) {
        const int p = p0 + lane;
        const uint32_t jk = __ldg(&g_pairs[n][min(p, pairs - 1)]);
        const int j = (int)(jk & 31u), k = (int)(jk >> 5);
        uint32_t keep = p < pairs ? (2u << min(j, n - 1)) - 1u : 0u;  // bit i: candidate (i, j, k)
        if (part) {
            const float4 qj = sm.Q[j], qk = sm.Q[k];
            const float vx = qj.x + qk.x, vy = qj.y + qk.y, vz = qj.z + qk.z, a = qj.w + qk.w;
            const float ca = c * a;
            float P = __fmaf_rn(0.5f, __fmaf_rn(vx, vx, __fmaf_rn(vy, vy, vz * vz)), tol);
            P = __fmaf_rn(ca, a - xs.w, P);
            P = __fmaf_rn(-2.0f * c * xs.w, qj.w, P);
            const float ca2 = 2.0f * ca;
            uint32_t out = 0;  // signs of s, i descending
#pragma unroll 1
            for (int i = (min(tm.shfl(j, TEAM - 1), n - 1) | 1) & some; i > 0; i -= 2) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float4 q = sm.Q[i - h];
                    const float s = __fmaf_rn(vx, q.x, __fmaf_rn(vy, q.y, __fmaf_rn(vz, q.z, __fmaf_rn(ca2, q.w, P + sm.G[i - h]))));
                    out = __funnelshift_l(__float_as_uint(s), out, 1);
                }
            }
            keep &= ~out;
        }
        // pack what is left, one i of every pair at a time
        for (unsigned b = tm.ballot(keep != 0u); b != 0u; b = tm.ballot(keep != 0u)) {
            if (keep) sm.queue[nq + __popc(b & below)] = (uint16_t)((__ffs(keep) - 1) << 10 | j << 5 | k);
            keep &= keep - 1u;
            nq += (uint32_t)__popc(b);
        }
    }
    tm.sync();
#pragma unroll 1
    for (uint32_t t = (uint32_t)lane; t < nq; t += TEAM) eval_key(sm, sm.queue[t], xs, cw, ob);
}

// The ordering along the principal axis is the first ordering of both
// compress3 and compress4 (cluster.rs:78-136 with the same axis and points),
// so compress4 takes it and its partial sums from compress3 when compress3
// built no later ordering over them.
struct SharedOrder {
    bool valid;  // S and hist[0] hold the principal-axis ordering
    int rank;    // this lane's point's position in it
    bool finite; // every dot product was finite
    uint32_t guess;  // points before 1/6, 1/2 and 5/6 of the projections' range (sweep4)
};

// ClusterFit::compress3 / compress4 (cluster.rs:152-417) for one team.
// best_err / best carry the ColourFit state across compress3 -> compress4.
// LEAN (BC1 IterativeClusterFit, whose two passes make the largest kernel and
// whose top stall is instruction fetch) trades unrolling for code size: the
// rank and partial-sum loops are unrolled 4 times instead of 16, and compress3's
// short lists go through the survivor sweep instead of a sweep of their own
// (1,557 vs 1,604 us for 2048x2048 when measured; the other kernels were faster
// without these changes).
template <int NC, int TEAM, int NITER, bool LEAN = false>
__device__ __forceinline__ void cluster_pass(const Team<TEAM> &tm, TeamSmem &sm, const uint32_t *tbl, int count,
                                             const float (&principal)[3], const float (&cw)[3], bool prune,
                                             const float (&var)[3],
                                             bool valid, int my_point, bool unit16, float &best_err, uint2 &best,
                                             SharedOrder &so) {
    const int lane = tm.lane;
    float run = best_err;
    float ba[3] = {0.0f, 0.0f, 0.0f}, bb[3] = {0.0f, 0.0f, 0.0f};
    uint32_t bentry = 0;
    int bit = 0, best_rank = 0;
    bool best_finite = false;
    float axis[3] = {principal[0], principal[1], principal[2]};
    const uint32_t ncand = (NC == 4) ? 0u : c_ncand3[count];
    float4 xs = make_float4(0.f, 0.f, 0.f, 0.f);

#pragma unroll 1
    for (int it = 0; it < NITER; ++it) {
        // construct_ordering (cluster.rs:78-136)
        int my_rank = 0;
        bool finite;
        uint32_t guess;
        if (NITER == 1 && so.valid) {  // (the iterative kernel measured faster rebuilding it)
            my_rank = so.rank;
            finite = so.finite;
            guess = so.guess;
        } else {
            float de = FLT_MAX;
            if (lane < count) de = sm.P[0][lane] * axis[0] + sm.P[1][lane] * axis[1] + sm.P[2][lane] * axis[2];
            const uint32_t ke = dps_key(de);
            {
                const bool p = lane < count;
                const uint32_t k0 = __reduce_min_sync(tm.mask, ke), k1 = __reduce_max_sync(tm.mask, p ? ke : 0u);
                auto value = [](uint32_t k) { return __uint_as_float(k ^ (~(uint32_t)((int32_t)k >> 31) | 0x80000000u)); };
                const float d0 = value(k0), r = value(k1) - d0;
                guess = (uint32_t)__popc(tm.ballot(p && de < __fmaf_rn(r, 1.0f / 6.0f, d0))) |
                        (uint32_t)__popc(tm.ballot(p && de < __fmaf_rn(r, 0.5f, d0))) << 5 |
                        (uint32_t)__popc(tm.ballot(p && de < __fmaf_rn(r, 5.0f / 6.0f, d0))) << 10;
            }
            if (lane < 16) sm.D[lane] = ke;
            tm.sync();
            if (lane < 16) {
                // stable rank: entries with a smaller key, or an equal key earlier
                int rank = 0;
                if (LEAN) {
#pragma unroll 4
                    for (int f = 0; f < 16; ++f) {
                        const uint32_t kf = sm.D[f];
                        rank += (kf < ke || (kf == ke && f < lane)) ? 1 : 0;
                    }
                } else {
#pragma unroll
                    for (int f = 0; f < 16; ++f) {
                        const uint32_t kf = sm.D[f];
                        rank += (kf < ke || (kf == ke && f < lane)) ? 1 : 0;
                    }
                }
                reinterpret_cast<uint8_t *>(sm.hist[it])[rank] = (uint8_t)(lane < count ? lane : 0);
                my_rank = rank;
            }
            // with every dot product finite, positions 0..count-1 hold each point once
            finite = tm.ballot(lane < count && ke == 0xFFFFFFFFu) == 0u;
            tm.sync();
            const int my_ord = (lane < 16) ? hist_get(sm, it, lane) : 0;
            bool repeated = false;
#pragma unroll 1
            for (int t = 0; t < it; ++t) repeated |= tm.all(lane >= 16 || hist_get(sm, t, lane) == my_ord);
            if (repeated) break;
            if (lane < count) {
                const float w = sm.P[3][my_ord];
                sm.PW[lane] = make_float4(sm.P[0][my_ord] * w, sm.P[1][my_ord] * w, sm.P[2][my_ord] * w, 1.0f * w);
            }
            tm.sync();
            // partial sums S(a,b) = pw[a] + ... + pw[b-1], accumulated from zero in
            // loop order exactly like part0/part1/part2 of the reference
            if (lane == 0) sm.S[tri_idx(count, count)] = make_float4(0.f, 0.f, 0.f, 0.f);
            {
                float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                float4 *row = sm.S + tri_idx(lane < 16 ? lane : 0, 0) + lane;  // &S(lane, lane)
                if (lane < count) row[0] = acc;
                if (LEAN) {
#pragma unroll 4
                    for (int s = 0; s < 16; ++s) {
                        if (s >= count) break;
                        if (lane + s < count) {
                            const float4 q = sm.PW[lane + s];
                            acc.x += q.x; acc.y += q.y; acc.z += q.z; acc.w += q.w;
                            row[s + 1] = acc;
                        }
                    }
                } else {
#pragma unroll
                    for (int s = 0; s < 16; ++s) {
                        if (s >= count) break;
                        if (lane + s < count) {
                            const float4 q = sm.PW[lane + s];
                            acc.x += q.x; acc.y += q.y; acc.z += q.z; acc.w += q.w;
                            row[s + 1] = acc;
                        }
                    }
                }
            }
            tm.sync();
            so.valid = it == 0;
            so.rank = my_rank;
            so.finite = finite;
            so.guess = guess;
        }
        xs = sm.S[count];  // S(0, count) == xsum_wsum

        // each lane's best starts at (run, 0): no entry is below 0, so a
        // candidate that only ties the running best never wins; NaN never
        // compares true
        LaneBest ob;
        ob.err = run;
        ob.ent = 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) { ob.a[c] = 0.0f; ob.b[c] = 0.0f; }
        uint32_t lean_nq = 0;  // LEAN: candidates queued for the exact sweep below
        if constexpr (NC == 4) {
            // (up to 5 points have 54 candidates)
            sweep4(tm, sm, count, xs, cw, var, prune && finite && count > 5, guess, ob);
        } else if (ncand <= 2u * TEAM || !prune) {
            if (LEAN) {
                uint32_t *queue = reinterpret_cast<uint32_t *>(sm.LB);
                for (uint32_t t = (uint32_t)lane; t < ncand; t += TEAM) queue[t] = t;
                lean_nq = ncand;
                tm.sync();
            } else {
                // short lists: the plain sweep, lane-strided over the candidates
                for (uint32_t t = (uint32_t)lane; t < ncand; t += TEAM) eval_candidate(sm, __ldg(tbl + t), xs, cw, ob);
            }
        } else {
            // 1. a lower bound of every candidate's error (see cand_bound)
            const BoundBlock bb = bound_block(xs, cw);
            float lmin = __int_as_float(0x7f800000);
            uint32_t tseed = 0xFFFFFFFFu;
            if (unit16) {
                const float4 *ub = g_ub3 + lane;
#pragma unroll (NITER > 1 ? 1 : 2)
                for (uint32_t t = (uint32_t)lane; t < ncand; t += TEAM, ub += TEAM) {
                    const float4 q = __ldg(ub);
                    const uint32_t o = __float_as_uint(q.w);
                    const float4 p0 = sm.S[o & 0xFFu];
                    const float4 p1 = sm.S[(o >> 8) & 0xFFu];
                    const float bnd = unit_bound(p0, p1, q, xs, cw, bb);
                    sm.LB[t] = bnd;
                    if (bnd < lmin) { lmin = bnd; tseed = t; }
                }
            } else {
#pragma unroll (NITER > 1 ? 1 : 2)
                for (uint32_t t = (uint32_t)lane; t < ncand; t += TEAM) {
                    const uint32_t e = __ldg(tbl + t);
                    const float4 p0 = sm.S[e & 0xFu];
                    const float4 p1 = sm.S[(e >> 4) & 0xFFu];
                    const float bnd = cand_bound(p0, p1, lb_terms(p0.w, p1.w, xs.w), cw, bb);
                    sm.LB[t] = bnd;
                    if (bnd < lmin) { lmin = bnd; tseed = t; }
                }
            }
            // 2. seeds: every lane's smallest bound, evaluated exactly; the
            // threshold is the smallest error reached (never above run)
            if (tseed != 0xFFFFFFFFu) {
                eval_candidate(sm, __ldg(tbl + tseed), xs, cw, ob);
                sm.LB[tseed] = __int_as_float(0x7f800000);  // already evaluated
            }
            const uint32_t ngroups = (ncand + 3u) >> 2;
            if (lane == 0) {
                for (uint32_t t = ncand; t < 4u * ngroups; ++t) sm.LB[t] = __int_as_float(0x7f800000);
                if (!unit16 && NITER == 1) {  // (the iterative kernels spill with it)
                    // one-cluster candidates: the flat bound of unit_terms with W =
                    // xs.w (their rounded alpha : beta : gamma are within a few u W of
                    // l^2 : (1-l)^2 : l(1-l), moving the error by at most 32 u W sum w
                    // on [0,1]^2, inside eps1; 2^-10 covers the approximate 1/W).  A
                    // seed among them may be written back to infinity, or evaluated
                    // again: either is harmless.
                    float rw;
                    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rw) : "f"(xs.w));
                    const float flat = __fmaf_rn(-(1.0f + 0x1p-10f) * bb.z, rw, -bb.eps1);
                    sm.LB[c_one3[count]] = flat;
                }
            }
            const float thr = tm.least(ob.err);
            tm.sync();
            // 3. survivors (bound not above thr; NaN = no bound) are packed in
            // place into the front of LB, four bounds per lane and round; a
            // round only writes slots that have already been read
            uint32_t *queue = reinterpret_cast<uint32_t *>(sm.LB);
            const float4 *lb4v = reinterpret_cast<const float4 *>(sm.LB);
            const unsigned below = (1u << lane) - 1u;
            uint32_t nq = 0;
            for (uint32_t r0 = 0; r0 < ngroups; r0 += TEAM) {
                const uint32_t g = r0 + (uint32_t)lane;
                float4 v = make_float4(__int_as_float(0x7f800000), __int_as_float(0x7f800000),
                                       __int_as_float(0x7f800000), __int_as_float(0x7f800000));
                if (g < ngroups) v = lb4v[g];
                const bool k0 = !(v.x > thr), k1 = !(v.y > thr), k2 = !(v.z > thr), k3 = !(v.w > thr);
                if (tm.ballot(k0 || k1 || k2 || k3) == 0u) continue;  // most rounds hold no survivor
                const unsigned b0 = tm.ballot(k0), b1 = tm.ballot(k1), b2 = tm.ballot(k2), b3 = tm.ballot(k3);
                const uint32_t n0 = (uint32_t)__popc(b0), n1 = (uint32_t)__popc(b1), n2 = (uint32_t)__popc(b2);
                if (k0) queue[nq + __popc(b0 & below)] = 4u * g;
                if (k1) queue[nq + n0 + __popc(b1 & below)] = 4u * g + 1u;
                if (k2) queue[nq + n0 + n1 + __popc(b2 & below)] = 4u * g + 2u;
                if (k3) queue[nq + n0 + n1 + n2 + __popc(b3 & below)] = 4u * g + 3u;
                nq += n0 + n1 + n2 + (uint32_t)__popc(b3);
            }
            tm.sync();
            // 4. exact errors of the survivors
            if (LEAN)
                lean_nq = nq;
            else
                for (uint32_t s = (uint32_t)lane; s < nq; s += TEAM) eval_candidate(sm, __ldg(tbl + queue[s]), xs, cw, ob);
        }
        if (LEAN && NC == 3) {
            const uint32_t *queue = reinterpret_cast<const uint32_t *>(sm.LB);
            for (uint32_t s = (uint32_t)lane; s < lean_nq; s += TEAM) eval_candidate(sm, __ldg(tbl + queue[s]), xs, cw, ob);
        }
        // lexicographic reduction of the lanes' bests; the winning lane (the
        // one holding the winning entry) supplies the endpoints
        const float lbest = tm.least(ob.err);
        const uint32_t lent = __reduce_min_sync(tm.mask, ob.err == lbest ? ob.ent : 0xFFFFFFFFu);
        if (lent != 0u) {
            const int src = __ffs(tm.ballot(ob.ent == lent)) - 1;
#pragma unroll
            for (int c = 0; c < 3; ++c) { ba[c] = tm.shfl(ob.a[c], src); bb[c] = tm.shfl(ob.b[c], src); }
            run = lbest;
            bentry = lent;
            bit = it;
            best_rank = my_rank;
            best_finite = finite;
        }
        tm.sync();  // the next ordering reuses the queue's shared memory
        if (bit != it) break;
        axis[0] = bb[0] - ba[0]; axis[1] = bb[1] - ba[1]; axis[2] = bb[2] - ba[2];
    }

    if (run < best_err) {
        int i, j, k;
        if (NC == 4) {
            i = (int)(bentry >> 10);
            j = (int)((bentry >> 5) & 31u);
            k = (int)(bentry & 31u);
        } else {
            decode_entry(bentry, i, j);
            k = 16;
        }
        uint32_t ind = 3;
        // position of this pixel's point in the winning ordering: its rank, or
        // (with non-finite dot products) the last position < count holding it
        int maxpos = tm.shfl(best_rank, my_point >= 0 ? my_point : 0);
        if (!best_finite) {
            maxpos = -1;
            for (int m = 0; m < count; ++m) maxpos = (hist_get(sm, bit, m) == my_point) ? m : maxpos;
        }
        if (valid) {
            if (NC == 4) ind = maxpos >= k ? 1u : maxpos >= j ? 3u : maxpos >= i ? 2u : 0u;
            else ind = maxpos >= j ? 1u : maxpos >= i ? 2u : 0u;
        }
        const uint32_t word = __reduce_or_sync(tm.mask, lane < 16 ? (ind << (2 * lane)) : 0u);
        const uint32_t a565 = pack_565(ba[0], ba[1], ba[2]), b565 = pack_565(bb[0], bb[1], bb[2]);
        best = (NC == 4) ? write4(a565, b565, word) : write3(a565, b565, word);
        best_err = run;
    }
}

// Per-CTA inputs of the team path: the candidate lists for sets of fewer than
// 16 colours and the exact u8 -> [0,1] and sqrt(count) tables in shared memory.
struct TeamTables {
    const uint32_t *cand3;
    const float *unorm, *sqrt;
};

template <int FMT, int TEAM, int NITER>
__device__ __forceinline__ uint2 colour_cluster_team(const Team<TEAM> &tm, TeamSmem &sm, const TeamTables &tt,
                                                     uint32_t px, bool inb, const DevParams &prm) {
    const uint32_t *tbl3 = tt.cand3;
    const int lane = tm.lane;
    const uint32_t a = px >> 24;
    const bool tr = (FMT == BC1) && inb && a < 128u;
    const bool valid = inb && !tr;
    const bool transparent = tm.ballot(tr) != 0u;
    const uint32_t key = valid ? (px & 0xFFFFFFu) : (0x01000000u | (uint32_t)lane);
    const unsigned eq = tm.match(key);
    const int first = __ffs(eq) - 1;
    const bool is_new = valid && first == lane;
    const unsigned newbits = tm.ballot(is_new);
    const int count = __popc(newbits);
    const int my_point = valid ? __popc(newbits & ((1u << first) - 1u)) : -1;

    // weights: count of equal pixels, or alpha weights summed in pixel order
    float wsum;
    if (!prm.alpha_weighted) {
        wsum = (float)__popc(eq);
    } else {
        const float wa = (float)(a + 1u) * (1.0f / 256.0f);
        const int fv = valid ? first : -1;
        wsum = 0.0f;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const float wq = tm.shfl(wa, q);
            const int fq = tm.shfl(fv, q);
            wsum = wsum + ((fq == lane) ? wq : 0.0f);
        }
    }
    if (is_new) {
        sm.P[0][my_point] = tt.unorm[px & 0xFFu];
        sm.P[1][my_point] = tt.unorm[(px >> 8) & 0xFFu];
        sm.P[2][my_point] = tt.unorm[(px >> 16) & 0xFFu];
        sm.P[3][my_point] = prm.alpha_weighted ? sqrt_rn(wsum) : tt.sqrt[__popc(eq)];
    }
    tm.sync();

    const uint32_t valid16 = tm.ballot(valid);
    if (count == 1) {
        return single_fit<FMT>(tm.shfl(px & 0xFFFFFFu, __ffs(newbits) - 1), valid16, transparent);
    }
    if (count == 0) {
        // RangeFit on an empty set (range.rs:67-98): start = end = 0, error 0.
        // BC1: compress3 writes (0, 0) with every pixel excluded -> index 3;
        // compress4 never wins against error 0.  BC2/3: write4 with a == b.
        return (FMT == BC1) ? make_uint2(0u, 0xFFFFFFFFu) : make_uint2(0u, 0u);
    }

    // Sym3x3::weighted_covariance (math.rs:44-73).  Lane k forms point k's
    // products; lane t then adds column t in point order, as the reference's
    // loop does.  Columns are padded with exact zeros to a multiple of 4
    // (x + 0 == x here: no running sum is -0, so no sign is lost).
    float *scr = sm.LB;  // free until the candidate sweep: [4][16] then [6][16]
    const int n4 = (count + 3) & ~3;
    float px3[3] = {0.f, 0.f, 0.f}, pw = 0.f;
    if (lane < count) { px3[0] = sm.P[0][lane]; px3[1] = sm.P[1][lane]; px3[2] = sm.P[2][lane]; pw = sm.P[3][lane]; }
    if (lane < 16) {
        scr[lane] = px3[0] * pw; scr[16 + lane] = px3[1] * pw; scr[32 + lane] = px3[2] * pw; scr[48 + lane] = pw;
    }
    tm.sync();
    const int col = lane < 10 ? lane : 0;
    auto column_sum = [&](const float *base) {
        float acc = 0.0f;
        for (int g = 0; g < n4; g += 4) {
            const float4 v = *reinterpret_cast<const float4 *>(base + 16 * col + g);
            acc = acc + v.x; acc = acc + v.y; acc = acc + v.z; acc = acc + v.w;
        }
        return acc;
    };
    const float sum1 = column_sum(scr);  // lanes 0-2: centroid sums, lane 3: total
    const float total = tm.shfl(sum1, 3);
    const float cdiv = total > FLT_EPSILON ? div_rn(sum1, total) : sum1;
    const float cen[3] = {tm.shfl(cdiv, 0), tm.shfl(cdiv, 1), tm.shfl(cdiv, 2)};
    if (lane < 16) {
        const float a0 = px3[0] - cen[0], a1 = px3[1] - cen[1], a2 = px3[2] - cen[2];
        const float b0 = a0 * pw, b1 = a1 * pw, b2 = a2 * pw;
        const bool in = lane < count;
        float *c2 = scr + 64;
        c2[lane] = in ? a0 * b0 : 0.f;      c2[16 + lane] = in ? a0 * b1 : 0.f;
        c2[32 + lane] = in ? a0 * b2 : 0.f; c2[48 + lane] = in ? a1 * b1 : 0.f;
        c2[64 + lane] = in ? a1 * b2 : 0.f; c2[80 + lane] = in ? a2 * b2 : 0.f;
    }
    tm.sync();
    const float cv = column_sum(scr + 64);
    float cov[6];
#pragma unroll
    for (int t = 0; t < 6; ++t) cov[t] = tm.shfl(cv, t);
    tm.sync();  // the scratch is reused by the ordering
    float principal[3];
    principle_component_team(tm, cov, principal);

    const float cw[3] = {prm.w[0], prm.w[1], prm.w[2]};
    float best_err = FLT_MAX;
    uint2 best = make_uint2(0u, 0u);
    // 16 distinct colours without alpha weighting: every weight is sqrt(1) = 1
    const bool unit16 = count == 16 && !prm.alpha_weighted;
    if (count == 16) tbl3 = g_cand16;
    // the error bound used for pruning holds for finite, non-negative weights
    const bool prune = cw[0] >= 0.0f && cw[1] >= 0.0f && cw[2] >= 0.0f && cw[0] <= FLT_MAX && cw[1] <= FLT_MAX &&
                       cw[2] <= FLT_MAX;
    // compress4's bound: ordinary weights (products of larger ones leave the f32 range)
    const bool part = prune && cw[0] <= 0x1p60f && cw[1] <= 0x1p60f && cw[2] <= 0x1p60f;
    const float var[3] = {cov[0], cov[3], cov[5]};
    SharedOrder so{false, 0, false, 0u};
    if (FMT == BC1) {
        cluster_pass<3, TEAM, NITER, (NITER > 1)>(tm, sm, tbl3, count, principal, cw, prune, var, valid, my_point, unit16, best_err,
                                     best, so);
        if (!transparent)
            cluster_pass<4, TEAM, NITER, (NITER > 1)>(tm, sm, nullptr, count, principal, cw, part, var, valid, my_point, unit16, best_err,
                                         best, so);
    } else {
        cluster_pass<4, TEAM, NITER>(tm, sm, nullptr, count, principal, cw, part, var, valid, my_point, unit16, best_err,
                                     best, so);
    }
    return best;
}

template <int TEAM>
__device__ __forceinline__ uint2 team_bc3_alpha(const Team<TEAM> &tm, uint32_t v, bool inb) {
    const int lane = tm.lane;
    int min7 = (int)__reduce_min_sync(tm.mask, inb ? v : 255u);
    int max7 = (int)__reduce_max_sync(tm.mask, inb ? v : 0u);
    int min5 = (int)__reduce_min_sync(tm.mask, (inb && v != 0u) ? v : 255u);
    int max5 = (int)__reduce_max_sync(tm.mask, (inb && v != 255u) ? v : 0u);
    if (min5 > max5) min5 = max5;
    if (min7 > max7) min7 = max7;
    fix_range(min5, max5, 5);
    fix_range(min7, max7, 7);
    int c5[8], c7[8];
    c5[0] = min5; c5[1] = max5;
#pragma unroll
    for (int i = 1; i < 5; ++i) c5[1 + i] = ((5 - i) * min5 + i * max5) / 5;
    c5[6] = 0; c5[7] = 255;
    c7[0] = min5; c7[1] = max5;
#pragma unroll
    for (int i = 1; i < 7; ++i) c7[1 + i] = ((7 - i) * min7 + i * max7) / 7;
    int i5 = 0, i7 = 0, d5 = abs((int)v - c5[0]), d7 = abs((int)v - c7[0]);
#pragma unroll
    for (int j = 1; j < 8; ++j) {
        const int e5 = abs((int)v - c5[j]), e7 = abs((int)v - c7[j]);
        if (e5 < d5) { d5 = e5; i5 = j; }
        if (e7 < d7) { d7 = e7; i7 = j; }
    }
    if (!inb) { i5 = 0; i7 = 0; d5 = 0; d7 = 0; }
    const uint32_t err5 = __reduce_add_sync(tm.mask, (uint32_t)(d5 * d5));
    const uint32_t err7 = __reduce_add_sync(tm.mask, (uint32_t)(d7 * d7));
    uint32_t a0, a1, idx;
    if (err5 <= err7) {
        a0 = (uint32_t)min5; a1 = (uint32_t)max5; idx = (uint32_t)i5;
        if (min5 > max5) {  // never true after fix_range (alpha.rs:146-165)
            a0 = (uint32_t)max5; a1 = (uint32_t)min5;
            idx = idx == 0 ? 1u : idx == 1 ? 0u : (idx <= 5 ? 7u - idx : idx);
        }
    } else {
        a0 = (uint32_t)min7; a1 = (uint32_t)max7; idx = (uint32_t)i7;
        if (min7 < max7) { a0 = (uint32_t)max7; a1 = (uint32_t)min7; idx = (9u - idx) & 7u; }
    }
    const uint32_t lo = __reduce_or_sync(tm.mask, (lane < 8) ? (idx << (3 * lane)) : 0u);
    const uint32_t hi = __reduce_or_sync(tm.mask, (lane >= 8 && lane < 16) ? (idx << (3 * (lane - 8))) : 0u);
    return make_uint2(a0 | (a1 << 8) | ((lo & 0xFFFFu) << 16), (lo >> 16) | (hi << 8));
}


// ===========================================================================
// block-level entry points

// Thread-per-block: encode and store block b (RangeFit / SingleColourFit path).
template <int FMT>
__device__ __forceinline__ void range_block(const SrcDesc &src, size_t b, const DevParams &prm, uint8_t *out,
                                            const float *s_unorm, const float *s_sqrt, const PointCol &pt) {
    uint32_t px[16];
    const uint32_t mask = load_block_rgba(src, b, px);
    // alpha first, so the alpha bytes are dead before the colour fit's registers peak
    uint2 al = make_uint2(0u, 0u);
    if (FMT == BC2) al = encode_bc2_alpha(px, mask);
    if (FMT == BC3) {
        uint32_t v[4];
        channel_words(px, 3, v);
        al = encode_bc3_alpha<false>(v, mask);
    }
    const uint2 col = colour_range_thread<FMT>(px, mask, prm, s_unorm, s_sqrt, pt);
    if (FMT == BC1) reinterpret_cast<uint2 *>(out)[b] = col;
    else reinterpret_cast<uint4 *>(out)[b] = make_uint4(al.x, al.y, col.x, col.y);
}

// Pixel p of block b for lane p < 16 of a team (RGBA8, pixel order), and
// whether it lies inside the image / is selected by the block's mask.
struct TeamPixel {
    uint32_t px;
    bool inb;
};

__device__ __forceinline__ TeamPixel load_team_pixel(const SrcDesc &src, size_t b, int p) {
    TeamPixel r{0u, false};
    if (p < 16) {
        if (src.mode == 1) {
            r.px = __ldg(reinterpret_cast<const uint32_t *>(src.base + 64 * b) + p);
            r.inb = src.masks ? ((__ldg(src.masks + b) >> p) & 1u) : true;
        } else {
            uint32_t bx, by;
            block_coords(src, b, bx, by);
            const uint32_t x = 4 * bx + (p & 3), y = 4 * by + (p >> 2);
            r.inb = x < src.width && y < src.height;
            if (r.inb) r.px = ld_u32_any(src.base + (size_t)y * src.pitch + 4 * (size_t)x);
        }
    }
    return r;
}

// Team-per-block: encode and store block b (ClusterFit path) from its pixels.
template <int FMT, int TEAM, int NITER>
__device__ __forceinline__ void cluster_block_px(const Team<TEAM> &tm, TeamSmem &sm, const TeamTables &tt,
                                                 const TeamPixel tp, size_t b, const DevParams &prm, uint8_t *out) {
    const int p = tm.lane;
    const uint32_t px = tp.px;
    const bool inb = tp.inb;
    uint2 al = make_uint2(0u, 0u);
    if (FMT == BC2) {
        const uint32_t q = inb ? bc2_quant(px >> 24) : 0u;
        al.x = __reduce_or_sync(tm.mask, p < 8 ? q << (4 * p) : 0u);
        al.y = __reduce_or_sync(tm.mask, (p >= 8 && p < 16) ? q << (4 * (p - 8)) : 0u);
    } else if (FMT == BC3) {
        al = team_bc3_alpha<TEAM>(tm, px >> 24, inb);
    }
    const uint2 col = colour_cluster_team<FMT, TEAM, NITER>(tm, sm, tt, px, inb, prm);
    if (p == 0) {
        if (FMT == BC1) reinterpret_cast<uint2 *>(out)[b] = col;
        else reinterpret_cast<uint4 *>(out)[b] = make_uint4(al.x, al.y, col.x, col.y);
    }
    tm.sync();
}

// Team-per-block: load, encode and store block b.
template <int FMT, int TEAM, int NITER>
__device__ __forceinline__ void cluster_block(const Team<TEAM> &tm, TeamSmem &sm, const TeamTables &tt,
                                              const SrcDesc &src, size_t b, const DevParams &prm, uint8_t *out) {
    const int p = tm.lane;
    uint32_t px = 0;
    bool inb = false;
    if (p < 16) {
        if (src.mode == 1) {
            px = __ldg(reinterpret_cast<const uint32_t *>(src.base + 64 * b) + p);
            inb = src.masks ? ((__ldg(src.masks + b) >> p) & 1u) : true;
        } else {
            uint32_t bx, by;
            block_coords(src, b, bx, by);
            const uint32_t x = 4 * bx + (p & 3), y = 4 * by + (p >> 2);
            inb = x < src.width && y < src.height;
            if (inb) px = ld_u32_any(src.base + (size_t)y * src.pitch + 4 * (size_t)x);
        }
    }
    uint2 al = make_uint2(0u, 0u);
    if (FMT == BC2) {
        const uint32_t q = inb ? bc2_quant(px >> 24) : 0u;
        al.x = __reduce_or_sync(tm.mask, p < 8 ? q << (4 * p) : 0u);
        al.y = __reduce_or_sync(tm.mask, (p >= 8 && p < 16) ? q << (4 * (p - 8)) : 0u);
    } else if (FMT == BC3) {
        al = team_bc3_alpha<TEAM>(tm, px >> 24, inb);
    }
    const uint2 col = colour_cluster_team<FMT, TEAM, NITER>(tm, sm, tt, px, inb, prm);
    if (p == 0) {
        if (FMT == BC1) reinterpret_cast<uint2 *>(out)[b] = col;
        else reinterpret_cast<uint4 *>(out)[b] = make_uint4(al.x, al.y, col.x, col.y);
    }
    tm.sync();
}

// (F1, r, C, offsets) of unit_bound from exact weight-lane terms w = (alpha,
// beta, gamma, factor) of a weight-1, 16-point set (W = 16): A = alpha + beta +
// 2 gamma, B = alpha + gamma, f = 1/det.  det of the f32 values is exact in
// double (products of two 24-bit significands); each term is rounded once.
//
// det = 0 exactly when every point is in one cluster (one interpolation
// weight l; the f32 constants keep alpha : beta : gamma = l^2 : (1-l)^2 :
// l(1-l) exactly, as 4/9 and 2/9 are 4 and 2 times 1/9 in f32).  The fit is
// then a single colour c = l a + (1-l) b, whose error sum_c w_c (W c^2 -
// 2 X c) is at least -Z/W; the reference's rounded ax, bx move it by at most
// 4 u sum_c w_c X_c (a, b in [0,1]), inside eps1.  So such a candidate gets
// the flat bound -(1 + 2^-10) Z/W - eps1 (F1 = 0), which the fitted
// endpoints of a textured block beat, instead of no bound.
__device__ __forceinline__ float4 unit_terms(const float4 w, uint32_t offs, bool one_cluster) {
    const double al = w.x, be = w.y, ga = w.z;
    const double det = al * be - ga * ga;
    const double A = al + be + 2.0 * ga;
    const float nan = __int_as_float(0x7fc00000);  // no bound
    if (!(det > 0.0))
        return one_cluster ? make_float4(0.0f, 0.0f, (float)(-(1.0 + 0x1p-10) / 16.0), __uint_as_float(offs))
                           : make_float4(nan, 0.0f, nan, __uint_as_float(offs));
    return make_float4((float)(-A / det), (float)(2.0 * (al + ga) / A), (float)(-(al + 0x1p-13) / det),
                       __uint_as_float(offs));
}

// Fill the bound terms g_ub3 from this TU's loop-order candidate
// list: the w-lane sums of a 16-point, weight-1 set are S(a,b).w = b - a
// (exact small integers), and wterms3 is the reference's f32 code.
static __global__ void k_unit_terms() {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < kCand3) {
        int i, j;
        decode_entry(g_cand16[t], i, j);
        const uint32_t offs = (uint32_t)tri_idx(0, i) | (uint32_t)tri_idx(i, j) << 8;
        const bool one = (i == 16) + (j - i == 16) + (16 - j == 16) == 1;
        g_ub3[t] = unit_terms(wterms3((float)i, (float)(j - i), 16.0f), offs, one);
    }
}

// ===========================================================================
// host side: candidate lists + upload of this TU's tables

// Build the candidate lists and single-colour tables and copy them to the
// current device.
static inline cudaError_t upload_tables_this_tu(const uint32_t lut[4][256][2]) {
    // compress3: (i, j), 0 <= i < 16, max(i,1) <= j <= 16
    struct C { int m, rank; uint32_t e; };
    C c3[kCand3];
    int n3 = 0;
    for (int i = 0; i < 16; ++i)
        for (int j = (i == 0 ? 1 : i); j <= 16; ++j) {
            const int m = i + 1 > j ? i + 1 : j;
            c3[n3].m = m;
            c3[n3].rank = n3;
            c3[n3].e = (uint32_t)i | ((uint32_t)tri_idx(i, j) << 4) | ((uint32_t)n3 << 20);
            ++n3;
        }
    if (n3 != kCand3) return cudaErrorInvalidValue;
    uint32_t loop_tbl[kCand3 + 1] = {}, tbl[kCand3 + 1] = {}, nc3[17] = {};
    for (int t = 0; t < kCand3; ++t) loop_tbl[t] = c3[t].e;
    for (int a = 1; a < n3; ++a) {  // stable insertion sort on m
        C t = c3[a];
        int b = a;
        while (b > 0 && c3[b - 1].m > t.m) { c3[b] = c3[b - 1]; --b; }
        c3[b] = t;
    }
    for (int t = 0; t < kCand3; ++t) tbl[t] = c3[t].e;
    for (int n = 0; n <= 16; ++n)
        for (int t = 0; t < kCand3; ++t) nc3[n] += c3[t].m <= n ? 1u : 0u;
    // position of the one-cluster candidate in the list each count uses
    uint16_t one3[17] = {};
    for (int n = 1; n <= 16; ++n) {
        const uint32_t *list = n == 16 ? loop_tbl : tbl;
        for (int t = 0; t < kCand3; ++t)
            if ((list[t] & 0xFFFu) == (uint32_t)tri_idx(0, n) << 4) one3[n] = (uint16_t)t;  // the i and S(i,j) fields
    }
    uint16_t pairs[17][kPairs] = {};
    for (int n = 1; n <= 16; ++n) {
        int t = 0;
        for (int j = 0; j <= n; ++j)
            for (int k = j == 0 ? 1 : j; k <= n; ++k) pairs[n][t++] = (uint16_t)(j | k << 5);
    }
    cudaError_t e;
    if ((e = cudaMemcpyToSymbol(g_cand, tbl, sizeof(tbl))) != cudaSuccess) return e;
    if ((e = cudaMemcpyToSymbol(g_cand16, loop_tbl, sizeof(loop_tbl))) != cudaSuccess) return e;
    if ((e = cudaMemcpyToSymbol(c_ncand3, nc3, sizeof(nc3))) != cudaSuccess) return e;
    if ((e = cudaMemcpyToSymbol(c_one3, one3, sizeof(one3))) != cudaSuccess) return e;
    if ((e = cudaMemcpyToSymbol(g_pairs, pairs, sizeof(pairs))) != cudaSuccess) return e;
    k_unit_terms<<<1, 256>>>();
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    k_unorm_tables<<<1, 256>>>();
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = cudaDeviceSynchronize()) != cudaSuccess) return e;
    return cudaMemcpyToSymbol(g_lut, lut, sizeof(g_lut));
}


}  // namespace tx
