// tx_cluster_lanes.cuh -- ClusterFit of BC2 and BC3 blocks with one block per
// thread (lib/src/colourfit/cluster.rs:33-136, :267-417).
//
// The team form (tx_colour.cuh) gives a block to 32 lanes and is bound by
// instruction issue: of its 2,670 warp instructions per block about half set the
// block up (colour set, covariance, axis, ordering, partial sums, alpha half),
// where a warp has at most 16 lanes' worth of work, and a candidate's bound
// takes 33.  Here a thread sets a block up (160 warp instructions per block);
// the bound of a candidate is a four-term dot product in registers, two
// candidates per paired instruction; and only the candidates that the bound
// cannot exclude (6 per block of a noisy ramp texture) are pooled over the warp
// and evaluated exactly, 32 at a time.  Bound now: instruction issue and, with
// 205 KB of code of which every warp runs a third, instruction fetch, which is
// why the phases are separated by barriers (the warps of a CTA then fetch the
// same code; 408 -> 366 us) and the sweeps are rolled loops (an unrolled sweep
// stalled on fetches for 6 of 10 cycles).
//
// BC3 2048x2048, noisy ramps: 340 us (alpha-weighted 354) where the team form took
// 735 (941) before this one and takes 588 now; smooth fields of nearly flat blocks,
// which take the grid filter: 1,320, 1,338 and 1,219.
#pragma once
#include "tx_colour.cuh"

namespace tx {

constexpr int kLaneThreads = 256;  // threads (= blocks in flight) per CTA
constexpr int kRowCap = 38;        // queued candidate rows per lane

// Shared memory of a CTA.  Column t of pts holds thread t's points: pixel order
// while the block is set up, then (x w, y w, z w, w) in the current ordering,
// zero past the last point.  For the sweeps the columns are dealt out again,
// sorted by their number of points (deal()).
struct LaneSmem {
    float4 pts[16 * kLaneThreads];
    float4 xs[kLaneThreads];                // per column: variances and least weight, then S(0, count)
    unsigned long long best[kLaneThreads];  // per column: order_key(error) << 32 | candidate
    uint32_t meta[kLaneThreads];            // per column: points, finite, first guess (deal())
    uint32_t dealt[kLaneThreads];           // thread -> column
    uint32_t rows[kRowCap * kLaneThreads];  // per thread: queued rows: mask of k (row_k) | j << 16 | i << 21
    uint32_t bins[64];
};

// "No candidate" in the low half of LaneSmem::best: above every candidate.
constexpr uint32_t kNone = 0x7FFFu;

// f32 -> unsigned with the same order (-0 and +0 equal); not for NaN.
__device__ __forceinline__ uint32_t order_key(float x) {
    const uint32_t u = __float_as_uint(x + 0.0f);
    return u ^ ((uint32_t)((int32_t)u >> 31) | 0x80000000u);
}
__device__ __forceinline__ float order_unkey(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k ^ 0x80000000u) : ~k);
}

// Paired fused multiply-add (used for the bounds only, where fusing is wanted).
__device__ __forceinline__ float2 fma2_rn(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{.reg .b64 ra, rb, rc, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\t"
        "mov.b64 rb, {%4, %5};\n\t"
        "mov.b64 rc, {%6, %7};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rc;\n\t"
        "mov.b64 {%0, %1}, rd;}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

__device__ __forceinline__ float rcp_fast(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float max3_abs(float a, float b, float c) {
    float d;
    asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Exact error and endpoints of candidate (i, j, k) of the ordered points in
// column `col` (cluster.rs:315-372): part sums accumulated from zero in order
// (0 + x = x), then the reference's fit.  Lanes hold different candidates, so
// every point goes through the three sums under predicates, with all loads in
// flight, instead of through loops of different lengths.
__device__ __forceinline__ float lane_exact(const float4 *col, const float4 xs, int i, int j, int k,
                                            const float (&cw)[3], float (&a)[3], float (&b)[3]) {
    float4 p0 = make_float4(0.f, 0.f, 0.f, 0.f), p1 = p0, p2 = p0;
#pragma unroll
    for (int t = 0; t < 16; ++t) {
        const float4 q = col[t * kLaneThreads];
        const bool in0 = t < i, in1 = t >= i && t < j, in2 = t >= j && t < k;
        p0.x = in0 ? p0.x + q.x : p0.x; p0.y = in0 ? p0.y + q.y : p0.y;
        p0.z = in0 ? p0.z + q.z : p0.z; p0.w = in0 ? p0.w + q.w : p0.w;
        p1.x = in1 ? p1.x + q.x : p1.x; p1.y = in1 ? p1.y + q.y : p1.y;
        p1.z = in1 ? p1.z + q.z : p1.z; p1.w = in1 ? p1.w + q.w : p1.w;
        p2.x = in2 ? p2.x + q.x : p2.x; p2.y = in2 ? p2.y + q.y : p2.y;
        p2.z = in2 ? p2.z + q.z : p2.z; p2.w = in2 ? p2.w + q.w : p2.w;
    }
    return eval4<true>(p0, p1, p2, xs, wterms4(p0.w, p1.w, p2.w, xs.w), cw, a, b);
}

// The k of bit `bit` of a row mask: odd k = 15, 13, .. 1 at bits 0-7, even
// k = 16, 14, .. 2 at bits 8-15.
__device__ __forceinline__ int row_k(int bit) { return bit < 8 ? 15 - 2 * bit : 32 - 2 * bit; }
// Row masks of the k >= j, and of the k <= n.
__host__ __device__ constexpr uint32_t row_from(int j) {
    uint32_t m = 0;
    for (int bit = 0; bit < 16; ++bit) m |= ((bit < 8 ? 15 - 2 * bit : 32 - 2 * bit) >= j ? 1u : 0u) << bit;
    return m;
}
__device__ __forceinline__ uint32_t row_from_dyn(int j) {  // 1 <= j <= 16
    return (0xFFu >> (j >> 1)) | ((0xFFu >> ((j - 1) >> 1)) << 8);
}
__device__ __forceinline__ uint32_t row_upto(int n) {
    return ((0xFFu << ((16 - n) >> 1)) & 0xFFu) | (((0xFFu << ((17 - n) >> 1)) & 0xFFu) << 8);
}

// When the least-squares bound keeps rows in a plane (one i) this many times
// over the lanes of a warp, the plane goes through the grid filter instead.
constexpr unsigned kGridRows = 96;
// Row mask of k = 16, which completes the one-cluster candidates (0, 0, 16) and
// (0, 16, 16).
constexpr uint32_t kOneCluster = 1u << 8;
// Blocks of a smaller weighted variance than this mostly need the grid filter.
constexpr float kFlat = 4e-3f;
// k >= j as a row mask, j = 0 .. 16 (row_from).
static __constant__ uint32_t c_row_from[17] = {
    row_from(0), row_from(1), row_from(2), row_from(3), row_from(4), row_from(5), row_from(6), row_from(7), row_from(8),
    row_from(9), row_from(10), row_from(11), row_from(12), row_from(13), row_from(14), row_from(15), row_from(16)};

// ---------------------------------------------------------------------------
// Bounds.  With v_t = w_t x_t the ordered weighted points (f32, as the reference
// rounds them) and X, W the reference's f32 sums of them, candidate (i, j, k)
// gives the points the weights l = 1, 2/3, 1/3, 0 towards endpoint a.  Let
// A' = sum l_t (v_t - w_t c), c = X / W, alpha = sum w l^2, B = sum w l and
// det = W alpha - B^2.  The error of endpoints a, b is then, channel by channel
// and exactly,
//     E = base + alpha a'^2 + beta b'^2 + 2 gamma a' b' - 2 A' (a' - b'),
// base = -X^2 / W, a' = a - c, b' = b - c, gamma = B - alpha,
// beta = W - 2 B + alpha: least (over real a, b) at a' - b' = d = A' W / det,
// where it is base - gain, gain = W A'^2 / det.  With Q(t) the prefix sums of
// the centred points and w(t) those of the weights, 3 A' = Q(i) + Q(j) + Q(k),
// 3 B = w(i) + w(j) + w(k) = u and 9 alpha = 5 w(i) + 3 w(j) + w(k) = v, so
//     gain = W |Q(i) + Q(j) + Q(k)|^2 / den,   den = 9 det = W v - u^2,
// |.|^2 weighted by the channel weights: centred, no term of the block's mean
// colour remains to be lost in rounding.
//
// A candidate can reach an error thr only if gain >= g = -(thr + base) - eps, eps
// bounding the rounding of the reference's own evaluation.  Multiplied out with
// c = g / (2 W) this is s = |Q(i) + Q(j) + Q(k)|^2 / 2 + tol - c den >= 0, and
//     s = r + qg(k) + (w_c V_c) . Q(k) + 2 c u_ij w(k),   V = Q(i) + Q(j),
// r for the row (i, j) and qg(k) = |Q(k)|^2 / 2 + c w(k) (w(k) - W) for the
// column: one addition and four fused multiply-adds per candidate.
//
// Rounding (R = 2^-24).  D >= |a - b|, |a - c|, |b - c| and e >= a, b: in a
// channel of variance var_c, d^2 det / W <= var_c, and W / det <= kappa =
// 9 W / (wmin (W - wmin)) unless all points are in one cluster; snapping moves
// d by less than one grid step.  So D = sqrt(kappa var_c) + step, e = c + D (at
// most 1).  S = sum of the prefix sums of v, S_w of w.
//   eps, per channel and times w_c R: the part sums are off by at most S in
//     total, the same in ax and (but for X, which is used as it is) in bx, which
//     moves E by 2 D S, and 2 D S_w e through the weights; the other roundings of
//     ax and bx move it by 10 e X, of the weight terms by 5.2 e^2 W, of the error
//     itself by 8 e^2 W + 14 e X; here c and base are off by 6 D X + 9 c X.  In
//     all e (14 e W + 25 X) + 9 c X + D (2.1 (S + S_w e) + 6 e W).
//   tol: the terms of s are at most 8 W T in size (T the weighted variance,
//     c W <= T / 2) with 8 roundings, the prefix weights move it by 60 W T and
//     the centred prefix sums by 144 W T (times R): 512 R W T is taken.
//   Candidates with every point in one cluster have no least-squares fit; their
//     error is at least base less 124 R W sum w_c (eps with e = D = 1).
//   The grid filter's E is off by at most tolp = R (1024 T + 32 W sum w_c D^2).
//     The reference's endpoint is (ax beta - bx gamma) / det, in f32 off by at
//     most slope (3 (S + 10 X) + 54 W e) R, slope the larger of (3 W - u) / den
//     and u / den, and by slope (18 X + 12 S_w e) R more if the weights are not
//     all 1.  The filter's own endpoint, centred, is off by slope (9 X + 6 W e) R
//     through c and the last rounding, and through its slope and sums by slope 32
//     W D R, 202 W D for weights other than 1 (u, v and the prefix weights within
//     24 W R and 72 W R, so den within 216 W^2 R, which moves a' by its share of
//     a').  An endpoint nearer to a rounding boundary than all this is in
//     doubt, and its candidate is kept.
struct LaneBound {
    float2 qx[8], qy[8], qz[8], qw[8];  // centred prefix sums and weights, prefixes 1..16 in pairs
    float2 qg[8];                       // |Q|^2 / 2 + c w (w - W)
    float W, rw, cx, cy, cz;
    float base, eps, eps1, tol, tolp, doubt;
    float c, cutp;
};

// Where the projections of the points cross 1/6, 1/2 and 5/6 of their range: a
// first guess of a good candidate.
struct LaneGuess {
    int i, j, k;
};

// The per-thread code of the kernel, with the CTA's shared memory and the
// channel weights.
struct ClusterLanes {
    LaneSmem &sm;
    const int tid, lane;
    int col;  // the column this thread sweeps
    float cw[3], sq[3];  // channel weights and their square roots

    __device__ __forceinline__ ClusterLanes(LaneSmem &s, const DevParams &p)
        : sm(s), tid(threadIdx.x), lane(threadIdx.x & 31), col(threadIdx.x) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            cw[c] = p.w[c];
            asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(sq[c]) : "f"(cw[c]));
        }
    }

    // construct_ordering (cluster.rs:78-136) of the pixel-ordered points in the
    // lane's column, which is replaced by the ordered weighted points.  Keys
    // tie in pixel order; entries that are not points stand for the reference's
    // padding (key of FLT_MAX, point 0).  Returns whether every dot product is
    // finite; ord receives the pixel at every position, four bits each.
    __device__ __forceinline__ bool order(const ColourSet &cs, const float (&axis)[3], uint32_t (&ord)[2],
                                          LaneGuess &g) const {
        float4 *pt = sm.pts + tid;
        float4 q[16];
        uint32_t key[16];
        float dmin = FLT_MAX, dmax = -FLT_MAX;
        bool finite = true;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            q[i] = pt[i * kLaneThreads];
            const bool p = (cs.newbits >> i) & 1u;
            const float d = p ? q[i].x * axis[0] + q[i].y * axis[1] + q[i].z * axis[2] : FLT_MAX;
            key[i] = dps_key(d);
            finite = finite && key[i] != 0xFFFFFFFFu;
            dmin = fminf(dmin, d);
            dmax = fmaxf(dmax, p ? d : -FLT_MAX);
        }
        const float r = dmax - dmin;
        const uint32_t k6 = dps_key(dmin + r * (1.0f / 6.0f)), k2 = dps_key(dmin + r * 0.5f),
                       k56 = dps_key(dmin + r * (5.0f / 6.0f));
        g.i = g.j = g.k = 0;
        int rank[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            rank[i] = i;
            g.i += key[i] < k6 ? 1 : 0;
            g.j += key[i] < k2 ? 1 : 0;
            g.k += key[i] < k56 ? 1 : 0;
        }
#pragma unroll
        for (int i = 1; i < 16; ++i)
#pragma unroll
            for (int j = 0; j < i; ++j) {
                const bool after = key[j] > key[i];
                rank[j] += after ? 1 : 0;
                rank[i] -= after ? 1 : 0;
            }
        ord[0] = ord[1] = 0u;
        const int first = __ffs(cs.newbits) - 1;
        float4 q0 = q[0];
#pragma unroll
        for (int i = 1; i < 16; ++i)
            if (first == i) q0 = q[i];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const bool p = (cs.newbits >> i) & 1u;
            const float4 v = p ? q[i] : q0;
            const bool in = rank[i] < cs.count;
            pt[rank[i] * kLaneThreads] = in ? make_float4(v.x * v.w, v.y * v.w, v.z * v.w, v.w)
                                            : make_float4(0.f, 0.f, 0.f, 0.f);
            const uint32_t e = (uint32_t)(p ? i : first) << (4 * (rank[i] & 7));
            if (rank[i] < 8) ord[0] |= e;
            else ord[1] |= e;
        }
        return finite;
    }

    // Sums, prefix tables and error terms of the column's ordering.  sm.xs holds
    // the weighted variances sum_t w_t (x_t - mean)^2 of its points per channel
    // and their least weight.
    __device__ __forceinline__ void prefixes(LaneBound &B, bool finite) const {
        const float4 *pt = sm.pts + col;
        const float4 vw = sm.xs[col];
        const float var[3] = {vw.x, vw.y, vw.z}, wmin = vw.w;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        float r = 0.f, rw = 0.f;  // sums of the prefix sums (largest channel; weights)
#pragma unroll 4
        for (int t = 0; t < 16; ++t) {  // in order from zero: the reference's xsum_wsum (pads add +0)
            const float4 q = pt[t * kLaneThreads];
            s.x += q.x; s.y += q.y; s.z += q.z; s.w += q.w;
            r += fmaxf(s.x, fmaxf(s.y, s.z));
            rw += s.w;
        }
        sm.xs[col] = s;
        const float W = s.w, iw = rcp_fast(W);
        B.W = W;
        B.rw = iw;
        B.cx = s.x * iw; B.cy = s.y * iw; B.cz = s.z * iw;
        float ax = 0.f, ay = 0.f, az = 0.f, aw = 0.f;
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            const float4 q = pt[t * kLaneThreads];
            ax += __fmaf_rn(-B.cx, q.w, q.x);
            ay += __fmaf_rn(-B.cy, q.w, q.y);
            az += __fmaf_rn(-B.cz, q.w, q.z);
            aw += q.w;
            if (t & 1) { B.qx[t >> 1].y = ax; B.qy[t >> 1].y = ay; B.qz[t >> 1].y = az; B.qw[t >> 1].y = aw; }
            else { B.qx[t >> 1].x = ax; B.qy[t >> 1].x = ay; B.qz[t >> 1].x = az; B.qw[t >> 1].x = aw; }
        }
        const float u = 5.9604645e-8f;  // 2^-24
        const float T = (cw[0] * var[0] + cw[1] * var[1] + cw[2] * var[2]) * 1.01f;
        const float kappa = 9.01f * W * rcp_fast(wmin * (W - wmin));
        const float c3[3] = {B.cx, B.cy, B.cz}, X3[3] = {s.x, s.y, s.z};
        float e1 = 0.f, d2 = 0.f, wsum = 0.f, emax = 0.f, dmax = 0.f;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            float D;
            asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(D) : "f"(var[c] * 1.01f * kappa));
            D = fminf(1.0f, D + (c == 1 ? 0.017f : 0.033f));
            const float e = fminf(1.0001f, c3[c] + D);
            e1 += cw[c] * (e * (14.0f * e * W + 25.0f * X3[c]) + 9.0f * c3[c] * X3[c] + D * (2.1f * (r + rw * e) + 6.0f * e * W));
            d2 += cw[c] * D * D;
            wsum += cw[c];
            emax = fmaxf(emax, e);
            dmax = fmaxf(dmax, D);
        }
        B.base = ((cw[0] * s.x) * s.x + (cw[1] * s.y) * s.y + (cw[2] * s.z) * s.z) * iw;
        B.eps = u * e1;
        B.eps1 = u * W * wsum * 124.0f;
        // with repeated points (a non-finite dot product) var says nothing and all is kept
        B.tol = finite ? __fmaf_rn(512.0f * u * W, T, 1e-30f) : 1e30f;
        B.tolp = 1024.0f * u * T + 32.0f * u * W * d2;
        const float xm = fmaxf(s.x, fmaxf(s.y, s.z));
        const bool ones = wmin == 1.0f && W == (float)(int)W && rw == 0.5f * W * (W + 1.0f) + (16.0f - W) * W;
        const float dw = ones ? 32.0f * W * dmax : 18.0f * xm + 12.0f * rw * emax + 202.0f * W * dmax;
        B.doubt = finite ? 63.0f * u * (3.0f * (r + 13.0f * xm) + 60.0f * W * emax + dw) : 1e30f;
    }

    // Take a new least error: the gain a candidate needs for it is
    // -(thr + base) - eps, and the row terms that depend on it.
    __device__ __forceinline__ void set_cut(LaneBound &B, float thr) const {
        const float g = -(thr + B.base) - B.eps;
        B.c = g > 0.0f ? g * (0.4999995f * B.rw) : 0.0f;
        B.cutp = thr + B.base + B.eps + B.tolp;
        const float2 cx = make_float2(0.5f * cw[0], 0.5f * cw[0]), cy = make_float2(0.5f * cw[1], 0.5f * cw[1]),
                     cz = make_float2(0.5f * cw[2], 0.5f * cw[2]), C = make_float2(B.c, B.c), NW = make_float2(-B.W, -B.W);
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            float2 h = mul2_rn(mul2_rn(cx, B.qx[p]), B.qx[p]);
            h = fma2_rn(mul2_rn(cy, B.qy[p]), B.qy[p], h);
            h = fma2_rn(mul2_rn(cz, B.qz[p]), B.qz[p], h);
            B.qg[p] = fma2_rn(mul2_rn(C, B.qw[p]), add2_rn(B.qw[p], NW), h);
        }
    }

    // Prefix t of the register tables for a t that is the same in every lane.
    __device__ __forceinline__ float4 prefix(const LaneBound &B, int t) const {
        switch (t) {
#define TX_CASE(T, P, F) case T: return make_float4(B.qx[P].F, B.qy[P].F, B.qz[P].F, B.qw[P].F);
            TX_CASE(1, 0, x) TX_CASE(2, 0, y) TX_CASE(3, 1, x) TX_CASE(4, 1, y)
            TX_CASE(5, 2, x) TX_CASE(6, 2, y) TX_CASE(7, 3, x) TX_CASE(8, 3, y)
            TX_CASE(9, 4, x) TX_CASE(10, 4, y) TX_CASE(11, 5, x) TX_CASE(12, 5, y)
            TX_CASE(13, 6, x) TX_CASE(14, 6, y) TX_CASE(15, 7, x) TX_CASE(16, 7, y)
#undef TX_CASE
        default: return make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }

    // Row mask of the candidates the least-squares bound keeps among the
    // prefixes k > 2 P0 that complete the row of V (u = its weight):
    // acc + tol - c den = r + qg(k) + w_c V_c Q_c(k) + 2 c u w(k) >= 0.
    template <int P0>
    __device__ __forceinline__ uint32_t row(const LaneBound &B, float r, float vx, float vy, float vz, float u2) const {
        uint32_t mx = 0, my = 0;
        const float2 VX = make_float2(vx, vx), VY = make_float2(vy, vy), VZ = make_float2(vz, vz);
        const float2 R2 = make_float2(r, r), E2 = make_float2(u2, u2);
#pragma unroll
        for (int p = P0; p < 8; ++p) {
            const float2 s = fma2_rn(VX, B.qx[p], fma2_rn(VY, B.qy[p], fma2_rn(VZ, B.qz[p],
                                     fma2_rn(E2, B.qw[p], add2_rn(R2, B.qg[p])))));
            mx = __funnelshift_l(__float_as_uint(s.x), mx, 1);
            my = __funnelshift_l(__float_as_uint(s.y), my, 1);
        }
        return ~(mx | (my << 8));
    }

    // The row's candidates as entries of their own.
    __device__ __forceinline__ void push_each(uint32_t m, int i, int j, int &pos) const {
        while (m) {
            const uint32_t low = m & (0u - m);
            m ^= low;
            sm.rows[pos++ * kLaneThreads + tid] = low | ((uint32_t)j << 16) | ((uint32_t)i << 21);
        }
    }

    // Centred point t of the lane's ordering and its weight.
    __device__ __forceinline__ float4 centred(const LaneBound &B, int t) const {
        const float4 q = sm.pts[t * kLaneThreads + col];
        return make_float4(__fmaf_rn(-B.cx, q.w, q.x), __fmaf_rn(-B.cy, q.w, q.y), __fmaf_rn(-B.cz, q.w, q.z), q.w);
    }

    // Rows (i, j), j = j0 .. min(maxc, J1), of one i for four codes; only
    // prefixes k > 2 P0 are looked at (j0 > 2 P0).  V holds Q(i) + Q(j0) and
    // its weight on entry, Q(i) + Q(j + 1) on return.
    template <int P0, int J1>
    __device__ __forceinline__ void rows(const LaneBound &B, float4 &V, float ki, int i, int &j, int maxc,
                                          uint32_t kmask, int &pos) const {
        const int j1 = min(maxc, J1);
#pragma unroll 1
        for (; j <= j1; ++j) {
            const float vx = cw[0] * V.x, vy = cw[1] * V.y, vz = cw[2] * V.z;
            const float n = __fmaf_rn(vx, V.x, __fmaf_rn(vy, V.y, vz * V.z));
            const float cu = B.c * V.w;
            const float r = __fmaf_rn(cu, __fmaf_rn(-3.0f, B.W, V.w), __fmaf_rn(0.5f, n, ki));
            const uint32_t m = row<P0>(B, r, vx, vy, vz, 2.0f * cu) & kmask & c_row_from[j];
            if (m) sm.rows[pos++ * kLaneThreads + tid] = m | (uint32_t)(j << 16 | i << 21);
            if (j < 16) {
                const float4 q = centred(B, j);
                V.x += q.x; V.y += q.y; V.z += q.z; V.w += q.w;
            }
        }
    }

    __device__ __forceinline__ void push(uint32_t m, int i, int j, int &pos) const {
        if (m) sm.rows[pos++ * kLaneThreads + tid] = m | ((uint32_t)j << 16) | ((uint32_t)i << 21);
    }

    // Prefixes 2 p + 1 and 2 p + 2 for a p that is the same in every lane.
    __device__ __forceinline__ void prefix_pair(const LaneBound &B, int p, float2 (&q)[3], float2 &w) const {
        switch (p) {
#define TX_CASE(P) case P: q[0] = B.qx[P]; q[1] = B.qy[P]; q[2] = B.qz[P]; w = B.qw[P]; break;
            TX_CASE(0) TX_CASE(1) TX_CASE(2) TX_CASE(3) TX_CASE(4) TX_CASE(5) TX_CASE(6)
        default: TX_CASE(7)
#undef TX_CASE
        }
    }

    // The grid filter of the row that prefixes k >= from complete (V: sum of the
    // row's prefixes and their weight; v0: its 5 w(i) + 3 w(j)): every
    // candidate's endpoints are snapped to the 5:6:5 grid as the reference snaps
    // them, and its error on the grid (less -base) is formed in fast arithmetic.
    // Kept are the candidates whose error is below B.cutp and those whose
    // snapping is in doubt.  least takes in the certain errors.
    __device__ __forceinline__ uint32_t grid_row(const LaneBound &B, const float4 V, float v0, int from, float &least) const {
        const float M = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer
        const float grid[3] = {31.0f, 63.0f, 31.0f}, rgrid[3] = {1.0f / 31.0f, 1.0f / 63.0f, 1.0f / 31.0f};
        const float c3[3] = {B.cx, B.cy, B.cz}, V3[3] = {V.x, V.y, V.z};
        uint32_t mx = 0, my = 0;
        auto both = [](float x) { return make_float2(x, x); };
#pragma unroll 1
        for (int p = (from - 1) >> 1; p < 8; ++p) {
            float2 q3[3], w;
            prefix_pair(B, p, q3, w);
            const float2 u = add2_rn(both(V.w), w), v = add2_rn(both(v0), w);
            const float2 nu = make_float2(-u.x, -u.y);
            const float2 den = fma2_rn(nu, u, mul2_rn(both(B.W), v));
            const float2 r = make_float2(rcp_fast(den.x), rcp_fast(den.y));
            const float2 sa = mul2_rn(add2_rn(both(3.0f * B.W), nu), r), sb = mul2_rn(nu, r);
            const float2 al = mul2_rn(both(1.0f / 9.0f), v);
            const float2 g2 = fma2_rn(both(2.0f / 3.0f), u, mul2_rn(both(-2.0f), al));              // 2 gamma
            const float2 be = add2_rn(fma2_rn(both(2.0f / 3.0f), nu, both(B.W)), al);               // beta
            float2 E = make_float2(0.f, 0.f);  // sum_c w_c (alpha a^2 + beta b^2 + 2 gamma a b - 2 A' (a - b)), centred
            float2 d[6];  // distances of the endpoints from their grid values
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float2 A = add2_rn(both(V3[c]), q3[c]);
                float2 ends[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float2 sl = h ? sb : sa;
                    float2 x;  // clamped endpoint
                    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(x.x) : "f"(sl.x), "f"(A.x), "f"(c3[c]));
                    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(x.y) : "f"(sl.y), "f"(A.y), "f"(c3[c]));
                    const float2 t = fma2_rn(x, both(grid[c]), both(M));
                    const float2 n = fma2_rn(t, both(-1.0f), both(M));  // -(rounded grid value)
                    d[2 * c + h] = fma2_rn(x, both(grid[c]), n);
                    ends[h] = fma2_rn(n, both(-rgrid[c] * sq[c]), both(-c3[c] * sq[c]));
                }
                const float2 A2 = mul2_rn(both(2.0f / 3.0f * sq[c]), A), nA2 = mul2_rn(both(-2.0f / 3.0f * sq[c]), A);
                E = fma2_rn(ends[0], fma2_rn(al, ends[0], fma2_rn(g2, ends[1], nA2)), E);
                E = fma2_rn(ends[1], fma2_rn(be, ends[1], A2), E);
            }
            // certain: no endpoint within its error bound of a rounding boundary
            const float2 e = mul2_rn(both(B.doubt), make_float2(fmaxf(fabsf(sa.x), fabsf(sb.x)), fmaxf(fabsf(sa.y), fabsf(sb.y))));
            const bool sx = max3_abs(max3_abs(d[0].x, d[1].x, d[2].x), max3_abs(d[3].x, d[4].x, d[5].x), 0.0f) + fabsf(e.x) <= 0.4999f;
            const bool sy = max3_abs(max3_abs(d[0].y, d[1].y, d[2].y), max3_abs(d[3].y, d[4].y, d[5].y), 0.0f) + fabsf(e.y) <= 0.4999f;
            if (2 * p + 1 >= from) least = fminf(least, sx ? E.x : 1e30f);
            least = fminf(least, sy ? E.y : 1e30f);
            const float2 k = add2_rn(make_float2(sx ? E.x : -1e30f, sy ? E.y : -1e30f), both(-B.cutp));  // kept: negative
            mx = __funnelshift_l(__float_as_uint(k.x), mx, 1);
            my = __funnelshift_l(__float_as_uint(k.y), my, 1);
        }
        return mx | (my << 8);
    }

    // Evaluate every queued candidate of the warp exactly and fold it into its
    // lane's best; empties the queues.
    __device__ __forceinline__ void drain(int &pos) {
        __syncwarp();
        uint32_t n = 0;
        for (int r = 0; r < pos; ++r) n += (uint32_t)__popc(sm.rows[r * kLaneThreads + tid] & 0xFFFFu);
        uint32_t incl = n;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, off);
            if (lane >= off) incl += v;
        }
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
        const bool single = __all_sync(0xFFFFFFFFu, n == (uint32_t)pos);
        for (uint32_t base = 0; base < total; base += 32u) {
            // owner of item base + lane: the first lane whose inclusive count exceeds it
            const uint32_t item = min(base + (uint32_t)lane, total - 1u);
            int own = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const uint32_t c = __shfl_sync(0xFFFFFFFFu, incl, own + step - 1);
                own += c <= item ? step : 0;
            }
            uint32_t rem = item - (__shfl_sync(0xFFFFFFFFu, incl, own) - __shfl_sync(0xFFFFFFFFu, n, own));
            const uint32_t *q = sm.rows + (tid - lane) + own;
            uint32_t e, m;
            if (single) {
                e = q[rem * kLaneThreads];
                m = e & 0xFFFFu;
            } else {
                e = *q;
                uint32_t c = (uint32_t)__popc(e & 0xFFFFu);
                while (rem >= c) {
                    rem -= c;
                    q += kLaneThreads;
                    e = *q;
                    c = (uint32_t)__popc(e & 0xFFFFu);
                }
                m = e & 0xFFFFu;
                while (rem--) m &= m - 1u;
            }
            const int i = (int)(e >> 21), j = (int)((e >> 16) & 31u), k = row_k(__ffs((int)m) - 1);
            const int o = __shfl_sync(0xFFFFFFFFu, col, own);
            float a[3], b[3];
            const float err = lane_exact(sm.pts + o, sm.xs[o], i, j, k, cw, a, b);
            // least (error, candidate) per owner: errors first, then the candidates
            // that have the least error
            const uint32_t hi = err == err ? order_key(err) : 0xFFFFFFFFu, lo = (uint32_t)(i << 10 | j << 5 | k);
            uint32_t *best = reinterpret_cast<uint32_t *>(&sm.best[o]);  // low half: candidate, high half: error
            const uint32_t before = best[1];
            __syncwarp();
            if (hi < before) atomicMin(best + 1, hi);
            __syncwarp();
            const uint32_t after = best[1];
            if (hi == after && after < before) best[0] = kNone;
            __syncwarp();
            if (hi == after) atomicMin(best, lo);
            __syncwarp();
        }
        pos = 0;
    }

    __device__ __forceinline__ float best_err() const { return order_unkey((uint32_t)(sm.best[col] >> 32)); }

    // Climb from a guess to a candidate of larger gain, one boundary moved by
    // one position at a time: its exact error is then a good first threshold
    // (14 -> 6 exact evaluations per block).
    __device__ __forceinline__ void climb(const LaneBound &B, int count, int &i, int &j, int &k) const {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);  // Q(i) + Q(j) + Q(k) and u
        float v = 0.f;
#pragma unroll 4
        for (int t = 0; t < 16; ++t) {
            const float4 q = centred(B, t);
            const float m = (t < i ? 1.0f : 0.0f) + (t < j ? 1.0f : 0.0f) + (t < k ? 1.0f : 0.0f);
            const float d = (t < i ? 5.0f : 0.0f) + (t < j ? 3.0f : 0.0f) + (t < k ? 1.0f : 0.0f);
            a.x = __fmaf_rn(m, q.x, a.x); a.y = __fmaf_rn(m, q.y, a.y); a.z = __fmaf_rn(m, q.z, a.z);
            a.w = __fmaf_rn(m, q.w, a.w);
            v = __fmaf_rn(d, q.w, v);
        }
        auto gain = [&](float x, float y, float z, float u, float vv) {
            const float n = __fmaf_rn(cw[0] * x, x, __fmaf_rn(cw[1] * y, y, (cw[2] * z) * z));
            return n * rcp_fast(__fmaf_rn(-u, u, B.W * vv));
        };
        float best = gain(a.x, a.y, a.z, a.w, v);
#pragma unroll 1
        for (int step = 0; step < 5; ++step) {
            int move = 0;
            float4 na = a;
            float nv = v;
            auto attempt = [&](bool ok, int t, float sign, float n, int id) {
                const float4 q = centred(B, t & 15);
                const float x = __fmaf_rn(sign, q.x, a.x), y = __fmaf_rn(sign, q.y, a.y), z = __fmaf_rn(sign, q.z, a.z);
                const float u = __fmaf_rn(sign, q.w, a.w), vv = __fmaf_rn(sign * n, q.w, v);
                const float g = gain(x, y, z, u, vv);
                if (ok && g > best) { best = g; move = id; na = make_float4(x, y, z, u); nv = vv; }
            };
            attempt(i < j && i + 1 < count, i, 1.0f, 5.0f, 1);
            attempt(i > 0, i - 1, -1.0f, 5.0f, 2);
            attempt(k < count, k, 1.0f, 1.0f, 3);
            attempt(k > j && k > 1, k - 1, -1.0f, 1.0f, 4);
            attempt(j < k, j, 1.0f, 3.0f, 5);
            attempt(j > i, j - 1, -1.0f, 3.0f, 6);
            if (__all_sync(0xFFFFFFFFu, move == 0)) break;
            i += move == 1 ? 1 : move == 2 ? -1 : 0;
            k += move == 3 ? 1 : move == 4 ? -1 : 0;
            j += move == 5 ? 1 : move == 6 ? -1 : 0;
            a = na;
            v = nv;
        }
    }

    // The rest of a sweep, planes i and up, through the grid filter.  A likely
    // plane is looked at first for a low error.
    __device__ __forceinline__ void sweep_grid(LaneBound &B, int count, int maxc, int i, int likely, float &thr, int &pos) {
        const int resume = i;
        bool scout = true;
        uint32_t record = 0;  // the likely plane's row that brought the lowest error
        B.cutp = thr + B.base;
        int j = i = likely;
        float4 V = make_float4(0.f, 0.f, 0.f, 0.f);  // Q(i) + Q(j) of the next row
#pragma unroll 1
        for (;;) {
            float least = 1e30f;
            const float4 qi = prefix(B, i);
            const uint32_t kmask = i < count ? row_upto(count) : 0u;
            if (j == i) V = make_float4(2.0f * qi.x, 2.0f * qi.y, 2.0f * qi.z, 2.0f * qi.w);
            // rows to the end of the plane, or until a queue may overflow
#pragma unroll 1
            do {
                const int from = max(j, 1);
                uint32_t m = grid_row(B, V, __fmaf_rn(3.0f, V.w, 2.0f * qi.w), from, least) & kmask & c_row_from[from];
                if (i == 0 && (j == 0 || j == 16)) m &= ~kOneCluster;
                if (scout) {
                    if (m) record = m | (uint32_t)j << 16;
                    B.cutp = fminf(B.cutp, least);
                } else {
                    push_each(m, i, j, pos);
                    B.cutp = fminf(B.cutp, least + 2.0f * (B.eps + B.tolp));
                }
                const float4 q = centred(B, min(j, 15));
                V.x += q.x; V.y += q.y; V.z += q.z; V.w += q.w;
                ++j;
            } while (j <= maxc && !__any_sync(0xFFFFFFFFu, pos > kRowCap - 19));
            const bool plane = j > maxc;  // the plane is complete
            if (scout && plane) push_each(record & 0xFFFFu, i, (int)(record >> 16), pos);
            // (the filter's own errors tighten the cut, so a queue can fill: 32 cost 1 %)
            if ((plane && (scout || __reduce_add_sync(0xFFFFFFFFu, (unsigned)pos) >= 192u)) ||
                __any_sync(0xFFFFFFFFu, pos > kRowCap - 19))
                drain(pos);
            thr = fminf(thr, fminf(best_err(), least - B.base + B.eps + B.tolp));
            B.cutp = thr + B.base + B.eps + B.tolp;
            if (plane) {
                if (!scout && i + 1 >= maxc) break;
                i = j = scout ? resume : i + 1;
                scout = false;
            }
        }
    }

    // The candidate sweep over the column's ordering (cluster.rs:315-372), by
    // planes of equal i.  Columns of count 0 take part with no candidate.  On
    // return sm.best[col] holds the column's least (error, candidate).
    __device__ __forceinline__ void sweep(LaneBound &B, int count, LaneGuess g) {
        const int maxc = (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)count);
        sm.best[col] = (unsigned long long)order_key(FLT_MAX) << 32 | kNone;
        if (maxc == 0) return;
        int pos = 0;
        g.i = min(g.i, max(count - 1, 0));
        g.j = min(max(g.j, g.i), count);
        g.k = min(max(max(g.k, g.j), 1), max(count, 1));
        climb(B, count, g.i, g.j, g.k);
        if (count > 0) push(row_from_dyn(g.k) & row_upto(g.k), g.i, g.j, pos);
        drain(pos);
        float thr = best_err();
        set_cut(B, thr);
        int i = 0;
        bool grid = false;
#pragma unroll 1
        for (; i < maxc; ++i) {
            const int pos0 = pos;
            const float4 qi = prefix(B, i);
            const uint32_t kmask = i < count ? row_upto(count) : 0u;
            const float ki = __fmaf_rn(-2.0f * B.c * B.W, qi.w, B.tol);
            float4 V = make_float4(2.0f * qi.x, 2.0f * qi.y, 2.0f * qi.z, 2.0f * qi.w);
            int j = i;
            if (i == 0) {
                push(row<0>(B, ki, 0.f, 0.f, 0.f, 0.f) & kmask & ~kOneCluster, 0, 0, pos);
                V = centred(B, 0);
                j = 1;
            }
            rows<0, 4>(B, V, ki, i, j, maxc, kmask, pos);
            rows<2, 8>(B, V, ki, i, j, maxc, kmask, pos);
            rows<4, 12>(B, V, ki, i, j, maxc, kmask, pos);
            rows<6, 16>(B, V, ki, i, j, i == 0 ? min(maxc, 15) : maxc, kmask, pos);
            const unsigned sum = __reduce_add_sync(0xFFFFFFFFu, (unsigned)pos);
            if (sum - __reduce_add_sync(0xFFFFFFFFu, (unsigned)pos0) >= kGridRows) {
                pos = pos0;  // the bound does not separate these blocks' candidates
                grid = true;
                break;
            }
            // evaluate when a queue may overflow in the next plane (17 rows and the
            // two below), or when there is enough to fill the warp (what it finds
            // tightens the bound for the rest)
            if (sum >= 32u || __any_sync(0xFFFFFFFFu, pos > kRowCap - 19)) {
                drain(pos);
                const float t = fminf(thr, best_err());
                if (__any_sync(0xFFFFFFFFu, t < thr)) {
                    thr = t;
                    set_cut(B, thr);
                }
            }
        }
        if (grid) {
            sweep_grid(B, count, maxc, i, min((int)(__reduce_add_sync(0xFFFFFFFFu, (unsigned)g.i) >> 5), maxc - 1), thr, pos);
            thr = fminf(thr, best_err());
        }
        // the one-cluster candidates, unless their own bound excludes them
        if (count == 16 && -(thr + B.base) - B.eps1 <= 0.0f) {
            push(kOneCluster, 0, 0, pos);
            push(kOneCluster, 0, 16, pos);
        }
        drain(pos);
    }

    // The colour half from candidate e of the thread's own column.
    __device__ __forceinline__ uint2 winner(uint32_t e, const ColourSet &cs, const uint32_t (&ord)[2]) const {
        const int i = (int)((e >> 10) & 31u), j = (int)((e >> 5) & 31u), k = (int)(e & 31u);
        float a[3], b[3];
        lane_exact(sm.pts + tid, sm.xs[tid], i, j, k, cw, a, b);
        // the last position that holds a point decides (cluster.rs:397-405)
        uint32_t closest = 0;
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const uint32_t o = 2u * ((ord[m >> 3] >> (4 * (m & 7))) & 15u);
            const uint32_t code = m >= k ? 1u : m >= j ? 3u : m >= i ? 2u : 0u;
            if (m < cs.count) closest = (closest & ~(3u << o)) | (code << o);
        }
        return write4(pack_565(a[0], a[1], a[2]), pack_565(b[0], b[1], b[2]), remap_thread(cs, closest));
    }

    // Deal the CTA's columns out to its threads by kind: a warp's sweep takes as
    // long as its largest set of points, and the grid filter runs for a warp if
    // some of its blocks need it, so blocks of few points, of none and of
    // nearly one colour go together (smooth fields: -6 %).
    __device__ __forceinline__ void deal(int count, bool finite, const LaneGuess &g, bool flat, float4 vw) {
        sm.meta[tid] = (uint32_t)count | (finite ? 32u : 0u) | (uint32_t)g.i << 6 | (uint32_t)g.j << 11 | (uint32_t)g.k << 16;
        sm.xs[tid] = vw;
        if (tid < 64) sm.bins[tid] = 0u;
        __syncthreads();
        const int key = count ? (flat ? 17 : 0) + count : 0;  // 0 .. 33
        const uint32_t at = atomicAdd(&sm.bins[key], 1u);
        __syncthreads();
        if (tid < 32) {  // exclusive sums over the bins
            const uint32_t v0 = sm.bins[lane], v1 = sm.bins[32 + lane];
            uint32_t s0 = v0, s1 = v1;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, s0, off), b = __shfl_up_sync(0xFFFFFFFFu, s1, off);
                if (lane >= off) { s0 += a; s1 += b; }
            }
            sm.bins[lane] = s0 - v0;
            sm.bins[32 + lane] = __shfl_sync(0xFFFFFFFFu, s0, 31) + s1 - v1;
        }
        __syncthreads();
        sm.dealt[sm.bins[key] + at] = (uint32_t)tid;
        __syncthreads();
        col = (int)sm.dealt[tid];
    }

    // The colour half of one block per thread (mask 0: none); every thread of
    // the CTA calls it.
    __device__ __forceinline__ uint2 fit(uint32_t (&px)[16], uint32_t mask, bool aw, const float *unorm,
                                         const float *sqrt_count) {
        const PointCol pt{sm.pts + tid, kLaneThreads};
        ColourSet cs;
        uint2 best = make_uint2(0u, 0u);  // no points: RangeFit on none (range.rs:67-98), as in colour_cluster_team
        float m[6], axis[3], wmin = 1.0f;
        LaneGuess g{0, 0, 0};
        uint32_t ord[2] = {0u, 0u};
        bool finite = true;
        {
            uint32_t a4[4];
            colour_set_thread<BC3>(px, mask, aw, a4, cs);
            if (cs.count == 1) best = single_thread<BC3>(px, cs);
            if (cs.count < 2) cs.count = 0;
            if (cs.count) {
                colour_points_thread(px, a4, cs, aw, unorm, sqrt_count, pt);
                covariance_thread(pt, m);
                principle_component(m, axis);
                if (aw) {
                    wmin = FLT_MAX;
#pragma unroll
                    for (int t = 0; t < 16; ++t)
                        if ((cs.newbits >> t) & 1u) wmin = fminf(wmin, pt[t].w);
                }
                finite = order(cs, axis, ord, g);
            } else {
#pragma unroll
                for (int t = 0; t < 16; ++t) pt[t] = make_float4(0.f, 0.f, 0.f, t < 2 ? 1.0f : 0.0f);
                m[0] = m[3] = m[5] = 0.0f;
            }
        }
        deal(cs.count, finite, g, cw[0] * m[0] + cw[1] * m[3] + cw[2] * m[5] < kFlat, make_float4(m[0], m[3], m[5], wmin));
        const uint32_t meta = sm.meta[col];
        LaneBound B;
        prefixes(B, (meta & 32u) != 0u);
        __syncthreads();
        sweep(B, (int)(meta & 31u), LaneGuess{(int)(meta >> 6 & 31u), (int)(meta >> 11 & 31u), (int)(meta >> 16 & 31u)});
        __syncthreads();
        const uint32_t e = (uint32_t)sm.best[tid];
        return cs.count && e != kNone ? winner(e, cs, ord) : best;
    }
};

}  // namespace tx
