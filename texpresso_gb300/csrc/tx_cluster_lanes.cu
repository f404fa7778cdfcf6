// tx_cluster_lanes.cu -- single-texture ClusterFit kernel of BC2 and BC3 with one
// block per thread (device code in tx_cluster_lanes.cuh).
#include "tx_cluster_lanes.cuh"
#include "tx_internal.h"

namespace tx {

template <int FMT>
__global__ void __launch_bounds__(kLaneThreads, 512 / kLaneThreads) k_cluster_lanes(SrcDesc src, DevParams prm,
                                                                                    uint8_t *__restrict__ out,
                                                                                    size_t nblocks) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ClusterLanes cl(*reinterpret_cast<LaneSmem *>(smem_raw), prm);
    const size_t b = (size_t)blockIdx.x * kLaneThreads + threadIdx.x;
    uint32_t px[16], mask = 0;
    if (b < nblocks) {
        mask = load_block_rgba(src, b, px);
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) px[i] = 0u;
    }
    uint2 al;
    if (FMT == BC2) {
        al = encode_bc2_alpha(px, mask);
    } else {
        uint32_t v[4];
        channel_words(px, 3, v);
        al = encode_bc3_alpha<false>(v, mask);
    }
    __syncthreads();
    const uint2 col = cl.fit(px, mask, prm.alpha_weighted, g_unorm8, g_sqrt_count);
    if (b < nblocks) reinterpret_cast<uint4 *>(out)[b] = make_uint4(al.x, al.y, col.x, col.y);
}

cudaError_t upload_cluster_lane_tables(const uint32_t lut[4][256][2]) { return upload_tables_this_tu(lut); }

// Whether a launch of n blocks goes to this kernel.
//   Size: its CTAs stay for the whole launch or a third of it (one wave of SMs x
//     512 blocks takes 106 us on noisy ramps and 435 us on smooth fields, full or
//     not), so a launch that leaves more than 16 % of its waves' blocks empty goes
//     to the team form, which scales down.  BC3, team / this, noisy ramps: 2048 x
//     2048 (84 % of four waves) 588 / 340 us, 1024 x 1024 (84 % of one) 155 / 106,
//     1000 x 1000 (80 %) 147 / 106, 900 x 900 (65 %) 121 / 102; smooth fields:
//     1,219 / 1,320, 414 / 435, 396 / 444, 332 / 430.  (The line was drawn where
//     smooth fields broke even before the team form left out their bounds.)
//   Weights: the bounds are derived for weights of ordinary size, zero or
//     2^-20 .. 2^20 with one of them not zero (products of smaller or larger ones
//     leave the range where f32 rounding is relative).
bool cluster_lanes_take(int fmt, const DevParams &prm, size_t n, int sm_count) {
    if (fmt != BC2 && fmt != BC3) return false;
    bool any = false;
    for (int c = 0; c < 3; ++c) {
        const float w = prm.w[c];
        if (w == 0.0f) continue;
        if (!(w >= 0x1p-20f && w <= 0x1p20f)) return false;
        any = true;
    }
    const size_t wave = (size_t)sm_count * 512;
    if (!any || wave == 0 || n > 0x7FFFFFFFull * kLaneThreads) return false;
    return n >= (n + wave - 1) / wave * wave / 25 * 21;
}

template <int FMT>
static cudaError_t launch_t(const SrcDesc &src, const DevParams &prm, uint8_t *out, size_t nblocks, cudaStream_t st) {
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 64 || !attr_set[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(k_cluster_lanes<FMT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)sizeof(LaneSmem));
        if (e != cudaSuccess) return e;
        if (dev < 64) attr_set[dev] = true;
    }
    const size_t grid = (nblocks + kLaneThreads - 1) / kLaneThreads;
    k_cluster_lanes<FMT><<<(unsigned)grid, kLaneThreads, sizeof(LaneSmem), st>>>(src, prm, out, nblocks);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_cluster_lanes(int fmt, const SrcDesc &src, const DevParams &prm, uint8_t *out, size_t nblocks,
                                 cudaStream_t st) {
    return fmt == BC2 ? launch_t<BC2>(src, prm, out, nblocks, st) : launch_t<BC3>(src, prm, out, nblocks, st);
}

}  // namespace tx
