// tx_decode.cu -- BCn decoders (Format::decompress, lib/src/lib.rs:124-156;
// decompress_block, lib/src/lib.rs:240-277; colourblock::decompress,
// lib/src/colourblock.rs:97-169; alpha::decompress_bc2/bc3,
// lib/src/alpha.rs:53-68, :258-304).  One thread per block; integer only.
#include "tx_device.cuh"
#include "tx_internal.h"

namespace tx {

__device__ __forceinline__ uint32_t expand565(uint32_t v) {
    const uint32_t r = (v >> 11) & 0x1Fu, g = (v >> 5) & 0x3Fu, b = v & 0x1Fu;
    return ((r << 3) | (r >> 2)) | (((g << 2) | (g >> 4)) << 8) | (((b << 3) | (b >> 2)) << 16) | 0xFF000000u;
}

// 16 RGBA8 pixels of a BC1/BC2/BC3 colour block.  The colour of an index is
// picked by selects: an indexed array would live in local memory.
__device__ __forceinline__ void decode_colour(uint2 blk, bool is_bc1, uint32_t (&px)[16]) {
    const uint32_t a = blk.x & 0xFFFFu, b = blk.x >> 16;
    const uint32_t c0 = expand565(a), c1 = expand565(b);
    uint32_t c2 = 0, c3 = 0;
    const bool three = is_bc1 && a <= b;
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
        const uint32_t c = (c0 >> (8 * ch)) & 0xFFu, d = (c1 >> (8 * ch)) & 0xFFu;
        if (three) { c2 |= ((c + d) / 2) << (8 * ch); }
        else { c2 |= ((2 * c + d) / 3) << (8 * ch); c3 |= ((c + 2 * d) / 3) << (8 * ch); }
    }
    c2 |= 0xFF000000u;
    if (!three) c3 |= 0xFF000000u;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const bool lo = (blk.y >> (2 * i)) & 1u, hi = (blk.y >> (2 * i + 1)) & 1u;
        px[i] = hi ? (lo ? c3 : c2) : (lo ? c1 : c0);
    }
}

// The values of a BC3/BC4/BC5 alpha block: byte c of v[r] is pixel 4 r + c.  The
// 8 codes are the bytes of two words, picked four pixels at a time by prmt.
__device__ __forceinline__ void decode_alpha8(uint2 blk, uint32_t (&v)[4]) {
    const uint32_t a0 = blk.x & 0xFFu, a1 = (blk.x >> 8) & 0xFFu;
    uint32_t code[8];
    code[0] = a0; code[1] = a1;
    if (a0 <= a1) {
#pragma unroll
        for (uint32_t i = 1; i < 5; ++i) code[1 + i] = ((5 - i) * a0 + i * a1) / 5;
        code[6] = 0; code[7] = 255;
    } else {
#pragma unroll
        for (uint32_t i = 1; i < 7; ++i) code[1 + i] = ((7 - i) * a0 + i * a1) / 7;
    }
    const uint32_t lo = code[0] | code[1] << 8 | code[2] << 16 | code[3] << 24;
    const uint32_t hi = code[4] | code[5] << 8 | code[6] << 16 | code[7] << 24;
    const uint32_t f[4] = {(blk.x >> 16) & 0xFFFu, (blk.x >> 28 | blk.y << 4) & 0xFFFu, (blk.y >> 8) & 0xFFFu, blk.y >> 20};
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        uint32_t sel = (f[r] & 0x03Fu) | ((f[r] & 0xFC0u) << 2);  // 3-bit fields to nibbles
        sel = (sel & 0x0707u) | ((sel & 0x3838u) << 1);
        v[r] = prmt(lo, hi, sel);
    }
}

// One block per thread.  Bound by HBM (8 or 16 bytes in, 64 out) as long as the
// stores are wide: each full row of a block is one 16-byte store (vec: the image
// and its pitch are 16-byte aligned), so a warp writes 512 contiguous bytes;
// edge blocks and other alignments store pixel by pixel.  BC3 2048x2048: 35.2 us
// with byte stores and indexed codes in local memory, 8.3 us now (2.5 TB/s).
template <int FMT>
__global__ void __launch_bounds__(128) k_decode(const uint8_t *__restrict__ data, SrcDesc div, size_t blocks_wide,
                                                size_t block_rows, size_t width, size_t height,
                                                uint8_t *__restrict__ out, size_t out_pitch, size_t out_len, bool vec) {
    const size_t b = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= blocks_wide * block_rows) return;
    size_t bx, by;
    if (div.blocks_wide) {
        uint32_t x, y;
        block_coords(div, b, x, y);
        bx = x;
        by = y;
    } else {
        bx = b % blocks_wide;
        by = b / blocks_wide;
    }
    uint32_t px[16];
    const uint2 *blk = reinterpret_cast<const uint2 *>(data + b * block_bytes(FMT));
    const uint2 first = blk[0];
    if (FMT == BC1) decode_colour(first, true, px);
    if (FMT == BC2 || FMT == BC3) decode_colour(blk[1], false, px);
    if (FMT == BC2) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const uint32_t q = ((i < 8 ? first.x : first.y) >> (4 * (i & 7))) & 0xFu;
            px[i] = (px[i] & 0x00FFFFFFu) | (q * 0x11u << 24);
        }
    } else if (FMT == BC3 || FMT == BC4) {
        uint32_t v[4];
        decode_alpha8(first, v);
#pragma unroll
        for (int i = 0; i < 16; ++i)
            px[i] = FMT == BC3 ? prmt(px[i], v[i >> 2], 0x4210u + 0x1000u * (uint32_t)(i & 3))
                               : prmt(v[i >> 2], 0xFFu, 0x4000u + 0x111u * (uint32_t)(i & 3));
    } else if (FMT == BC5) {
        uint32_t r[4], g[4];
        decode_alpha8(first, r);
        decode_alpha8(blk[1], g);
#pragma unroll
        for (int i = 0; i < 16; ++i)
            px[i] = (prmt(r[i >> 2], g[i >> 2], 0x40u + 0x11u * (uint32_t)(i & 3)) & 0xFFFFu) | 0xFF000000u;
    }
#pragma unroll
    for (int py = 0; py < 4; ++py) {
        const size_t y = 4 * by + py;
        if (y >= height) continue;
        const size_t o = y * out_pitch + 16 * bx;
        if (vec && 4 * bx + 4 <= width && o + 16 <= out_len) {
            *reinterpret_cast<uint4 *>(out + o) = make_uint4(px[4 * py], px[4 * py + 1], px[4 * py + 2], px[4 * py + 3]);
            continue;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (4 * bx + c < width && o + 4 * c + 4 <= out_len) {
                uint8_t *d = out + o + 4 * c;
                const uint32_t v = px[4 * py + c];
                if ((reinterpret_cast<uintptr_t>(d) & 3u) == 0) {
                    *reinterpret_cast<uint32_t *>(d) = v;
                } else {
                    d[0] = (uint8_t)v; d[1] = (uint8_t)(v >> 8); d[2] = (uint8_t)(v >> 16); d[3] = (uint8_t)(v >> 24);
                }
            }
        }
    }
}

cudaError_t launch_decode(int fmt, const uint8_t *data, size_t blocks_wide, size_t block_rows, size_t width,
                          size_t height, uint8_t *out, size_t out_pitch, size_t out_len, cudaStream_t st) {
    const size_t n = blocks_wide * block_rows;
    if (n == 0) return cudaSuccess;
    const unsigned grid = (unsigned)((n + 127) / 128);
    const bool vec = reinterpret_cast<uintptr_t>(out) % 16 == 0 && out_pitch % 16 == 0;
    SrcDesc div{};  // only its division by blocks_wide
    if (blocks_wide <= 0xFFFFFFFFull) set_blocks_wide(div, (uint32_t)blocks_wide);
    auto go = [&](auto kernel) {
        kernel<<<grid, 128, 0, st>>>(data, div, blocks_wide, block_rows, width, height, out, out_pitch, out_len, vec);
    };
    switch (fmt) {
    case BC1: go(k_decode<BC1>); break;
    case BC2: go(k_decode<BC2>); break;
    case BC3: go(k_decode<BC3>); break;
    case BC4: go(k_decode<BC4>); break;
    case BC5: go(k_decode<BC5>); break;
    default: return cudaErrorInvalidValue;
    }
    note_launch();
    return cudaGetLastError();
}

}  // namespace tx
