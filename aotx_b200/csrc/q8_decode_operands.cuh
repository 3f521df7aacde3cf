// What the kernels that multiply from registers (q8_decode_warp.cu, q8_decode_rows.cu) share: the layout of x in shared
// memory and the operands of the MMA.
#pragma once

#include "q8_tile.cuh"
#include "q8_warp_ptx.cuh"

namespace q8 {

constexpr uint32_t kWarpXRow = 528;        // bytes of a row of x in a stage: 256 halves and a shift of 16 bytes

// Bring a row piece of x into the order of the weights and store it: `v` holds halves 8 lane ..
// 8 lane + 7 of the segment.  Blocks of 32 weights are 4 lanes; even blocks are turned by two
// halves (one word), so a lane needs its neighbour's first word.
template <bool BF>
__device__ __forceinline__ void stage_x_row(uint4 v, uint32_t row_at, uint32_t lane)
{
    if (BF) {
        v.x = bf16x2_to_f16x2(v.x);
        v.y = bf16x2_to_f16x2(v.y);
        v.z = bf16x2_to_f16x2(v.z);
        v.w = bf16x2_to_f16x2(v.w);
    }
    const uint32_t next = __shfl_sync(0xFFFFFFFFu, v.x, (int)((lane & ~3u) | ((lane + 1u) & 3u)));
    if ((lane & 4u) == 0u) {
        v = make_uint4(v.y, v.z, v.w, next);
    }
    // step = two per block, lane t of the MMA: halves 4t .. 4t+3 of the step's sixteen
    const uint32_t step = ((lane >> 2) & 1u) * 2u + ((lane >> 1) & 1u);
    const uint32_t at = row_at + (lane >> 3) * 128u + (lane & 1u) * 64u + step * 8u;
    st_shared_v2(at, v.x, v.y);
    st_shared_v2(at + 32u, v.z, v.w);
}

// The halves of one 32-weight block of rows g and g + 8 as the two steps' A operands.
__device__ __forceinline__ void block_operands(const uint32_t (&first)[2], const uint32_t (&second)[2],
                                               const uint32_t (&d_bits)[2], uint32_t (&a)[2][4])
{
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const __half2 d2 = *reinterpret_cast<const __half2 *>(&d_bits[r]);
        const uint32_t f0 = first[r] ^ 0x80808080u;
        const uint32_t f1 = second[r] ^ 0x80808080u;
        a[0][r] = dequant_pair<0>(f0, d2);
        a[0][r + 2] = dequant_pair<1>(f0, d2);
        a[1][r] = dequant_pair<0>(f1, d2);
        a[1][r + 2] = dequant_pair<1>(f1, d2);
    }
}

// Block b of a segment of two rows of w as the two steps' A operands; `row0` and `row1` are the segment's first word of the
// rows, and the lane's (t) word further.
__device__ __forceinline__ void block_of_rows(const unsigned char *row0, const unsigned char *row1, uint32_t t, uint32_t turn,
                                              uint32_t b, uint32_t (&a)[2][4])
{
    // the block's scale is in word 0 (low half) or 8 (high half) of its pair
    const uint32_t word0 = (b / 2u) * 68u + (b & 1u) * 32u;
    uint32_t first[2], second[2], d_bits[2];
#pragma unroll
    for (uint32_t r = 0; r < 2u; ++r) {
        const unsigned char *row = (r == 0u ? row0 : row1) + word0;
        const uint32_t scale = *reinterpret_cast<const uint32_t *>(row - 4u * t);
        first[r] = *reinterpret_cast<const uint32_t *>(row + 4u);
        second[r] = *reinterpret_cast<const uint32_t *>(row + 20u);
        if ((b & 1u) == 0u) {
            second[r] = prmt(second[r], scale, turn);
            d_bits[r] = prmt(scale, scale, 0x1010u);
        } else {
            d_bits[r] = prmt(scale, scale, 0x3232u);
        }
    }
    block_operands(first, second, d_bits, a);
}

} // namespace q8
