// What the one-block-per-SM kernels with converter groups (q8_mid.cu, q8_pair.cu) share: the hand-back
// check of a raw stage and the stores of finished sums.
#pragma once

#include "q8_tile.cuh"
#include "q8_warp_ptx.cuh"

namespace q8 {

// 16 columns of the sums at taddr: what the chains of accumulators, `stride` columns apart, hold together.
__device__ __forceinline__ void load_sums(uint32_t taddr, uint32_t chains, uint32_t stride, uint32_t (&v)[16])
{
    tmem_ld_32x16(taddr, v);
    tmem_ld_wait();
#pragma unroll 1
    for (uint32_t c = 1u; c < chains; ++c) {
        uint32_t more[16];
        taddr += stride;
        tmem_ld_32x16(taddr, more);
        tmem_ld_wait();
#pragma unroll
        for (uint32_t i = 0; i < 16u; ++i) {
            v[i] = __float_as_uint(__uint_as_float(v[i]) + __uint_as_float(more[i]));
        }
    }
}

// Where finished sums go, and what becomes of them (the epilogue codes of q8_launch.h).
struct RowStore {
    void *y;
    const unsigned int *row_map;       // rows of y of the rows of x, or null
    unsigned int ldy;
    unsigned int epilogue;
};

// Every lane has the words of its row, not only asked for them, when the raw stage goes back
// (raw_words_present in q8_tile.cuh says why); true about once in 2^32 loads, and then does nothing.
__device__ __forceinline__ void row_words_present(const uint32_t (&raw)[36], unsigned int *status)
{
    uint32_t all = 0x5F3759DFu;
#pragma unroll
    for (int i = 0; i < 36; ++i) {
        all ^= raw[i];
    }
    if (__any_sync(0xFFFFFFFFu, all == 0u)) {
        atomicOr(status, 0u);
    }
}

// silu(gate) * up (cuda/model/norm.cu:92-105).  The quotient gate / (1 + e^-gate) by a reciprocal and one
// correction of the quotient by its remainder (Markstein's division step) in place of the division
// operator, whose branches kept a storing warp from working on several values at a time: 1300 cycles per
// 8 values a lane, 16 x 32 sums, against 280 for a plain store.  Where the step has no meaning - an infinite gate, a
// divisor that overflows (gate below -88.7) - the remainder is NaN and the quotient stands as it is: infinite, or
// zero, as the operator gives it.
__device__ __forceinline__ float gated_unit(float gate, float up)
{
    const float divisor = 1.0f + expf(-gate);
    const float r = rcp_approx(divisor);
    const float quotient = gate * r;
    const float closer = fmaf(fmaf(-quotient, divisor, gate), r, quotient);
    return (closer == closer ? closer : quotient) * up;
}

// The partial sums of one piece (16 rows of x by 32 rows of w) that other blocks have left in `slots` (one slot
// every `stride` floats, `count` of them) added to v in order; two slots' loads are on their way at a time.
__device__ __forceinline__ void add_partial_sums(uint32_t (&v)[16], const float *slots, unsigned long long stride, uint32_t count)
{
#pragma unroll 1
    for (uint32_t c = 0; c < count; c += 2u) {
        const bool two = c + 1u < count;
        const float *first = slots + c * stride;
        const float *second = two ? first + stride : first;
#pragma unroll
        for (uint32_t h = 0; h < 16u; h += 8u) {
            float a[8], b[8];
#pragma unroll
            for (uint32_t i = 0; i < 8u; ++i) {
                a[i] = __ldcg(first + (h + i) * kRows);
                b[i] = two ? __ldcg(second + (h + i) * kRows) : 0.0f;
            }
#pragma unroll
            for (uint32_t i = 0; i < 8u; ++i) {
                v[h + i] = __float_as_uint(__uint_as_float(v[h + i]) + a[i] + b[i]);
            }
        }
    }
}

// A flag counts the warps that have published their part of a quarter of a partial tile; this many make it whole
// (one warp alone counts for all).
constexpr uint32_t kPublishers = 5;

// What one finished value becomes: stored, added to the float stream (cuda/model/norm.cu:78-89).
template <typename YT>
__device__ __forceinline__ void store_value(const RowStore &to, size_t at, float value)
{
    if (to.epilogue == kEpilogueAdd) {
        float *sum = static_cast<float *>(to.y) + at;
        *sum = *sum + value;
    } else {
        store_out<YT>(static_cast<YT *>(to.y), at, value);
    }
}

// The same values without the detour of store_rows_staged, for columns that are no multiple of four: each lane its
// column (`gated`: each pair of lanes) of ROWS rows of x; `mine` of the warp's 32 rows of w are inside the tensor.
template <typename YT, int ROWS>
__device__ __forceinline__ void store_rows_direct(const RowStore &to, bool gated, uint32_t lane, uint32_t mine, uint32_t first_col,
                                                  uint32_t first_row, uint32_t row_limit, const uint32_t (&v)[ROWS])
{
#pragma unroll
    for (uint32_t i = 0; i < (uint32_t)ROWS; ++i) {
        float value = __uint_as_float(v[i]);
        if (gated) {
            const float other = __shfl_xor_sync(0xFFFFFFFFu, value, 1u);
            value = gated_unit(value, other);
        }
        const uint32_t row_x = first_row + i;
        if (row_x < row_limit && lane < mine && (!gated || (lane & 1u) == 0u)) {
            const uint32_t row_y = to.row_map != nullptr ? to.row_map[row_x] : row_x;
            store_value<YT>(to, (size_t)row_y * to.ldy + first_col + (gated ? lane / 2u : lane), value);
        }
    }
}

// ROWS (16 or 8) rows of x by this warp's 32 columns of y, every lane one column: turned round in shared memory of
// the warp's own and written four values per lane, 2 to 4 store instructions instead of 16 (the
// number of store instructions is what a store costs here, see q8_tile.cuh).  GATED: neighbouring
// lanes hold gate and up of one column (cuda/model/norm.cu:92-105); 16 columns then.
// `columns`: how many of the 32 (16) are inside the tensor, a multiple of four.  MAPPED: row i of x goes to row
// `mapped` of lane i of y, which the caller has from before the sums were there (fetched here, the row map's latency
// came to every 16 rows: q8_mid.cu); else to the row of the same number.
template <typename YT, bool GATED, bool MAPPED, int ROWS>
__device__ __forceinline__ void store_rows_staged(const RowStore &to, uint32_t stage, uint32_t lane, uint32_t first_col,
                                                 uint32_t columns, uint32_t first_row, uint32_t row_limit,
                                                 const uint32_t (&v)[ROWS], uint32_t mapped = 0u)
{
    constexpr uint32_t kColumns = GATED ? 16u : 32u;
    constexpr uint32_t kRowBytes = kColumns * sizeof(YT);
    constexpr uint32_t kLanesPerRow = kColumns / 4u;
    constexpr uint32_t kRowsPerStep = 32u / kLanesPerRow;      // 4 or 8
    constexpr uint32_t kSteps = (uint32_t)ROWS / kRowsPerStep;
    const uint32_t column = GATED ? lane / 2u : lane;
#pragma unroll
    for (uint32_t i = 0; i < (uint32_t)ROWS; ++i) {
        float value = __uint_as_float(v[i]);
        if (GATED) {
            const float other = __shfl_xor_sync(0xFFFFFFFFu, value, 1u);
            value = gated_unit(value, other);
        }
        if (!GATED || (lane & 1u) == 0u) {
            if (sizeof(YT) == 4) {
                st_shared_b32(stage + i * kRowBytes + column * 4u, __float_as_uint(value));
            } else {
                st_shared_b16(stage + i * kRowBytes + column * 2u, out_bits<YT>(value));
            }
        }
    }
    __syncwarp();
    const uint32_t part = lane % kLanesPerRow;
    const bool adds = !GATED && sizeof(YT) == 4 && to.epilogue == kEpilogueAdd;
    YT *at[kSteps];
#pragma unroll
    for (uint32_t step = 0; step < kSteps; ++step) {
        const uint32_t local = step * kRowsPerStep + lane / kLanesPerRow;
        const uint32_t row_x = first_row + local;
        const uint32_t row_y = MAPPED ? __shfl_sync(0xFFFFFFFFu, mapped, local) : row_x;
        at[step] = nullptr;
        if (row_x < row_limit && part * 4u < columns) {
            at[step] = static_cast<YT *>(to.y) + (size_t)row_y * to.ldy + first_col + part * 4u;
        }
    }
    float4 before[kSteps];
    if (adds) {
        // one rounded add per value; the old values are fetched together, before the first store
#pragma unroll
        for (uint32_t step = 0; step < kSteps; ++step) {
            before[step] = at[step] != nullptr ? *reinterpret_cast<const float4 *>(at[step]) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
#pragma unroll
    for (uint32_t step = 0; step < kSteps; ++step) {
        const uint32_t from = stage + (step * kRowsPerStep + lane / kLanesPerRow) * kRowBytes + part * 4u * sizeof(YT);
        if (sizeof(YT) == 4) {
            uint32_t a, b, c, d;
            ld_shared_v4(from, a, b, c, d);
            float4 piece = make_float4(__uint_as_float(a), __uint_as_float(b), __uint_as_float(c), __uint_as_float(d));
            if (adds) {
                piece = make_float4(before[step].x + piece.x, before[step].y + piece.y, before[step].z + piece.z,
                                    before[step].w + piece.w);
            }
            if (at[step] != nullptr) {
                *reinterpret_cast<float4 *>(at[step]) = piece;
            }
        } else {
            uint32_t a, b;
            ld_shared_v2(from, a, b);
            if (at[step] != nullptr) {
                *reinterpret_cast<uint2 *>(at[step]) = make_uint2(a, b);
            }
        }
    }
}

} // namespace q8
