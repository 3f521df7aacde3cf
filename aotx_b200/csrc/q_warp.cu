// Products with the block types and shapes that the TMA kernels do not take, on the warp-level
// tensor path: Q8_0 rows of any multiple of 32 weights at any even address, and Q4_0, Q4_1, Q5_0,
// Q5_1, Q4_K, Q5_K, Q6_K.  (F32, F16, Q2_K, Q3_K and unaligned activations stay with the decoders on
// the ordinary cores, q_generic.cu and q8_simt_gemv.cuh.)
//
// A weight of these formats is s * q + o with one scale s (and offset o) per 32 weights, 16 in
// Q6_K, and q a small whole number.  The whole numbers go through the MMA as they are - exact in
// binary16 and in bfloat16, so x is read in whichever of the two it comes - and a block's sums
// are scaled in float afterwards: sum += s * (q . x) + o * (1 . x).  No weight is rounded to 16
// bits, as in the reference's memory-bound kernel (cuda/model/matrix.cuh:493-670).
//
// HBM-bound at these batches: rows are read once per 16 rows of x (the passes of a longer batch
// run side by side and meet the row in L2).  The rows of one MMA operand (16) belong to a block,
// whose 8 warps split the depth; a warp keeps its own ring of pieces of 128 or 256 weights per
// row in flight with 16-byte asynchronous copies - rows start at any even address, so a piece is
// copied as the 16-byte units that cover it and read from its own offset - and needs no other
// warp until the 8 partial sums of a row group are added.  Two blocks of 8 warps per SM keep about
// 100 KB in flight.  The kernels on the ordinary cores read a row two bytes per lane and 34 bytes
// apart: 5003 x 2912 at 7 rows took 137 us, Q4_K 14336 x 4096 at 4 rows 86 us.
#include "q8_launch.h"
#include "q8_tile.cuh"
#include "q8_warp_ptx.cuh"
#include "q_blocks.cuh"

namespace q8 {

constexpr uint32_t kAnyWarps = 8;
constexpr uint32_t kAnyRows = 16;

template <uint32_t TYPE>
struct AnyShape {
    static constexpr bool super = TYPE == kTypeQ4_K || TYPE == kTypeQ5_K || TYPE == kTypeQ6_K;
    static constexpr bool offset = TYPE == kTypeQ4_1 || TYPE == kTypeQ5_1 || TYPE == kTypeQ4_K || TYPE == kTypeQ5_K;
    static constexpr bool sixteens = TYPE == kTypeQ6_K;          // a scale per 16 weights
    // rows (and everything in them) start on multiples of 4 when the tensor does
    static constexpr bool words = TYPE == kTypeQ4_1 || TYPE == kTypeQ5_1 || TYPE == kTypeQ4_K || TYPE == kTypeQ5_K;
    static constexpr uint32_t block_bytes = TYPE == kTypeQ4_0   ? 18
                                            : TYPE == kTypeQ4_1 ? 20
                                            : TYPE == kTypeQ5_0 ? 22
                                            : TYPE == kTypeQ5_1 ? 24
                                            : TYPE == kTypeQ8_0 ? 34
                                            : TYPE == kTypeQ4_K ? 144
                                            : TYPE == kTypeQ5_K ? 176
                                                                : 210;
    static constexpr uint32_t piece_runs = super ? 8 : 4;        // runs of 32 weights per piece
    static constexpr uint32_t piece_bytes = super ? block_bytes : 4 * block_bytes;
    static constexpr uint32_t units = (piece_bytes + 14 + 15) / 16;   // 16-byte units that can touch a piece
    static constexpr uint32_t slot = 16 * (units | 1u);          // 8 rows of a slot start 4 * odd words apart
    static constexpr uint32_t stage = kAnyRows * slot;
};

// A warp's ring: four pieces in flight or in use, three where four would leave room for one block on an SM only (Q6_K,
// and Q5_K at 16 rows of x: the grid below has two blocks per SM, which then ran one behind the other; Q6_K 14336 x
// 4096, 4 rows, 25.8 us against 18.2, 16 rows, 36.4 against 30.0).
template <uint32_t TYPE, uint32_t TILES>
struct AnyRing {
    static constexpr uint32_t sums_bytes = 2u * kAnyWarps * 8u * TILES * kAnyRows * 4u;
    static constexpr uint32_t most_bytes = (228u * 1024u) / 2u - 1024u;      // two blocks' shared memory on one SM
    static constexpr uint32_t depth = kAnyWarps * 4u * AnyShape<TYPE>::stage + sums_bytes <= most_bytes ? 4u : 3u;
    static constexpr uint32_t warp_bytes = depth * AnyShape<TYPE>::stage;
    static constexpr uint32_t smem_bytes = kAnyWarps * warp_bytes;
    static_assert(smem_bytes + sums_bytes <= most_bytes, "two blocks' shared memory on one SM");
};

// Four codes of 8 bits as the two operand words of an MMA step.  Codes are whole numbers below 64
// (bias 0, 8, 16 or 32 is taken away), or signed bytes.
template <uint32_t TYPE, bool BF>
__device__ __forceinline__ void codes_to_operands(uint32_t codes, uint32_t &low, uint32_t &high)
{
    constexpr uint32_t bias = TYPE == kTypeQ4_0 ? 8u : TYPE == kTypeQ5_0 ? 16u : TYPE == kTypeQ6_K ? 32u : 0u;
    if (BF) {
        // 0x4300 is 128, one unit per step of the mantissa: 128 + code is exact
        const uint32_t a = prmt(codes, 0x43434343u, 0x4140u);
        const uint32_t b = prmt(codes, 0x43434343u, 0x4342u);
        if (TYPE == kTypeQ8_0) {
            // a signed byte: 128 + (q & 127), less 128 or (q negative) 256 = 0x4380
            const uint32_t a7 = a & 0xFF7FFF7Fu, a8 = a & 0xFF80FF80u, b7 = b & 0xFF7FFF7Fu, b8 = b & 0xFF80FF80u;
            const __nv_bfloat162 l = __hsub2(*reinterpret_cast<const __nv_bfloat162 *>(&a7), *reinterpret_cast<const __nv_bfloat162 *>(&a8));
            const __nv_bfloat162 h = __hsub2(*reinterpret_cast<const __nv_bfloat162 *>(&b7), *reinterpret_cast<const __nv_bfloat162 *>(&b8));
            low = *reinterpret_cast<const uint32_t *>(&l);
            high = *reinterpret_cast<const uint32_t *>(&h);
        } else {
            const uint32_t zero = 0x43004300u + bias * 0x00010001u;
            const __nv_bfloat162 z = *reinterpret_cast<const __nv_bfloat162 *>(&zero);
            const __nv_bfloat162 l = __hsub2(*reinterpret_cast<const __nv_bfloat162 *>(&a), z);
            const __nv_bfloat162 h = __hsub2(*reinterpret_cast<const __nv_bfloat162 *>(&b), z);
            low = *reinterpret_cast<const uint32_t *>(&l);
            high = *reinterpret_cast<const uint32_t *>(&h);
        }
    } else {
        // 0x6400 is 1024, one unit per step of the mantissa
        const uint32_t c = TYPE == kTypeQ8_0 ? codes ^ 0x80808080u : codes;
        const uint32_t a = prmt(c, 0x64646464u, 0x4140u);
        const uint32_t b = prmt(c, 0x64646464u, 0x4342u);
        const uint32_t zero = 0x64006400u + (TYPE == kTypeQ8_0 ? 128u : bias) * 0x00010001u;
        const __half2 z = *reinterpret_cast<const __half2 *>(&zero);
        const __half2 l = __hsub2(*reinterpret_cast<const __half2 *>(&a), z);
        const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&b), z);
        low = *reinterpret_cast<const uint32_t *>(&l);
        high = *reinterpret_cast<const uint32_t *>(&h);
    }
}

__device__ __forceinline__ float half_bits(uint32_t bits)
{
    return __half2float(__ushort_as_half((unsigned short)bits));
}

// Where a row of a piece lies in the warp's ring: a word index, and whether its bytes start in the
// middle of that word (rows start at any even address).  Every read below is then at a constant
// distance from that index, and a word that straddles two is put together with a selector that is
// one of two constants per row.
struct RowAt {
    const uint32_t *words;         // the word that holds (or precedes by two bytes) the first byte
    const unsigned char *bytes;    // the first byte
    uint32_t even, odd;            // selectors of a word at a distance of 4 i and 4 i + 2 bytes
};

// The word `C` + 4 * t bytes from the start of the row's piece (C even).
template <bool WORDS, uint32_t C>
__device__ __forceinline__ uint32_t word_at(const RowAt &row, uint32_t t)
{
    if constexpr (WORDS) {
        return row.words[C / 4u + t];
    } else {
        return prmt(row.words[C / 4u + t], row.words[C / 4u + t + 1u], C % 4u == 0u ? row.even : row.odd);
    }
}

template <uint32_t C>
__device__ __forceinline__ uint32_t u16_at(const RowAt &row)
{
    return reinterpret_cast<const unsigned short *>(row.bytes)[C / 2u];
}

// Bits b0..b3 of `four` as bit 4 of the four bytes of a word.
__device__ __forceinline__ uint32_t fifth_bits(uint32_t four)
{
    four &= 15u;
    return ((four | (four << 7) | (four << 14) | (four << 21)) & 0x01010101u) << 4;
}

// Which weights of a run of 32 a lane takes does not matter to the sum, as long as x goes with them.  WIDE: 8t ..
// 8t + 7, so that a lane's x of a run is one load of 16 bytes; else 4t .. 4t + 3 and 16 + 4t .. + 3, two loads of 8.
// What a warp's load of x costs is its 8 rows, not its bytes; what the wide form costs is two weight words from
// one nibble plane, and rows of words two apart.  Measured, wide against not: Q8_0 30000 x 2912, 7 rows, 30.5 us
// against 34.0, 5003 x 2912, 40 rows, 26.7 against 28.2; Q4_K 14336 x 4096, 4 rows, 15.3 against 16.3, 30 rows
// (two columns of eight) 49.1 against 47.9; Q4_0, 4 rows, 17.2 against 16.0.  Q6_K has a scale per step.
template <uint32_t TYPE, uint32_t TILES>
__host__ __device__ constexpr bool any_wide()
{
    return TYPE == kTypeQ8_0 || (TILES == 1u && (TYPE == kTypeQ4_K || TYPE == kTypeQ5_K));
}

// One run of 32 weights of the formats whose block is a run (run R of the piece).
template <uint32_t TYPE, uint32_t R>
__device__ __forceinline__ void one_run(const RowAt &row, uint32_t t, uint32_t (&codes)[4][2], float (&scale)[8], float (&off)[4])
{
    using S = AnyShape<TYPE>;
    constexpr bool W = S::words;
    constexpr uint32_t at = R * S::block_bytes;
    scale[R] = half_bits(u16_at<at>(row));
    if constexpr (TYPE == kTypeQ8_0) {
        codes[R][0] = word_at<W, at + 2u>(row, 2u * t);
        codes[R][1] = word_at<W, at + 6u>(row, 2u * t);
    } else {
        constexpr bool five = TYPE == kTypeQ5_0 || TYPE == kTypeQ5_1;
        constexpr uint32_t head = S::offset ? 4u : 2u;
        if constexpr (S::offset) {
            off[R] = half_bits(u16_at<at + 2u>(row));
        }
        const uint32_t pairs = word_at<W, at + head + (five ? 4u : 0u)>(row, t);
        codes[R][0] = pairs & 0x0F0F0F0Fu;
        codes[R][1] = (pairs >> 4) & 0x0F0F0F0Fu;
        if constexpr (five) {
            const uint32_t bits = word_at<W, at + head>(row, 0u);
            codes[R][0] |= fifth_bits(bits >> (4u * t));
            codes[R][1] |= fifth_bits(bits >> (16u + 4u * t));
        }
    }
}

// The codes of four runs of 32 weights (runs 4 * HALF .. + 3 of the piece) that lane t of a
// row's four lanes holds: codes[run][step], weights 16 step + 4t .. + 3 or (WIDE) 8t + 4 step .. + 3; and the runs' scales and
// offsets (Q6_K: scale[2 * run + step]).
template <uint32_t TYPE, uint32_t HALF, bool WIDE>
__device__ __forceinline__ void four_runs(const RowAt &row, uint32_t t, uint32_t (&codes)[4][2], float (&scale)[8],
                                          float (&off)[4])
{
    using S = AnyShape<TYPE>;
    constexpr bool W = S::words;
    if constexpr (!S::super) {
        one_run<TYPE, 0>(row, t, codes, scale, off);
        one_run<TYPE, 1>(row, t, codes, scale, off);
        one_run<TYPE, 2>(row, t, codes, scale, off);
        one_run<TYPE, 3>(row, t, codes, scale, off);
    } else if constexpr (TYPE == kTypeQ4_K || TYPE == kTypeQ5_K) {
        const float d = half_bits(row.words[0] & 0xFFFFu);
        const float dmin = half_bits(row.words[0] >> 16);
        // twelve bytes of 6-bit scales and minima: words p0 (scales 0-3 and two bits of 4-7), p1
        // (minima likewise), p2 (four bits each of scales and minima 4-7)
        const uint32_t p0 = row.words[1];
        const uint32_t p1 = row.words[2];
        uint32_t sc = p0 & 0x3F3F3F3Fu;
        uint32_t mn = p1 & 0x3F3F3F3Fu;
        if constexpr (HALF != 0u) {
            const uint32_t p2 = row.words[3];
            sc = (p2 & 0x0F0F0F0Fu) | ((p0 >> 2) & 0x30303030u);
            mn = ((p2 >> 4) & 0x0F0F0F0Fu) | ((p1 >> 2) & 0x30303030u);
        }
#pragma unroll
        for (uint32_t r = 0; r < 4u; ++r) {
            // 0x4B000000 is 2^23, one unit per step of the mantissa: a whole number by a byte permute and an
            // exact subtraction; the conversion instruction runs at a quarter of their rate
            scale[r] = d * (__uint_as_float(prmt(sc, 0x4B000000u, 0x7650u + r)) - 8388608.0f);
            off[r] = dmin * (8388608.0f - __uint_as_float(prmt(mn, 0x4B000000u, 0x7650u + r)));
        }
        constexpr uint32_t nibbles = (TYPE == kTypeQ5_K ? 48u : 16u) + HALF * 64u;
#pragma unroll
        for (uint32_t c = 0; c < 2u; ++c) {
#pragma unroll
            for (uint32_t step = 0; step < 2u; ++step) {
                const uint32_t w = row.words[nibbles / 4u + c * 8u + (WIDE ? 2u * t + step : step * 4u + t)];
                codes[2u * c][step] = w & 0x0F0F0F0Fu;
                codes[2u * c + 1u][step] = (w >> 4) & 0x0F0F0F0Fu;
            }
        }
        if constexpr (TYPE == kTypeQ5_K) {
#pragma unroll
            for (uint32_t step = 0; step < 2u; ++step) {
                const uint32_t w = row.words[4u + (WIDE ? 2u * t + step : step * 4u + t)] >> (4u * HALF);
#pragma unroll
                for (uint32_t r = 0; r < 4u; ++r) {
                    codes[r][step] |= ((w >> r) & 0x01010101u) << 4;
                }
            }
        }
    } else {
        // Q6_K: the half's 128 weights are four quarters of 32
        const float d = half_bits(u16_at<208>(row));
#pragma unroll
        for (uint32_t step = 0; step < 2u; ++step) {
            const uint32_t n0 = step == 0u ? word_at<W, HALF * 64u>(row, t) : word_at<W, HALF * 64u + 16u>(row, t);
            const uint32_t n1 = step == 0u ? word_at<W, HALF * 64u + 32u>(row, t) : word_at<W, HALF * 64u + 48u>(row, t);
            const uint32_t up = step == 0u ? word_at<W, 128u + HALF * 32u>(row, t) : word_at<W, 144u + HALF * 32u>(row, t);
            codes[0][step] = (n0 & 0x0F0F0F0Fu) | ((up << 4) & 0x30303030u);
            codes[1][step] = (n1 & 0x0F0F0F0Fu) | ((up << 2) & 0x30303030u);
            codes[2][step] = ((n0 >> 4) & 0x0F0F0F0Fu) | (up & 0x30303030u);
            codes[3][step] = ((n1 >> 4) & 0x0F0F0F0Fu) | ((up >> 2) & 0x30303030u);
        }
        const uint32_t s0 = word_at<W, 192u + 8u * HALF>(row, 0u);
        const uint32_t s1 = word_at<W, 196u + 8u * HALF>(row, 0u);
#pragma unroll
        for (uint32_t i = 0; i < 4u; ++i) {
            scale[i] = d * (float)(int)(signed char)(s0 >> (8u * i));
            scale[4u + i] = d * (float)(int)(signed char)(s1 >> (8u * i));
        }
    }
}

struct AnyArgs {
    const unsigned char *w;
    const void *x;
    void *y;
    const unsigned int *m_dev;
    unsigned long long row_bytes;
    uint32_t n, k, m_max;
    uint32_t y_dtype, epilogue;
    uint32_t wide_x;               // x starts on a 16-byte boundary
};

// One product weight by weight by a warp, as the kernels on the ordinary cores form it (lanes take runs 32 apart, their
// parts are added in a tree): what a sum in whole-number form is replaced by when it is not finite.  There s * q and
// o of one weight meet x apart, so an infinite x can give NaN where the weight times x is infinite, and q * x can
// leave the float range where s * q * x does not.
template <uint32_t TYPE, bool BF>
__device__ __noinline__ float sum_by_weights(const unsigned char *row, const unsigned short *x, uint32_t runs)
{
    float sum = 0.0f;
#pragma unroll 1
    for (uint32_t run = threadIdx.x & 31u; run < runs; run += 32u) {
        float values[32];
        decode_run(TYPE, row, run, values);
#pragma unroll
        for (uint32_t i = 0; i < 32u; ++i) {
            const uint32_t bits = x[run * 32u + i];
            sum = fmaf(values[i], BF ? __uint_as_float(bits << 16) : half_bits(bits), sum);
        }
    }
#pragma unroll
    for (uint32_t step = 16u; step != 0u; step >>= 1) {
        sum += __shfl_down_sync(0xFFFFFFFFu, sum, step);
    }
    return __shfl_sync(0xFFFFFFFFu, sum, 0);
}

template <uint32_t TYPE, bool BF, uint32_t TILES>
__global__ void __launch_bounds__(kAnyWarps * 32u, 2)
q_gemv_any_kernel_warp(const AnyArgs args)
{
    using S = AnyShape<TYPE>;
    using R = AnyRing<TYPE, TILES>;
    constexpr uint32_t kAnyDepth = R::depth;
    constexpr bool kWide = any_wide<TYPE, TILES>();
    extern __shared__ __align__(16) unsigned char any_smem_[];
    __shared__ float parts[2][kAnyWarps][8u * TILES][kAnyRows];   // partial sums of the 8 warps, two row groups in turn
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t g = lane >> 2;
    const uint32_t t = lane & 3u;
    const uint32_t runs = args.k / 32u;
    const uint32_t pieces = (runs + S::piece_runs - 1u) / S::piece_runs;
    const uint32_t first_piece = pieces * warp / kAnyWarps;
    const uint32_t my_pieces = pieces * (warp + 1u) / kAnyWarps - first_piece;
    const uint32_t groups = (args.n + kAnyRows - 1u) / kAnyRows;
    const uint32_t my_groups = (groups - blockIdx.y + gridDim.y - 1u) / gridDim.y;
    const uint32_t items = my_groups * my_pieces;   // the host keeps this below 2^32
    const uint32_t ring_at = smem_u32(any_smem_) + warp * R::warp_bytes;

    // Item i of this warp: piece first_piece + i % my_pieces of the rows of group i / my_pieces.
    // Neighbouring lanes copy neighbouring 16-byte units of a row, then those of the next row.  (Two
    // lanes to a row, every other unit each, saves the address arithmetic below and is slower: an
    // instruction then touches 16 rows, and the copies queue up: 15.2 us against 12.9 at 5003 x 2912.)
    constexpr uint32_t kLaneCopies = (kAnyRows * S::units + 31u) / 32u;
    uint32_t copy_from[kLaneCopies];     // distance of this lane's rows from the group's first one
#pragma unroll
    for (uint32_t i = 0; i < kLaneCopies; ++i) {
        copy_from[i] = (lane + 32u * i) / S::units * (uint32_t)args.row_bytes;
    }
    uint32_t ahead_group = blockIdx.y;
    uint32_t ahead_piece = 0u;
    const unsigned long long group_bytes = args.row_bytes * kAnyRows;
    const unsigned char *ahead_rows = args.w + ahead_group * group_bytes + (unsigned long long)first_piece * S::piece_bytes;
    auto issue = [&](uint32_t item) {
        if (item < items) {
            const unsigned char *base = ahead_rows + ahead_piece * S::piece_bytes;
            // the last piece of a row can be short; rows past the last copy nothing
            uint32_t bytes = S::piece_bytes;
            if (!S::super && first_piece + ahead_piece + 1u == pieces) {
                bytes = (runs - (pieces - 1u) * S::piece_runs) * S::block_bytes;
            }
            const uint32_t rows = args.n - ahead_group * kAnyRows;
            const uint32_t to = ring_at + (item % kAnyDepth) * S::stage;
#pragma unroll
            for (uint32_t i = 0; i < kLaneCopies; ++i) {
                const uint32_t row = (lane + 32u * i) / S::units;
                const uint32_t unit = (lane + 32u * i) % S::units;
                const unsigned char *from = base + copy_from[i];
                const uint32_t shift = (uint32_t)reinterpret_cast<uintptr_t>(from) & 15u;
                // only units that hold a byte of the piece: nothing past the tensor's own 16-byte units
                if (row < rows && row < kAnyRows && unit * 16u < shift + bytes) {
                    copy_async_16(to + row * S::slot + unit * 16u, from - shift + unit * 16u);
                }
            }
            if (++ahead_piece == my_pieces) {
                ahead_piece = 0u;
                ahead_group += gridDim.y;
                ahead_rows += gridDim.y * group_bytes;
            }
        }
        copy_async_commit();
    };
    // Everything may come from the launch before this one, the weights too.  Until it has ended the first pieces are
    // only asked for into L2, where a write that is still to come finds them.  (Copied before the wait they saved
    // another microsecond: 5003 x 2912, 7 rows, 8.0 us against 9.1; but a caller may write the weights just before.)
    if (lane / 2u < args.n - ahead_group * kAnyRows) {
        // two lanes to a row, every other line each
        const uint32_t begin = first_piece * S::piece_bytes;
        uint32_t end = begin + (my_pieces < kAnyDepth - 1u ? my_pieces : kAnyDepth - 1u) * S::piece_bytes;
        end = end < (uint32_t)args.row_bytes ? end : (uint32_t)args.row_bytes;
#pragma unroll 1
        for (uint32_t at = begin + (lane & 1u) * 128u; at < end; at += 256u) {
            prefetch_l2(ahead_rows + lane / 2u * (uint32_t)args.row_bytes + (at - begin));
        }
    }
    grid_dependency_wait();
    grid_launch_dependents();
#pragma unroll
    for (uint32_t i = 0; i < kAnyDepth - 1u; ++i) {
        issue(i);
    }
    uint32_t m = args.m_max;
    if (args.m_dev != nullptr) {
        const uint32_t live = *args.m_dev;
        m = live < m ? live : m;
    }
    const uint32_t token0 = blockIdx.x * 8u * TILES;
    if (token0 >= m) {
        copy_async_wait<0>();
        return;
    }

    // this lane's row of x per column of eight (past the batch: the last row; those sums are not
    // stored), from the warp's first weight on
    const unsigned short *x_row[TILES];
#pragma unroll
    for (uint32_t j = 0; j < TILES; ++j) {
        const uint32_t token = token0 + 8u * j + g;
        x_row[j] = static_cast<const unsigned short *>(args.x) + (size_t)(token < m ? token : m - 1u) * args.k
                 + first_piece * S::piece_runs * 32u + (kWide ? 8u : 4u) * t;
    }
    // where this lane's rows g and g + 8 start modulo 16 bytes, at the warp's first piece of a group
    const uint32_t row_shift = (uint32_t)(reinterpret_cast<uintptr_t>(args.w) + g * args.row_bytes
                                          + (unsigned long long)first_piece * S::piece_bytes);
    const uint32_t eight_rows = (uint32_t)(8u * args.row_bytes);
    uint32_t item = 0u;
    for (uint32_t turn = 0; turn < my_groups; ++turn) {
        const uint32_t group = blockIdx.y + turn * gridDim.y;
        const uint32_t group_shift = row_shift + group * (uint32_t)group_bytes;
        float acc[TILES][4];
#pragma unroll
        for (uint32_t j = 0; j < TILES; ++j) {
#pragma unroll
            for (uint32_t i = 0; i < 4u; ++i) {
                acc[j][i] = 0.0f;
            }
        }
#pragma unroll 1
        for (uint32_t piece = 0; piece < my_pieces; ++piece, ++item) {
            const uint32_t run0 = (first_piece + piece) * S::piece_runs;
            // a short last piece: its missing runs hold whatever the slot held before and are passed over
            const uint32_t live_runs = S::super ? 8u : (runs - run0 < 4u ? runs - run0 : 4u);
            uint2 xv[TILES][4][2];
            auto fetch_x = [&](uint32_t half) {
#pragma unroll
                for (uint32_t j = 0; j < TILES; ++j) {
                    const uint2 *from = reinterpret_cast<const uint2 *>(x_row[j] + piece * (S::piece_runs * 32u) + half * 128u);
#pragma unroll
                    for (uint32_t r = 0; r < 4u; ++r) {
                        if (!S::super && r >= live_runs) {
                            continue;
                        }
                        if (kWide && args.wide_x != 0u) {
                            const uint4 both = *reinterpret_cast<const uint4 *>(from + r * 8u);
                            xv[j][r][0] = make_uint2(both.x, both.y);
                            xv[j][r][1] = make_uint2(both.z, both.w);
                        } else {
                            xv[j][r][0] = from[r * 8u];
                            xv[j][r][1] = from[r * 8u + (kWide ? 1u : 4u)];
                        }
                    }
                }
            };
            fetch_x(0u);
            copy_async_wait<kAnyDepth - 2>();
            __syncwarp();
            issue(item + kAnyDepth - 1u);
            RowAt rows[2];
#pragma unroll
            for (uint32_t r = 0; r < 2u; ++r) {
                const uint32_t shift = (group_shift + r * eight_rows + piece * S::piece_bytes) & 15u;
                const uint32_t at = warp * R::warp_bytes + (item % kAnyDepth) * S::stage + (g + 8u * r) * S::slot + shift;
                rows[r].bytes = any_smem_ + at;
                rows[r].words = reinterpret_cast<const uint32_t *>(any_smem_ + (at & ~3u));
                rows[r].even = (at & 2u) != 0u ? 0x5432u : 0x3210u;
                rows[r].odd = (at & 2u) != 0u ? 0x7654u : 0x5432u;
            }
#pragma unroll
            for (uint32_t half = 0; half < S::piece_runs / 4u; ++half) {
                if (half != 0u) {
                    fetch_x(half);
                }
                uint32_t codes[2][4][2];
                float scale[2][8];
                float off[2][4];
                if (half == 0u) {
                    four_runs<TYPE, 0, kWide>(rows[0], t, codes[0], scale[0], off[0]);
                    four_runs<TYPE, 0, kWide>(rows[1], t, codes[1], scale[1], off[1]);
                } else {
                    four_runs<TYPE, 1, kWide>(rows[0], t, codes[0], scale[0], off[0]);
                    four_runs<TYPE, 1, kWide>(rows[1], t, codes[1], scale[1], off[1]);
                }
#pragma unroll
                for (uint32_t r = 0; r < 4u; ++r) {
                    if (!S::super && r >= live_runs) {
                        continue;
                    }
                    uint32_t a[2][4];
#pragma unroll
                    for (uint32_t step = 0; step < 2u; ++step) {
                        codes_to_operands<TYPE, BF>(codes[0][r][step], a[step][0], a[step][2]);
                        codes_to_operands<TYPE, BF>(codes[1][r][step], a[step][1], a[step][3]);
                    }
                    const uint32_t one = BF ? 0x3F803F80u : 0x3C003C00u;
                    const uint32_t ones[4] = {one, one, one, one};
#pragma unroll
                    for (uint32_t j = 0; j < TILES; ++j) {
                        float d[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
                        float e[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                        for (uint32_t step = 0; step < 2u; ++step) {
                            float (&into)[4] = d[S::sixteens ? step : 0u];
                            if (BF) {
                                mma_16816_bf16(into, a[step], xv[j][r][step].x, xv[j][r][step].y);
                            } else {
                                mma_16816(into, a[step], xv[j][r][step].x, xv[j][r][step].y);
                            }
                            if (S::offset) {
                                if (BF) {
                                    mma_16816_bf16(e, ones, xv[j][r][step].x, xv[j][r][step].y);
                                } else {
                                    mma_16816(e, ones, xv[j][r][step].x, xv[j][r][step].y);
                                }
                            }
                        }
#pragma unroll
                        for (uint32_t i = 0; i < 4u; ++i) {
                            if (S::sixteens) {
                                acc[j][i] = fmaf(scale[i >> 1][2u * r], d[0][i], acc[j][i]);
                                acc[j][i] = fmaf(scale[i >> 1][2u * r + 1u], d[1][i], acc[j][i]);
                            } else {
                                acc[j][i] = fmaf(scale[i >> 1][r], d[0][i], acc[j][i]);
                            }
                            if (S::offset) {
                                acc[j][i] = fmaf(off[i >> 1][r], e[i], acc[j][i]);
                            }
                        }
                    }
                }
            }
        }
        // the 8 warps' parts of the row group, added in order of depth
        float (&mine)[kAnyWarps][8u * TILES][kAnyRows] = parts[turn & 1u];
#pragma unroll
        for (uint32_t j = 0; j < TILES; ++j) {
#pragma unroll
            for (uint32_t i = 0; i < 4u; ++i) {
                mine[warp][8u * j + 2u * t + (i & 1u)][g + 8u * (i >> 1)] = acc[j][i];
            }
        }
        __syncthreads();   // two buffers: a warp that runs ahead writes the other one
        for (uint32_t at = threadIdx.x; at < 8u * TILES * kAnyRows; at += kAnyWarps * 32u) {
            const uint32_t row = at % kAnyRows;
            const uint32_t token = token0 + at / kAnyRows;
            float sum = mine[0][at / kAnyRows][row];
#pragma unroll
            for (uint32_t v = 1; v < kAnyWarps; ++v) {
                sum += mine[v][at / kAnyRows][row];
            }
            const uint32_t j = group * kAnyRows + row;
            uint32_t open = __ballot_sync(0xFFFFFFFFu, !(fabsf(sum) <= 3.402823466e38f) && token < m && j < args.n);
            while (open != 0u) {
                const uint32_t who = __ffs(open) - 1u;
                open &= open - 1u;
                const uint32_t its_row = __shfl_sync(0xFFFFFFFFu, j, who);
                const uint32_t its_token = __shfl_sync(0xFFFFFFFFu, token, who);
                const float again = sum_by_weights<TYPE, BF>(args.w + its_row * args.row_bytes,
                                                             static_cast<const unsigned short *>(args.x) + (size_t)its_token * args.k, runs);
                sum = lane == who ? again : sum;
            }
            uint32_t columns = args.n;
            uint32_t column = j;
            bool writes = token < m && j < args.n;
            if (args.epilogue == kEpilogueSwiglu) {
                // rows 2p and 2p + 1 are the gate and up rows of column p (cuda/model/norm.cu:92-105)
                const float up = __shfl_xor_sync(0xFFFFFFFFu, sum, 1u);
                sum = sum / (1.0f + expf(-sum)) * up;
                columns = args.n / 2u;
                column = j / 2u;
                writes = writes && (row & 1u) == 0u;
            }
            if (writes) {
                const size_t where = (size_t)token * columns + column;
                if (args.epilogue == kEpilogueAdd) {
                    // one rounded add into the float residual stream (cuda/model/norm.cu:78-89)
                    static_cast<float *>(args.y)[where] += sum;
                } else if (args.y_dtype == 0u) {
                    static_cast<float *>(args.y)[where] = sum;
                } else if (args.y_dtype == 1u) {
                    static_cast<__half *>(args.y)[where] = __float2half_rn(sum);
                } else {
                    static_cast<__nv_bfloat16 *>(args.y)[where] = __float2bfloat16_rn(sum);
                }
            }
        }
    }
    copy_async_wait<0>();
}

template <uint32_t TYPE, bool BF, uint32_t TILES>
static cudaError_t launch_any_tiles(cudaStream_t stream, bool overlap, const AnyArgs &args)
{
    using S = AnyRing<TYPE, TILES>;
    static unsigned long long configured = 0ull;
    cudaError_t err = allow_shared_memory(q_gemv_any_kernel_warp<TYPE, BF, TILES>, S::smem_bytes, &configured, true);
    if (err != cudaSuccess) {
        return err;
    }
    const uint32_t passes = (args.m_max + 8u * TILES - 1u) / (8u * TILES);
    const uint32_t groups = (args.n + kAnyRows - 1u) / kAnyRows;
    // Two blocks per SM where the rows are enough for it, some with a group more than others.  (As few blocks as
    // give all the same number of groups leave half of the SMs with one block: 14336 rows, 896 groups: 224
    // blocks of four against 296 of three or four.)
    const uint32_t wave = (2u * kSmCount + passes - 1u) / passes;
    const uint32_t blocks = groups < wave ? groups : wave;
    return launch_kernel_early(overlap, q_gemv_any_kernel_warp<TYPE, BF, TILES>, dim3(passes, blocks), kAnyWarps * 32u, S::smem_bytes,
                         stream, args);
}

template <uint32_t TYPE>
static cudaError_t launch_any_type(cudaStream_t stream, bool overlap, const AnyArgs &args, bool bf)
{
    // 8 rows of x to a pass, or 16
    if (args.m_max <= 8u) {
        return bf ? launch_any_tiles<TYPE, true, 1u>(stream, overlap, args) : launch_any_tiles<TYPE, false, 1u>(stream, overlap, args);
    }
    return bf ? launch_any_tiles<TYPE, true, 2u>(stream, overlap, args) : launch_any_tiles<TYPE, false, 2u>(stream, overlap, args);
}

bool warp_any_supports(const void *w, unsigned int type, unsigned int n, unsigned int k, const void *x, unsigned int m)
{
    const bool words = type == kTypeQ4_1 || type == kTypeQ5_1 || type == kTypeQ4_K || type == kTypeQ5_K;
    const bool known = words || type == kTypeQ8_0 || type == kTypeQ4_0 || type == kTypeQ5_0 || type == kTypeQ6_K;
    // grids of at most 65535 blocks of rows (turns take care of that) by 2^31 passes; row groups by
    // pieces in 32 bits
    return known && (reinterpret_cast<uintptr_t>(x) & 7u) == 0u && (!words || (reinterpret_cast<uintptr_t>(w) & 3u) == 0u)
        && m <= (1u << 20) && (unsigned long long)((n + 15u) / 16u) * (k / 32u) < (1ull << 31);
}

cudaError_t launch_warp_any(cudaStream_t stream, const void *w, unsigned int type, unsigned int n, unsigned int k,
                            const void *x, int x_bf16, unsigned int m, const unsigned int *m_dev, void *y, int y_dtype,
                            unsigned int epilogue, bool overlap)
{
    if (y_dtype < 0 || y_dtype > 2 || (epilogue == kEpilogueAdd && y_dtype != 0)
        || (epilogue == kEpilogueSwiglu && (n & 1u) != 0u) || epilogue > kEpilogueSwiglu) {
        return cudaErrorInvalidValue;
    }
    AnyArgs args = {};
    args.w = static_cast<const unsigned char *>(w);
    args.x = x;
    args.y = y;
    args.m_dev = m_dev;
    args.row_bytes = block_row_bytes(type, k);
    args.n = n;
    args.k = k;
    args.m_max = m;
    args.y_dtype = (uint32_t)y_dtype;
    args.epilogue = epilogue;
    args.wide_x = (reinterpret_cast<uintptr_t>(x) & 15u) == 0u ? 1u : 0u;
    const bool bf = x_bf16 != 0;
    switch (type) {
    case kTypeQ8_0: return launch_any_type<kTypeQ8_0>(stream, overlap, args, bf);
    case kTypeQ4_0: return launch_any_type<kTypeQ4_0>(stream, overlap, args, bf);
    case kTypeQ4_1: return launch_any_type<kTypeQ4_1>(stream, overlap, args, bf);
    case kTypeQ5_0: return launch_any_type<kTypeQ5_0>(stream, overlap, args, bf);
    case kTypeQ5_1: return launch_any_type<kTypeQ5_1>(stream, overlap, args, bf);
    case kTypeQ4_K: return launch_any_type<kTypeQ4_K>(stream, overlap, args, bf);
    case kTypeQ5_K: return launch_any_type<kTypeQ5_K>(stream, overlap, args, bf);
    case kTypeQ6_K: return launch_any_type<kTypeQ6_K>(stream, overlap, args, bf);
    default: return cudaErrorInvalidValue;
    }
}

} // namespace q8
