// The prefill-regime kernel: batches above 128 rows of x.  y[i][j] = sum_c x[i][c] * w[j][c], float sums, w
// dequantised to binary16, or (bfloat16 x) rounded once to bfloat16.
//
// Tensor-bound.  A tile is 256 rows of w by up to 256 rows of x, and two blocks on neighbouring SMs
// (cta_group::2) work on it together: each dequantises 128 rows of w into its own tensor memory and
// brings half of the tile's rows of x into its own shared memory, which the MMA reads in both.  What
// bounds the one-block form of this tile (128 x 256, q8_wide.cu) is shared memory: 256 deep, a block
// writes and reads 34 KB of weights twice over (544 cycles of its 128 bytes) and writes and reads 128 KB of
// x (2048 cycles) under 2048 cycles of MMAs.  Sharing x halves the second part.
//
//   * Weights: converter warps in two groups of eight that take segments in turn, as in q8_mid.cu.
//   * One accumulator (256 columns; the other 256 are two segments of A), so the MMAs of a tile wait until
//     the sums of the one before are out of tensor memory: the storing warps first turn all of them
//     into rows in shared memory (64 KB for the four warps), give the accumulator back and store
//     from there beside the next tile.
//   * The first tiles are dealt whole, one after the other to every pair; what is left for less than a turn of
//     all pairs is cut (pair_split in q8_schedule.cuh).  A cut tile is finished by the pair that holds its
//     first segment, each block its own rows (that is a pair's last piece and all its warps store), or by all of its
//     holders, each a run of its rows of x (kPairShareMore and pair_undecided say when).
//   * The first weights are on their way before the live batch is known; the accumulator goes back before a part of a
//     cut tile is published.
//   * The tile's rows of x are the batch in equal parts of at most 256, rounded up to 32.
//
// 23 warps per block, one block per SM: 0-3 store, 4-19 convert, 20 copies weights, 21 copies x, 22 of the
// first block issues the MMAs.  Every wait is bounded and raises a status bit when it runs out.
// Measured against q8_wide.cu: gate+up 28672 x 4096, 2048 rows, bfloat16, 489 -> 350 us (1377 TFLOP/s); the
// fused layer of 2560 by 9728, 300 rows, 365 -> 112 us (120 before the shares, and the first weights and the accumulator's
// return as above).  Reference kernel replaced: cuda/model/gemm.cuh:55-189.
#include <cuda.h>

#include "q8_launch.h"
#include "q8_rows.cuh"
#include "q8_schedule.cuh"

namespace q8 {

constexpr uint32_t kPairThreads = 23 * 32;
constexpr uint32_t kPairGroups = 2;
constexpr uint32_t kPairGroupWarps = 8;
constexpr uint32_t kPairWeightWarp = 20;
constexpr uint32_t kPairInputWarp = 21;
constexpr uint32_t kPairMmaWarp = 22;
constexpr uint32_t kPairTok = 256;          // rows of x per tile, at most
constexpr uint32_t kPairMaxRaw = 4;
constexpr uint32_t kPairMaxX = 8;
constexpr uint32_t kPairAStages = 2;
constexpr uint32_t kPairAColumns = kSegK / 2;
constexpr uint32_t kPairBars = 3 * kPairMaxRaw + 2 * kPairMaxX + 2 * kPairAStages + 2 + 1 + 1;
constexpr uint32_t kPairWarpStage = 16384;  // per storing warp: its 32 columns of the tile's rows of x
constexpr uint32_t kPairPlanBytes = 128;
constexpr uint32_t kPairTail = kEpilogueWarps * kPairWarpStage + kPairBars * 8 + 16 + kPairPlanBytes;
constexpr uint32_t kPairSmem = 227u * 1024u;
constexpr uint32_t kPairRings = (kPairSmem - 1024u - kPairTail) / 1024u * 1024u;
struct PairArgs {
    unsigned int n, k, m_max;
    const unsigned int *m_dev;
    RowStore to;
    unsigned int *status;
    unsigned int ntok;                 // rows of x per tile
    unsigned int b_bf16;
    float *partial;                    // per block: [row of x][row of w], and its flags
    unsigned int *flags;
    unsigned long long tile_floats;
    unsigned int x_stages, raw_stages;
    unsigned int x_pieces;             // of x, 64 deep, per stage of its ring: 1 or 2
    PairSplit split;                   // of the whole batch's tiles
};

// Up to this many rows of x per tile a value has two accumulators, which successive pieces of x take in turn (an MMA
// truncates the sum it adds to; q8_mid.cu says more).
constexpr uint32_t kPairTwoChains = kPairTok / 2;

// The sums of a whole tile's `rows` rows of x (accumulator columns) and this warp's 32 rows of w: into rows in the
// warp's own shared memory, then - `release` is called in between - 16 bytes per lane to y.  Everything
// is inside the tensor and on 16-byte boundaries (pair_drain_fits).  GATED: rows of w in pairs, gate and up of one
// column (arithmetic of cuda/model/norm.cu:92-105); of two rows of x the even lane forms the first's
// value and the odd lane the second's.
template <typename YT, bool GATED, typename Release>
__device__ __forceinline__ void pair_drain(const RowStore &to, uint32_t stage, uint32_t lane_taddr, uint32_t lane,
                                           uint32_t chains, uint32_t first_col, uint32_t first_row, uint32_t rows,
                                           Release release)
{
    constexpr uint32_t kRowBytes = (GATED ? 16u : 32u) * sizeof(YT);
    constexpr uint32_t kRound = kPairWarpStage / kRowBytes < kPairTok ? kPairWarpStage / kRowBytes : kPairTok;
    constexpr uint32_t kLanesPerRow = kRowBytes / 16u;
    constexpr uint32_t kRowsPerStep = 32u / kLanesPerRow;
    constexpr uint32_t kTogether = 4u;
    const bool odd = (lane & 1u) != 0u;
    for (uint32_t base = 0; base < rows; base += kRound) {
        const uint32_t here = rows - base < kRound ? rows - base : kRound;
#pragma unroll 1
        for (uint32_t c0 = 0; c0 < here; c0 += 16u) {
            uint32_t v[16];
            load_sums(lane_taddr + base + c0, chains, kPairTwoChains, v);
            const uint32_t at = stage + c0 * kRowBytes;
            if (GATED) {
#pragma unroll
                for (uint32_t i = 0; i < 16u; i += 2u) {
                    const float give = __uint_as_float(odd ? v[i] : v[i + 1u]);
                    const float keep = __uint_as_float(odd ? v[i + 1u] : v[i]);
                    const float got = __shfl_xor_sync(0xFFFFFFFFu, give, 1u);
                    const float gate = odd ? got : keep;
                    const float up = odd ? keep : got;
                    const float value = gated_unit(gate, up);
                    const uint32_t cell = at + (i + (odd ? 1u : 0u)) * kRowBytes + lane / 2u * sizeof(YT);
                    if (sizeof(YT) == 4) {
                        st_shared_b32(cell, __float_as_uint(value));
                    } else {
                        st_shared_b16(cell, out_bits<YT>(value));
                    }
                }
            } else {
#pragma unroll
                for (uint32_t i = 0; i < 16u; ++i) {
                    if (sizeof(YT) == 4) {
                        st_shared_b32(at + i * kRowBytes + lane * 4u, v[i]);
                    } else {
                        st_shared_b16(at + i * kRowBytes + lane * 2u, out_bits<YT>(__uint_as_float(v[i])));
                    }
                }
            }
        }
        if (base + kRound >= rows) {
            release();
        }
        __syncwarp();
        const uint32_t part = lane % kLanesPerRow;
        const bool adds = !GATED && sizeof(YT) == 4 && to.epilogue == kEpilogueAdd;
        for (uint32_t r0 = lane / kLanesPerRow; r0 < here; r0 += kRowsPerStep * kTogether) {
            float4 before[kTogether];
            YT *y[kTogether];
#pragma unroll
            for (uint32_t i = 0; i < kTogether; ++i) {
                const uint32_t r = r0 + i * kRowsPerStep;
                y[i] = r < here ? static_cast<YT *>(to.y) + (size_t)(first_row + base + r) * to.ldy + first_col + part * (16u / sizeof(YT))
                                : nullptr;
                before[i] = adds && y[i] != nullptr ? *reinterpret_cast<const float4 *>(y[i]) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
#pragma unroll
            for (uint32_t i = 0; i < kTogether; ++i) {
                uint4 piece;
                const uint32_t r = r0 + i * kRowsPerStep;
                ld_shared_v4(stage + (r < here ? r : 0u) * kRowBytes + part * 16u, piece.x, piece.y, piece.z, piece.w);
                if (adds) {
                    // one rounded add per value (cuda/model/norm.cu:78-89)
                    piece.x = __float_as_uint(before[i].x + __uint_as_float(piece.x));
                    piece.y = __float_as_uint(before[i].y + __uint_as_float(piece.y));
                    piece.z = __float_as_uint(before[i].z + __uint_as_float(piece.z));
                    piece.w = __float_as_uint(before[i].w + __uint_as_float(piece.w));
                }
                if (y[i] != nullptr) {
                    *reinterpret_cast<uint4 *>(y[i]) = piece;
                }
            }
        }
        __syncwarp();
    }
}

// A cut tile that a pair holds a piece of: the tile and its holders, `holders` pairs from `first` on.
struct PairCut {
    uint32_t tile, first, holders;
};

__device__ __forceinline__ PairCut pair_cut(const PairWork &work, uint32_t id)
{
    PairCut cut;
    cut.tile = work.tile;
    cut.first = pair_first_holder(work, id, work.tile);
    cut.holders = pair_last_holder(work, cut.first, work.tile) + 1u - cut.first;
    return cut;
}

// What a block works on.  One thread works it out and the roles read it from shared memory: the divisions take a
// microsecond, and kept in registers across the roles it costs the converters theirs.
struct PairPlan {
    uint32_t m;                 // live rows of x
    PairWork work;
    uint32_t share_from;        // from this many holders on a cut tile may be finished by all of them
    PairCut begun, begins;      // the cut tiles that the pair has pieces of: begun by another pair, and by itself
};
static_assert(sizeof(PairPlan) <= kPairPlanBytes, "room for the plan");

__device__ __forceinline__ void pair_plan_cuts(PairPlan *plan, uint32_t id)
{
    plan->begun.holders = plan->begins.holders = 0u;
    plan->share_from = pair_share_from(plan->work);
    PairWork ahead = plan->work;
    ahead.whole_left = 0u;
    while (ahead.next()) {
        if (ahead.s0 != 0u) {
            plan->begun = pair_cut(ahead, id);
        } else if (ahead.s1 != ahead.segs) {
            plan->begins = pair_cut(ahead, id);
        }
    }
}

// Where a block's part of a cut tile lies: a block has two slots (the context's scratch is sized for two blocks per
// SM), for the tile that it begins and for the one that others began.
__device__ __forceinline__ uint32_t pair_slot(uint32_t block, bool begins)
{
    return begins ? gridDim.x + block : block;
}

__device__ __forceinline__ uint32_t pair_cut_slot(const PairCut &cut, uint32_t holder, uint32_t rank)
{
    return pair_slot(2u * (cut.first + holder) + rank, holder == 0u);
}

// Words of a quarter of a cut tile that its holders may finish together, behind the flags of the first two holders'
// parts: how many warps have published and seen what they need, and which holders have begun (kPairAlone).
__device__ __forceinline__ unsigned int *pair_count(unsigned int *flags, const PairCut &cut, uint32_t rank, uint32_t lanes)
{
    return flags + kFlagWords * pair_cut_slot(cut, 0u, rank) + kEpilogueWarps + lanes;
}

__device__ __forceinline__ unsigned int *pair_begun(unsigned int *flags, const PairCut &cut, uint32_t rank, uint32_t lanes)
{
    return flags + kFlagWords * pair_cut_slot(cut, 1u, rank) + kEpilogueWarps + lanes;
}

// This block runs: for the tiles that it may have to finish together with others.  (By a thread that counts itself in
// pair_count later on, so that nothing is added to a word after it has been cleared.)
__device__ __forceinline__ void pair_say_begun(unsigned int *flags, const PairPlan &plan, uint32_t rank, uint32_t lanes)
{
    if (plan.begun.holders >= plan.share_from) {
        atomicAdd(pair_begun(flags, plan.begun, rank, lanes), 1u);
    }
    if (plan.begins.holders >= plan.share_from) {
        atomicAdd(pair_begun(flags, plan.begins, rank, lanes), 1u);
    }
}

// Of which of a pair's cut tiles all holders have begun by now: bit 0 the tile that others began, bit 1 its own.
__device__ __forceinline__ uint32_t pair_all_begun(unsigned int *flags, const PairPlan &plan, uint32_t rank, uint32_t lanes)
{
    const uint32_t first = plan.begun.holders >= plan.share_from ? ld_relaxed_gpu(pair_begun(flags, plan.begun, rank, lanes)) : 0u;
    const uint32_t second = plan.begins.holders >= plan.share_from ? ld_relaxed_gpu(pair_begun(flags, plan.begins, rank, lanes)) : 0u;
    return (__all_sync(0xFFFFFFFFu, first == plan.begun.holders) ? 1u : 0u)
         | (__all_sync(0xFFFFFFFFu, second == plan.begins.holders) ? 2u : 0u);
}

// Whether all holders finish a quarter of a cut tile; else the one that began the tile does.
__device__ __forceinline__ bool pair_together(unsigned int *word, uint32_t holders)
{
    uint32_t seen = ld_relaxed_gpu(word);
    while (pair_undecided(seen, holders)) {
        const uint32_t now = atomicCAS(word, seen, seen | kPairAlone);
        seen = now == seen ? seen | kPairAlone : now;
    }
    return seen == holders;
}

// A partial sum that another block has left, past the first-level cache.  Volatile, so that the loads of a piece are
// issued one after the other before the first is used: a round trip is 0.7 us.
__device__ __forceinline__ float ld_partial(const float *from)
{
    float v;
    asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(from) : "memory");
    return v;
}

// The parts of one run of rows that the holders after the first have left (a slot every `stride` floats, `count` of
// them), added to v in order; two of them are on their way at a time.
__device__ __forceinline__ void add_parts(uint32_t (&v)[16], const float *slots, unsigned long long stride, uint32_t count)
{
#pragma unroll 1
    for (uint32_t c = 0; c < count; c += 2u) {
        const bool two = c + 1u < count;
        float a[16], b[16];
#pragma unroll
        for (uint32_t i = 0; i < 16u; ++i) {
            a[i] = ld_partial(slots + i * kRows);
        }
        slots += two ? stride : 0ull;
#pragma unroll
        for (uint32_t i = 0; i < 16u; ++i) {
            b[i] = ld_partial(slots + i * kRows);
        }
        slots += stride;
#pragma unroll
        for (uint32_t i = 0; i < 16u; ++i) {
            v[i] = __float_as_uint(__uint_as_float(v[i]) + a[i] + (two ? b[i] : 0.0f));
        }
    }
}

// Add to v the 16 columns of sums at taddr (load_sums in q8_rows.cuh).
__device__ __forceinline__ void add_sums(uint32_t taddr, uint32_t chains, uint32_t stride, uint32_t (&v)[16])
{
#pragma unroll 1
    for (uint32_t c = 0; c < chains; ++c, taddr += stride) {
        uint32_t more[16];
        tmem_ld_32x16(taddr, more);
        tmem_ld_wait();
#pragma unroll
        for (uint32_t i = 0; i < 16u; ++i) {
            v[i] = __float_as_uint(__uint_as_float(v[i]) + __uint_as_float(more[i]));
        }
    }
}

// Wait until the holders from `from` on have published their part of this quarter of the tile.
__device__ __forceinline__ void wait_for_parts(const PairArgs &args, const PairCut &at, uint32_t from, uint32_t rank, uint32_t lanes,
                                               uint32_t lane, volatile uint32_t *abort_flag)
{
    for (uint32_t h = from + lane; h < at.holders; h += 32u) {
        const unsigned int *flag = args.flags + kFlagWords * pair_cut_slot(at, h, rank) + lanes;
        const long long begin = clock64();
        while (ld_acquire_gpu(flag) < kPublishers) {
            if (clock64() - begin > Q8_WAIT_CYCLES || *abort_flag != 0u) {
                atomicOr(args.status, Q8_DEV_FLAG_TIMEOUT);
                break;
            }
        }
    }
    __syncwarp();
}

// Rows of x that a warp finishes of a cut tile at a time.
constexpr uint32_t kPairShareRows = 8;

// The parts of a cut tile's holders, `partial` being this lane's place in slot 0, added in order; the loads of four
// holders are on their way at a time.
__device__ __forceinline__ void sum_of_parts(uint32_t (&v)[kPairShareRows], const float *partial, unsigned long long tile_floats,
                                             const PairCut &cut, uint32_t rank)
{
    constexpr uint32_t kTogether = 4u;
    float sum[kPairShareRows];
#pragma unroll
    for (uint32_t i = 0; i < kPairShareRows; ++i) {
        sum[i] = 0.0f;
    }
#pragma unroll 1
    for (uint32_t h0 = 0; h0 < cut.holders; h0 += kTogether) {
        float part[kTogether][kPairShareRows];
#pragma unroll
        for (uint32_t h = 0; h < kTogether; ++h) {
            const bool there = h0 + h < cut.holders;
            const float *from = partial + pair_cut_slot(cut, there ? h0 + h : h0, rank) * tile_floats;
#pragma unroll
            for (uint32_t i = 0; i < kPairShareRows; ++i) {
                part[h][i] = ld_partial(from + i * kRows);
            }
        }
#pragma unroll
        for (uint32_t h = 0; h < kTogether; ++h) {
#pragma unroll
            for (uint32_t i = 0; i < kPairShareRows; ++i) {
                sum[i] += h0 + h < cut.holders ? part[h][i] : 0.0f;
            }
        }
    }
#pragma unroll
    for (uint32_t i = 0; i < kPairShareRows; ++i) {
        v[i] = __float_as_uint(sum[i]);
    }
}

template <bool BF>
__device__ __forceinline__ void pair_convert(uint32_t half, const uint32_t (&raw)[36], uint32_t taddr)
{
    if (half == 0u) {
        convert_stage_tmem<0, 0, BF>(raw, taddr);
        convert_stage_tmem<0, 1, BF>(raw, taddr + kSubK / 2u);
    } else {
        convert_stage_tmem<1, 0, BF>(raw, taddr);
        convert_stage_tmem<1, 1, BF>(raw, taddr + kSubK / 2u);
    }
}

// What the thread that issues a pair's MMAs knows.
struct PairIssue {
    uint32_t x_full, x_empty, a_full, a_empty, acc_full, acc_empty;     // barriers
    uint32_t tmem_base, a_column0, smem0, x_piece_bytes, x_stages, idesc, chains;
    unsigned int *status;
};

// All of a pair's MMAs.  PIECES: of x per stage of its ring (launch_pair_kernel).  Every wait stands where it is needed:
// asking for the next stage before the MMAs of this one cost more than it hid, because the answer is waited for where it
// is asked for (2048 rows, layer 782 -> 773 us without).
template <uint32_t PIECES>
__device__ __forceinline__ void pair_issue(PairWork &work, const PairIssue &at, volatile uint32_t *abort_flag)
{
    uint32_t xst = 0u, xph = 0u;
    uint32_t ast = 0u, aph = 0u;
    for (uint32_t turn = 0; work.next(); ++turn) {
        if (!mbar_wait_hot(at.acc_empty, (turn & 1u) ^ 1u, abort_flag, at.status)) {
            return;
        }
        tc_fence_after_sync();
        for (uint32_t s = work.s0; s < work.s1; ++s) {
            if (!mbar_wait_hot(at.a_full + 8u * ast, aph, abort_flag, at.status)) {
                return;
            }
            const uint32_t a_tmem = at.tmem_base + at.a_column0 + ast * kPairAColumns;
#pragma unroll 1
            for (uint32_t j0 = 0; j0 < kSubs; j0 += PIECES) {
                if (!mbar_wait_hot(at.x_full + 8u * xst, xph, abort_flag, at.status)) {
                    return;
                }
                tc_fence_after_sync();
                const uint32_t x_stage = at.smem0 + xst * (PIECES * at.x_piece_bytes);
#pragma unroll
                for (uint32_t i = 0; i < PIECES; ++i) {
                    const uint32_t j = j0 + i;
                    const uint64_t b_desc = umma_desc_sw128(x_stage + i * at.x_piece_bytes);
#pragma unroll
                    for (uint32_t kk = 0; kk < kSubK / 16u; ++kk) {
                        // 16 halves: 8 columns of A, 32 bytes along the swizzled row of x
                        pair_mma_f16_ts(at.tmem_base + (j & (at.chains - 1u)) * kPairTwoChains, a_tmem + j * (kSubK / 2u) + 8u * kk,
                                        b_desc + 2u * kk, at.idesc, s != work.s0 || j >= at.chains || kk != 0u ? 1u : 0u);
                    }
                }
                pair_commit(at.x_empty + 8u * xst);
                xst = xst + 1u == at.x_stages ? 0u : xst + 1u;
                xph ^= xst == 0u ? 1u : 0u;
            }
            pair_commit(at.a_empty + 8u * ast);
            if (++ast == kPairAStages) {
                ast = 0u;
                aph ^= 1u;
            }
        }
        pair_commit(at.acc_full);
    }
}

template <typename YT>
__global__ void __launch_bounds__(kPairThreads, 1)
q8_wide_kernel_pair(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const PairArgs args)
{
    extern __shared__ unsigned char smem_raw_[];
    const uint32_t smem0 = (smem_u32(smem_raw_) + 1023u) & ~1023u;
    unsigned char *const smem = smem_raw_ + (smem0 - smem_u32(smem_raw_));
    const uint32_t ntok = args.ntok;
    const uint32_t x_piece_bytes = ntok * (kSubK * 2u) / 2u;      // this block's half of the rows, 64 deep
    const uint32_t x_stage_bytes = x_piece_bytes * args.x_pieces;
    const uint32_t raw_base = smem0 + args.x_stages * x_stage_bytes;
    const uint32_t stage_base = smem0 + kPairRings;
    const uint32_t raw_full = stage_base + kEpilogueWarps * kPairWarpStage;
    const uint32_t raw_empty = raw_full + 16u * kPairMaxRaw;      // two full barriers per stage (q8_mid.cu says why)
    const uint32_t raw_turns = 2u * args.raw_stages;
    const uint32_t x_full = raw_empty + 8u * kPairMaxRaw;         // the first block's: both halves have landed
    const uint32_t x_empty = x_full + 8u * kPairMaxX;
    const uint32_t a_full = x_empty + 8u * kPairMaxX;             // the first block's: both blocks' weights are there
    const uint32_t a_empty = a_full + 8u * kPairAStages;
    const uint32_t acc_full = a_empty + 8u * kPairAStages;
    const uint32_t acc_empty = acc_full + 8u;                     // the first block's: both blocks' sums are out
    const uint32_t drain_bar = acc_empty + 8u;
    const uint32_t cuts_bar = drain_bar + 8u;                     // plan->begun and plan->begins are there
    const uint32_t tmem_slot = cuts_bar + 8u;
    volatile uint32_t *tmem_slot_ptr = reinterpret_cast<volatile uint32_t *>(smem + (tmem_slot - smem0));
    volatile uint32_t *abort_flag = tmem_slot_ptr + 1;

    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t rank = cluster_ctarank();

    grid_launch_dependents();
    const uint32_t segs = args.k / kSegK;
    const uint32_t pairs = gridDim.x / 2u;
    const uint32_t row_tiles = (args.n + 2u * kRows - 1u) / (2u * kRows);   // below 2^31 units: the host checks
    const uint32_t pair_id = blockIdx.x / 2u;
    PairPlan *plan = reinterpret_cast<PairPlan *>(smem + (tmem_slot + 16u - smem0));

    uint32_t early = 0u;
    if (warp == kPairWeightWarp && elect_one()) {
        tma_prefetch_desc(&tmap_w);
        tma_prefetch_desc(&tmap_x);
        for (uint32_t i = 0; i < args.raw_stages; ++i) {
            mbar_init(raw_full + 8u * i, 1u);
            mbar_init(raw_full + 8u * (i + args.raw_stages), 1u);
            mbar_init(raw_empty + 8u * i, kPairGroupWarps);
        }
        for (uint32_t i = 0; i < args.x_stages; ++i) {
            mbar_init(x_full + 8u * i, 1u);
            mbar_init(x_empty + 8u * i, 1u);
        }
        for (uint32_t i = 0; i < kPairAStages; ++i) {
            mbar_init(a_full + 8u * i, 2u * kPairGroupWarps);
            mbar_init(a_empty + 8u * i, 1u);
        }
        mbar_init(acc_full, 1u);
        mbar_init(acc_empty, 2u * kEpilogueWarps);
        mbar_init(drain_bar, 1u);
        mbar_init(cuts_bar, 1u);
        *abort_flag = 0u;
        mbar_init_fence();
        fence_proxy_async_smem();
        // the first weights: only this block's own barriers have to be there
        PairWork ahead;
        const uint32_t tok_tiles = (args.m_max + ntok - 1u) / ntok;
        pair_work(&ahead, args.split, pair_id, pairs, segs);
        const uint32_t total = ahead.whole_left * segs + ahead.left;
        uint32_t s = 0u;
        ahead.s1 = 0u;
        for (; early < args.raw_stages && early < total; ++early, ++s) {
            if (s == ahead.s1) {
                ahead.next();
                s = ahead.s0;
            }
            mbar_expect_tx(raw_full + 8u * early, kRawStageBytes);
            tma_load_2d(raw_base + early * kRawStageBytes, &tmap_w, raw_full + 8u * early, (int)(s * kSegWords),
                        (int)((ahead.tile / tok_tiles * 2u + rank) * kRows));
        }
        // The live batch decides how many tiles there are, and is known when the launch before this one has ended.
        // The first weights are on their way by then, as the whole batch wants them; where it has more tiles than
        // the live one, they land first and their barriers are made anew.
        if (args.m_dev != nullptr) {
            grid_dependency_wait();
            const unsigned int live = *args.m_dev;
            if (live < args.m_max && (live + ntok - 1u) / ntok != tok_tiles) {
                uint32_t local_abort = 0;
                for (uint32_t i = 0; i < early; ++i) {
                    mbar_wait(raw_full + 8u * i, 0u, &local_abort, nullptr);
                    mbar_inval(raw_full + 8u * i);
                    mbar_init(raw_full + 8u * i, 1u);
                }
                mbar_init_fence();
                fence_proxy_async_smem();
                early = 0u;
            }
        }
    }
    if (threadIdx.x == 0u) {
        PairWork work;
        uint32_t m = args.m_max;
        if (args.m_dev != nullptr) {
            prefetch_l2(args.m_dev);
            grid_dependency_wait();
            const unsigned int live = *args.m_dev;
            m = live < m ? live : m;
        }
        if ((m + ntok - 1u) / ntok == (args.m_max + ntok - 1u) / ntok) {
            pair_work(&work, args.split, pair_id, pairs, segs);
        } else {
            pair_deal(&work, pair_id, pairs, row_tiles * ((m + ntok - 1u) / ntok), segs);
        }
        plan->m = m;
        plan->work = work;
    }
    if (warp == kPairMmaWarp) {
        pair_tmem_alloc(tmem_slot, 512u);
        pair_tmem_relinquish();
    }
    // both blocks' barriers are there before either signals the other's (the fence after their
    // initialisation orders it)
    __syncwarp();
    cluster_arrive_relaxed();
    cluster_wait_acquire();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot_ptr;
    const uint32_t m = plan->m;
    const uint32_t tok_tiles = (m + ntok - 1u) / ntok;
    const uint32_t a_column0 = kPairTok;
    const uint32_t chains = ntok <= kPairTwoChains ? 2u : 1u;

    if (warp == kPairWeightWarp) {
        // ---------------------------------------------------------------- weight copies
        if (elect_one()) {
            uint32_t g = 0;
            bool ok = true;
            uint32_t full = 0u;
            PairWork work = plan->work;
            uint32_t st = 0u, ph = 1u;
            while (ok && work.next()) {
                const uint32_t w_row = (work.tile / tok_tiles * 2u + rank) * kRows;
                for (uint32_t s = work.s0; s < work.s1; ++s, ++g) {
                    if (g >= early) {
                        if (!mbar_wait(raw_empty + 8u * st, ph, abort_flag, args.status)) {
                            ok = false;
                            break;
                        }
                        mbar_expect_tx(raw_full + 8u * full, kRawStageBytes);
                        tma_load_2d(raw_base + st * kRawStageBytes, &tmap_w, raw_full + 8u * full, (int)(s * kSegWords),
                                    (int)w_row);
                    }
                    full = full + 1u == raw_turns ? 0u : full + 1u;
                    if (++st == args.raw_stages) {
                        st = 0u;
                        ph ^= 1u;
                    }
                }
            }
            // Let every copy this thread started land before the block ends.
            uint32_t local_abort = 0;
            const uint32_t issued = g > early ? g : early;
            const uint32_t first = issued > args.raw_stages ? issued - args.raw_stages : 0u;
            for (uint32_t i = first; i < issued; ++i) {
                mbar_wait(raw_full + 8u * (i % raw_turns), (i / raw_turns) & 1u, &local_abort, nullptr);
            }
        }
    } else if (warp == kPairInputWarp) {
        // ---------------------------------------------------------------- x copies
        // each block its half of the tile's rows, both signalling the first block's barrier
        if (elect_one()) {
            uint32_t q = 0;
            grid_dependency_wait();
            bool ok = true;
            uint32_t st = 0u, ph = 1u;
            const uint32_t signal = mapa_shared(x_full, 0u);
            PairWork work = plan->work;
            while (ok && work.next()) {
                const uint32_t row = work.tile % tok_tiles * ntok + rank * (ntok / 2u);
                for (uint32_t sub = work.s0 * kSubs; sub < work.s1 * kSubs; sub += args.x_pieces, ++q) {
                    if (!mbar_wait_hot(x_empty + 8u * st, ph, abort_flag, args.status)) {
                        ok = false;
                        break;
                    }
                    if (rank == 0u) {
                        mbar_expect_tx(x_full + 8u * st, 2u * x_stage_bytes);
                    }
                    // (a loop over the pieces in place of the two: 0.6 % slower over 110 shapes of 96 to 540 rows)
                    pair_tma_load_2d(smem0 + st * x_stage_bytes, &tmap_x, signal + 8u * st, (int)(sub * kSubK), (int)row);
                    if (args.x_pieces > 1u) {
                        pair_tma_load_2d(smem0 + st * x_stage_bytes + x_piece_bytes, &tmap_x, signal + 8u * st,
                                         (int)((sub + 1u) * kSubK), (int)row);
                    }
                    if (++st == args.x_stages) {
                        st = 0u;
                        ph ^= 1u;
                    }
                }
            }
            if (rank == 0u) {
                // both blocks' copies (the second block stays until the first has seen this)
                uint32_t local_abort = 0;
                const uint32_t first = q > args.x_stages ? q - args.x_stages : 0u;
                for (uint32_t i = first; i < q; ++i) {
                    mbar_wait(x_full + 8u * (i % args.x_stages), (i / args.x_stages) & 1u, &local_abort, nullptr);
                }
            }
        }
    } else if (warp == kPairMmaWarp) {
        // ---------------------------------------------------------------- MMA issue, for both blocks
        if (rank == 0u && elect_one()) {
            const uint32_t idesc = umma_idesc(2u * kRows, ntok, args.b_bf16, args.b_bf16);
            PairWork work = plan->work;
            const bool works = !work.last();
            const PairIssue at = {x_full, x_empty, a_full, a_empty, acc_full, acc_empty, tmem_base, a_column0, smem0, x_piece_bytes,
                                  args.x_stages, idesc, chains, args.status};
            if (args.x_pieces == 1u) {
                pair_issue<1u>(work, at, abort_flag);
            } else {
                pair_issue<2u>(work, at, abort_flag);
            }
            if (works) {
                // Every MMA has finished: what the helping warps of both blocks wait for.  This thread waits as
                // well; a pair without work issues none, because nobody would wait for its arrivals, and they
                // must not come to a shared memory that the blocks have left.
                uint32_t local_abort = 0;
                pair_commit(drain_bar);
                mbar_wait(drain_bar, 0u, &local_abort, nullptr);
            }
        }
    } else if (warp >= kConvertWarp0) {
        // ---------------------------------------------------------------- dequantise
        const uint32_t cw = warp - kConvertWarp0;
        const uint32_t group = cw / kPairGroupWarps;
        const uint32_t half = (cw >> 2) & 1u;
        const uint32_t row_at = ((cw & 3u) * 32u + lane) * kSegBytes;
        const uint32_t lane_base = tmem_base + (((cw & 3u) * 32u) << 16) + a_column0 + half * (kSegK / 4u);
        const uint32_t signal = mapa_shared(a_full, 0u);
        const PairWork work = plan->work;
        const uint32_t total = work.whole_left * segs + work.left;    // segments of weights
        uint32_t full = group, fph = 0, ast = group, aph = 0;
        for (uint32_t g = group; g < total; g += kPairGroups) {
            if (!__all_sync(0xFFFFFFFFu, mbar_wait_hot(raw_full + 8u * full, fph, abort_flag, args.status))) {
                break;
            }
            const uint32_t rst = full < args.raw_stages ? full : full - args.raw_stages;
            uint32_t raw[36];
            const uint32_t raw_row = raw_base + rst * kRawStageBytes + row_at;
            if (half == 0u) {
                load_raw<0>(raw_row, raw);
            } else {
                load_raw<1>(raw_row, raw);
            }
            row_words_present(raw, args.status);
            if (lane == 0u) {
                mbar_arrive(raw_empty + 8u * rst);
            }
            if (!__all_sync(0xFFFFFFFFu, mbar_wait_hot(a_empty + 8u * ast, aph ^ 1u, abort_flag, args.status))) {
                break;
            }
            const uint32_t taddr = lane_base + ast * kPairAColumns;
            tc_fence_after_sync();
            if (args.b_bf16 != 0u) {
                pair_convert<true>(half, raw, taddr);
            } else {
                pair_convert<false>(half, raw, taddr);
            }
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0u) {
                mbar_arrive_cluster(signal + 8u * ast);
            }
            full += kPairGroups;
            if (full >= raw_turns) {
                full -= raw_turns;
                fph ^= 1u;
            }
            // two stages, two groups: each group keeps its own
            aph ^= 1u;
        }
    }

    if (warp < kPairWeightWarp) {
        // ---------------------------------------------------------------- read sums, store
        const uint32_t lanes = warp & 3u;
        const uint32_t helper = warp >> 2;                       // 0: the storing warps
        const uint32_t lane_taddr = tmem_base + ((lanes * 32u) << 16);
        const bool gated = args.to.epilogue == kEpilogueSwiglu;
        PairWork work = plan->work;
        if (threadIdx.x == 0u) {
            pair_plan_cuts(plan, pair_id);
            mbar_arrive(cuts_bar);
        }
        __syncwarp();
        const uint32_t stage = helper == 0u ? stage_base + warp * kPairWarpStage : smem0 + (warp - kEpilogueWarps) * 4096u;
        const uint32_t release_bar = mapa_shared(acc_empty, 0u);
        uint32_t flip = 0u;      // the two turns of a helper's staging buffer
        grid_dependency_wait();
        if (helper == 0u) {
            mbar_wait_hot(cuts_bar, 0u, abort_flag, args.status);
            if (lane == 0u) {
                pair_say_begun(args.flags, *plan, rank, lanes);
            }
            __syncwarp();
        }
        uint32_t all_begun = 0u;      // bits: of which of the pair's two cut tiles all holders are known to have begun
        // rows of y on a boundary of 16 bytes (the drain of a whole tile) or of four values (the others)
        const bool aligned16 = ((size_t)args.to.ldy * sizeof(YT)) % 16u == 0u && (reinterpret_cast<uintptr_t>(args.to.y) % 16u) == 0u;
        const bool aligned4 = (args.to.ldy % 4u) == 0u && (reinterpret_cast<uintptr_t>(args.to.y) % (4u * sizeof(YT))) == 0u;
        for (uint32_t turn = 0; work.next(); ++turn) {
            const bool last = work.last();
            const bool owner = work.s0 == 0u;
            const bool helped = last;
            const bool cut = !owner || work.s1 != segs;
            if (helper != 0u && !helped) {
                continue;
            }
            const uint32_t row_tile = work.tile / tok_tiles;
            const uint32_t tok0 = (work.tile - row_tile * tok_tiles) * ntok;
            const uint32_t rows = m - tok0 < ntok ? m - tok0 : ntok;                     // live rows of x of the tile
            const uint32_t j = (row_tile * 2u + rank) * kRows + lanes * 32u;             // this warp's first row of w
            const uint32_t inside = args.n > j ? args.n - j : 0u;                        // ... and how many are there
            const uint32_t mine = inside < 32u ? inside : 32u;
            const uint32_t columns = gated ? mine / 2u : mine;
            const uint32_t col = gated ? j / 2u : j;
            uint32_t others = 0u;          // holders whose parts this pair adds to its own
            bool publish = false;
            if (cut) {
                mbar_wait_hot(cuts_bar, 0u, abort_flag, args.status);
                const PairCut at = owner ? plan->begins : plan->begun;
                publish = !owner || at.holders >= plan->share_from;
                if (!publish) {
                    // The pairs right after this one; they met the tile at the start of their runs of units.
                    others = at.holders - 1u;
                    wait_for_parts(args, at, 1u, rank, lanes, lane, abort_flag);
                }
            }
            auto add_others = [&](uint32_t (&v)[16], uint32_t first_row) {
                add_parts(v, args.partial + (2ull * pair_id + 2u + rank) * args.tile_floats + first_row * kRows + lanes * 32u + lane,
                                 2u * args.tile_floats, others);
            };
            const uint32_t step = helped ? kPairWeightWarp / 4u : 1u;
            uint32_t c0 = helped ? helper * 16u : 0u;
            uint32_t v[16] = {};
            if (others != 0u && c0 < rows && mine != 0u) {
                // the others' parts of this warp's first run of rows, before its own sums are there
                add_others(v, c0);
            }
            if (last && cut) {
                // asked before the last sums are there, so that the answer is
                all_begun = pair_all_begun(args.flags, *plan, rank, lanes);
            }
            // (a helper has seen none of the pieces before, so it does not ask for a parity of their barrier)
            if (!__all_sync(0xFFFFFFFFu, helper == 0u ? mbar_wait_hot(acc_full, turn & 1u, abort_flag, args.status)
                                                      : mbar_wait_hot(drain_bar, 0u, abort_flag, args.status))) {
                break;
            }
            tc_fence_after_sync();
            auto release = [&]() {
                // The accumulator is free again.
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0u) {
                    mbar_arrive_cluster(release_bar);
                }
            };
            if (!last && owner && aligned16 && mine == 32u) {
                if (gated) {
                    pair_drain<YT, true>(args.to, stage, lane_taddr, lane, chains, col, tok0, rows, release);
                } else {
                    pair_drain<YT, false>(args.to, stage, lane_taddr, lane, chains, col, tok0, rows, release);
                }
                continue;
            }
            const bool staged = aligned4 && (columns % 4u) == 0u;
#pragma unroll 1
            for (; c0 < rows && mine != 0u; c0 += 16u * step) {
                add_sums(lane_taddr + c0, chains, kPairTwoChains, v);
                if (publish) {
                    float *to = args.partial + (unsigned long long)pair_slot(blockIdx.x, owner) * args.tile_floats + c0 * kRows
                              + lanes * 32u + lane;
#pragma unroll
                    for (uint32_t i = 0; i < 16u; ++i) {
                        __stcg(to + i * kRows, __uint_as_float(v[i]));
                    }
                } else if (staged) {
                    const uint32_t buffer = stage + flip;
                    flip ^= 2048u;
                    if (gated) {
                        store_rows_staged<YT, true, false>(args.to, buffer, lane, col, columns, tok0 + c0, tok0 + rows, v);
                    } else {
                        // in two halves: the old values of an add take as many registers as the sums
                        uint32_t half[8];
#pragma unroll
                        for (uint32_t h = 0; h < 16u; h += 8u) {
#pragma unroll
                            for (uint32_t i = 0; i < 8u; ++i) {
                                half[i] = v[h + i];
                            }
                            store_rows_staged<YT, false, false>(args.to, buffer + h * 32u * sizeof(YT), lane, col, columns, tok0 + c0 + h,
                                                         tok0 + rows, half);
                        }
                    }
                } else {
                    store_rows_direct<YT>(args.to, gated, lane, mine, col, tok0 + c0, tok0 + rows, v);
                }
#pragma unroll
                for (uint32_t i = 0; i < 16u; ++i) {
                    v[i] = 0u;
                }
                if (others != 0u && c0 + 16u * step < rows) {
                    add_others(v, c0 + 16u * step);
                }
            }
            if (!last) {
                release();
            }
            if (publish) {
                // Publish this warp's quarter; every lane makes its own stores visible first.
                __threadfence();
                __syncwarp();
                if (lane == 0u) {
                    red_release_gpu_add(args.flags + kFlagWords * pair_slot(blockIdx.x, owner) + lanes, helped ? 1u : kPublishers);
                }
            }
        }
        // ------------------------------------------------------------ tiles of many holders
        // Every holder finishes a share of the tile's rows of x: the parts of all holders, its own among them, added
        // in the order of the depth.  A pair has published all it has before it waits here, and waits only where all
        // holders have begun: it holds its SMs while it waits, and a launch of another stream may hold those that a
        // holder yet needs.  Where not all have begun when the first comes here, the pair that began the tile
        // finishes it and the others go, as with few holders.  (tests/schedule_check.cu, point 9)
        mbar_wait_hot(cuts_bar, 0u, abort_flag, args.status);
#pragma unroll 1
        for (uint32_t which = 0; which < 2u; ++which) {
            const PairCut at = which == 0u ? plan->begun : plan->begins;
            if (at.holders < plan->share_from) {
                continue;
            }
            const uint32_t row_tile = at.tile / tok_tiles;
            const uint32_t tok0 = (at.tile - row_tile * tok_tiles) * ntok;
            const uint32_t rows = m - tok0 < ntok ? m - tok0 : ntok;
            const uint32_t j = (row_tile * 2u + rank) * kRows + lanes * 32u;
            const uint32_t inside = args.n > j ? args.n - j : 0u;
            const uint32_t mine = inside < 32u ? inside : 32u;
            const uint32_t columns = gated ? mine / 2u : mine;
            const uint32_t col = gated ? j / 2u : j;
            const bool staged = aligned4 && (columns % 4u) == 0u;
            const uint32_t runs = (rows + kPairShareRows - 1u) / kPairShareRows;
            if (((all_begun >> which) & 1u) == 0u) {
                const bool together = lane == 0u && pair_together(pair_begun(args.flags, at, rank, lanes), at.holders);
                all_begun |= (__any_sync(0xFFFFFFFFu, together) ? 1u : 0u) << which;
            }
            uint32_t run, end;
            pair_share(((all_begun >> which) & 1u) != 0u, pair_id - at.first, at.holders, runs, &run, &end);
            run += helper;
            if (mine == 0u) {
                run = end;
            }
            if (run < end) {
                wait_for_parts(args, at, 0u, rank, lanes, lane, abort_flag);
            }
            // This warp has published, and has seen what it needs of the others: lane 0, which has published for the warp, says
            // so, and the last warp of the holders to say so clears their flags and both counts.  Release here and
            // acquire there, so that every publication lies before the clearing, those of warps that had nothing to
            // wait for among them (no rows of w or of x left for them).
            unsigned int *count = pair_count(args.flags, at, rank, lanes);
            uint32_t came = 0u;
            if (lane == 0u) {
                __threadfence();
                came = atomicAdd(count, 1u) + 1u;
            }
            __syncwarp();
#pragma unroll 1
            for (; run < end; run += kPairWeightWarp / 4u) {
                const uint32_t c0 = run * kPairShareRows;
                const uint32_t slot = c0 * kRows + lanes * 32u + lane;
                uint32_t v[kPairShareRows];
                sum_of_parts(v, args.partial + slot, args.tile_floats, at, rank);
                if (staged) {
                    const uint32_t buffer = stage + flip;
                    flip ^= 2048u;
                    if (gated) {
                        store_rows_staged<YT, true, false>(args.to, buffer, lane, col, columns, tok0 + c0, tok0 + rows, v);
                    } else {
                        store_rows_staged<YT, false, false>(args.to, buffer, lane, col, columns, tok0 + c0, tok0 + rows, v);
                    }
                    continue;
                }
                store_rows_direct<YT>(args.to, gated, lane, mine, col, tok0 + c0, tok0 + rows, v);
            }
            if (__shfl_sync(0xFFFFFFFFu, came, 0) == at.holders * kPublishers) {
                __threadfence();
                for (uint32_t h = lane; h < at.holders; h += 32u) {
                    *reinterpret_cast<volatile unsigned int *>(args.flags + kFlagWords * pair_cut_slot(at, h, rank) + lanes) = 0u;
                }
                if (lane == 0u) {
                    *reinterpret_cast<volatile unsigned int *>(count) = 0u;
                    *reinterpret_cast<volatile unsigned int *>(pair_begun(args.flags, at, rank, lanes)) = 0u;
                }
            }
        }
    }

    // Neither block leaves while the other may still signal its barriers or read its shared memory.
    // (Nothing is handed over here, so the arrival need not wait for what a thread has in flight.)
    __syncwarp();
    tc_fence_before_sync();
    cluster_arrive_relaxed();
    cluster_wait_acquire();
    if (warp < kEpilogueWarps) {
        // The slots that an owner alone has read go back for the next launch that uses this set (every warp has passed
        // its waits; ordered by the end of the kernel).
        const PairCut at = plan->begins;
        for (uint32_t h = 1u + lane; at.holders < plan->share_from && h < at.holders; h += 32u) {
            *reinterpret_cast<volatile unsigned int *>(args.flags + kFlagWords * pair_cut_slot(at, h, rank) + warp) = 0u;
        }
    }
    if (warp == kPairMmaWarp) {
        tc_fence_after_sync();
        pair_tmem_dealloc(tmem_base, 512u);
    }
}

template <typename YT>
static cudaError_t launch_pair_typed(cudaStream_t stream, const CUtensorMap &tw, const CUtensorMap &tx, const PairArgs &args,
                                     unsigned int grid, bool overlap)
{
    static unsigned long long configured = 0ull;
    cudaError_t err = allow_shared_memory(q8_wide_kernel_pair<YT>, kPairSmem, &configured);
    if (err != cudaSuccess) {
        return err;
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(grid, 1, 1);
    config.blockDim = dim3(kPairThreads, 1, 1);
    config.dynamicSmemBytes = kPairSmem;
    config.stream = stream;
    cudaLaunchAttribute attribute[2];
    unsigned int count = 0;
    attribute[count].id = cudaLaunchAttributeClusterDimension;
    attribute[count].val.clusterDim.x = 2;
    attribute[count].val.clusterDim.y = 1;
    attribute[count].val.clusterDim.z = 1;
    ++count;
    if (overlap) {
        attribute[count].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attribute[count].val.programmaticStreamSerializationAllowed = 1;
        ++count;
    }
    config.attrs = attribute;
    config.numAttrs = count;
    return cudaLaunchKernelEx(&config, q8_wide_kernel_pair<YT>, tw, tx, args);
}

// Rows of x per tile: the batch in equal parts of at most 256, a multiple of 32 (what an MMA of two blocks
// takes).
unsigned int pair_token_tile(unsigned int m)
{
    const unsigned int parts = (m + kPairTok - 1u) / kPairTok;
    return ((m + parts - 1u) / parts + 31u) / 32u * 32u;
}

cudaError_t launch_pair_kernel(cudaStream_t stream, const CUtensorMap &tw, const CUtensorMap &tx, unsigned int ntok,
                               unsigned int sm_count, unsigned int n, unsigned int k, bool x_bf16, unsigned int m,
                               const unsigned int *m_dev, void *y, int y_dtype, unsigned int ldy, unsigned int epilogue,
                               float *partial, unsigned int *flags, unsigned long long tile_floats, unsigned int *status,
                               bool overlap)
{
    PairArgs args = {};
    args.n = n;
    args.k = k;
    args.m_max = m;
    args.m_dev = m_dev;
    args.to.y = y;
    args.to.ldy = ldy;
    args.to.epilogue = epilogue;
    args.status = status;
    args.ntok = ntok;
    args.b_bf16 = x_bf16 ? 1u : 0u;
    args.partial = partial;
    args.flags = flags;
    args.tile_floats = tile_floats;
    // Shared memory: two raw segments and as many stages of x as fit, three where that leaves five of one piece.
    // A wait, even for what is there, and a commit take the thread that issues the MMAs as long as four MMAs of 160
    // columns, one piece: so few columns have two pieces to a stage, and a raw segment less to make room for them.  Us with
    // one piece and with two: 28672 x 4096, 96 rows, 38.5 and 35.9, 128 rows 39.7 and 37.6 (three raw segments beside two
    // pieces: the same), 150 rows 42.0 and 40.3, 300 rows (160 columns) 71.0 and 69.1; four pieces below 128 columns: the same
    // as two.  192 columns: three stages of two hold less than seven of one, which one token tile feels (20480 x 4096, 192 rows,
    // 35.5 and 36.3, 28672 x 4096 44.7 and 45.1, 14336 x 4096 26.5 and 26.3) and several do not (28672 x 4096, 370 rows, 78.0
    // and 77.4, 540 rows 110.4 and 109.3, 24000 x 4096, 540 rows, 90.5 and 89.2).  224 columns: 28672 x 4096, 224 rows, 47.3
    // and 48.2; 256: 250 rows 55.0 and 60.7.
    args.x_pieces = ntok <= (m > ntok ? 192u : 160u) ? 2u : 1u;
    const unsigned int x_stage = ntok * kSubK * args.x_pieces;
    args.raw_stages = args.x_pieces == 1u && 3u * kRawStageBytes + 5u * x_stage <= kPairRings ? 3u : 2u;
    const unsigned int x_stages = (kPairRings - args.raw_stages * kRawStageBytes) / x_stage;
    args.x_stages = x_stages < kPairMaxX ? x_stages : kPairMaxX;
    const unsigned long long units = (unsigned long long)((n + 2u * kRows - 1u) / (2u * kRows)) * ((m + ntok - 1u) / ntok) * (k / kSegK);
    const unsigned int pairs = units < sm_count / 2u ? (unsigned int)units : sm_count / 2u;
    args.split = pair_split(pairs, (n + 2u * kRows - 1u) / (2u * kRows) * ((m + ntok - 1u) / ntok), k / kSegK);
    switch (y_dtype) {
    case 0:
        return launch_pair_typed<float>(stream, tw, tx, args, 2u * pairs, overlap);
    case 1:
        return launch_pair_typed<__half>(stream, tw, tx, args, 2u * pairs, overlap);
    case 2:
        return launch_pair_typed<__nv_bfloat16>(stream, tw, tx, args, 2u * pairs, overlap);
    default:
        return cudaErrorInvalidValue;
    }
}

} // namespace q8
