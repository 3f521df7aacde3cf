// The Q8_0 product for 17 to 128 rows of x, and the grouped products of the routed experts:
// y[i][j] = sum_c x[i][c] * half(q[j][c] * d[j][c / 32]), float sums.
//
// Between the two regimes: the weights cross HBM once (HBM-bound up to about 64 rows), but x,
// read again for every piece of w, weighs as much as they do, and the arithmetic is too much for the
// warp-level MMA of q8_decode_warp.cu.  Weights are dequantised into tensor memory and multiplied
// by tcgen05.mma (128 x N x 16, N = the batch rounded up to 16), as in q8_stream.cu; what is
// different there cost half the time of these products:
//
//   * Few rows of w (at most 256 per cluster of four): they are dealt in SLABS of at most 128 rows, all
//     of one size, to clusters; each block takes a run of the depth, and the parts are added through
//     distributed shared memory.  More rows: tiles of two slabs, as many to every block; or, where that
//     would leave the last of the blocks' turns too empty (kMidCutUnits), tiles of 128-row slabs cut
//     into (tile, segment) units that are dealt evenly, a cut tile finished by the block that holds
//     its first segment.
//   * A segment of x (256 deep) in shared memory meets two slabs, one after the other: half the x
//     traffic, which at 64 rows was as many bytes as the weights.
//   * 16 converter warps in two groups that take segments in turn (thread = row, half a segment).
//   * The first copies of weights go out before anything else is set up.
//   * No long chains of MMAs into one accumulator: each truncates the sum it adds to.  Two or four accumulators per
//     value (`chains`), or, in a cluster, an accumulator that is emptied into a sum of its own every few segments
//     (`run_segs`).  mid_accuracy says how many.
//
// 23 warps, one block per SM: 0-3 store (and before that turn bfloat16 x into binary16, mid_converts_x), 4-19 convert, 20 copies weights, 21 copies x, 22 issues the MMAs.  Every wait is bounded and raises a
// status bit when it runs out.  Reference kernels replaced: as q8_stream.cu.
#include <cuda.h>

#include "q8_launch.h"
#include "q8_rows.cuh"
#include "q8_schedule.cuh"

namespace q8 {

constexpr uint32_t kMidThreads = 23 * 32;
constexpr uint32_t kMidGroups = 2;         // of converter warps, which take segments in turn
constexpr uint32_t kMidGroupWarps = 8;
constexpr uint32_t kMidWeightWarp = 20;
constexpr uint32_t kMidInputWarp = 21;
constexpr uint32_t kMidMmaWarp = 22;
constexpr uint32_t kMidMaxRaw = 12;        // stages of the rings, at most
constexpr uint32_t kMidMaxX = 8;
constexpr uint32_t kMidMaxA = 3;
constexpr uint32_t kMidBars = 3 * kMidMaxRaw + 3 * kMidMaxX + 2 * kMidMaxA + 4 + 1;
constexpr uint32_t kMidStageBytes = 4 * 2 * 2048;   // per storing warp: two turns of 16 rows of x by 32 columns, floats
constexpr uint32_t kMidTail = kMidStageBytes + kMidBars * 8 + 16;
constexpr uint32_t kMidConvertStep = kEpilogueWarps * 32u * 16u;      // bytes of x that the storing warps convert at a time
constexpr uint32_t kMidSmem = 227u * 1024u;
constexpr uint32_t kMidRings = (kMidSmem - 1024u - kMidTail) / 1024u * 1024u;   // both rings' shared memory

// Cutting tiles into units evens the blocks out and costs them the hand-over of the cut tiles, more
// stores at the wrong moment and a longer end: about as long as five units (of two slabs) take.
// Measured with and without: 28672 x 4096, 64 rows, 12.1 units against 16: 33.5 us against 30.6;
// 151936 x 8192, 64 rows, 128.3 against 144: 249 us against 269; routed experts, 512 tokens, 21
// against 24: 262 us against 217.
constexpr uint32_t kMidCutUnits = 5;

struct MidArgs {
    unsigned int n, k, m_max;
    const unsigned int *m_dev;
    RowStore to;
    unsigned int *status;
    const GroupTile *group_tiles;      // grouped mode: the device's table, else null
    const unsigned int *group_count;
    unsigned int ntok;                 // columns of an accumulator: rows of x, a multiple of 16
    unsigned int slab_rows;            // rows of w per slab (a multiple of 4)
    unsigned int pair;                 // slabs that share a segment of x: 1 or 2
    unsigned int table_late;           // grouped: the launch before this one writes the table
    unsigned int tiles;                // of `pair` slabs each (not in grouped mode)
    unsigned int turns;                // whole tiles per block; 0: units (not in grouped mode)
    // unit schedule: a block's partial tile, [slab][row of x][row of w], and its flags
    float *partial;
    unsigned int *flags;
    unsigned long long tile_floats;
    unsigned int x_stages, raw_stages, a_stages, acc_buffers;
    unsigned int raw_offset, raw_stride;
    unsigned int chains;               // accumulators of a value, which parts of a segment take in turn: 1, 2 or 4
    unsigned int run_segs;             // segments per run of a cluster's block, fewer than it has; 0: one run
    // Columns of tensor memory: of one accumulator of a tile, of a buffer of `chains` of them (and of the sum of a
    // cluster's runs so far, behind them); where the segments of A begin.
    unsigned int acc_columns, buffer_columns, a_column0;
    unsigned int x_bf16;               // x is bfloat16 and becomes binary16 in shared memory (one piece per block only)
    unsigned int read_chains;          // accumulators, and the sum of the runs, that make a finished sum
};

// The MMAs of one segment of A against one of x: `chains` accumulators, `stride` columns apart, which the segment's
// four parts (64 deep) take in turn; `later`: not the first segment of its piece.
__device__ __forceinline__ void multiply_segment(uint32_t d_tmem, uint32_t stride, uint32_t chains, uint32_t a_tmem, uint32_t x_seg,
                                                 uint32_t x_seg_bytes, uint32_t idesc, bool later)
{
#pragma unroll
    for (uint32_t j = 0; j < kSubs; ++j) {
        const uint64_t b_desc = umma_desc_sw128(x_seg + j * (x_seg_bytes / kSubs));
        const uint32_t d = d_tmem + (j & (chains - 1u)) * stride;
#pragma unroll
        for (uint32_t kk = 0; kk < kSubK / 16u; ++kk) {
            // 16 halves: 8 columns of A, 32 bytes along the swizzled row of x
            umma_f16_ts(d, a_tmem + j * (kSubK / 2u) + 8u * kk, b_desc + 2u * kk, idesc,
                        kk != 0u || j >= chains || later ? 1u : 0u);
        }
    }
}

// The sums of all runs but the last (`turns` of them) of a cluster's block, added up behind the accumulators by the
// storing warps; the readers at the end find them there.  (The MMAs of a run wait for what is done here with the
// one before, which orders it for who waits for the MMAs.)  Out of line: few launches need it, and a short
// launch fetches its code cold.
__device__ __noinline__ void add_up_runs(uint32_t lane_taddr, uint32_t columns, uint32_t chains, uint32_t turns, uint32_t acc_full,
                                         uint32_t acc_empty, volatile uint32_t *abort_flag, unsigned int *status)
{
    for (uint32_t turn = 0; turn < turns; ++turn) {
        if (!__all_sync(0xFFFFFFFFu, mbar_wait_hot(acc_full, turn & 1u, abort_flag, status))) {
            return;
        }
        tc_fence_after_sync();
#pragma unroll 1
        for (uint32_t c0 = 0; c0 < columns; c0 += 16u) {
            uint32_t v[16];
            load_sums(lane_taddr + c0, turn != 0u ? chains + 1u : chains, columns, v);
            tmem_st_32x16(lane_taddr + chains * columns + c0, v);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if ((threadIdx.x & 31u) == 0u) {
            mbar_arrive(acc_empty);
        }
    }
}

// TWIN (grouped, pair 2): the second slab of a tile is the same rows of a second tensor, and what is stored is
// the gated unit of the two.
template <typename YT, bool TWIN>
__global__ void __launch_bounds__(kMidThreads, 1)
q8_stream_kernel_mid(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_second,
                     const __grid_constant__ CUtensorMap tmap_x, const MidArgs args)
{
    extern __shared__ unsigned char smem_raw_[];
    const uint32_t smem0 = (smem_u32(smem_raw_) + 1023u) & ~1023u;
    unsigned char *const smem = smem_raw_ + (smem0 - smem_u32(smem_raw_));
    const uint32_t raw_base = smem0 + args.raw_offset;
    const uint32_t stage_base = smem0 + kMidRings;
    const uint32_t raw_full = stage_base + kMidStageBytes;
    // Two barriers per raw stage, for its uses in turn: a barrier then belongs to one group of
    // converters.  (With one barrier and an odd number of stages the groups alternate on it, and a
    // group that comes to a stage's second use while the first copy is still on its way - copies may
    // land out of order - finds the parity it waits for: that of the use before the first.)
    const uint32_t raw_empty = raw_full + 16u * kMidMaxRaw;
    const uint32_t raw_turns = 2u * args.raw_stages;
    const uint32_t x_full = raw_empty + 8u * kMidMaxRaw;
    const uint32_t x_empty = x_full + 8u * kMidMaxX;
    const uint32_t a_full = x_empty + 8u * kMidMaxX;
    const uint32_t a_empty = a_full + 8u * kMidMaxA;
    const uint32_t acc_full = a_empty + 8u * kMidMaxA;
    const uint32_t acc_empty = acc_full + 16u;
    const uint32_t drain_bar = acc_empty + 16u;
    const uint32_t x_ready = drain_bar + 8u;      // x is binary16
    const uint32_t tmem_slot = x_ready + 8u * kMidMaxX;
    volatile uint32_t *tmem_slot_ptr = reinterpret_cast<volatile uint32_t *>(smem + (tmem_slot - smem0));
    volatile uint32_t *abort_flag = tmem_slot_ptr + 1;

    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31u;
    const bool grouped = args.group_tiles != nullptr;
    const uint32_t segs = args.k / kSegK;
    const uint32_t pair = args.pair;
    const uint32_t ntok = args.ntok;
    const uint32_t x_seg_bytes = ntok * (kSegK * 2u);
    const uint32_t raw_bytes = args.slab_rows * kSegBytes;
    const uint32_t csize = cluster_nctarank();
    const uint32_t crank = cluster_ctarank();
    // Clusters: one tile each, a run of its segments per block.  Else (tile, segment) units dealt evenly,
    // the same arithmetic as the decode kernel's.  (The table of the grouped products, and its length, are
    // there already unless the launch before this one writes them.  That launch is then waited for before
    // the next one may start, so that the next one finds the table, too.)
    if (args.table_late != 0u) {
        grid_dependency_wait();
    }
    // table entries per tile, and from the first slab's to the second's
    const uint32_t entries = TWIN ? 1u : pair;
    constexpr uint32_t second = TWIN ? 0u : 1u;
    const uint32_t tiles = grouped ? *reinterpret_cast<const volatile unsigned int *>(args.group_count) / entries : args.tiles;
    const uint32_t units = tiles * segs;      // the host refuses products with 2^31 units or more
    const uint32_t blocks = units < gridDim.x ? units : gridDim.x;
    uint32_t turns = args.turns;
    if (grouped) {
        turns = (tiles + gridDim.x - 1u) / gridDim.x;
        if (turns * segs > units / gridDim.x + kMidCutUnits) {
            turns = 0u;
        }
    }
    MidWork work;
    mid_deal(&work, blockIdx.x, gridDim.x, csize, crank, tiles, segs, turns, args.run_segs);
    const uint32_t total = work.left * pair;   // segments of weights

    grid_launch_dependents();

    uint32_t early = 0u;
    if (warp == kMidWeightWarp && elect_one()) {
        tma_prefetch_desc(&tmap_w);
        if (TWIN) {
            tma_prefetch_desc(&tmap_second);
        }
        tma_prefetch_desc(&tmap_x);
        for (uint32_t i = 0; i < args.raw_stages; ++i) {
            mbar_init(raw_full + 8u * i, 1u);
            mbar_init(raw_full + 8u * (i + args.raw_stages), 1u);
            mbar_init(raw_empty + 8u * i, kMidGroupWarps);
        }
        for (uint32_t i = 0; i < args.x_stages; ++i) {
            mbar_init(x_full + 8u * i, 1u);
            mbar_init(x_empty + 8u * i, 1u);
            mbar_init(x_ready + 8u * i, kEpilogueWarps);
        }
        for (uint32_t i = 0; i < args.a_stages; ++i) {
            mbar_init(a_full + 8u * i, kMidGroupWarps);
            mbar_init(a_empty + 8u * i, 1u);
        }
        for (uint32_t i = 0; i < 2u; ++i) {
            mbar_init(acc_full + 8u * i, 1u);
            mbar_init(acc_empty + 8u * i, kEpilogueWarps);
        }
        mbar_init(drain_bar, 1u);
        *abort_flag = 0u;
        mbar_init_fence();
        fence_proxy_async_smem();
        // the first weights: only the barriers they signal have to be there
        uint32_t tile = work.next_tile, s = work.next_seg, p = 0u;
        for (; early < args.raw_stages && early < total; ++early) {
            const uint32_t w_row = grouped ? args.group_tiles[(size_t)tile * entries + p * second].w_row
                                           : (tile * pair + p) * args.slab_rows;
            mbar_expect_tx(raw_full + 8u * early, raw_bytes);
            tma_load_2d(raw_base + early * args.raw_stride, TWIN && p != 0u ? &tmap_second : &tmap_w,
                        raw_full + 8u * early, (int)(s * kSegWords), (int)w_row);
            if (++p == pair) {
                p = 0u;
                if (++s == segs) {
                    s = 0u;
                    tile += work.stride;
                }
            }
        }
    }
    if (warp == kMidMmaWarp) {
        tmem_alloc(tmem_slot, 512u);
        tmem_relinquish();
    }
    if (csize > 1u) {
        __syncwarp();
        cluster_arrive_relaxed();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot_ptr;

    unsigned int m_live = args.m_max;

    if (warp == kMidWeightWarp) {
        // ---------------------------------------------------------------- weight copies
        if (elect_one()) {
            uint32_t g = 0;
            bool ok = true;
            uint32_t full = 0u;                    // g modulo the full barriers
            uint32_t st = 0u, ph = 1u;             // g modulo the stages, and the parity of the use before
            while (ok && work.next()) {
                uint32_t w_row[2];
                if (grouped) {
                    const GroupTile *entry = args.group_tiles + (size_t)work.tile * entries;
                    w_row[0] = entry[0].w_row;
                    w_row[1] = pair > 1u ? entry[second].w_row : 0u;
                } else {
                    w_row[0] = work.tile * pair * args.slab_rows;
                    w_row[1] = w_row[0] + args.slab_rows;
                }
                for (uint32_t s = work.s0; ok && s < work.s1; ++s) {
                    for (uint32_t p = 0; p < pair; ++p, ++g) {
                        if (g >= early) {
                            if (!mbar_wait(raw_empty + 8u * st, ph, abort_flag, args.status)) {
                                ok = false;
                                break;
                            }
                            mbar_expect_tx(raw_full + 8u * full, raw_bytes);
                            tma_load_2d(raw_base + st * args.raw_stride, TWIN && p != 0u ? &tmap_second : &tmap_w,
                                        raw_full + 8u * full, (int)(s * kSegWords), (int)(p == 0u ? w_row[0] : w_row[1]));
                        }
                        full = full + 1u == raw_turns ? 0u : full + 1u;
                        if (++st == args.raw_stages) {
                            st = 0u;
                            ph ^= 1u;
                        }
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
    } else if (warp == kMidInputWarp) {
        // ---------------------------------------------------------------- x copies
        if (elect_one()) {
            uint32_t g = 0;
            grid_dependency_wait();
            bool ok = true;
            uint32_t st = 0u, ph = 1u;
            while (ok && work.next()) {
                const uint32_t tok0 = grouped ? args.group_tiles[(size_t)work.tile * entries].tok0 : 0u;
                for (uint32_t s = work.s0; s < work.s1; ++s, ++g) {
                    if (!mbar_wait(x_empty + 8u * st, ph, abort_flag, args.status)) {
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(x_full + 8u * st, x_seg_bytes);
#pragma unroll
                    for (uint32_t j = 0; j < kSubs; ++j) {
                        tma_load_2d(smem0 + st * x_seg_bytes + j * (x_seg_bytes / kSubs), &tmap_x, x_full + 8u * st,
                                    (int)(s * kSegK + j * kSubK), (int)tok0);
                    }
                    if (++st == args.x_stages) {
                        st = 0u;
                        ph ^= 1u;
                    }
                }
            }
            uint32_t local_abort = 0;
            const uint32_t first = g > args.x_stages ? g - args.x_stages : 0u;
            for (uint32_t i = first; i < g; ++i) {
                mbar_wait(x_full + 8u * (i % args.x_stages), (i / args.x_stages) & 1u, &local_abort, nullptr);
            }
        }
    } else if (warp == kMidMmaWarp) {
        // ---------------------------------------------------------------- MMA issue
        // (Asking for the next segments before the MMAs of this one, so that the answer is there when they are issued, was
        // slower: the answer is waited for where it is asked for, and the MMAs behind it.  Layer of 32 rows 73.7 -> 72.8 us,
        // of 100 rows 105.1 -> 103.4, routed experts, 512 tokens, 199 -> 197 without.)
        if (elect_one()) {
            const uint32_t idesc = umma_idesc(kRows, ntok, 0u, 0u);
            const uint32_t x_bar = args.x_bf16 != 0u ? x_ready : x_full;
            // (counted up, not divided: a division by a number that only the launch knows takes longer
            // than the MMAs of a segment)
            uint32_t xst = 0u, xph = 0u;
            uint32_t ast = 0u, aph = 0u;
            bool ok = true;
            for (uint32_t turn = 0; ok && work.next(); ++turn) {
                const uint32_t buf = args.acc_buffers > 1u ? turn & 1u : 0u;
                const uint32_t uses = args.acc_buffers > 1u ? turn >> 1 : turn;
                if (!mbar_wait(acc_empty + 8u * buf, (uses & 1u) ^ 1u, abort_flag, args.status)) {
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                for (uint32_t s = work.s0; ok && s < work.s1; ++s) {
                    if (!mbar_wait_hot(x_bar + 8u * xst, xph, abort_flag, args.status)) {
                        ok = false;
                        break;
                    }
                    for (uint32_t p = 0; p < pair; ++p) {
                        if (!mbar_wait_hot(a_full + 8u * ast, aph, abort_flag, args.status)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after_sync();
                        const uint32_t d_tmem = tmem_base + buf * args.buffer_columns + p * ntok;
                        const uint32_t a_tmem = tmem_base + args.a_column0 + ast * (kSegK / 2u);
                        const uint32_t x_seg = smem0 + xst * x_seg_bytes;
                        const bool later = s != work.s0;
                        multiply_segment(d_tmem, args.acc_columns, args.chains, a_tmem, x_seg, x_seg_bytes, idesc, later);
                        umma_commit(a_empty + 8u * ast);
                        if (++ast == args.a_stages) {
                            ast = 0u;
                            aph ^= 1u;
                        }
                    }
                    if (ok) {
                        umma_commit(x_empty + 8u * xst);
                        if (++xst == args.x_stages) {
                            xst = 0u;
                            xph ^= 1u;
                        }
                    }
                }
                if (ok) {
                    umma_commit(acc_full + 8u * buf);
                }
            }
            if (total != 0u) {
                // Every MMA has finished: what the helping warps wait for.  This thread waits as well, whoever
                // else does: the arrival must not come to a shared memory that the block has left, nor may
                // tensor memory go back under outstanding MMAs.  (A block without work issues none.)
                uint32_t local_abort = 0;
                umma_commit(drain_bar);
                mbar_wait(drain_bar, 0u, &local_abort, nullptr);
            }
        }
    } else if (warp >= kConvertWarp0) {
        // ---------------------------------------------------------------- dequantise
        // Two groups of eight warps take segments in turn: while one group waits for its raw segment, for
        // its stage of tensor memory or for its loads, the other has the arithmetic.  (Sixteen warps
        // on one segment go through these phases together and leave the schedulers idle in between.)
        const uint32_t cw = warp - kConvertWarp0;
        const uint32_t group = cw / kMidGroupWarps;
        const uint32_t half = (cw >> 2) & 1u;
        const uint32_t row = (cw & 3u) * 32u + lane;
        // rows past the slab repeat its last one (their sums are not stored)
        const uint32_t row_at = (row < args.slab_rows ? row : args.slab_rows - 1u) * kSegBytes;
        const uint32_t lane_base = tmem_base + (((cw & 3u) * 32u) << 16) + args.a_column0 + half * (kSegK / 4u);
        uint32_t full = group, fph = 0, ast = group, aph = 0;
        for (uint32_t g = group; g < total; g += kMidGroups) {
            if (!__all_sync(0xFFFFFFFFu, mbar_wait_hot(raw_full + 8u * full, fph, abort_flag, args.status))) {
                break;
            }
            const uint32_t rst = full < args.raw_stages ? full : full - args.raw_stages;
            uint32_t raw[36];
            const uint32_t raw_row = raw_base + rst * args.raw_stride + row_at;
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
            const uint32_t taddr = lane_base + ast * (kSegK / 2u);
            tc_fence_after_sync();
            if (half == 0u) {
                convert_stage_tmem<0, 0>(raw, taddr);
                convert_stage_tmem<0, 1>(raw, taddr + kSubK / 2u);
            } else {
                convert_stage_tmem<1, 0>(raw, taddr);
                convert_stage_tmem<1, 1>(raw, taddr + kSubK / 2u);
            }
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0u) {
                mbar_arrive(a_full + 8u * ast);
            }
            full += kMidGroups;
            if (full >= raw_turns) {
                full -= raw_turns;
                fph ^= 1u;
            }
            ast += kMidGroups;
            if (ast >= args.a_stages) {
                ast -= args.a_stages;
                aph ^= 1u;
            }
        }
    } else if (args.x_bf16 != 0u) {
        // ---------------------------------------------------------------- x to binary16
        // The storing warps have nothing to store before the block's one piece is done.
        uint32_t st = 0u, ph = 0u;
        for (uint32_t g = 0; g < work.left; ++g) {
            if (!__all_sync(0xFFFFFFFFu, mbar_wait_hot(x_full + 8u * st, ph, abort_flag, args.status))) {
                break;
            }
            const uint32_t mine = smem0 + st * x_seg_bytes + threadIdx.x * 16u;
#pragma unroll 1
            for (uint32_t at = mine; at < mine + x_seg_bytes; at += 4u * kMidConvertStep) {
                uint32_t v[4][4];
#pragma unroll
                for (uint32_t i = 0; i < 4u; ++i) {
                    ld_shared_v4(at + i * kMidConvertStep, v[i][0], v[i][1], v[i][2], v[i][3]);
                }
#pragma unroll
                for (uint32_t i = 0; i < 4u; ++i) {
                    st_shared_v4(at + i * kMidConvertStep, bf16x2_to_f16x2(v[i][0]), bf16x2_to_f16x2(v[i][1]),
                                 bf16x2_to_f16x2(v[i][2]), bf16x2_to_f16x2(v[i][3]));
                }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0u) {
                mbar_arrive(x_ready + 8u * st);
            }
            if (++st == args.x_stages) {
                st = 0u;
                ph ^= 1u;
            }
        }
    }

    uint32_t last_cc = blockIdx.x;      // the last block whose partial sums this one takes
    if (csize == 1u && warp < kMidWeightWarp && total != 0u) {
        // ---------------------------------------------------------------- read sums, store
        // Warps 0-3 store every piece but the last beside the work of the next.  In the last one nothing
        // is left to convert and the converters help: four warps alone took 4.6 us (64 rows) and 7 us
        // (100 rows) at the end of launches of 30 and 40 us.  Their staging buffers lie over the
        // rings, which are idle once the last sums are there.
        //
        // A tile that is cut between blocks belongs to the block that holds its first segment: that
        // block's last piece, while the other holders - the blocks right after it - meet the tile at the
        // start of their ranges and have published their sums long before.  The owner adds them in
        // block order.
        const uint32_t lanes = warp & 3u;
        const uint32_t helper = warp >> 2;                       // 0: the storing warps
        const uint32_t lane_taddr = tmem_base + ((lanes * 32u) << 16);
        const bool gated = args.to.epilogue == kEpilogueSwiglu && !TWIN;
        const uint32_t buffers = helper == 0u ? stage_base + warp * (kMidStageBytes / 4u)
                                              : smem0 + (warp - kEpilogueWarps) * (kMidStageBytes / 4u);
        uint32_t flip = 0u;      // the two turns of the warp's staging buffer
        grid_dependency_wait();
        if (args.m_dev != nullptr) {
            const unsigned int live = *args.m_dev;
            m_live = live < m_live ? live : m_live;
        }
        // rows of y start on a boundary of four values
        const bool aligned = (args.to.ldy % 4u) == 0u && (reinterpret_cast<uintptr_t>(args.to.y) % (4u * sizeof(YT))) == 0u;
        for (uint32_t turn = 0; work.next(); ++turn) {
            const bool last = work.left == 0u;
            const bool owner = work.s0 == 0u;
            const bool helped = last;
            if (helper != 0u && !helped) {
                continue;
            }
            const uint32_t buf = args.acc_buffers > 1u ? turn & 1u : 0u;
            const uint32_t uses = args.acc_buffers > 1u ? turn >> 1 : turn;
            // where the tile goes (in grouped mode the entry of its first slab; the second slab is the next 128 rows
            // of the same expert, TWIN the same rows of the other tensor): asked for before the wait
            GroupTile place = {};
            if (grouped) {
                place = args.group_tiles[(size_t)work.tile * entries];
            } else {
                place.j0 = work.tile * pair * args.slab_rows;
                place.j_limit = args.n;
                place.tok_limit = m_live;
            }
            // The rows of y of the tile's rows of x (both slabs have the same), lane i those of rows i, 32 + i, ..: asked for
            // before the wait as well (TWIN: the same numbers).  Where each store of 16 rows fetched its own, 1400 cycles
            // each, the routed experts' down product waited for its four storing warps: 512 tokens, 8 of 128
            // experts, 2048 x 768, the whole step 204.7 -> 197.1 us.
            uint32_t rows_of[kRows / 32u];
#pragma unroll
            for (uint32_t i = 0; i < kRows / 32u; ++i) {
                const uint32_t row_x = place.tok0 + 32u * i + lane;
                rows_of[i] = !TWIN && args.to.row_map != nullptr && row_x < place.tok_limit ? args.to.row_map[row_x] : row_x;
            }
            if (owner && work.s1 != segs) {
                last_cc = decode_holder((work.tile + 1u) * segs - 1u, blocks, units);
                for (uint32_t base = blockIdx.x + 1u; base <= last_cc; base += 32u) {
                    const uint32_t cc = base + lane;
                    if (cc <= last_cc) {
                        const unsigned int *flag = args.flags + kFlagWords * cc + lanes;
                        const long long begin = clock64();
                        while (ld_acquire_gpu(flag) < kPublishers) {
                            if (clock64() - begin > Q8_WAIT_CYCLES || *abort_flag != 0u) {
                                atomicOr(args.status, Q8_DEV_FLAG_TIMEOUT);
                                break;
                            }
                        }
                    }
                }
                __syncwarp();
            }
            // (a helper has seen none of the pieces before, so it does not ask for a parity of their barrier)
            if (!__all_sync(0xFFFFFFFFu, helper == 0u ? mbar_wait(acc_full + 8u * buf, uses & 1u, abort_flag, args.status)
                                                      : mbar_wait(drain_bar, 0u, abort_flag, args.status))) {
                break;
            }
            tc_fence_after_sync();
            // pieces of 16 rows of x, dealt to the warps of the same lanes where they help
            const uint32_t step = helped ? kMidWeightWarp / 4u : 1u;
            uint32_t piece = helped ? helper : 0u;
#pragma unroll 1
            for (uint32_t p = 0; p < (TWIN && owner ? 1u : pair); ++p) {
                const uint32_t rows = place.tok_limit > place.tok0 ? place.tok_limit - place.tok0 : 0u;
                const uint32_t live = (rows < ntok ? rows + 15u : ntok) / 16u;           // pieces with a row to store
                const uint32_t j0 = place.j0 + (TWIN ? 0u : p * args.slab_rows);
                const uint32_t j_limit = j0 + args.slab_rows < place.j_limit ? j0 + args.slab_rows : place.j_limit;
                const uint32_t j = j0 + lanes * 32u;                                     // this warp's first row of w
                const uint32_t inside = j_limit > j ? j_limit - j : 0u;                  // ... and how many are there
                const uint32_t mine = inside < 32u ? inside : 32u;
                const uint32_t columns = gated ? mine / 2u : mine;
                const uint32_t col = gated ? j / 2u : j;
                const bool staged = aligned && (columns % 4u) == 0u;
#pragma unroll 1
                for (; piece < live; piece += step) {
                    if (mine == 0u) {
                        continue;
                    }
                    const uint32_t c0 = piece * 16u;
                    const uint32_t slot = (p * ntok + c0) * kRows + lanes * 32u + lane;
                    uint32_t v[16];
                    load_sums(lane_taddr + buf * args.buffer_columns + p * ntok + c0, args.read_chains, args.acc_columns, v);
                    if (!owner) {
                        float *to = args.partial + (unsigned long long)blockIdx.x * args.tile_floats + slot;
#pragma unroll
                        for (uint32_t i = 0; i < 16u; ++i) {
                            __stcg(to + i * kRows, __uint_as_float(v[i]));
                        }
                        continue;
                    }
                    const uint32_t holders = last_cc - blockIdx.x;   // none for a whole tile
                    const float *others = args.partial + (unsigned long long)(blockIdx.x + 1u) * args.tile_floats + slot;
                    add_partial_sums(v, others, args.tile_floats, holders);
                    if (TWIN) {
                        // gate and up of the same columns lie in the two slabs' sums
                        uint32_t up[16];
                        load_sums(lane_taddr + buf * args.buffer_columns + ntok + c0, args.read_chains, args.acc_columns, up);
                        add_partial_sums(up, others + ntok * kRows, args.tile_floats, holders);
#pragma unroll
                        for (uint32_t i = 0; i < 16u; ++i) {
                            v[i] = __float_as_uint(gated_unit(__uint_as_float(v[i]), __uint_as_float(up[i])));
                        }
                    }
                    if (staged) {
                        const uint32_t buffer = buffers + flip;
                        flip ^= kMidStageBytes / 8u;
                        const uint32_t two_pieces = c0 < 64u ? (c0 < 32u ? rows_of[0] : rows_of[1]) : (c0 < 96u ? rows_of[2] : rows_of[3]);
                        const uint32_t mapped = __shfl_sync(0xFFFFFFFFu, two_pieces, (c0 & 16u) + (lane & 15u));
                        if (gated) {
                            store_rows_staged<YT, true, !TWIN>(args.to, buffer, lane, col, columns, place.tok0 + c0, place.tok_limit, v, mapped);
                        } else {
                            store_rows_staged<YT, false, !TWIN>(args.to, buffer, lane, col, columns, place.tok0 + c0, place.tok_limit, v, mapped);
                        }
                        continue;
                    }
                    store_rows_direct<YT>(args.to, gated, lane, mine, col, place.tok0 + c0, place.tok_limit, v);
                }
                piece -= live;
            }
            if (!owner) {
                // Publish this warp's quarter; every lane makes its own stores visible first.
                __threadfence();
                __syncwarp();
                if (lane == 0u) {
                    red_release_gpu_add(args.flags + kFlagWords * blockIdx.x + lanes, helped ? 1u : kPublishers);
                }
            }
            if (!last) {
                // The accumulators are free again.
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0u) {
                    mbar_arrive(acc_empty + 8u * buf);
                }
            }
        }
    }

    __syncwarp();
    if (csize > 1u) {
        // ------------------------------------------------------------ sum of a cluster's parts
        // One pair of slabs per cluster.  The rows of x are dealt to its blocks in runs of `share`;
        // every block writes its part's sums into their owners' shared memory, over the rings, which are
        // idle by then: [sender][slab][run of four rows of x][row of w], 16 bytes at a time.  The owner adds the parts in block order.
        if (args.run_segs != 0u && warp < kEpilogueWarps) {
            add_up_runs(tmem_base + ((warp * 32u) << 16), args.acc_columns, args.chains, (work.left - 1u) / args.run_segs, acc_full,
                        acc_empty, abort_flag, args.status);
        }
        bool there = true;
        if (warp < kMidWeightWarp) {
            there = mbar_wait(drain_bar, 0u, abort_flag, args.status);
            tc_fence_after_sync();
        }
        const uint32_t share = ntok / csize;
        __syncwarp();
        cluster_wait_acquire();      // every block has started ...
        cluster_arrive_relaxed();    // ... and is done with its rings
        cluster_wait_acquire();
        if (warp < kMidWeightWarp) {
            const uint32_t quarter_lanes = warp & 3u;
            const uint32_t lane_taddr = tmem_base + ((quarter_lanes * 32u) << 16);
            const uint32_t row = quarter_lanes * 32u + lane;
            const uint32_t chunks = quarter_lanes * 32u < args.slab_rows ? pair * ntok / 16u : 0u;     // (rows of w past the slab)
            for (uint32_t c = warp >> 2; c < chunks; c += kMidWeightWarp / 4u) {
                const uint32_t p = c / (ntok / 16u);
                const uint32_t c0 = (c - p * (ntok / 16u)) * 16u;
                uint32_t v[16];
                load_sums(lane_taddr + p * ntok + c0, args.read_chains, args.acc_columns, v);
                uint32_t owner = c0 / share;
                uint32_t run = (c0 - owner * share) / 4u;
#pragma unroll
                for (uint32_t i = 0; i < 16u; i += 4u) {
                    const uint32_t at = smem0 + (((crank * pair + p) * (share / 4u) + run) * kRows + row) * 16u;
                    st_shared_cluster_v4_f32(mapa_shared(at, owner), __uint_as_float(v[i]), __uint_as_float(v[i + 1u]),
                                             __uint_as_float(v[i + 2u]), __uint_as_float(v[i + 3u]));
                    if (++run == share / 4u) {
                        run = 0u;
                        ++owner;
                    }
                }
            }
            tc_fence_before_sync();
        }
        __syncwarp();
        cluster_arrive_release();
        cluster_wait_acquire();
        grid_dependency_wait();
        if (args.m_dev != nullptr) {
            const unsigned int live = *args.m_dev;
            m_live = live < m_live ? live : m_live;
        }
        if (!there) {
            m_live = 0u;
        }
        const float4 *recv = reinterpret_cast<const float4 *>(smem);
        const bool gated = args.to.epilogue == kEpilogueSwiglu;
        const uint32_t runs = pair * (share / 4u);                      // runs of four rows of x per sender
        // warp = 32 rows of w of one run
        for (uint32_t at = warp; at < runs * (kRows / 32u); at += kMidThreads / 32u) {
            const uint32_t local = at / (kRows / 32u);                  // slab * (share / 4) + run within the share
            const uint32_t row = (at % (kRows / 32u)) * 32u + lane;
            if (row - lane >= args.slab_rows) {
                continue;
            }
            const uint32_t p = local / (share / 4u);
            const uint32_t token = crank * share + (local - p * (share / 4u)) * 4u;
            float4 four = recv[local * kRows + row];
            for (uint32_t src = 1; src < csize; ++src) {
                const float4 more = recv[(src * runs + local) * kRows + row];
                four = make_float4(four.x + more.x, four.y + more.y, four.z + more.z, four.w + more.w);
            }
            const uint32_t j = (blockIdx.x / csize * pair + p) * args.slab_rows + row;
            const float sums[4] = {four.x, four.y, four.z, four.w};
#pragma unroll
            for (uint32_t i = 0; i < 4u; ++i) {
                float sum = sums[i];
                if (gated) {
                    const float up = __shfl_xor_sync(0xFFFFFFFFu, sum, 1u);
                    sum = gated_unit(sum, up);
                }
                if (token + i < m_live && row < args.slab_rows && j < args.n && (!gated || (row & 1u) == 0u)) {
                    store_value<YT>(args.to, (size_t)(token + i) * args.to.ldy + (gated ? j / 2u : j), sum);
                }
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp < kEpilogueWarps) {
        // Hand the consumed slots back for the next launch that uses this set (every warp has passed its
        // waits; ordered by the end of the kernel).
        for (uint32_t cc = blockIdx.x + 1u + lane; cc <= last_cc; cc += 32u) {
            *reinterpret_cast<volatile unsigned int *>(args.flags + kFlagWords * cc + warp) = 0u;
        }
    }
    if (warp == kMidMmaWarp) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512u);
    }
}

template <typename YT, bool TWIN>
static cudaError_t launch_mid_typed(cudaStream_t stream, const CUtensorMap &tw, const CUtensorMap &tw2, const CUtensorMap &tx, const MidArgs &args,
                                    unsigned int grid, unsigned int cluster, bool overlap)
{
    static unsigned long long configured = 0ull;
    cudaError_t err = allow_shared_memory(q8_stream_kernel_mid<YT, TWIN>, kMidSmem, &configured);
    if (err != cudaSuccess) {
        return err;
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(grid, 1, 1);
    config.blockDim = dim3(kMidThreads, 1, 1);
    config.dynamicSmemBytes = kMidSmem;
    config.stream = stream;
    cudaLaunchAttribute attribute[2];
    unsigned int count = 0;
    if (overlap) {
        attribute[count].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attribute[count].val.programmaticStreamSerializationAllowed = 1;
        ++count;
    }
    if (cluster > 1u) {
        attribute[count].id = cudaLaunchAttributeClusterDimension;
        attribute[count].val.clusterDim.x = cluster;
        attribute[count].val.clusterDim.y = 1;
        attribute[count].val.clusterDim.z = 1;
        ++count;
    }
    config.attrs = attribute;
    config.numAttrs = count;
    return cudaLaunchKernelEx(&config, q8_stream_kernel_mid<YT, TWIN>, tw, tw2, tx, args);
}

static cudaError_t launch_mid(cudaStream_t stream, const CUtensorMap &tw, const CUtensorMap *tw_second,
                              const CUtensorMap &tx, MidArgs &args, unsigned int grid, unsigned int cluster, bool overlap, int y_dtype)
{
    // Tensor memory: accumulators in two buffers where a block has several pieces and they leave room for
    // two segments of A.  (One piece: nothing to overlap its store with, and a third segment of A instead
    // is worth 4 %: 28672 x 4096, 64 rows, 31.9 -> 30.4 us; 4096 x 14336, 100 rows, 24.4 -> 23.5.)
    const bool one_piece = cluster > 1u || args.turns == 1u;
    args.acc_columns = args.pair * args.ntok;
    args.read_chains = args.chains + (args.run_segs != 0u ? 1u : 0u);
    args.buffer_columns = args.read_chains * args.acc_columns;
    args.acc_buffers = !one_piece && 2u * args.buffer_columns <= 256u ? 2u : 1u;
    args.a_column0 = args.acc_buffers * args.buffer_columns;
    const unsigned int a_stages = (512u - args.a_column0) / (kSegK / 2u);
    args.a_stages = a_stages < kMidMaxA ? a_stages : kMidMaxA;
    // Shared memory: up to four segments of x, as far as they leave about 100 KB to the weights (three
    // full slabs; 104 KB in flight per SM read memory at 6.8 TB/s), the rest to the weights.
    const unsigned int x_seg = args.ntok * kSegK * 2u;
    args.raw_stride = (args.slab_rows * kSegBytes + 127u) / 128u * 128u;
    unsigned int x_stages = 4u;
    while (x_stages > 2u && x_stages * x_seg + 3u * kRawStageBytes > kMidRings) {
        --x_stages;
    }
    args.x_stages = x_stages;
    args.raw_offset = x_stages * x_seg;
    const unsigned int raw_stages = (kMidRings - args.raw_offset) / args.raw_stride;
    args.raw_stages = raw_stages < kMidMaxRaw ? raw_stages : kMidMaxRaw;
    if (tw_second != nullptr) {
        return y_dtype == 1 ? launch_mid_typed<__half, true>(stream, tw, *tw_second, tx, args, grid, cluster, overlap)
                            : cudaErrorInvalidValue;
    }
    switch (y_dtype) {
    case 0:
        return launch_mid_typed<float, false>(stream, tw, tw, tx, args, grid, cluster, overlap);
    case 1:
        return launch_mid_typed<__half, false>(stream, tw, tw, tx, args, grid, cluster, overlap);
    case 2:
        return launch_mid_typed<__nv_bfloat16, false>(stream, tw, tw, tx, args, grid, cluster, overlap);
    default:
        return cudaErrorInvalidValue;
    }
}

// How many clusters of four blocks run at once (clusters do not cross the boundaries of the GPU's
// processing clusters, so it is fewer than a quarter of the SMs); once per device.
static unsigned int clusters_of_four(unsigned int sm_count)
{
    static unsigned int known[64] = {};
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) {
        return sm_count / 5u;
    }
    if (known[device] == 0u) {
        static unsigned long long configured = 0ull;
        int found = 0;
        cudaLaunchConfig_t config = {};
        config.gridDim = dim3(4u * (sm_count / 4u), 1, 1);
        config.blockDim = dim3(kMidThreads, 1, 1);
        config.dynamicSmemBytes = kMidSmem;
        cudaLaunchAttribute attribute[1];
        attribute[0].id = cudaLaunchAttributeClusterDimension;
        attribute[0].val.clusterDim.x = 4;
        attribute[0].val.clusterDim.y = 1;
        attribute[0].val.clusterDim.z = 1;
        config.attrs = attribute;
        config.numAttrs = 1;
        if (allow_shared_memory(q8_stream_kernel_mid<float, false>, kMidSmem, &configured) != cudaSuccess
            || cudaOccupancyMaxActiveClusters(&found, q8_stream_kernel_mid<float, false>, &config) != cudaSuccess || found <= 0) {
            found = (int)(sm_count / 5u);
        }
        known[device] = (unsigned int)found;
    }
    return known[device];
}

// How the sums of a product are kept exact.  An MMA truncates the sum it adds to, so the error grows with the MMAs that
// go into one accumulator one after the other.  The measure is the run of depth that a place for a block gets
// where all (128 rows, segment) units are dealt evenly: `m` above 32 rows one place per SM, up to 32 two places
// and two accumulators.  Blocks here get longer runs - all of a tile's depth, or a quarter or a half in a
// cluster - and make up for it by accumulators in turn, as far as they leave two segments of A (256 columns),
// or by runs.  4096 x 4096, 32 rows, 12.5e-7 of the result with one accumulator, 3.5e-7 so; 28672 x 4096, 32 rows,
// 48.6e-7 and 12.6e-7; 512 x 16384, 64 rows, 48.6e-7 and 3.5e-7.  It costs a third segment of A or a second buffer
// where those would fit, and the reads at the end: 28672 x 4096, 32 rows, 30.9 -> 31.8 us; 4096 x 14336, 100 rows,
// 26.1 -> 27.9; in runs 300 x 16384, 128 rows, 30 -> 58.
static void mid_accuracy(MidPlan &plan, unsigned int n, unsigned int segs, unsigned int sm_count)
{
    const unsigned int tiles = (n + kRows - 1u) / kRows;
    const unsigned int acc_columns = plan.pair * plan.ntok;
    plan.chains = 1u;
    plan.run_segs = 0u;
    if (plan.ntok <= 32u) {
        // (units dealt to as many places as here, or clusters of four where there were four blocks: two)
        plan.chains = plan.cluster == 4u && plan.pair == 2u ? 2u : 4u;
        if (plan.cluster == 1u && plan.turns == 0u) {
            plan.chains = 2u;
        }
        return;
    }
    if (plan.cluster > 1u) {
        // (two slabs to a cluster: it has no more depth than an even share)
        const unsigned int depth = (segs + plan.cluster - 1u) / plan.cluster;
        if (plan.pair == 1u && depth > 1u && depth * sm_count > tiles * segs) {
            if (depth * sm_count <= 2u * tiles * segs || depth == 2u) {
                plan.chains = 2u;
            } else {
                plan.chains = plan.ntok <= 48u ? 4u : plan.ntok <= 80u ? 2u : 1u;
                const unsigned int share = plan.chains * tiles * segs / sm_count;
                plan.run_segs = share > plan.chains ? share : plan.chains;
                const unsigned int least = segs / plan.cluster;        // 2 at least: the depth is above two
                plan.run_segs = plan.run_segs < least ? plan.run_segs : least - 1u;
            }
        }
        return;
    }
    // whole tiles in one or two turns: a third of them would be cut
    if ((plan.turns == 1u || plan.turns == 2u) && 2u * acc_columns <= 256u) {
        plan.chains = 2u;
    }
}

// Where the storing warps are free until the block's last sums are there they turn bfloat16 x into binary16 as it comes,
// and no launch has to do it before this one.  Four warps do 32 rows beside everything else (6144 x 4096 14.6 -> 13.6 us,
// 28672 x 4096 32.2 -> 30.0; 13.2 with binary16 x); 64 rows where a segment of x meets two whole slabs (28672 x 4096
// 34.8 -> 33.4), not in a cluster (4096 x 14336 22.0 -> 23.3); 100 rows take longer than the launch did (27.8 -> 32.3).
bool mid_converts_x(const MidPlan &plan)
{
    return (plan.cluster > 1u ? plan.ntok <= 32u : plan.turns == 1u && plan.ntok <= 64u) && plan.run_segs == 0u;
}

MidPlan mid_plan(unsigned int n, unsigned int k, unsigned int m, unsigned int sm_count, unsigned long long tile_floats,
                 unsigned int epilogue)
{
    MidPlan plan = {};
    plan.ntok = (m + 15u) / 16u * 16u;
    const unsigned int segs = k / kSegK;
    const unsigned int step = epilogue == kEpilogueSwiglu ? 8u : 4u;
    // Few rows: clusters of four or two, at most two slabs to a cluster, all of one size so that every
    // cluster has work.  (Cutting them into units instead leaves pieces of a few segments and as many
    // hand-overs through memory: 16384 x 4096, 100 rows, 28.9 us against 24.5.)
    for (unsigned int size = 4u; size >= 2u; size /= 2u) {
        const unsigned int clusters = size == 4u ? clusters_of_four(sm_count) : sm_count / 2u;
        if (segs < size || n > clusters * 2u * kRows) {
            continue;
        }
        plan.cluster = size;
        plan.pair = n > clusters * kRows ? 2u : 1u;
        const unsigned int all = clusters * plan.pair;
        plan.slab_rows = ((n + all - 1u) / all + step - 1u) / step * step;
        const unsigned int used = (n + plan.slab_rows - 1u) / plan.slab_rows;
        plan.tiles = (used + plan.pair - 1u) / plan.pair;
        plan.grid = plan.tiles * plan.cluster;
        mid_accuracy(plan, n, segs, sm_count);
        return plan;
    }
    plan.cluster = 1u;
    // (the fixed scratch of aotx_q8_matmul_static holds one slab)
    plan.pair = n > kRows && 2ull * kRows * plan.ntok <= tile_floats ? 2u : 1u;
    plan.slab_rows = kRows;
    plan.tiles = (n + plan.pair * kRows - 1u) / (plan.pair * kRows);
    const unsigned long long units = (unsigned long long)plan.tiles * segs;
    plan.grid = units < sm_count ? (unsigned int)units : sm_count;
    // Whole tiles, all of one size and as many to every block, unless cutting them is cheaper.
    const unsigned int turns = (plan.tiles + sm_count - 1u) / sm_count;
    if ((unsigned long long)turns * segs <= units / plan.grid + kMidCutUnits) {
        const unsigned int all = sm_count * turns * plan.pair;
        plan.turns = turns;
        plan.slab_rows = ((n + all - 1u) / all + step - 1u) / step * step;
        plan.tiles = (n + plan.pair * plan.slab_rows - 1u) / (plan.pair * plan.slab_rows);
        plan.grid = plan.tiles < sm_count ? plan.tiles : sm_count;
    }
    mid_accuracy(plan, n, segs, sm_count);
    return plan;
}

cudaError_t launch_mid_product(cudaStream_t stream, const CUtensorMap &tw, const CUtensorMap &tx, const MidPlan &plan,
                               unsigned int n, unsigned int k, unsigned int m, const unsigned int *m_dev, void *y, int y_dtype,
                               unsigned int ldy, unsigned int epilogue, float *partial, unsigned int *flags,
                               unsigned long long tile_floats, unsigned int *status, bool overlap, bool x_bf16)
{
    MidArgs args = {};
    args.x_bf16 = x_bf16 ? 1u : 0u;
    args.n = n;
    args.k = k;
    args.m_max = m;
    args.m_dev = m_dev;
    args.to.y = y;
    args.status = status;
    args.to.ldy = ldy;
    args.to.epilogue = epilogue;
    args.ntok = plan.ntok;
    args.slab_rows = plan.slab_rows;
    args.pair = plan.pair;
    args.tiles = plan.tiles;
    args.turns = plan.turns;
    args.chains = plan.chains;
    args.run_segs = plan.run_segs;
    args.partial = partial;
    args.flags = flags;
    args.tile_floats = tile_floats;
    return launch_mid(stream, tw, nullptr, tx, args, plan.grid, plan.cluster, overlap, y_dtype);
}

cudaError_t launch_mid_grouped(cudaStream_t stream, const CUtensorMap &tw, const CUtensorMap *tw_second,
                               const CUtensorMap &tx, bool table_late, unsigned int grid, unsigned int k, unsigned int ntok, const GroupTile *tiles, const unsigned int *count_dev,
                               const unsigned int *row_map, void *y, unsigned int ldy, int y_dtype, unsigned int epilogue,
                               float *partial, unsigned int *flags, unsigned long long tile_floats, unsigned int *status,
                               bool overlap)
{
    MidArgs args = {};
    args.k = k;
    args.partial = partial;
    args.flags = flags;
    args.tile_floats = tile_floats;
    args.to.y = y;
    args.status = status;
    args.to.ldy = ldy;
    args.to.epilogue = epilogue;
    args.group_tiles = tiles;
    args.table_late = table_late ? 1u : 0u;
    args.group_count = count_dev;
    args.to.row_map = row_map;
    args.ntok = ntok;
    args.slab_rows = kRows;
    args.pair = 2u;
    args.chains = ntok <= 32u ? 2u : 1u;      // two buffers of them fit beside two segments of A
    return launch_mid(stream, tw, tw_second, tx, args, grid, 1u, overlap, y_dtype);
}

} // namespace q8
