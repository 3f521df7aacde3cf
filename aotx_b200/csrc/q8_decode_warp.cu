// The decode-regime kernel of the Q8_0 product for batches of up to 16 rows of x:
// y[i][j] = sum_c x[i][c] * half(q[j][c] * d[j][c / 32]), float sums.
//
// HBM-bound: a launch moves n * (k / 32) * 34 bytes of weights once, and an SM has to turn about
// 21 weights per cycle into products to keep up with memory.  The weights therefore go from
// shared memory straight into the registers of the warp that multiplies them (mma.sync
// m16n8k16, 951 products per cycle and SM measured, 21 x 16 needed at 16 rows): one hand-over
// per segment (copy lands -> warps read) where a kernel on tensor memory has five, each a
// fraction of a microsecond long.
//
//   * Two blocks of 12 warps per SM.  Warps 0-7 multiply; warps 8-11 bring x in, and one lane of
//     warp 8 issues the bulk tensor copies of the weights: segments [128 rows x 272 B] into a
//     two-deep ring (2 blocks x 2 segments in flight read memory at 6.85 TB/s without any
//     arithmetic; one contiguous piece of 34 KB per copy reads 7.0).
//   * Rows of a segment lie 68 words apart in shared memory, 4 modulo the 32 banks, so the 8 rows
//     by 4 lanes of an MMA operand are read without conflicts when the lanes of a row take
//     neighbouring WORDS.  Two blocks of 32 weights are 17 words: w0 = d | q0 q1, w1..w7, w8 =
//     q30 q31 | d', w9..w16.  Lane t takes w(1+t) and w(5+t) of the even block - lane 3's second
//     word is w8's low half with w0's high half - and w(9+t), w(13+t) of the odd one.  The order
//     of the weights along k is then 2, 3, .. 31, 0, 1 in even blocks; x is laid out in the same
//     order, and the sum does not care.
//   * x (half, or bfloat16 turned into half once per block and segment) is stored so that a lane
//     reads its four words of a block's two MMA steps as 16 bytes: row stride 528 bytes, lane t
//     of a pair of blocks at 32 t.
//   * A warp takes 16 rows of w over the whole segment.  (At 32 rows of x, warps of 32 rows over half a segment
//     each, this kernel is bound by its instructions: q8_mid.cu is as fast there and needs no second form.)
//   * Schedule as in q8_decode.cu: few row tiles run as a cluster per tile, each block one run of
//     its segments, pieces added through distributed shared memory in block order; larger
//     tensors run (tile, segment) units dealt evenly, the first holder of a cut tile owns it.
//
// Against the kernel on tensor memory that these batches ran on before (q8_decode.cu): 4096 x 4096, one row,
// 7.9 -> 6.5 us in a graph; the four products of a layer of 4096 by 14336, 8 rows, 95 -> 60 us; 151936 x 8192,
// 8 rows, 328 -> 246 us (5.4 TB/s with a cold L2 full of changed lines, 6.3 without).  What is left of a
// small product is its start and end: the first copy's latency, the exchange in the cluster.
//
// Every wait is bounded and raises a status bit when it runs out.  Reference kernels replaced:
// ptx/gemv_q8.ptx:18-223, cuda/model/gemv.cuh:33-145 (and the three-node switch of
// cuda/model/graph_host.cu:31-39 for these batches).
#include <cuda.h>

#include "q8_decode_operands.cuh"
#include "q8_launch.h"
#include "q8_tile.cuh"
#include "q8_warp_ptx.cuh"

namespace q8 {

constexpr uint32_t kWarpThreads = 384;
constexpr uint32_t kWarpCompute = 8;       // multiplying warps
constexpr uint32_t kWarpLoaders = 4;       // warps that bring x in

template <int NTOK>
struct WarpShape {
    static constexpr uint32_t tiles = NTOK / 8;                   // MMA columns of 8 rows of x
    // Sums that successive steps take in turn.  An MMA truncates the sum it adds to, so the error of a product
    // grows with the steps that go into one sum: 4096 x 4096, one row, 3.5e-7 of the result with two sums,
    // 2.0e-7 with four; 28672 x 4096, 8 rows, 15.3e-7 and 7.9e-7; the time is the same within 1.4 %.
    static constexpr uint32_t chains = 4;
    static constexpr uint32_t stages = 2;
    static constexpr uint32_t held = tiles * 4;                   // finished sums per thread
    static constexpr uint32_t x_stage_bytes = NTOK * kWarpXRow;
    static constexpr uint32_t raw_offset = 0;
    static constexpr uint32_t x_offset = stages * kRawStageBytes;
    // what the blocks of a cluster send: a tile of floats, beside the rings, so that a block may receive
    // while it still multiplies
    static constexpr uint32_t recv_bytes = kRows * NTOK * 4;
    static constexpr uint32_t recv_offset = x_offset + stages * x_stage_bytes;
    static constexpr uint32_t bar_offset = recv_offset + recv_bytes;
    static constexpr uint32_t bar_count = 3 * stages + 1;
    static constexpr uint32_t smem_bytes = bar_offset + bar_count * 8 + 16 + 1024;
    static_assert(2u * (smem_bytes + 1024u) <= 228u * 1024u, "two blocks' shared memory on one SM");
};

// Finished sums: value `i` of a thread belongs to row row_of(i) of the tile and row token_of(i) of x.
static __device__ __forceinline__ uint32_t row_of(uint32_t i, uint32_t warp, uint32_t g)
{
    return warp * 16u + g + ((i >> 1) & 1u) * 8u;
}

static __device__ __forceinline__ uint32_t token_of(uint32_t i, uint32_t t)
{
    return i / 4u * 8u + 2u * t + (i & 1u);
}

// Store the sums of a tile that lie in fragment order (pairs of rows of x in d0, d1 and d2, d3).
template <int NTOK, typename YT>
__device__ __forceinline__ void store_fragments(const UmmaArgs &args, uint32_t tile, uint32_t m_live, uint32_t warp,
                                                uint32_t lane, float (&v)[WarpShape<NTOK>::held])
{
    using S = WarpShape<NTOK>;
    const uint32_t g = lane >> 2;
    const uint32_t t = lane & 3u;
    const uint32_t n = args.n;
    const size_t ldy = args.ldy;
    YT *y = static_cast<YT *>(args.y);
    const bool odd = (g & 1u) != 0u;
    if (args.epilogue == kEpilogueSwiglu || (sizeof(YT) == 2 && args.epilogue == kEpilogueStore && (ldy & 1u) == 0u
                                             && (reinterpret_cast<uintptr_t>(y) & 3u) == 0u)) {
        // rows g and g ^ 1 of w meet: the even lane takes the first of the two rows of x, the odd
        // lane the second, each with both rows of w
#pragma unroll
        for (uint32_t i = 0; i < S::held; i += 2u) {
            const float give = odd ? v[i] : v[i + 1u];
            const float keep = odd ? v[i + 1u] : v[i];
            const float got = __shfl_xor_sync(0xFFFFFFFFu, give, 4u);
            const float low = odd ? got : keep;
            const float high = odd ? keep : got;
            const uint32_t token = token_of(i, t) + (odd ? 1u : 0u);
            const uint32_t row = tile * kRows + (row_of(i, warp, g) & ~1u);
            if (token < m_live && row < n) {
                if (args.epilogue == kEpilogueSwiglu) {
                    // gate and up rows of one column (the arithmetic of cuda/model/norm.cu:92-105)
                    store_out<YT>(y, (size_t)token * ldy + (row >> 1), low / (1.0f + expf(-low)) * high);
                } else if (row + 1u < n) {
                    *reinterpret_cast<uint32_t *>(y + (size_t)token * ldy + row) =
                        out_bits<YT>(low) | (out_bits<YT>(high) << 16);
                } else {
                    store_out<YT>(y, (size_t)token * ldy + row, low);
                }
            }
        }
        return;
    }
    if (args.epilogue == kEpilogueAdd) {
        // y is the float residual stream: one rounded add per value (cuda/model/norm.cu:78-89), the
        // old values fetched together
        float *sums = static_cast<float *>(args.y);
        float before[S::held];
#pragma unroll
        for (uint32_t i = 0; i < S::held; ++i) {
            const uint32_t token = token_of(i, t);
            const uint32_t row = tile * kRows + row_of(i, warp, g);
            before[i] = token < m_live && row < n ? sums[(size_t)token * ldy + row] : 0.0f;
        }
#pragma unroll
        for (uint32_t i = 0; i < S::held; ++i) {
            const uint32_t token = token_of(i, t);
            const uint32_t row = tile * kRows + row_of(i, warp, g);
            if (token < m_live && row < n) {
                sums[(size_t)token * ldy + row] = before[i] + v[i];
            }
        }
        return;
    }
#pragma unroll
    for (uint32_t i = 0; i < S::held; ++i) {
        const uint32_t token = token_of(i, t);
        const uint32_t row = tile * kRows + row_of(i, warp, g);
        if (token < m_live && row < n) {
            store_out<YT>(y, (size_t)token * ldy + row, v[i]);
        }
    }
}

template <int NTOK, bool BF, typename YT>
__global__ void __launch_bounds__(kWarpThreads, 2)
q8_decode_kernel_warp(const __grid_constant__ CUtensorMap tmap_w, const void *x_any, const UmmaArgs args)
{
    using S = WarpShape<NTOK>;
    extern __shared__ unsigned char smem_raw_[];
    const uint32_t smem0 = (smem_u32(smem_raw_) + 1023u) & ~1023u;
    unsigned char *const smem = smem_raw_ + (smem0 - smem_u32(smem_raw_));
    const uint32_t raw_base = smem0 + S::raw_offset;
    const uint32_t x_base = smem0 + S::x_offset;
    const uint32_t raw_full = smem0 + S::bar_offset;
    const uint32_t x_full = raw_full + 8u * S::stages;
    const uint32_t empty = x_full + 8u * S::stages;
    const uint32_t received = empty + 8u * S::stages;     // the pieces of this block's sums are here
    volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(smem + S::bar_offset + 8u * S::bar_count);

    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31u;

    grid_launch_dependents();

    const uint32_t segs = args.k / kSegK;
    const uint32_t row_tiles = (args.n + kRows - 1u) / kRows;
    const uint32_t units = row_tiles * segs; // the host refuses products with 2^31 units or more
    const bool split = args.split != 0u;
    uint32_t crank = 0u;
    uint32_t csize = 1u;
    uint32_t blocks = gridDim.x;
    uint32_t u_begin, u_end;
    if (split) {
        // one tile per cluster, one run of its segments per block
        csize = cluster_nctarank();
        crank = cluster_ctarank();
        const uint32_t tile = blockIdx.x / csize;
        u_begin = tile * segs + crank * segs / csize;
        u_end = tile * segs + (crank + 1u) * segs / csize;
    } else {
        blocks = units < gridDim.x ? units : gridDim.x;
        if (blockIdx.x >= blocks) {
            return;
        }
        decode_range(blockIdx.x, blocks, units, &u_begin, &u_end);
    }
    const uint32_t tile_begin = u_begin / segs;
    const uint32_t seg_begin = u_begin - tile_begin * segs;
    const uint32_t total = u_end - u_begin;

    if (threadIdx.x == kWarpCompute * 32u) {
        tma_prefetch_desc(&tmap_w);
        for (uint32_t i = 0; i < S::stages; ++i) {
            mbar_init(raw_full + 8u * i, 1u);
            mbar_init(x_full + 8u * i, kWarpLoaders);
            mbar_init(empty + 8u * i, kWarpCompute);
        }
        mbar_init(received, 1u);
        *abort_flag = 0u;
        mbar_init_fence();
        fence_proxy_async_smem();
        if (split) {
            mbar_expect_tx(received, S::recv_bytes);
        }
        // the first segments of weights: nothing but the barriers they signal is needed for them
        uint32_t tile = tile_begin;
        uint32_t s = seg_begin;
        for (uint32_t i = 0; i < S::stages && i < total; ++i) {
            mbar_expect_tx(raw_full + 8u * i, kRawStageBytes);
            tma_load_2d(raw_base + i * kRawStageBytes, &tmap_w, raw_full + 8u * i, (int)(s * kSegWords),
                        (int)(tile * kRows));
            if (++s == segs) {
                s = 0u;
                ++tile;
            }
        }
    }
    if (split) {
        // every block of the cluster has started (its shared memory may be written) before the exchange
        __syncwarp();
        cluster_arrive_relaxed();
    }
    __syncthreads();

    unsigned int m_live = 0u;
    bool ok = true;
    float acc[S::chains][S::tiles][4];

    if (warp >= kWarpCompute) {
        // ---------------------------------------------------------------- x, and the weight copies
        const uint32_t loader = warp - kWarpCompute;
        constexpr uint32_t kRowsEach = NTOK / kWarpLoaders;
        const uint4 *x = static_cast<const uint4 *>(x_any) + lane;
        const uint32_t row_chunks = args.k / 8u;
        const bool issuer = loader == 0u && lane == 0u;
        // the next segment that this lane copies, two ahead of the segment of x it stores
        uint32_t w_tile = tile_begin;
        uint32_t w_seg = seg_begin + S::stages;
        while (w_seg >= segs) {
            w_seg -= segs;
            ++w_tile;
        }
        uint4 v[kRowsEach];
        uint32_t seg = seg_begin;
        grid_dependency_wait();
        auto fetch = [&](uint32_t s) {
#pragma unroll
            for (uint32_t i = 0; i < kRowsEach; ++i) {
                const uint32_t r = loader + kWarpLoaders * i;
                v[i] = r < args.m_max ? __ldcg(x + (size_t)r * row_chunks + s * (kSegK / 8u)) : make_uint4(0u, 0u, 0u, 0u);
            }
        };
        fetch(seg);
        uint32_t issued = S::stages < total ? S::stages : total;
        for (uint32_t g = 0; g < total; ++g) {
            const uint32_t st = g % S::stages;
            const uint32_t ph = (g / S::stages) & 1u;
            if (!__all_sync(0xFFFFFFFFu, mbar_wait_hot(empty + 8u * st, ph ^ 1u, abort_flag, args.status))) {
                break;
            }
            if (g >= S::stages) {
                if (issuer) {
                    mbar_expect_tx(raw_full + 8u * st, kRawStageBytes);
                    tma_load_2d(raw_base + st * kRawStageBytes, &tmap_w, raw_full + 8u * st, (int)(w_seg * kSegWords),
                                (int)(w_tile * kRows));
                }
                issued = g + 1u;
                if (++w_seg == segs) {
                    w_seg = 0u;
                    ++w_tile;
                }
            }
#pragma unroll
            for (uint32_t i = 0; i < kRowsEach; ++i) {
                stage_x_row<BF>(v[i], x_base + st * S::x_stage_bytes + (loader + kWarpLoaders * i) * kWarpXRow, lane);
            }
            __syncwarp();
            if (lane == 0u) {
                mbar_arrive(x_full + 8u * st);
            }
            if (++seg == segs) {
                seg = 0u;
            }
            if (g + 1u < total) {
                fetch(seg);
            }
        }
        if (issuer) {
            // Let every copy this thread started land before the block ends.
            uint32_t local_abort = 0;
            const uint32_t first = issued > S::stages ? issued - S::stages : 0u;
            for (uint32_t i = first; i < issued; ++i) {
                mbar_wait(raw_full + 8u * (i % S::stages), (i / S::stages) & 1u, &local_abort, nullptr);
            }
        }
    } else {
        // ---------------------------------------------------------------- multiply, store
        const uint32_t g8 = lane >> 2;
        const uint32_t t = lane & 3u;
        const uint32_t turn = t == 3u ? 0x7610u : 0x3210u;     // lane 3's second word of an even block
        // this lane's first row and first pair of blocks, and its x
        const unsigned char *w_lane = smem + S::raw_offset + (warp * 16u + g8) * kSegBytes + 4u * t;
        const unsigned char *x_lane = smem + S::x_offset + g8 * kWarpXRow + 32u * t;
        uint32_t g = 0;
        uint32_t tile = tile_begin;
        uint32_t s0 = seg_begin;
        bool first_piece = true;
        for (uint32_t u = u_begin; ok && u < u_end;) {
            const uint32_t left = u_end - u;
            const uint32_t s1 = (segs - s0) < left ? segs : s0 + left;
#pragma unroll
            for (uint32_t c = 0; c < S::chains; ++c) {
#pragma unroll
                for (uint32_t j = 0; j < S::tiles; ++j) {
#pragma unroll
                    for (uint32_t i = 0; i < 4u; ++i) {
                        acc[c][j][i] = 0.0f;
                    }
                }
            }
#pragma unroll 1
            for (uint32_t s = s0; s < s1; ++s, ++g) {
                const uint32_t st = g % S::stages;
                const uint32_t ph = (g / S::stages) & 1u;
                ok = mbar_wait_hot(raw_full + 8u * st, ph, abort_flag, args.status)
                  && mbar_wait_hot(x_full + 8u * st, ph, abort_flag, args.status);
                ok = __all_sync(0xFFFFFFFFu, ok) != 0;
                if (!ok) {
                    break;
                }
                const unsigned char *w_at = w_lane + st * kRawStageBytes;
                const unsigned char *x_at = x_lane + st * S::x_stage_bytes;
#pragma unroll
                for (uint32_t b = 0; b < kSegK / 32u; ++b) {
                    uint32_t a[2][4];
                    block_of_rows(w_at, w_at + 8u * kSegBytes, t, turn, b, a);
                    // one step of all columns before the next: an MMA that adds to the sums of the one
                    // before it waits for them, about four MMAs' time
                    uint4 xv[S::tiles];
#pragma unroll
                    for (uint32_t j = 0; j < S::tiles; ++j) {
                        xv[j] = *reinterpret_cast<const uint4 *>(x_at + j * 8u * kWarpXRow + (b / 2u) * 128u + (b & 1u) * 16u);
                    }
#pragma unroll
                    for (uint32_t j = 0; j < S::tiles; ++j) {
                        mma_16816(acc[2u * (b & 1u)][j], a[0], xv[j].x, xv[j].y);
                    }
#pragma unroll
                    for (uint32_t j = 0; j < S::tiles; ++j) {
                        mma_16816(acc[2u * (b & 1u) + 1u][j], a[1], xv[j].z, xv[j].w);
                    }
                }
                // The stage goes back when the words of every lane have arrived, not only been asked
                // for (the next copy overwrites it): the vote needs sums that every load of the
                // segment went into.  It is true about once in 2^32 segments, and then does nothing.
                uint32_t seen = __float_as_uint(acc[2][0][0]) ^ __float_as_uint(acc[3][0][2]);
#pragma unroll
                for (uint32_t j = 0; j < S::tiles; ++j) {
                    seen ^= __float_as_uint(acc[3][j][1]) ^ __float_as_uint(acc[0][j][3]) ^ __float_as_uint(acc[1][j][3]);
                }
                if (__any_sync(0xFFFFFFFFu, seen == 0x7FB1A5C3u)) {
                    atomicOr(args.status, 0u);
                }
                if (lane == 0u) {
                    mbar_arrive(empty + 8u * st);
                }
            }
            if (!ok) {
                break;
            }
            float v[S::held];
#pragma unroll
            for (uint32_t i = 0; i < S::held; ++i) {
                v[i] = (acc[0][i / 4u][i % 4u] + acc[1][i / 4u][i % 4u]) + (acc[2][i / 4u][i % 4u] + acc[3][i / 4u][i % 4u]);
            }
            if (first_piece) {
                first_piece = false;
                grid_dependency_wait();
                m_live = args.m_max;
                if (args.m_dev != nullptr) {
                    const unsigned int live = *args.m_dev;
                    m_live = live < m_live ? live : m_live;
                }
            }
            if (split) {
#pragma unroll
                for (uint32_t i = 0; i < S::held; ++i) {
                    acc[0][i / 4u][i % 4u] = v[i];
                }
                break;
            }
            const bool owner = s0 == 0u;
            const bool whole = owner && s1 == segs;
            const uint32_t thread = warp * 32u + lane;
            if (!owner) {
                // publish this warp's part of the partial tile for the block that owns it
                float *slot = args.partial + (unsigned long long)blockIdx.x * args.tile_floats + thread;
#pragma unroll
                for (uint32_t i = 0; i < S::held; ++i) {
                    __stcg(slot + i * 256u, v[i]);
                }
                __threadfence();
                __syncwarp();
                if (lane == 0u) {
                    st_release_gpu(args.flags + 8u * blockIdx.x + warp, 1u);
                }
            } else {
                if (!whole) {
                    // The other holders of this tile are the blocks right after this one; they met
                    // it at the start of their ranges.
                    const unsigned int last_cc = decode_holder((tile + 1u) * segs - 1u, blocks, units);
                    for (unsigned int base = blockIdx.x + 1u; base <= last_cc; base += 32u) {
                        const unsigned int cc = base + lane;
                        if (cc <= last_cc) {
                            const unsigned int *flag = args.flags + 8u * cc + warp;
                            const long long begin = clock64();
                            while (ld_acquire_gpu(flag) == 0u) {
                                if (clock64() - begin > Q8_WAIT_CYCLES || *abort_flag != 0u) {
                                    atomicOr(args.status, Q8_DEV_FLAG_TIMEOUT);
                                    break;
                                }
                            }
                        }
                    }
                    __syncwarp();
#pragma unroll 1
                    for (unsigned int cc = blockIdx.x + 1u; cc <= last_cc; ++cc) {
                        const float *slot = args.partial + (unsigned long long)cc * args.tile_floats + thread;
                        float part[S::held];
#pragma unroll
                        for (uint32_t i = 0; i < S::held; ++i) {
                            part[i] = __ldcg(slot + i * 256u);
                        }
#pragma unroll
                        for (uint32_t i = 0; i < S::held; ++i) {
                            v[i] += part[i];
                        }
                    }
                    // hand the consumed slots back for the next launch that uses this set (ordered
                    // by the end of the kernel)
                    for (unsigned int base = blockIdx.x + 1u; base <= last_cc; base += 32u) {
                        const unsigned int cc = base + lane;
                        if (cc <= last_cc) {
                            *reinterpret_cast<volatile unsigned int *>(args.flags + 8u * cc + warp) = 0u;
                        }
                    }
                }
                store_fragments<NTOK, YT>(args, tile, m_live, warp, lane, v);
            }
            u += s1 - s0;
            s0 = 0u;
            ++tile;
        }
    }
    if (!split) {
        return;
    }

    // ------------------------------------------------------------ sum of a cluster's pieces
    // The rows of x are dealt to the blocks of the cluster in runs of `share`; every block writes
    // its piece's sums into their owners' shared memory, [sender][row of x][row of w], and the
    // owner adds the pieces in block order and stores.
    __syncwarp();
    cluster_wait_acquire();
    const uint32_t share = (uint32_t)NTOK / csize;   // 1 to 16: the cluster size is a power of two up to 8
    if (warp < kWarpCompute) {
        const uint32_t g8 = lane >> 2;
        const uint32_t t = lane & 3u;
#pragma unroll
        for (uint32_t i = 0; i < S::held; ++i) {
            const uint32_t token = token_of(i, t);
            const uint32_t row = row_of(i, warp, g8);
            const uint32_t at = smem0 + S::recv_offset + ((crank * share + token % share) * kRows + row) * 4u;
            store_counted(mapa_shared(at, token / share), acc[0][i / 4u][i % 4u], mapa_shared(received, token / share));
        }
        // The stores count themselves on their owner's barrier, which is all it waits for.  (A barrier of the cluster with
        // release and acquire in its place: 4096 x 4096, 8 rows, 6.95 us against 6.62, 4096 x 14336 14.9 and 14.4, 2560 x
        // 9728, 12 rows, 11.9 and 11.3.)
        if (!__all_sync(0xFFFFFFFFu, mbar_wait_counted(received, 0u, abort_flag, args.status))) {
            // Pieces are missing, and may still be on their way into this block's shared memory: it stays until every
            // other thread of the cluster has ended or come here.
            cluster_arrive_relaxed();
            cluster_wait_acquire();
            return;
        }
        // thread = row of w (two threads per row where a block owns several rows of x)
        const uint32_t row = threadIdx.x & (kRows - 1u);
        const uint32_t tile = blockIdx.x / csize;
        const uint32_t j = tile * kRows + row;
        const float *recv = reinterpret_cast<const float *>(smem + S::recv_offset) + row;
        YT *y = static_cast<YT *>(args.y);
        const size_t ldy = args.ldy;
        for (uint32_t local = threadIdx.x / kRows; local < share; local += 2u) {
            const uint32_t token = crank * share + local;
            float sum = recv[local * kRows];
            for (uint32_t src = 1; src < csize; ++src) {
                sum += recv[(src * share + local) * kRows];
            }
            if (args.epilogue == kEpilogueSwiglu) {
                const float up = __shfl_xor_sync(0xFFFFFFFFu, sum, 1u);
                sum = sum / (1.0f + expf(-sum)) * up;
            }
            if (token < m_live && j < args.n) {
                if (args.epilogue == kEpilogueSwiglu) {
                    if ((row & 1u) == 0u) {
                        store_out<YT>(y, (size_t)token * ldy + (j >> 1), sum);
                    }
                } else if (args.epilogue == kEpilogueAdd) {
                    float *at = static_cast<float *>(args.y) + (size_t)token * ldy + j;
                    *at = *at + sum;
                } else {
                    store_out<YT>(y, (size_t)token * ldy + j, sum);
                }
            }
        }
    }
}

template <int NTOK, bool BF, typename YT>
static cudaError_t launch_warp_typed(cudaStream_t stream, const CUtensorMap &tw, const void *x, const UmmaArgs &args,
                                     unsigned int grid, unsigned int cluster)
{
    using S = WarpShape<NTOK>;
    static unsigned long long configured = 0ull;
    cudaError_t err = allow_shared_memory(q8_decode_kernel_warp<NTOK, BF, YT>, S::smem_bytes, &configured, true);
    if (err != cudaSuccess) {
        return err;
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(grid, 1, 1);
    config.blockDim = dim3(kWarpThreads, 1, 1);
    config.dynamicSmemBytes = S::smem_bytes;
    config.stream = stream;
    cudaLaunchAttribute attribute[2];
    unsigned int count = 0;
    if (args.overlap != 0u) {
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
    return cudaLaunchKernelEx(&config, q8_decode_kernel_warp<NTOK, BF, YT>, tw, x, args);
}

template <int NTOK, bool BF>
static cudaError_t launch_warp_out(cudaStream_t stream, const CUtensorMap &tw, const void *x, const UmmaArgs &args,
                                   unsigned int grid, unsigned int cluster, int y_dtype)
{
    switch (y_dtype) {
    case 0:
        return launch_warp_typed<NTOK, BF, float>(stream, tw, x, args, grid, cluster);
    case 1:
        return launch_warp_typed<NTOK, BF, __half>(stream, tw, x, args, grid, cluster);
    case 2:
        return launch_warp_typed<NTOK, BF, __nv_bfloat16>(stream, tw, x, args, grid, cluster);
    default:
        return cudaErrorInvalidValue;
    }
}

template <int NTOK>
static cudaError_t launch_warp_tile(cudaStream_t stream, const CUtensorMap &tw, const void *x, const UmmaArgs &args,
                                    unsigned int grid, unsigned int cluster, int y_dtype)
{
    return args.b_bf16 != 0u ? launch_warp_out<NTOK, true>(stream, tw, x, args, grid, cluster, y_dtype)
                             : launch_warp_out<NTOK, false>(stream, tw, x, args, grid, cluster, y_dtype);
}

cudaError_t launch_decode_warp(cudaStream_t stream, const CUtensorMap &tw, const void *x, const UmmaArgs &args,
                               unsigned int grid, unsigned int cluster, int y_dtype)
{
    if (args.m_max <= 8u) {
        return launch_warp_tile<8>(stream, tw, x, args, grid, cluster, y_dtype);
    }
    return launch_warp_tile<16>(stream, tw, x, args, grid, cluster, y_dtype);
}

} // namespace q8
