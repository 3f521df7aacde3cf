// The Q8_0 product for one to four rows of x with a tensor of few rows:
// y[i][j] = sum_c x[i][c] * half(q[j][c] * d[j][c / 32]), float sums.
//
// Such a launch is bound by its start and end.  q8_decode_warp.cu cuts a tile's depth between the blocks of a cluster,
// whose exchange of sums takes a microsecond of the seven that 4096 x 4096 takes; here nothing is cut between blocks:
//
//   * A block takes a tile of up to 16 rows of w over their whole depth.  The tile's segments, 256 deep, are dealt to
//     the block's eight warps in runs, and their sums are added up in shared memory at the end.
//   * Each warp works alone until then: it has its own ring of raw segments with its own barriers, copies into it
//     itself, and brings the segment of x that it needs into its own shared memory.  Weights and x lie there as in
//     q8_decode_warp.cu and go the same way through mma.sync.
//   * Two blocks per SM; a launch has as many as that or fewer.
//
// Every block reads all of x, and every warp turns its part round by itself, so it pays for few rows of x only, and a
// warp's own copies and hand-overs cost instructions, so it pays where a launch is short (rows_height has both sides).
// 4096 x 4096, one row, 7.3 -> 5.6 us (weights in L2, from call to call 6.7 -> 4.6); four rows 7.3 -> 6.2.  At 28672 x 4096,
// several such tiles to a block took 29 us against 26, and eight rows of x 31 against 25.  Every wait is bounded and raises a
// status bit when it runs out.  Reference kernels replaced: as q8_decode_warp.cu.
#include <cuda.h>

#include "q8_decode_operands.cuh"
#include "q8_launch.h"
#include "q8_tile.cuh"

namespace q8 {

constexpr uint32_t kRowsWarps = 8;
constexpr uint32_t kRowsThreads = kRowsWarps * 32;
constexpr uint32_t kRowsTokens = 4;            // rows of x, at most
constexpr uint32_t kRowsMaxStages = 4;
// Shared memory of a block: two blocks per SM.  Not three: a launch's blocks then come to lie unevenly, three on some SMs
// and one on others (4096 x 4096, one row, 5.6 and 6.4 us).
constexpr uint32_t kRowsMost = 112u * 1024u;
constexpr uint32_t kRowsLeast = 77u * 1024u;
// The sums of a warp in shared memory: [row of x][row of w], the rows 4 words longer than they are so that the MMA's
// fragments are stored without bank conflicts.
constexpr uint32_t kRowsPitch = 20;
// Where the lines lie, between this kernel and q8_decode_warp.cu: tiles of fewer rows multiply repeats, and with more depth
// it is memory that counts.  Above 32 tiles of 128 rows the clusters of eight of q8_decode_warp.cu do not all run at once,
// and any depth is faster here.  That kernel's us and this one's, launches in a graph, weights from memory:
//   rows a tile       8            10           11           13           14           15           16
//   one row of x
//     2048 deep   3.9   3.1    4.2   3.2    4.4   3.2    4.9   3.3    5.5   3.3    7.1   3.4    7.4   3.5
//     4096 deep   5.3   4.8    5.7   5.2    5.9   5.4    6.4   5.8    6.9   5.6    9.4   6.2   10.5   6.4
//     5120 deep   6.3   6.4    6.9   7.0    7.1   7.3    7.8   7.8    8.1   7.6   12.1   8.3   12.3   8.5
//     8192 deep   8.0   8.6    8.5   9.6    8.8  10.1    9.7   9.8   10.0   9.8   15.0  10.8   15.5  11.2
//    14336 deep  13.1  12.6   13.5  13.5   13.7  14.1   14.3  13.9   14.6  14.1   22.4  14.8   23.2  15.5
//   four
//     2048 deep   4.0   3.4    4.3   3.5    4.4   3.6    4.9   3.8    5.4   3.8    7.2   3.9    7.6   3.9
//     4096 deep   5.4   5.4    5.8   5.7    6.1   5.9    6.5   6.1    6.9   6.2    9.6   6.4   10.8   6.6
//     5120 deep   6.5   7.0    7.0   7.6    7.3   7.8    8.0   8.3    8.3   8.3   12.2   7.9   12.4   8.0
//     8192 deep   8.2   9.6    8.6  10.6    8.9  10.3    9.8  11.0   10.1  11.0   15.0  10.3   15.5  10.5
//    14336 deep  13.0  14.3   13.7  15.1   13.9  14.8   14.5  15.7   14.8  15.7   22.4  15.2   23.4  15.4
// (In the column of 14 rows the tensor has 4096.)  The lines are on the safe side: this kernel is no slower from 8 rows a tile
// on up to 4096 deep, nor at 1024 deep (8 rows a tile, one row of x, 3.1 and 2.4; 16, 3.6 and 2.6).
constexpr uint32_t kRowsHeight = 11;
constexpr uint32_t kRowsDepth = 4096;
constexpr uint32_t kRowsChains = 4;            // accumulators of a value (q8_decode_warp.cu says why)
constexpr uint32_t kRowsBarBytes = kRowsWarps * kRowsMaxStages * 8 + 16;

struct RowsArgs {
    unsigned int n, k, m_max;
    const unsigned int *m_dev;
    void *y;
    unsigned int *status;
    unsigned int ldy, epilogue;
    unsigned int height;               // rows of w per tile, up to 16
    unsigned int stages, stage_bytes;  // of a warp's ring
    unsigned int x_bytes;              // of a warp's x, and of its sums at the tile's end
};

template <bool BF, typename YT>
__global__ void __launch_bounds__(kRowsThreads, 2)
q8_stream_kernel_rows(const __grid_constant__ CUtensorMap tmap_w, const void *x_any, const RowsArgs args)
{
    extern __shared__ unsigned char smem_raw_[];
    const uint32_t smem0 = (smem_u32(smem_raw_) + 127u) & ~127u;
    unsigned char *const smem = smem_raw_ + (smem0 - smem_u32(smem_raw_));
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t ring_bytes = args.stages * args.stage_bytes;
    const uint32_t ring = smem0 + warp * ring_bytes;
    const uint32_t x_offset = kRowsWarps * ring_bytes + warp * args.x_bytes;
    const uint32_t bars = smem0 + kRowsWarps * (ring_bytes + args.x_bytes);
    const uint32_t full = bars + warp * args.stages * 8u;
    volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(smem + (bars - smem0) + kRowsWarps * kRowsMaxStages * 8u);

    grid_launch_dependents();

    const uint32_t segs = args.k / kSegK;
    const uint32_t height = args.height;
    const uint32_t item_bytes = height * kSegBytes;
    const uint32_t begin = warp * segs / kRowsWarps;                // this warp's segments of the block's tile
    const uint32_t end = (warp + 1u) * segs / kRowsWarps;
    uint32_t ahead = begin;            // the next that it copies
    auto copy_next = [&](uint32_t st) {
        mbar_expect_tx(full + 8u * st, item_bytes);
        tma_load_2d(ring + st * args.stage_bytes, &tmap_w, full + 8u * st, (int)(ahead * kSegWords),
                    (int)(blockIdx.x * height));
    };
    if (threadIdx.x == 0u) {
        *abort_flag = 0u;
    }
    if (elect_one()) {
        tma_prefetch_desc(&tmap_w);
        for (uint32_t i = 0; i < args.stages; ++i) {
            mbar_init(full + 8u * i, 1u);
        }
        mbar_init_fence();
        fence_proxy_async_smem();
    }
    __syncwarp();
    for (uint32_t i = 0; i < args.stages && ahead < end; ++i, ++ahead) {
        if (elect_one()) {
            copy_next(i);
        }
    }
    __syncthreads();      // (the abort flag)

    const uint32_t g8 = lane >> 2;
    const uint32_t t4 = lane & 3u;
    const uint32_t turn = t4 == 3u ? 0x7610u : 0x3210u;     // lane 3's second word of an even block
    // rows past the tile, and rows of x past the batch, repeat the last one (their sums are not stored)
    const uint32_t row0 = (g8 < height ? g8 : height - 1u) * kSegBytes + 4u * t4;
    const uint32_t row1 = (g8 + 8u < height ? g8 + 8u : height - 1u) * kSegBytes + 4u * t4;
    const uint32_t m_max = args.m_max;
    unsigned char *const x_mine = smem + x_offset;
    const unsigned char *x_lane = x_mine + (g8 < m_max ? g8 : m_max - 1u) * kWarpXRow + 32u * t4;
    const uint4 *x = static_cast<const uint4 *>(x_any) + lane;
    const uint32_t row_chunks = args.k / 8u;
    uint4 next_x[kRowsTokens];
    auto fetch_x = [&](uint32_t s) {
#pragma unroll
        for (uint32_t r = 0; r < kRowsTokens; ++r) {
            next_x[r] = r < m_max ? __ldcg(x + (size_t)r * row_chunks + s * (kSegK / 8u)) : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    grid_dependency_wait();
    if (begin != end) {
        fetch_x(begin);
    }
    unsigned int m_live = m_max;
    if (args.m_dev != nullptr) {
        const unsigned int live = *args.m_dev;
        m_live = live < m_live ? live : m_live;
    }

    uint32_t st = 0u, ph = 0u, taken = begin;
    float acc[kRowsChains][4] = {};
#pragma unroll 1
    for (; taken < end; ++taken) {
        // this segment of x, and the next one on its way
        __syncwarp();
#pragma unroll
        for (uint32_t r = 0; r < kRowsTokens; ++r) {
            if (r < m_max) {
                stage_x_row<BF>(next_x[r], smem0 + x_offset + r * kWarpXRow, lane);
            }
        }
        __syncwarp();
        if (taken + 1u < end) {
            fetch_x(taken + 1u);
        }
        if (!__all_sync(0xFFFFFFFFu, mbar_wait_hot(full + 8u * st, ph, abort_flag, args.status))) {
            break;
        }
        const unsigned char *w0 = smem + (ring - smem0) + st * args.stage_bytes + row0;
        const unsigned char *w1 = smem + (ring - smem0) + st * args.stage_bytes + row1;
#pragma unroll
        for (uint32_t b = 0; b < kSegK / 32u; ++b) {
            uint32_t a[2][4];
            block_of_rows(w0, w1, t4, turn, b, a);
            const uint4 xv = *reinterpret_cast<const uint4 *>(x_lane + (b / 2u) * 128u + (b & 1u) * 16u);
            mma_16816(acc[2u * (b & 1u)], a[0], xv.x, xv.y);
            mma_16816(acc[2u * (b & 1u) + 1u], a[1], xv.z, xv.w);
        }
        // The stage goes back when the words of every lane have arrived: the vote needs sums that every load of the
        // segment went into (q8_decode_warp.cu).
        const uint32_t seen = __float_as_uint(acc[0][0]) ^ __float_as_uint(acc[0][3]) ^ __float_as_uint(acc[1][1]) ^ __float_as_uint(acc[1][2])
                            ^ __float_as_uint(acc[2][0]) ^ __float_as_uint(acc[2][3]) ^ __float_as_uint(acc[3][1]) ^ __float_as_uint(acc[3][2]);
        if (__any_sync(0xFFFFFFFFu, seen == 0x7FB1A5C3u)) {
            atomicOr(args.status, 0u);
        }
        if (ahead < end) {
            if (elect_one()) {
                copy_next(st);
            }
            ++ahead;
        }
        if (++st == args.stages) {
            st = 0u;
            ph ^= 1u;
        }
    }
    // ---------------------------------------------------------------- the tile's sums
    __syncwarp();
    float *sums = reinterpret_cast<float *>(x_mine);
#pragma unroll
    for (uint32_t i = 0; i < 4u; ++i) {
        const uint32_t token = 2u * t4 + (i & 1u);
        if (token < kRowsTokens) {
            sums[token * kRowsPitch + g8 + (i >> 1) * 8u] = (acc[0][i] + acc[1][i]) + (acc[2][i] + acc[3][i]);
        }
    }
    __syncthreads();
    // half a warp = the tile's rows of one row of x
    if (warp * 2u < m_max) {
        YT *y = static_cast<YT *>(args.y);
        const uint32_t token = warp * 2u + (lane >> 4);
        const uint32_t row = lane & 15u;
        const float *from = reinterpret_cast<const float *>(smem + kRowsWarps * ring_bytes) + token * kRowsPitch + row;
        float sum = from[0];
#pragma unroll
        for (uint32_t w = 1; w < kRowsWarps; ++w) {
            sum += from[w * (args.x_bytes / 4u)];
        }
        const uint32_t j = blockIdx.x * height + row;
        const size_t ldy = args.ldy;
        const bool inside = token < m_live && row < height && j < args.n;
        if (args.epilogue == kEpilogueSwiglu) {
            // gate and up rows of one column (the arithmetic of cuda/model/norm.cu:92-105)
            const float up = __shfl_xor_sync(0xFFFFFFFFu, sum, 1u);
            if (inside && (row & 1u) == 0u) {
                store_out<YT>(y, (size_t)token * ldy + (j >> 1), sum / (1.0f + expf(-sum)) * up);
            }
        } else if (inside) {
            if (args.epilogue == kEpilogueAdd) {
                float *to = static_cast<float *>(args.y) + (size_t)token * ldy + j;
                *to = *to + sum;
            } else {
                store_out<YT>(y, (size_t)token * ldy + j, sum);
            }
        }
    }
    // Let every copy of this warp land before the block ends (a warp that gave up has some on their way).
    uint32_t local_abort = 0;
    for (; taken < ahead; ++taken) {
        mbar_wait(full + 8u * st, ph, &local_abort, nullptr);
        if (++st == args.stages) {
            st = 0u;
            ph ^= 1u;
        }
    }
}

template <bool BF, typename YT>
static cudaError_t launch_rows_typed(cudaStream_t stream, const CUtensorMap &tw, const void *x, const RowsArgs &args, unsigned int grid,
                                     unsigned int smem_bytes, bool overlap)
{
    static unsigned long long configured = 0ull;
    cudaError_t err = allow_shared_memory(q8_stream_kernel_rows<BF, YT>, kRowsMost, &configured, true);
    if (err != cudaSuccess) {
        return err;
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(grid, 1, 1);
    config.blockDim = dim3(kRowsThreads, 1, 1);
    config.dynamicSmemBytes = smem_bytes;
    config.stream = stream;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attribute;
    config.numAttrs = overlap ? 1u : 0u;
    return cudaLaunchKernelEx(&config, q8_stream_kernel_rows<BF, YT>, tw, x, args);
}

template <bool BF>
static cudaError_t launch_rows_out(cudaStream_t stream, const CUtensorMap &tw, const void *x, const RowsArgs &args, unsigned int grid,
                                   unsigned int smem_bytes, bool overlap, int y_dtype)
{
    switch (y_dtype) {
    case 0:
        return launch_rows_typed<BF, float>(stream, tw, x, args, grid, smem_bytes, overlap);
    case 1:
        return launch_rows_typed<BF, __half>(stream, tw, x, args, grid, smem_bytes, overlap);
    case 2:
        return launch_rows_typed<BF, __nv_bfloat16>(stream, tw, x, args, grid, smem_bytes, overlap);
    default:
        return cudaErrorInvalidValue;
    }
}

// The tiles' height (0: not by this kernel): one tile to every place for a block, two per SM.
unsigned int rows_height(unsigned int n, unsigned int k, unsigned int m, unsigned int sm_count, unsigned int epilogue)
{
    const unsigned int step = epilogue == kEpilogueSwiglu ? 2u : 1u;
    const unsigned int height = ((n + 2u * sm_count - 1u) / (2u * sm_count) + step - 1u) / step * step;
    const unsigned int deepest = n > 32u * kRows ? 4u * kRowsDepth : kRowsDepth;
    return m <= kRowsTokens && height >= kRowsHeight && height <= 16u && k >= kRowsWarps * kSegK && k <= deepest ? height : 0u;
}

cudaError_t launch_decode_rows(cudaStream_t stream, const CUtensorMap &tw, const void *x, bool x_bf16, unsigned int height,
                               const UmmaArgs &from, int y_dtype)
{
    RowsArgs args = {};
    args.n = from.n;
    args.k = from.k;
    args.m_max = from.m_max;
    args.m_dev = from.m_dev;
    args.y = from.y;
    args.status = from.status;
    args.ldy = from.ldy;
    args.epilogue = from.epilogue;
    args.height = height;
    args.stage_bytes = (height * kSegBytes + 127u) / 128u * 128u;
    const unsigned int x_bytes = args.m_max * kWarpXRow;
    const unsigned int sum_bytes = kRowsTokens * kRowsPitch * 4u;
    args.x_bytes = x_bytes > sum_bytes ? x_bytes : sum_bytes;
    // as many stages as a warp has segments and as fit
    const unsigned int fixed = kRowsWarps * args.x_bytes + kRowsBarBytes + 128u;
    const unsigned int ring = kRowsWarps * args.stage_bytes;
    const unsigned int most = (args.k / kSegK + kRowsWarps - 1u) / kRowsWarps;
    unsigned int stages = (kRowsMost - fixed) / ring;
    stages = stages < kRowsMaxStages ? stages : kRowsMaxStages;
    args.stages = stages < most ? stages : most;
    const unsigned int grid = (args.n + height - 1u) / height;
    const unsigned int wanted = fixed + args.stages * ring;
    const unsigned int smem_bytes = wanted > kRowsLeast ? wanted : kRowsLeast;
    const bool overlap = from.overlap != 0u;
    return x_bf16 ? launch_rows_out<true>(stream, tw, x, args, grid, smem_bytes, overlap, y_dtype)
                  : launch_rows_out<false>(stream, tw, x, args, grid, smem_bytes, overlap, y_dtype);
}

} // namespace q8
