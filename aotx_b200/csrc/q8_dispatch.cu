// Host side of the tensor-core products: which kernel serves a product, its tensor maps, its
// grid and its scratch.
//
//   rows of x     kernel                                                          file
//   1 .. 4        whole rows of w per block, where w has 11 to 16 rows to a block  q8_decode_rows.cu
//                 (148 SMs: 2961 to 4736) and is 2048 to 4096 deep, to 16384
//                 above 4096 rows
//   1 .. 16       weights through registers into mma.sync, two blocks per SM      q8_decode_warp.cu
//   17 .. 128     weights through tensor memory, one block per SM; also the       q8_mid.cu
//                 grouped products of the routed experts
//   129 ..        pairs of SMs, tiles of 256 rows of w by up to 256 of x; from    q8_pair.cu
//                 65 or 113 rows on where w has rows for every block
//
// Where the lines lie: at 17 rows mma.sync would need a third column of eight and is bound by its
// instructions at 32 (q8_decode_warp.cu); above 128 an accumulator of q8_mid.cu no longer fits
// beside two segments of A.  Products stored into several GPUs' copies of y, bfloat16 x without room for
// its binary16 copy, and the host emulation run on the kernels these replaced (q8_decode.cu up to 32 rows,
// q8_stream.cu up to 128, q8_wide.cu above).
//
// Shapes none of them takes (k not a multiple of 256, unaligned pointers) return
// cudaErrorNotSupported and the caller uses the general kernel (q8_simt.cu).  Reference: the
// regime switch of cuda/model/graph_host.cu:20-40 and cuda/model/product.cu:24-49, which this
// replaces with one launch per product.
#include <cuda.h>

#include "q8_launch.h"
#include "q8_tile.cuh"

namespace q8 {

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled()
{
#ifdef Q8_HOST_EMULATION
    return q8emu::encode_tiled; // the tests' stand-in: keeps the map's description for its copies
#endif
    static EncodeTiledFn fn = nullptr;
    if (fn == nullptr) {
        void *sym = nullptr;
        cudaDriverEntryPointQueryResult result;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &result) == cudaSuccess
            && result == cudaDriverEntryPointSuccess) {
            fn = reinterpret_cast<EncodeTiledFn>(sym);
        }
    }
    return fn;
}

unsigned int umma_token_tile(unsigned int m)
{
    if (m <= 16u) {
        return 16u;
    }
    if (m <= 32u) {
        return 32u;
    }
    if (m <= 64u) {
        return 64u;
    }
    // Batches above 128 rows run on the 256-row kernel with the weights in tensor memory
    // (q8_wide.cu), one token tile of 256 rows at a time.
    if (m > 128u) {
        return 256u;
    }
    return 128u;
}

// x as binary16, 16 bytes a step (the conversion the kernels apply to an x tile in shared
// memory: exact between 2^-14 and 65504, saturating above).  No __restrict__ on x, here and in every kernel that
// starts before the launch before it has ended: a read-only load wants data that does not change while
// the kernel lives, and the wait below does not hold it back.
__global__ void q8_x_to_f16_kernel(const uint4 *x, unsigned long long chunks, uint4 *out)
{
    grid_launch_dependents();   // the product this is part of: nothing is written here that it reads before its own wait
    grid_dependency_wait();     // x, and the products that still read the copy
    for (unsigned long long at = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; at < chunks;
         at += (unsigned long long)gridDim.x * blockDim.x) {
        uint4 v = x[at];
        v.x = bf16x2_to_f16x2(v.x);
        v.y = bf16x2_to_f16x2(v.y);
        v.z = bf16x2_to_f16x2(v.z);
        v.w = bf16x2_to_f16x2(v.w);
        out[at] = v;
    }
}

bool umma_supports(const void *w, unsigned int n, unsigned int k, const void *x, unsigned int m)
{
    if (n == 0u || m == 0u || k == 0u || (k % kSegK) != 0u) {
        return false;
    }
    if ((reinterpret_cast<uintptr_t>(w) & 15u) != 0u || (reinterpret_cast<uintptr_t>(x) & 15u) != 0u) {
        return false;
    }
    return true;
}

// The tensor map of a weight tensor's rows (boxes of box_rows rows by one segment) and of rows of x
// (boxes of box_rows rows by 64 values, 128-byte swizzle).
static bool map_weights(EncodeTiledFn encode, CUtensorMap *map, const void *w, unsigned int rows, unsigned int k,
                        unsigned int box_rows)
{
    const cuuint64_t row_b = row_bytes(k);
    const cuuint64_t dims[2] = {row_b / 4ull, rows};
    const cuuint64_t strides[1] = {row_b};
    const cuuint32_t box[2] = {kSegWords, box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void *>(w), dims, strides, box, elem,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
        == CUDA_SUCCESS;
}

static bool map_rows(EncodeTiledFn encode, CUtensorMap *map, const void *x, unsigned int rows, unsigned int k,
                     unsigned int box_rows, bool bf16)
{
    const cuuint64_t dims[2] = {k, rows};
    const cuuint64_t strides[1] = {(cuuint64_t)k * 2ull};
    const cuuint32_t box[2] = {kSubK, box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return encode(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(x),
                  dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
        == CUDA_SUCCESS;
}

// Two sets of slots and flags alternate between launches, so that a launch whose blocks start early
// never meets the slots of the launch before it.
static float *set_partial(const UmmaScratch &scratch, unsigned int set)
{
    return scratch.partial + (unsigned long long)(set & 1u) * scratch.blocks * scratch.tile_floats;
}

static unsigned int *set_flags(const UmmaScratch &scratch, unsigned int set)
{
    return scratch.flags + (unsigned long long)(set & 1u) * scratch.blocks * kFlagWords;
}

cudaError_t launch_umma(cudaStream_t stream, const UmmaScratch &scratch, unsigned int sm_count,
                        const void *w, unsigned int n, unsigned int k, const void *x, int x_bf16,
                        unsigned int m, const unsigned int *m_dev, void *y, int y_dtype, unsigned int set,
                        bool overlap, const PeerOut *out, unsigned int epilogue)
{
    if (!umma_supports(w, n, k, x, m)) {
        return cudaErrorNotSupported;
    }
    EncodeTiledFn encode = encode_tiled();
    if (encode == nullptr) {
        return cudaErrorNotSupported;
    }
    const unsigned int ntok = umma_token_tile(m);
    // bfloat16 activations at 17 to 128 rows become binary16: in the kernel as x comes (mid_converts_x), or by one pass
    // over x into the context's copy, 2.7 us between the launch before and the product.
    const bool copy_fits = scratch.x16 != nullptr && (unsigned long long)m * k * 2ull <= scratch.x16_bytes;
#ifdef Q8_HOST_EMULATION
    const bool mid = false;
#else
    // the kernel for 17 to 128 rows multiplies binary16 x
    const bool mid = ntok > 16u && ntok <= 128u && out == nullptr && (!x_bf16 || copy_fits)
                  && (unsigned long long)(n / kRows + 1u) * (k / kSegK) < (1ull << 31);
#endif
#ifdef Q8_HOST_EMULATION
    const bool warp_kernel = false; // cluster launches and warp-level MMA are not modelled
    const bool as_it_is = false;
#else
    // Up to 16 rows, one copy of y: the register-fed kernel; up to 128: q8_mid.cu.  Stores into the
    // peers' copies stay with the kernels they were measured on.
    const bool warp_kernel = ntok <= 16u && out == nullptr;
    // Above 112 rows q8_mid.cu has accumulators as wide as a pair's; with rows of w enough for every block a
    // pair of SMs, which reads half of x each, is then faster: 28672 x 4096, 128 rows, 42.0 -> 38.6 us,
    // 151936 x 8192 359 -> 341 (few rows of w: clusters, 24.1 against 26.1).  From 65 rows on where q8_mid.cu would
    // take whole tiles in one or two turns: a pair has room for a second accumulator per value, which such tiles
    // need (mid_accuracy), q8_mid.cu beside two slabs has not; 28672 x 4096, 100 rows, 36.8 us with one
    // accumulator in q8_mid.cu, 37.0 with two in a pair.
    MidPlan plan = {};
    if (mid) {
        plan = mid_plan(n, k, m, sm_count < scratch.blocks ? sm_count : scratch.blocks, scratch.tile_floats, epilogue);
    }
    const bool wide = ntok > 128u
                   || (mid && plan.cluster == 1u && (m > 112u || (m > 64u && (plan.turns == 1u || plan.turns == 2u))));
    const bool as_it_is = mid && !wide && mid_converts_x(plan);
#endif
    if (x_bf16 && !as_it_is && (mid || ntok >= 64u) && ntok <= 128u && copy_fits) {
        const unsigned long long chunks = (unsigned long long)m * k / 8ull;
        const unsigned int blocks = (unsigned int)((chunks + 255ull) / 256ull < 4ull * sm_count
                                                       ? (chunks + 255ull) / 256ull : 4ull * sm_count);
        cudaError_t turned = launch_kernel_early(overlap, q8_x_to_f16_kernel, blocks, 256, 0, stream,
                                           static_cast<const uint4 *>(x), chunks, static_cast<uint4 *>(scratch.x16));
        if (turned != cudaSuccess) {
            return turned;
        }
        x = scratch.x16;
        x_bf16 = 0;
    }
#ifndef Q8_HOST_EMULATION
    if (wide && out == nullptr && scratch.blocks >= 2u * sm_count && scratch.tile_floats >= 256ull * kRows
        && (unsigned long long)(n / (2u * kRows) + 1u) * (m / 128u + 1u) * (k / kSegK) < (1ull << 31)) {
        const unsigned int rows = pair_token_tile(m);
        CUtensorMap tw, tx;
        if (!map_weights(encode, &tw, w, n, k, kRows) || !map_rows(encode, &tx, x, m, k, rows / 2u, x_bf16 != 0)) {
            return cudaErrorInvalidValue;
        }
        return launch_pair_kernel(stream, tw, tx, rows, sm_count, n, k, x_bf16 != 0, m, m_dev, y, y_dtype,
                                  epilogue == kEpilogueSwiglu ? n / 2u : n, epilogue, set_partial(scratch, set),
                                  set_flags(scratch, set), scratch.tile_floats, scratch.status, overlap);
    }
    if (mid) {
        CUtensorMap tw, tx;
        if (!map_weights(encode, &tw, w, n, k, plan.slab_rows) || !map_rows(encode, &tx, x, m, k, plan.ntok, x_bf16 != 0)) {
            return cudaErrorInvalidValue;
        }
        return launch_mid_product(stream, tw, tx, plan, n, k, m, m_dev, y, y_dtype, epilogue == kEpilogueSwiglu ? n / 2u : n,
                                  epilogue, set_partial(scratch, set), set_flags(scratch, set), scratch.tile_floats,
                                  scratch.status, overlap, x_bf16 != 0);
    }
#endif

    CUtensorMap tw, tx;
#ifndef Q8_HOST_EMULATION
    const unsigned int height = warp_kernel ? rows_height(n, k, m, sm_count, epilogue) : 0u;
    const unsigned int box_rows = height != 0u ? height : kRows;
#else
    const unsigned int box_rows = kRows;
#endif
    if (!map_weights(encode, &tw, w, n, k, box_rows) || (!warp_kernel && !map_rows(encode, &tx, x, m, k, ntok, x_bf16 != 0))) {
        return cudaErrorInvalidValue;
    }

    const unsigned long long row_tiles = (n + kRows - 1u) / kRows;
    const unsigned long long tok_tiles = (m + ntok - 1u) / ntok;
    const unsigned long long units = row_tiles * tok_tiles * (k / kSegK);
    unsigned int grid = sm_count < scratch.blocks ? sm_count : scratch.blocks;
    if (units < grid) {
        grid = (unsigned int)units;
    }
    if (scratch.tile_floats < (unsigned long long)kRows * ntok) {
        return cudaErrorInvalidValue;
    }

    UmmaArgs args = {};
    args.n = n;
    args.k = k;
    args.m_max = m;
    args.m_dev = m_dev;
    args.y = y;
    args.partial = set_partial(scratch, set);
    args.flags = set_flags(scratch, set);
    args.overlap = overlap ? 1u : 0u;
    args.group_tiles = nullptr;
    args.group_count = nullptr;
    args.row_map = nullptr;
    args.epilogue = epilogue;
    args.ldy = epilogue == kEpilogueSwiglu ? n / 2u : n;
    args.peers = 0u;
    args.col0 = 0u;
    if (out != nullptr) {
        args.ldy = out->ldy;
        args.col0 = out->col0;
        args.peers = out->peers;
        for (unsigned int i = 0; i < 8u; ++i) {
            args.y_peer[i] = i < out->peers ? out->y_peer[i] : nullptr;
        }
    }
    args.status = scratch.status;
    args.tile_floats = scratch.tile_floats;
    args.b_bf16 = x_bf16 ? 1u : 0u;
    if (ntok <= 32u) {
        // one token tile: the decode kernel, two blocks per SM (q8_decode.cu); its unit
        // arithmetic is 32-bit
        if (units >= (1ull << 31)) {
            return cudaErrorNotSupported;
        }
        unsigned int cluster = 0u;
        const unsigned int decode_blocks = decode_grid((unsigned int)row_tiles, k / kSegK, sm_count,
                                                       scratch.blocks, &cluster);
        args.split = cluster;
#ifndef Q8_HOST_EMULATION
        if (height != 0u) {
            return launch_decode_rows(stream, tw, x, x_bf16 != 0, height, args, y_dtype);
        }
        if (warp_kernel) {
            // (One piece per tile, rows of one segment: no cluster is launched, and whole tiles are units as any others.  The
            // counted stores of a cluster's exchange are an illegal instruction in a launch without clusters.)
            args.split = cluster > 1u ? cluster : 0u;
            return launch_decode_warp(stream, tw, x, args, decode_blocks, cluster, y_dtype);
        }
#endif
        return launch_decode_kernel(stream, tw, tx, args, decode_blocks, cluster, ntok, y_dtype);
    }
    if (ntok <= 128u) {
        return launch_stream_kernel(stream, tw, tx, args, grid, ntok, y_dtype);
    }
    return launch_wide_kernel(stream, tw, tx, args, grid, y_dtype);
}

cudaError_t launch_umma_grouped(cudaStream_t stream, const UmmaScratch &scratch, unsigned int sm_count,
                                const void *w_stacked, unsigned int total_rows, unsigned int k,
                                const void *x_sorted, unsigned int x_rows, unsigned int ntok,
                                const GroupTile *tiles, const unsigned int *count_dev, unsigned int max_tiles,
                                const unsigned int *row_map, void *y, unsigned int ldy, int y_dtype,
                                unsigned int set, bool overlap, unsigned int epilogue, const void *w_second,
                                bool table_late)
{
    EncodeTiledFn encode = encode_tiled();
    if (encode == nullptr || (k % kSegK) != 0u || ntok > 128u) {
        return cudaErrorNotSupported;
    }
    if (max_tiles == 0u || x_rows == 0u) {
        return cudaSuccess;
    }
    CUtensorMap tw, tx;
    if (!map_weights(encode, &tw, w_stacked, total_rows, k, kRows) || !map_rows(encode, &tx, x_sorted, x_rows, k, ntok, false)) {
        return cudaErrorInvalidValue;
    }
#ifndef Q8_HOST_EMULATION
    {
        // every expert has an even number of weight row tiles (hidden and ffn are multiples of 256), so
        // the table's entries pair up (with a second tensor, an entry is a tile by itself)
        const unsigned int most = w_second != nullptr ? max_tiles : max_tiles / 2u;
        const unsigned int blocks = most < sm_count ? most : sm_count;
        CUtensorMap tw2;
        if (w_second != nullptr && !map_weights(encode, &tw2, w_second, total_rows, k, kRows)) {
            return cudaErrorInvalidValue;
        }
        return launch_mid_grouped(stream, tw, w_second != nullptr ? &tw2 : nullptr, tx, table_late, blocks, k, ntok, tiles, count_dev, row_map, y, ldy, y_dtype, epilogue,
                                  set_partial(scratch, set), set_flags(scratch, set), scratch.tile_floats, scratch.status,
                                  overlap);
    }
#endif
    if (w_second != nullptr) {
        return cudaErrorNotSupported;
    }
    (void)table_late;
    const unsigned long long units = (unsigned long long)max_tiles * (k / kSegK);
    unsigned int grid = sm_count < scratch.blocks ? sm_count : scratch.blocks;
    if (units < grid) {
        grid = (unsigned int)units;
    }
    UmmaArgs args = {};
    args.n = total_rows;
    args.k = k;
    args.m_max = x_rows;
    args.m_dev = nullptr;
    args.y = y;
    args.partial = set_partial(scratch, set);
    args.flags = set_flags(scratch, set);
    args.status = scratch.status;
    args.tile_floats = scratch.tile_floats;
    args.b_bf16 = 0u;
    args.overlap = overlap ? 1u : 0u;
    args.group_tiles = tiles;
    args.group_count = count_dev;
    args.row_map = row_map;
    args.ldy = ldy;
    args.peers = 0u;
    args.col0 = 0u;
    args.epilogue = epilogue;
    return launch_stream_kernel(stream, tw, tx, args, grid, ntok, y_dtype);
}

} // namespace q8
