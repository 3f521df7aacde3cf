// Routed experts as grouped products: the (token, rank) pairs are sorted by expert on the
// device, each expert's rows then form token tiles of up to 128, and the tensor-core kernel
// of q8_mid.cu runs over a table of (expert, token tile, weight row tile) entries, reading every
// expert's weights once for all of its tokens.  Five launches with the router and the sum, each of
// which starts while the one before it ends.
//
// The reference runs one single-row product per token and rank on the token's expert slice
// (cuda/model/expert_matrix.cu:8-27, loop cuda/model/experts_host.cu:99-111), which re-reads an
// expert's weights for every token routed to it.  The results are the same products; the
// rank-ordered weighted sum (cuda/model/experts.cu:77-98) is kept as it is.
#include <math.h>
#include <stdlib.h>

#include "q8_launch.h"
#include "q8_tile.cuh"

namespace q8 {

#define Q8_GROUP_THREADS 1024u
#define Q8_GROUP_MAX_EXPERTS 256u

#ifndef Q8_GROUP_TOKENS
#define Q8_GROUP_TOKENS 64u /* token tile of the grouped products */
#endif

// Token tile of the grouped products: the pairs an expert gets on average and two and a half standard
// deviations more, so that all but a few experts need one tile (an expert with more takes another
// tile, and its weights a second time), and no more columns than that.
static unsigned int group_tokens(unsigned int pairs, unsigned int experts)
{
#ifdef Q8_HOST_EMULATION
    (void)pairs;
    (void)experts;
    return Q8_GROUP_TOKENS;
#else
    const float mean = (float)pairs / (float)experts;
    const unsigned int want = (unsigned int)(mean + 2.5f * sqrtf(mean) + 1.0f);
    const unsigned int tile = (want + 15u) / 16u * 16u;
    return tile < 128u ? tile : 128u;
#endif
}

// One block.  Counts the pairs of every expert, places each pair in its expert's run of
// `sorted_pair` in ascending order of the pair index (a stable sort: the place of a pair, and
// with it the token tile it lands in and the points where that tile's sums are cut between
// blocks, is a function of the selections alone, so the results repeat bit for bit from run to
// run), and writes the two tile tables.
//
// Every warp takes one contiguous run of the pairs.  Pass 1 counts, per warp and expert, the
// warp's pairs (lanes that name the same expert find each other with a match); a scan over the
// warps turns the counts into each warp's first place within the expert; pass 2 walks the
// same run again and places the pairs, lanes in order within a step, steps in order within
// the warp, warps in order within the expert.
__global__ void __launch_bounds__(Q8_GROUP_THREADS)
q8_group_build_kernel(const unsigned int *__restrict__ ids, unsigned int tokens_max,
                      const unsigned int *tokens_dev, unsigned int used, unsigned int experts,
                      unsigned int ffn, unsigned int hidden, unsigned int *__restrict__ sorted_pair,
                      GroupTile *__restrict__ tiles_feed, GroupTile *__restrict__ tiles_down,
                      unsigned int *__restrict__ counts, unsigned int tile_tokens)
{
    __shared__ unsigned int count[Q8_GROUP_MAX_EXPERTS];
    __shared__ unsigned int offset[Q8_GROUP_MAX_EXPERTS];
    __shared__ unsigned int feed_base[Q8_GROUP_MAX_EXPERTS];
    __shared__ unsigned int down_base[Q8_GROUP_MAX_EXPERTS];
    __shared__ unsigned int placed;
    __shared__ unsigned int scan_pairs[Q8_GROUP_MAX_EXPERTS];
    __shared__ unsigned int scan_tiles[Q8_GROUP_MAX_EXPERTS];
    // per warp and expert: first the number of the warp's pairs, then the next free place of
    // the warp within the expert's run
    __shared__ unsigned int warp_place[Q8_GROUP_THREADS / 32u][Q8_GROUP_MAX_EXPERTS];
    unsigned int tokens = tokens_max;
    if (tokens_dev != nullptr) {
        unsigned int live = *tokens_dev;
        tokens = live < tokens_max ? live : tokens_max;
    }
    const unsigned int pairs = tokens * used;
    const unsigned int feed_rows = (ffn + kRows - 1u) / kRows;
    const unsigned int down_rows = (hidden + kRows - 1u) / kRows;
    const unsigned int warp = threadIdx.x >> 5;
    const unsigned int lane = threadIdx.x & 31u;
    const unsigned int warps = blockDim.x >> 5;
    // the warp's run of pairs, a whole number of steps of 32
    const unsigned int per_warp = ((pairs + warps - 1u) / warps + 31u) / 32u * 32u;
    const unsigned int run_begin = warp * per_warp < pairs ? warp * per_warp : pairs;
    const unsigned int run_end = run_begin + per_warp < pairs ? run_begin + per_warp : pairs;
    const unsigned int none = 0xFFFFFFFFu;

    for (unsigned int e = lane; e < experts; e += 32u) {
        warp_place[warp][e] = 0u;
    }
    __syncwarp();
    // A selection outside the expert table is left out of both passes (its result row is then
    // never written), rather than indexing past the tables.
    for (unsigned int first = run_begin; first < run_end; first += 32u) {
        const unsigned int p = first + lane;
        unsigned int e = p < run_end ? ids[p] : none;
        if (e >= experts) {
            e = none;
        }
        const unsigned int same = __match_any_sync(0xFFFFFFFFu, e);
        if (e != none && (same & ((1u << lane) - 1u)) == 0u) {
            warp_place[warp][e] += (unsigned int)__popc(same); // the lowest lane speaks for the expert
        }
        __syncwarp();
    }
    __syncthreads();
    for (unsigned int e = threadIdx.x; e < experts; e += blockDim.x) {
        unsigned int running = 0u;
        for (unsigned int w = 0u; w < warps; ++w) {
            const unsigned int here = warp_place[w][e];
            warp_place[w][e] = running;
            running += here;
        }
        count[e] = running;
    }
    __syncthreads();
    // running totals over the experts of the pairs and of the token tiles (a scan in shared
    // memory, one thread per expert): an expert's first place and first table entries
    {
        const unsigned int e = threadIdx.x;
        const unsigned int mine = e < experts ? count[e] : 0u;
        const unsigned int mine_tiles = (mine + tile_tokens - 1u) / tile_tokens;
        if (e < Q8_GROUP_MAX_EXPERTS) {
            scan_pairs[e] = mine;
            scan_tiles[e] = mine_tiles;
        }
        __syncthreads();
        for (unsigned int step = 1u; step < Q8_GROUP_MAX_EXPERTS; step <<= 1) {
            unsigned int add_pairs = 0u;
            unsigned int add_tiles = 0u;
            if (e < Q8_GROUP_MAX_EXPERTS && e >= step) {
                add_pairs = scan_pairs[e - step];
                add_tiles = scan_tiles[e - step];
            }
            __syncthreads();
            if (e < Q8_GROUP_MAX_EXPERTS) {
                scan_pairs[e] += add_pairs;
                scan_tiles[e] += add_tiles;
            }
            __syncthreads();
        }
        if (e < experts) {
            offset[e] = scan_pairs[e] - mine;
            feed_base[e] = (scan_tiles[e] - mine_tiles) * feed_rows;
            down_base[e] = (scan_tiles[e] - mine_tiles) * down_rows;
            if (e == experts - 1u) {
                counts[0] = scan_tiles[e] * feed_rows;
                counts[1] = scan_tiles[e] * down_rows;
                placed = scan_pairs[e];
            }
        }
    }
    __syncthreads();
    for (unsigned int first = run_begin; first < run_end; first += 32u) {
        const unsigned int p = first + lane;
        unsigned int e = p < run_end ? ids[p] : none;
        if (e >= experts) {
            e = none;
        }
        const unsigned int same = __match_any_sync(0xFFFFFFFFu, e);
        const unsigned int below = (unsigned int)__popc(same & ((1u << lane) - 1u));
        const unsigned int base = e != none ? warp_place[warp][e] : 0u;
        __syncwarp();
        if (e != none) {
            sorted_pair[offset[e] + base + below] = p;
            if (below == 0u) {
                warp_place[warp][e] = base + (unsigned int)__popc(same);
            }
        }
        __syncwarp();
    }
    // the places that pairs left out would have taken name no pair (the gather skips them)
    for (unsigned int at = placed + threadIdx.x; at < pairs; at += blockDim.x) {
        sorted_pair[at] = 0xFFFFFFFFu;
    }
    // the tile tables: a warp per expert, a lane per weight row tile
    for (unsigned int e = warp; e < experts; e += warps) {
        const unsigned int tok_tiles = (count[e] + tile_tokens - 1u) / tile_tokens;
        for (unsigned int tt = 0u; tt < tok_tiles; ++tt) {
            const unsigned int tok0 = offset[e] + tt * tile_tokens;
            unsigned int tok_limit = offset[e] + count[e];
            if (tok_limit > tok0 + tile_tokens) {
                tok_limit = tok0 + tile_tokens;
            }
            for (unsigned int r = lane; r < feed_rows; r += 32u) {
                GroupTile t;
                t.w_row = e * ffn + r * kRows;
                t.j0 = r * kRows;
                t.j_limit = ffn;
                t.tok0 = tok0;
                t.tok_limit = tok_limit;
                tiles_feed[feed_base[e] + tt * feed_rows + r] = t;
            }
            for (unsigned int r = lane; r < down_rows; r += 32u) {
                GroupTile t;
                t.w_row = e * hidden + r * kRows;
                t.j0 = r * kRows;
                t.j_limit = hidden;
                t.tok0 = tok0;
                t.tok_limit = tok_limit;
                tiles_down[down_base[e] + tt * down_rows + r] = t;
            }
        }
    }
}

// x_sorted[i] = x[sorted_pair[i] / used], rows of `hidden` halves, 16 bytes per thread step.
// Expert parallel: token t is row t % rows_per_part of array t / rows_per_part (the tokens of
// all GPUs, each GPU's in its own array, read through peer-mapped addresses).
__global__ void q8_gather_rows_kernel(const __grid_constant__ RowParts x, const unsigned int *__restrict__ sorted_pair,
                                      unsigned int tokens_max, const unsigned int *tokens_dev,
                                      unsigned int used, unsigned int row_chunks, uint4 *__restrict__ out)
{
    unsigned int tokens = tokens_max;
    if (tokens_dev != nullptr) {
        unsigned int live = *tokens_dev;
        tokens = live < tokens_max ? live : tokens_max;
    }
    const unsigned int pairs = tokens * used;
    for (unsigned int i = blockIdx.x; i < pairs; i += gridDim.x) {
        const unsigned int p = sorted_pair[i];
        if (p >= pairs) {
            continue; // no pair here: a selection outside the expert table was left out
        }
        unsigned int t = p / used;
        const uint4 *from = static_cast<const uint4 *>(x.base[0]);
        if (x.parts > 1u) {
            from = static_cast<const uint4 *>(x.base[t / x.rows_per_part]);
            t = t % x.rows_per_part;
        }
        for (unsigned int c = threadIdx.x; c < row_chunks; c += blockDim.x) {
            out[(size_t)i * row_chunks + c] = from[(size_t)t * row_chunks + c];
        }
    }
}

// ids_all[q * count + i] = ids_of_rank[q][i] - first: the selections of every GPU's tokens,
// numbered from this GPU's first expert (unsigned: an expert below it wraps to a number that
// names no local expert, like one above the last).
struct IdParts {
    const unsigned int *base[8];
};

__global__ void q8_collect_ids_kernel(const __grid_constant__ IdParts ids, unsigned int parts, unsigned int count,
                                      unsigned int first, unsigned int *__restrict__ ids_all)
{
    const unsigned int total = parts * count;
    for (unsigned int at = blockIdx.x * blockDim.x + threadIdx.x; at < total; at += gridDim.x * blockDim.x) {
        const unsigned int q = at / count;
        ids_all[at] = ids.base[q][at - q * count] - first;
    }
}

cudaError_t launch_collect_ids(cudaStream_t stream, const unsigned int *const *ids_of_rank, unsigned int parts,
                               unsigned int count, unsigned int first_expert, unsigned int *ids_all)
{
    IdParts ids = {};
    for (unsigned int q = 0; q < parts && q < 8u; ++q) {
        ids.base[q] = ids_of_rank[q];
    }
    const unsigned int total = parts * count;
    const unsigned int grid = (total + 255u) / 256u < 148u * 4u ? (total + 255u) / 256u : 148u * 4u;
    return launch_kernel(q8_collect_ids_kernel, grid, 256, 0, stream, ids, parts, count, first_expert, ids_all);
}

#ifndef Q8_HOST_EMULATION
// The same table, sort and gather as one launch over many blocks; what the routed-expert step runs on the
// GPU.  (The two kernels above are the serial form, which the host emulation steps through.)
//
// Latency bounds this step, not bytes: one block, with a launch of its own for the gather behind it, took
// 16 + 6 us for 512 tokens of 8 experts and 7 + 3.5 us for 8 tokens.  So every block counts all pairs by
// itself (a few steps per warp, their loads issued together), which leaves nothing to hand over between
// blocks; then the places of the sorted order are dealt to the blocks in equal runs - not by
// expert: one expert may hold most of the pairs - and a block writes and gathers its own run.
// The tile tables are dealt to all warps of the grid by expert.
constexpr unsigned int kGroupAhead = 4;   // pairs per lane whose loads are issued together
constexpr unsigned int kGroupFewPairs = 1024;  // up to here blocks of 512 threads
constexpr unsigned int kGroupRun = 1024;  // places of a block that are kept in shared memory as well

__device__ __forceinline__ void group_load_ids(const unsigned int *ids, unsigned int first, unsigned int end,
                                               unsigned int experts, unsigned int lane, unsigned int (&e)[kGroupAhead])
{
#pragma unroll
    for (unsigned int a = 0; a < kGroupAhead; ++a) {
        const unsigned int p = first + 32u * a + lane;
        e[a] = p < end ? ids[p] : 0xFFFFFFFFu;
    }
#pragma unroll
    for (unsigned int a = 0; a < kGroupAhead; ++a) {
        e[a] = e[a] < experts ? e[a] : 0xFFFFFFFFu;    // a selection outside the table is left out
    }
}

// The rows of one expert in a tile table: token tiles by 128-row tiles of its weights.
__device__ __forceinline__ void group_write_tiles(GroupTile *__restrict__ tiles, unsigned int expert, unsigned int rows,
                                                  unsigned int first_place, unsigned int pairs, unsigned int tile_tokens,
                                                  unsigned int lane)
{
    const unsigned int row_tiles = (rows + kRows - 1u) / kRows;
    const unsigned int entries = (pairs + tile_tokens - 1u) / tile_tokens * row_tiles;
    for (unsigned int i = lane; i < entries; i += 32u) {
        const unsigned int tt = i / row_tiles;
        const unsigned int r = i - tt * row_tiles;
        const unsigned int left = pairs - tt * tile_tokens;
        GroupTile t;
        t.w_row = expert * rows + r * kRows;
        t.j0 = r * kRows;
        t.j_limit = rows;
        t.tok0 = first_place + tt * tile_tokens;
        t.tok_limit = t.tok0 + (left < tile_tokens ? left : tile_tokens);
        tiles[i] = t;
    }
}

template <unsigned int THREADS>
__global__ void __launch_bounds__(THREADS, 1)
q8_group_build_kernel_many(const __grid_constant__ RowParts x, const unsigned int *ids, unsigned int tokens_max,
                       const unsigned int *tokens_dev, unsigned int used, unsigned int experts, unsigned int feed,
                       unsigned int hidden, unsigned int *sorted_pair, GroupTile *__restrict__ tiles_feed,
                       GroupTile *__restrict__ tiles_down, unsigned int *__restrict__ counts, unsigned int tile_tokens,
                       uint4 *__restrict__ x_sorted)
{
    constexpr unsigned int kWarps = THREADS / 32u;
    // per warp and expert: the number of the warp's pairs, then the next free place of the warp in the order
    __shared__ unsigned int warp_place[kWarps][Q8_GROUP_MAX_EXPERTS];
    __shared__ unsigned int scan_pairs[Q8_GROUP_MAX_EXPERTS];       // up to and with the expert
    __shared__ unsigned int scan_tiles[Q8_GROUP_MAX_EXPERTS];
    __shared__ unsigned int edge[2];
    __shared__ unsigned int run[kGroupRun];
    __shared__ unsigned int warp_pairs[kWarps];
    __shared__ unsigned int warp_tiles[kWarps];
    const unsigned int warp = threadIdx.x >> 5;
    const unsigned int lane = threadIdx.x & 31u;
    for (unsigned int e = lane; e < experts; e += 32u) {
        warp_place[warp][e] = 0u;
    }
    if (threadIdx.x == 0u) {
        edge[0] = 1u;     // none: the first is after the last
        edge[1] = 0u;
    }
    __syncwarp();
    grid_dependency_wait();
    grid_launch_dependents();
    unsigned int tokens = tokens_max;
    if (tokens_dev != nullptr) {
        const unsigned int live = *tokens_dev;
        tokens = live < tokens_max ? live : tokens_max;
    }
    const unsigned int pairs = tokens * used;
    // the warp's run of pairs, a whole number of steps of 32
    const unsigned int per_warp = ((pairs + kWarps - 1u) / kWarps + 31u) / 32u * 32u;
    const unsigned int run_begin = warp * per_warp < pairs ? warp * per_warp : pairs;
    const unsigned int run_end = run_begin + per_warp < pairs ? run_begin + per_warp : pairs;

    // the block's run of places
    const unsigned int per_block = (pairs + gridDim.x - 1u) / gridDim.x;
    const unsigned int place_begin = blockIdx.x * per_block < pairs ? blockIdx.x * per_block : pairs;
    const unsigned int place_end = place_begin + per_block < pairs ? place_begin + per_block : pairs;
    unsigned int e[kGroupAhead];
    for (unsigned int first = run_begin; first < run_end; first += 32u * kGroupAhead) {
        group_load_ids(ids, first, run_end, experts, lane, e);
#pragma unroll
        for (unsigned int a = 0; a < kGroupAhead; ++a) {
            if (e[a] != 0xFFFFFFFFu) {
                atomicAdd(&warp_place[warp][e[a]], 1u);
            }
        }
    }
    __syncthreads();
    // One thread per expert: its pairs, and the running totals over the experts of pairs and token tiles.
    {
        const unsigned int ex = threadIdx.x;
        unsigned int mine = 0u;
        if (ex < experts) {
#pragma unroll 8
            for (unsigned int w = 0u; w < kWarps; ++w) {
                const unsigned int here = warp_place[w][ex];
                warp_place[w][ex] = mine;
                mine += here;
            }
        }
        const unsigned int mine_tiles = (mine + tile_tokens - 1u) / tile_tokens;
        unsigned int run_pairs = mine;
        unsigned int run_tiles = mine_tiles;
#pragma unroll
        for (unsigned int step = 1u; step < 32u; step <<= 1) {
            const unsigned int below_pairs = __shfl_up_sync(0xFFFFFFFFu, run_pairs, step);
            const unsigned int below_tiles = __shfl_up_sync(0xFFFFFFFFu, run_tiles, step);
            if (lane >= step) {
                run_pairs += below_pairs;
                run_tiles += below_tiles;
            }
        }
        if (lane == 31u) {
            warp_pairs[warp] = run_pairs;
            warp_tiles[warp] = run_tiles;
        }
        __syncthreads();
        if (ex < Q8_GROUP_MAX_EXPERTS) {
            for (unsigned int w = 0u; w < warp; ++w) {
                run_pairs += warp_pairs[w];
                run_tiles += warp_tiles[w];
            }
            scan_pairs[ex] = run_pairs;
            scan_tiles[ex] = run_tiles;
            // the experts that hold the first and the last of the block's places
            const unsigned int begin = run_pairs - mine;
            if (begin <= place_begin && place_begin < run_pairs) {
                edge[0] = ex;
            }
            if (begin < place_end && place_begin < run_pairs) {
                atomicMax(&edge[1], ex);
            }
        }
        __syncthreads();
    }
    const unsigned int placed = scan_pairs[experts - 1u];
    const unsigned int feed_rows = (feed + kRows - 1u) / kRows;
    const unsigned int down_rows = (hidden + kRows - 1u) / kRows;
    if (blockIdx.x == 0u && threadIdx.x == 0u) {
        counts[0] = scan_tiles[experts - 1u] * feed_rows;
        counts[1] = scan_tiles[experts - 1u] * down_rows;
    }
    for (unsigned int ex = blockIdx.x + gridDim.x * warp; ex < experts; ex += gridDim.x * kWarps) {
        const unsigned int place = ex != 0u ? scan_pairs[ex - 1u] : 0u;
        const unsigned int tile = ex != 0u ? scan_tiles[ex - 1u] : 0u;
        const unsigned int mine = scan_pairs[ex] - place;
        group_write_tiles(tiles_feed + (size_t)tile * feed_rows, ex, feed, place, mine, tile_tokens, lane);
        group_write_tiles(tiles_down + (size_t)tile * down_rows, ex, hidden, place, mine, tile_tokens, lane);
    }
    // Only the few experts of the block's run matter here: a ballot per expert and step tells the pairs'
    // places, steps in order within the warp, warps in order within the expert.
    const unsigned int edge_first = edge[0];
    const unsigned int edge_last = edge[1];
    if (edge_first <= edge_last && place_begin < placed) {
        for (unsigned int first = run_begin; first < run_end; first += 32u * kGroupAhead) {
            if (per_warp > 32u * kGroupAhead) {
                group_load_ids(ids, first, run_end, experts, lane, e);     // else they are still there
            }
            for (unsigned int ex = edge_first; ex <= edge_last; ++ex) {
                const unsigned int in_expert = warp_place[warp][ex];
                unsigned int place = (ex != 0u ? scan_pairs[ex - 1u] : 0u) + in_expert;
                unsigned int seen = 0u;
#pragma unroll
                for (unsigned int a = 0; a < kGroupAhead; ++a) {
                    const unsigned int same = __ballot_sync(0xFFFFFFFFu, e[a] == ex);
                    const unsigned int at = place + seen + (unsigned int)__popc(same & ((1u << lane) - 1u));
                    if (e[a] == ex && at >= place_begin && at < place_end) {
                        sorted_pair[at] = first + 32u * a + lane;
                        if (at - place_begin < kGroupRun) {
                            run[at - place_begin] = first + 32u * a + lane;
                        }
                    }
                    seen += (unsigned int)__popc(same);
                }
                __syncwarp();
                if (lane == 0u) {
                    warp_place[warp][ex] = in_expert + seen;
                }
            }
            __syncwarp();
        }
    }
    // the places that pairs left out would have taken name no pair
    for (unsigned int at = (placed > place_begin ? placed : place_begin) + threadIdx.x; at < place_end; at += blockDim.x) {
        sorted_pair[at] = 0xFFFFFFFFu;
    }
    __syncthreads();
    // the rows of x of the block's places, 16 bytes per thread step
    const unsigned int row_chunks = hidden / 8u;
    const unsigned int last = placed < place_end ? placed : place_end;
    const unsigned int total = last > place_begin ? (last - place_begin) * row_chunks : 0u;
#pragma unroll 4
    for (unsigned int i = threadIdx.x; i < total; i += THREADS) {
        const unsigned int at = i / row_chunks;
        const unsigned int c = i - at * row_chunks;
        unsigned int t = (at < kGroupRun ? run[at] : sorted_pair[place_begin + at]) / used;
        const uint4 *from = static_cast<const uint4 *>(x.base[0]);
        if (x.parts > 1u) {
            const unsigned int part = t / x.rows_per_part;
            from = static_cast<const uint4 *>(x.base[part]);
            t -= part * x.rows_per_part;
        }
        x_sorted[(size_t)(place_begin + at) * row_chunks + c] = from[(size_t)t * row_chunks + c];
    }
}

static cudaError_t launch_group_gather(cudaStream_t stream, bool overlap, unsigned int sm_count, const RowParts &rows,
                                       const unsigned int *ids, unsigned int tokens, const unsigned int *tokens_dev,
                                       unsigned int used, unsigned int experts, unsigned int feed, unsigned int hidden,
                                       unsigned char *workspace, const MoeWorkspace &ws, unsigned int tile_tokens)
{
    const unsigned int pairs = tokens * used;
    const unsigned int blocks = pairs < sm_count ? pairs : sm_count;
    auto launch = [&](auto kernel, unsigned int threads) {
        return launch_kernel_early(overlap, kernel, blocks, threads, 0, stream, rows, ids, tokens,
                                   tokens_dev, used, experts, feed, hidden,
                                   reinterpret_cast<unsigned int *>(workspace + ws.sorted_pair),
                                   reinterpret_cast<GroupTile *>(workspace + ws.tiles_feed),
                                   reinterpret_cast<GroupTile *>(workspace + ws.tiles_down),
                                   reinterpret_cast<unsigned int *>(workspace + ws.counts), tile_tokens,
                                   reinterpret_cast<uint4 *>(workspace + ws.x_sorted));
    };
    // Few pairs: half the threads, which find room beside the blocks of the router (whole step, 8 tokens of 8 of 128
    // experts, 74.1 -> 73.4 us, 1 token 40.1 -> 39.7, 127 of 8 of 32 54.2 -> 53.9, 100 of 8 of 128 the same; 512 tokens
    // 195 -> 199, so not where there is something to count).
    return pairs <= kGroupFewPairs ? launch(q8_group_build_kernel_many<512u>, 512u) : launch(q8_group_build_kernel_many<1024u>, 1024u);
}
#endif

// act = half(silu(gate) * up), silu(g) = g / (1 + exp(-g))  (cuda/model/norm.cu:92-105)
__global__ void q8_swiglu_kernel(const float *__restrict__ gate, const float *__restrict__ up,
                                 unsigned int tokens_max, const unsigned int *tokens_dev, unsigned int used,
                                 unsigned int ffn, __half *__restrict__ act)
{
    unsigned int tokens = tokens_max;
    if (tokens_dev != nullptr) {
        unsigned int live = *tokens_dev;
        tokens = live < tokens_max ? live : tokens_max;
    }
    const size_t total = (size_t)tokens * used * ffn;
    for (size_t at = (size_t)blockIdx.x * blockDim.x + threadIdx.x; at < total;
         at += (size_t)gridDim.x * blockDim.x) {
        float g = gate[at];
        float unit = g / (1.0f + expf(-g));
        act[at] = __float2half_rn(unit * up[at]);
    }
}

bool moe_grouped_supports(const void *w_gate, const void *w_up, const void *w_down, const void *x,
                          unsigned int hidden, unsigned int ffn, unsigned int experts)
{
    auto aligned16 = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0u; };
    return (hidden % kSegK) == 0u && (ffn % kSegK) == 0u && experts <= Q8_GROUP_MAX_EXPERTS && aligned16(w_gate)
        && aligned16(w_up) && aligned16(w_down) && aligned16(x);
}

static size_t up256(size_t v)
{
    return (v + 255u) / 256u * 256u;
}

MoeWorkspace moe_workspace_layout(unsigned int tokens, unsigned int used, unsigned int hidden,
                                  unsigned int ffn, unsigned int experts)
{
    MoeWorkspace ws;
    const size_t pairs = (size_t)tokens * used;
    const size_t tok_tiles = pairs / 16u + experts; /* room for the smallest token tile */
    /* room for the interleaved gate+up form as well, which has twice the rows */
    ws.max_feed = (unsigned int)(tok_tiles * ((2u * ffn + kRows - 1u) / kRows));
    ws.max_down = (unsigned int)(tok_tiles * ((hidden + kRows - 1u) / kRows));
    size_t at = 0;
    ws.act = at;
    at += up256(pairs * ffn * sizeof(unsigned short));
    ws.proj = at;
    at += up256(pairs * hidden * sizeof(float));
    ws.sorted_pair = at;
    at += up256(pairs * sizeof(unsigned int));
    ws.counts = at;
    at += 256;
    ws.tiles_feed = at;
    at += up256((size_t)ws.max_feed * sizeof(GroupTile));
    ws.tiles_down = at;
    at += up256((size_t)ws.max_down * sizeof(GroupTile));
    ws.x_sorted = at;
    at += up256(pairs * hidden * sizeof(unsigned short));
    ws.gate = at;
    at += up256(pairs * ffn * sizeof(float));
    ws.up = at;
    at += up256(pairs * ffn * sizeof(float));
    ws.bytes = at;
    return ws;
}

cudaError_t launch_moe_grouped(cudaStream_t stream, const UmmaScratch &scratch, unsigned int sm_count,
                               unsigned int *launches, bool overlap, const void *w_gate, const void *w_up,
                               const void *w_down, unsigned int experts, unsigned int hidden,
                               unsigned int ffn, const void *x, const unsigned int *ids, unsigned int tokens,
                               const unsigned int *tokens_dev, unsigned int used, unsigned char *workspace,
                               const MoeWorkspace &ws, const RowParts *x_parts, float *proj_out)
{
    const unsigned int pairs = tokens * used;
    // (several GPUs: the pairs of all, of which this GPU's experts get their part)
    const unsigned int tile_tokens = group_tokens(x_parts != nullptr ? pairs / x_parts->parts : pairs, experts);
    unsigned int *sorted_pair = reinterpret_cast<unsigned int *>(workspace + ws.sorted_pair);
    unsigned int *counts = reinterpret_cast<unsigned int *>(workspace + ws.counts);
    GroupTile *tiles_feed = reinterpret_cast<GroupTile *>(workspace + ws.tiles_feed);
    GroupTile *tiles_down = reinterpret_cast<GroupTile *>(workspace + ws.tiles_down);
    __half *x_sorted = reinterpret_cast<__half *>(workspace + ws.x_sorted);
    float *gate = reinterpret_cast<float *>(workspace + ws.gate);
    float *up = reinterpret_cast<float *>(workspace + ws.up);
    __half *act = reinterpret_cast<__half *>(workspace + ws.act);
    float *proj = proj_out != nullptr ? proj_out : reinterpret_cast<float *>(workspace + ws.proj);
    RowParts rows = {};
    rows.base[0] = x;
    rows.parts = 1u;
    if (x_parts != nullptr) {
        rows = *x_parts;
    }

#ifndef Q8_HOST_EMULATION
    cudaError_t err = launch_group_gather(stream, overlap, sm_count, rows, ids, tokens, tokens_dev, used, experts, ffn,
                                          hidden, workspace, ws, tile_tokens);
    if (err != cudaSuccess) {
        return err;
    }
    // Gate and up in one launch: a tile's two slabs are the same rows of the two tensors, and the store
    // applies the gated unit.  (Two products, their sums through memory as floats and an elementwise
    // kernel took 2 x 50 + 14 us for 512 tokens of 8 of 128 experts, 2048 x 768.)
    err = launch_umma_grouped(stream, scratch, sm_count, w_gate, experts * ffn, hidden, x_sorted, pairs, tile_tokens,
                              tiles_feed, counts + 0, ws.max_feed, nullptr, act, ffn, 1, (*launches)++, overlap,
                              kEpilogueSwiglu, w_up, true);
    if (err != cudaSuccess) {
        return err;
    }
    (void)gate;
    (void)up;
#else
    cudaError_t err = launch_kernel(q8_group_build_kernel, 1, Q8_GROUP_THREADS, 0, stream, ids, tokens, tokens_dev,
                                    used, experts, ffn, hidden, sorted_pair, tiles_feed, tiles_down, counts,
                                    tile_tokens);
    if (err != cudaSuccess) {
        return err;
    }
    const unsigned int wave = pairs < 148u * 16u ? pairs : 148u * 16u;
    err = launch_kernel(q8_gather_rows_kernel, wave, 128, 0, stream, rows, sorted_pair, tokens,
                        tokens_dev, used, hidden / 8u, reinterpret_cast<uint4 *>(x_sorted));
    if (err != cudaSuccess) {
        return err;
    }
    err = launch_umma_grouped(stream, scratch, sm_count, w_gate, experts * ffn, hidden, x_sorted, pairs,
                              tile_tokens, tiles_feed, counts + 0, ws.max_feed, nullptr, gate, ffn, 0,
                              (*launches)++, overlap);
    if (err != cudaSuccess) {
        return err;
    }
    err = launch_umma_grouped(stream, scratch, sm_count, w_up, experts * ffn, hidden, x_sorted, pairs,
                              tile_tokens, tiles_feed, counts + 0, ws.max_feed, nullptr, up, ffn, 0,
                              (*launches)++, overlap);
    if (err != cudaSuccess) {
        return err;
    }
    err = launch_kernel(q8_swiglu_kernel, 148 * 8, 256, 0, stream, gate, up, tokens, tokens_dev, used, ffn, act);
    if (err != cudaSuccess) {
        return err;
    }
#endif
    return launch_umma_grouped(stream, scratch, sm_count, w_down, experts * hidden, ffn, act, pairs,
                               tile_tokens, tiles_down, counts + 1, ws.max_down, sorted_pair, proj, hidden,
                               0, (*launches)++, overlap);
}

// The same step with gate and up in one tensor, rows interleaved (row 2r of an expert is its
// gate row r, row 2r + 1 its up row r): one grouped product whose store applies the gated unit
// and writes the half activations, then the down product.  Two tensor-core launches instead of
// three and an elementwise kernel, and no float gate / up round trip.
cudaError_t launch_moe_grouped_fused(cudaStream_t stream, const UmmaScratch &scratch, unsigned int sm_count,
                                     unsigned int *launches, bool overlap, const void *w_gate_up,
                                     const void *w_down, unsigned int experts, unsigned int hidden,
                                     unsigned int ffn, const void *x, const unsigned int *ids,
                                     unsigned int tokens, const unsigned int *tokens_dev, unsigned int used,
                                     unsigned char *workspace, const MoeWorkspace &ws)
{
    const unsigned int pairs = tokens * used;
    const unsigned int tile_tokens = group_tokens(pairs, experts);
    unsigned int *sorted_pair = reinterpret_cast<unsigned int *>(workspace + ws.sorted_pair);
    unsigned int *counts = reinterpret_cast<unsigned int *>(workspace + ws.counts);
    GroupTile *tiles_feed = reinterpret_cast<GroupTile *>(workspace + ws.tiles_feed);
    GroupTile *tiles_down = reinterpret_cast<GroupTile *>(workspace + ws.tiles_down);
    __half *x_sorted = reinterpret_cast<__half *>(workspace + ws.x_sorted);
    __half *act = reinterpret_cast<__half *>(workspace + ws.act);
    float *proj = reinterpret_cast<float *>(workspace + ws.proj);

    RowParts rows = {};
    rows.base[0] = x;
    rows.parts = 1u;
    // the feed table is built over the 2 * ffn interleaved rows of every expert
#ifndef Q8_HOST_EMULATION
    cudaError_t err = launch_group_gather(stream, overlap, sm_count, rows, ids, tokens, tokens_dev, used, experts, 2u * ffn,
                                          hidden, workspace, ws, tile_tokens);
    const bool table_late = true;
#else
    cudaError_t err = launch_kernel(q8_group_build_kernel, 1, Q8_GROUP_THREADS, 0, stream, ids, tokens, tokens_dev,
                                    used, experts, 2u * ffn, hidden, sorted_pair, tiles_feed, tiles_down, counts,
                                    tile_tokens);
    if (err != cudaSuccess) {
        return err;
    }
    const unsigned int wave = pairs < 148u * 16u ? pairs : 148u * 16u;
    err = launch_kernel(q8_gather_rows_kernel, wave, 128, 0, stream, rows, sorted_pair, tokens,
                        tokens_dev, used, hidden / 8u, reinterpret_cast<uint4 *>(x_sorted));
    const bool table_late = false;
#endif
    if (err != cudaSuccess) {
        return err;
    }
    err = launch_umma_grouped(stream, scratch, sm_count, w_gate_up, experts * 2u * ffn, hidden, x_sorted, pairs,
                              tile_tokens, tiles_feed, counts + 0, ws.max_feed, nullptr, act, ffn, 1,
                              (*launches)++, overlap, kEpilogueSwiglu, nullptr, table_late);
    if (err != cudaSuccess) {
        return err;
    }
    return launch_umma_grouped(stream, scratch, sm_count, w_down, experts * hidden, ffn, act, pairs,
                               tile_tokens, tiles_down, counts + 1, ws.max_down, sorted_pair, proj, hidden,
                               0, (*launches)++, overlap);
}

} // namespace q8
