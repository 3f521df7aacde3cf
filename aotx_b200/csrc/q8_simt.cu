// General-shape kernels of the Q8_0 path on the ordinary cores: dequantisation, the
// any-shape product (depth any multiple of 32, any alignment the block layout allows), the
// expert router, the per-pair expert products and the ordered expert sum.
//
// The kernels behind q8_dispatch.cu take products with a depth of a multiple of 256 and 16-byte
// aligned rows, q_warp.cu the others with x on an 8-byte boundary; the product here serves what is
// left, so that the library covers the whole contract of the reference's kernels:
//   cuda/model/dequant.cu:9-70      -> q8_dequant_kernel
//   cuda/model/gemv.cuh:33-145      -> q8_gemv_simt_kernel
//   cuda/model/experts.cu:10-75     -> q8_route_kernel (many tokens: q8_route.cu)
//   cuda/model/expert_matrix.cu:8-27, cuda/model/norm.cu:92-105 -> q8_expert_feed_kernel / q8_expert_down_kernel
//   cuda/model/experts.cu:77-98     -> q8_expert_sum_kernel
#include "q8_common.cuh"
#include "q8_launch.h"
#include "q8_route.cuh"
#include "q8_simt_gemv.cuh"
#ifndef Q8_HOST_EMULATION
#include "q8_warp_ptx.cuh"
#endif

namespace q8 {

// ---------------------------------------------------------------------------------------
// Dequantisation.  The rows [first, first + rows) are one contiguous run of 34-byte
// blocks, so the kernel walks blocks, not rows: one thread turns 8 weights of one block
// into 8 halves and stores them with one 16-byte store.  HBM-bound, if enough loads are on
// their way: a thread asks for four pieces before it turns the first.
// ---------------------------------------------------------------------------------------
template <unsigned int TOGETHER>
__device__ __forceinline__ void dequant_body(const unsigned char *w, unsigned long long blocks,
                                             __half *__restrict__ out, int wide_store)
{
    const unsigned long long total = blocks * 4ull;
    const unsigned int step = blockDim.x;    // neighbouring threads, neighbouring pieces
    // The next launch starts after the wait: it may read its weights at once, and what was written two launches
    // before it is there by then.
    grid_dependency_wait();
    grid_launch_dependents();
    for (unsigned long long first = (unsigned long long)blockIdx.x * blockDim.x * TOGETHER + threadIdx.x;
         first < total; first += (unsigned long long)gridDim.x * blockDim.x * TOGETHER) {
        unsigned short scale[TOGETHER];
        unsigned short codes[TOGETHER][4];
#pragma unroll
        for (unsigned int j = 0; j < TOGETHER; ++j) {
            const unsigned long long at = first + j * step;
            const unsigned char *one = w + (at < total ? at >> 2 : 0ull) * Q8_BLOCK_BYTES;
            const unsigned short *src = reinterpret_cast<const unsigned short *>(one + 2u + (unsigned int)(at & 3ull) * 8u);
            scale[j] = *reinterpret_cast<const unsigned short *>(one);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                codes[j][i] = src[i];
            }
        }
#pragma unroll
        for (unsigned int j = 0; j < TOGETHER; ++j) {
            const unsigned long long at = first + j * step;
            if (at >= total) {
                break;
            }
            const __half2 d2 = __half2half2(*reinterpret_cast<const __half *>(&scale[j]));
            uint32_t packed[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t flipped = (uint32_t)codes[j][i] ^ 0x8080u;
                packed[i] = dequant_pair<0>(flipped, d2);
            }
            __half *dst = out + (at >> 2) * Q8_BLOCK + (unsigned int)(at & 3ull) * 8u;
            if (wide_store) {
                *reinterpret_cast<uint4 *>(dst) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    *reinterpret_cast<__half2 *>(dst + 2 * i) = *reinterpret_cast<__half2 *>(&packed[i]);
                }
            }
        }
    }
}

#define Q8_DEQUANT_TOGETHER 4u
__global__ void q8_dequant_kernel(const unsigned char *w, unsigned long long blocks,
                                  __half *__restrict__ out, int wide_store)
{
    dequant_body<1u>(w, blocks, out, wide_store);
}

__global__ void q8_dequant_kernel_many(const unsigned char *w, unsigned long long blocks,
                                       __half *__restrict__ out, int wide_store)
{
    dequant_body<Q8_DEQUANT_TOGETHER>(w, blocks, out, wide_store);
}

// ---------------------------------------------------------------------------------------
// Expert router.  Logits are float dot products of the float router rows with the half
// activations: lanes 32 apart along the row, then a shuffle tree; the softmax takes the maximum
// away; the experts come out in order of probability, equal ones the lower index first.  Every
// sum runs in the same order as the reference kernel's, so the probabilities are the same floats.
//
// A cluster of blocks shares TOKENS tokens: each block takes its share of the experts, a warp
// EXPERTS of them at a time, and the logits of a token are gathered in the shared memory of the
// block that finishes it.  What bounds it is the latency of the router rows (1 MB from L2 at 128
// experts of 2048) as long as tokens are few, and the float additions (tokens * experts * hidden)
// when they are many: so few tokens per cluster and many loads of a row in flight for a short
// batch, many tokens per row value for a long one.  One block for all experts of four tokens,
// one row of eight loads per warp at a time, took 78 us at any number of tokens up to
// 512 (140 us with the router cold in L2); this takes 7 us for 8 tokens and
// 22 us for 512 (128 experts, hidden 2048), for which q8_route.cu takes 17: above 148 tokens these kernels
// are left with a live count on the device, rows off a 16-byte boundary or of no multiple of 32 values, and the numbers of
// experts and widths for which they are the faster ones (route_tiles_pay in q8_route.cuh).
// ---------------------------------------------------------------------------------------
#define Q8_ROUTE_THREADS 256u     // of the emulated launch
#define Q8_ROUTE_GPU_THREADS 512u

// Activations of a group in shared memory, [position along the row][token], rows padded so that
// 16-byte reads of 8 neighbouring lanes meet 32 different banks.
template <unsigned int TOKENS>
struct RouteShape {
    static constexpr unsigned int stride = TOKENS <= 4u ? TOKENS : TOKENS + 4u;
};

// One position of the rows: EXPERTS router values by TOKENS activations.
template <unsigned int TOKENS, unsigned int EXPERTS>
__device__ __forceinline__ void route_step(const float *at, const float (&r)[EXPERTS], float (&dot)[EXPERTS][TOKENS])
{
    constexpr unsigned int kTogether = TOKENS < 4u ? TOKENS : 4u;
#pragma unroll
    for (unsigned int g0 = 0; g0 < TOKENS; g0 += kTogether) {
        float xv[kTogether];
        if (TOKENS >= 4u) {
            const float4 four = *reinterpret_cast<const float4 *>(at + g0);
            xv[0] = four.x;
            xv[1u % kTogether] = four.y;
            xv[2u % kTogether] = four.z;
            xv[3u % kTogether] = four.w;
        } else {
#pragma unroll
            for (unsigned int g = 0; g < kTogether; ++g) {
                xv[g] = at[g];
            }
        }
#pragma unroll
        for (unsigned int g = 0; g < kTogether; ++g) {
#pragma unroll
            for (unsigned int e = 0; e < EXPERTS; ++e) {
                // the reference's own expression; both compile to one fused multiply-add
                dot[e][g0 + g] += r[e] * xv[g];
            }
        }
    }
}

__device__ __forceinline__ void route_arrive()
{
#ifdef Q8_HOST_EMULATION
    cluster_arrive_release();
#else
    cluster_arrive_relaxed();
#endif
}

template <unsigned int TOKENS, unsigned int EXPERTS, unsigned int AHEAD>
__device__ __forceinline__ void route_body(const __half *x, const float *router,
                                           unsigned int tokens_max, const unsigned int *tokens_dev,
                                           unsigned int hidden, unsigned int experts, unsigned int used,
                                           float *__restrict__ prob, unsigned int *__restrict__ ids, float *route_x,
                                           float (&probability)[TOKENS][Q8_ROUTE_EXPERTS])
{
    constexpr unsigned int kStride = RouteShape<TOKENS>::stride;
    unsigned int tokens = tokens_max;
    if (tokens_dev != nullptr) {
        unsigned int live = *tokens_dev;
        tokens = live < tokens_max ? live : tokens_max;
    }
    const unsigned int lane = threadIdx.x & 31u;
    const unsigned int warp = threadIdx.x >> 5;
    const unsigned int warps = blockDim.x >> 5;
    const unsigned int csize = cluster_nctarank();
    const unsigned int crank = cluster_ctarank();
    const unsigned int first_expert = crank * experts / csize;
    const unsigned int last_expert = (crank + 1u) * experts / csize;
    if (csize > 1u) {
        // every block has started before another writes into its shared memory (nothing is handed over:
        // a relaxed arrival, which spares the 2400 cycles of a cluster-scope release); waited for below
        route_arrive();
    }
    bool others_started = csize == 1u;
    // the blocks of a cluster take the same groups, so they leave this loop together
    for (unsigned int t0 = blockIdx.x / csize * TOKENS; t0 < tokens; t0 += gridDim.x / csize * TOKENS) {
        const unsigned int group = tokens - t0 < TOKENS ? tokens - t0 : TOKENS;
        // one value of every token at a time: the loads of several positions go out together, and the
        // stores of a warp fill whole bank rows
#pragma unroll 4
        for (unsigned int d = threadIdx.x; d < hidden; d += blockDim.x) {
            float in[TOKENS];
#pragma unroll
            for (unsigned int g = 0; g < TOKENS; ++g) {
                in[g] = g < group ? __half2float(x[(size_t)(t0 + g) * hidden + d]) : 0.0f;
            }
            if (TOKENS >= 4u) {
#pragma unroll
                for (unsigned int g = 0; g < TOKENS; g += 4u) {
                    *reinterpret_cast<float4 *>(route_x + d * kStride + g) =
                        make_float4(in[g], in[(g + 1u) % TOKENS], in[(g + 2u) % TOKENS], in[(g + 3u) % TOKENS]);
                }
            } else {
#pragma unroll
                for (unsigned int g = 0; g < TOKENS; ++g) {
                    route_x[d * kStride + g] = in[g];
                }
            }
        }
        __syncthreads();
        if (!others_started) {
            cluster_wait_acquire();
            others_started = true;
        }
        for (unsigned int ex = first_expert + warp * EXPERTS; ex < last_expert; ex += warps * EXPERTS) {
            // rows past the end repeat the last one; their sums are not used
            const float *row[EXPERTS];
#pragma unroll
            for (unsigned int e = 0; e < EXPERTS; ++e) {
                row[e] = router + (size_t)(ex + e < last_expert ? ex + e : last_expert - 1u) * hidden;
            }
            float dot[EXPERTS][TOKENS];
#pragma unroll
            for (unsigned int e = 0; e < EXPERTS; ++e) {
#pragma unroll
                for (unsigned int g = 0; g < TOKENS; ++g) {
                    dot[e][g] = 0.0f;
                }
            }
            // Whole rounds of AHEAD positions per lane: the values of the next round are on their way
            // while this one's are used, and every address is a register and a constant.
            const unsigned int rounds = hidden / (32u * AHEAD);
            float next[AHEAD][EXPERTS];
            if (rounds != 0u) {
#pragma unroll
                for (unsigned int a = 0; a < AHEAD; ++a) {
#pragma unroll
                    for (unsigned int e = 0; e < EXPERTS; ++e) {
                        next[a][e] = row[e][lane + 32u * a];
                    }
                }
            }
            const float *at = route_x + lane * kStride;
            for (unsigned int round = 0; round < rounds; ++round) {
                float here[AHEAD][EXPERTS];
#pragma unroll
                for (unsigned int a = 0; a < AHEAD; ++a) {
#pragma unroll
                    for (unsigned int e = 0; e < EXPERTS; ++e) {
                        here[a][e] = next[a][e];
                    }
                }
                if (round + 1u < rounds) {
#pragma unroll
                    for (unsigned int e = 0; e < EXPERTS; ++e) {
                        row[e] += 32u * AHEAD;
#pragma unroll
                        for (unsigned int a = 0; a < AHEAD; ++a) {
                            next[a][e] = row[e][lane + 32u * a];
                        }
                    }
                }
#pragma unroll
                for (unsigned int a = 0; a < AHEAD; ++a) {
                    route_step<TOKENS, EXPERTS>(at + 32u * a * kStride, here[a], dot);
                }
                at += 32u * AHEAD * kStride;
            }
            for (unsigned int d = rounds * 32u * AHEAD + lane; d < hidden; d += 32u) {
                float here[EXPERTS];
#pragma unroll
                for (unsigned int e = 0; e < EXPERTS; ++e) {
                    here[e] = router[(size_t)(ex + e < last_expert ? ex + e : last_expert - 1u) * hidden + d];
                }
                route_step<TOKENS, EXPERTS>(route_x + d * kStride, here, dot);
            }
#pragma unroll
            for (unsigned int e = 0; e < EXPERTS; ++e) {
#pragma unroll
                for (unsigned int g = 0; g < TOKENS; ++g) {
                    for (unsigned int step = 16u; step != 0u; step >>= 1) {
                        dot[e][g] += __shfl_down_sync(0xFFFFFFFFu, dot[e][g], step);
                    }
                    if (lane == 0u && ex + e < last_expert) {
                        if (csize == 1u) {
                            probability[g][ex + e] = dot[e][g];
                        } else {
                            st_shared_cluster_f32(mapa_shared(smem_u32(&probability[g][ex + e]), g % csize), dot[e][g]);
                        }
                    }
                }
            }
        }
        // every logit of the group lies with the block that finishes its token
        if (csize == 1u) {
            __syncthreads();
        } else {
            __syncwarp();
            cluster_arrive_release();
            cluster_wait_acquire();
        }
        for (unsigned int g = crank + csize * warp; g < group; g += csize * warps) {
            route_choose(probability[g], t0 + g, experts, used, prob, ids);
        }
        // the next group's activations and logits come after everyone has read this one's
        if (t0 + gridDim.x / csize * TOKENS >= tokens) {
            break;
        }
        if (csize == 1u) {
            __syncthreads();
        } else {
            __syncwarp();
            cluster_arrive_release();
            cluster_wait_acquire();
        }
    }
    if (!others_started) {
        cluster_wait_acquire();
    }
}

#define Q8_ROUTE_KERNEL(NAME, TOKENS, EXPERTS, AHEAD)                                                               \
    __global__ void __launch_bounds__(Q8_ROUTE_GPU_THREADS, 2)                                                      \
    NAME(const __half *x, const float *router, unsigned int tokens_max,                                             \
         const unsigned int *tokens_dev, unsigned int hidden, unsigned int experts, unsigned int used,              \
         float *__restrict__ prob, unsigned int *__restrict__ ids)                                                  \
    {                                                                                                               \
        Q8_ROUTE_DYNAMIC                                                                                            \
        __shared__ float probability[TOKENS][Q8_ROUTE_EXPERTS];                                                     \
        grid_dependency_wait();                                                                                     \
        grid_launch_dependents();                                                                                   \
        route_body<TOKENS, EXPERTS, AHEAD>(x, router, tokens_max, tokens_dev, hidden, experts, used, prob, ids,     \
                                           route_x, probability);                                                   \
    }
#ifdef Q8_HOST_EMULATION
#define Q8_ROUTE_DYNAMIC float *route_x = emulated_dynamic_shared;
#else
#define Q8_ROUTE_DYNAMIC extern __shared__ __align__(16) float route_x[];
#endif
// middling batches, and rows too long for eight tokens in shared memory; short batches; long ones
Q8_ROUTE_KERNEL(q8_route_kernel, 4u, 1u, 8u)
Q8_ROUTE_KERNEL(q8_route_kernel_few, 2u, 1u, 16u)
Q8_ROUTE_KERNEL(q8_route_kernel_many, 8u, 2u, 3u)

// ---------------------------------------------------------------------------------------
// Per-pair expert products (pair = token t, rank r; index t * used + r).  These re-read an
// expert's slice for every pair, like the reference's per-token kernel; the grouped
// tensor-core kernels replace them for the shapes those support.
// ---------------------------------------------------------------------------------------

// act[pair][f] = half(silu(gate) * up), gate = x[t] . Wg[e][f], up = x[t] . Wu[e][f].
__global__ void __launch_bounds__(Q8_SIMT_WARPS * 32u)
q8_expert_feed_kernel(const unsigned char *__restrict__ w_gate, const unsigned char *__restrict__ w_up,
                      unsigned int hidden, unsigned int ffn, const __half *__restrict__ x,
                      const unsigned int *__restrict__ ids, unsigned int experts, unsigned int tokens_max,
                      const unsigned int *tokens_dev, unsigned int used, __half *__restrict__ act)
{
    unsigned int tokens = tokens_max;
    if (tokens_dev != nullptr) {
        unsigned int live = *tokens_dev;
        tokens = live < tokens_max ? live : tokens_max;
    }
    unsigned int lane = threadIdx.x & 31u;
    unsigned int warp = threadIdx.x >> 5;
    unsigned long long stride = row_bytes(hidden);
    unsigned int f = blockIdx.x * Q8_SIMT_WARPS + warp;
    if (f >= ffn) {
        return;
    }
    for (unsigned int pair = blockIdx.y; pair < tokens * used; pair += gridDim.y) {
        unsigned int t = pair / used;
        unsigned int expert = ids[pair];
        if (expert >= experts) {
            continue; // a selection outside the expert table: left out, as in the grouped path
        }
        const unsigned char *gate_row = w_gate + ((unsigned long long)expert * ffn + f) * stride;
        const unsigned char *up_row = w_up + ((unsigned long long)expert * ffn + f) * stride;
        float gate[Q8_SIMT_TAKE];
        float up[Q8_SIMT_TAKE];
        simt_row<__half>(gate_row, hidden, x + (size_t)t * hidden, hidden, 1u, gate);
        simt_row<__half>(up_row, hidden, x + (size_t)t * hidden, hidden, 1u, up);
        if (lane == 0u) {
            float unit = gate[0] / (1.0f + expf(-gate[0]));
            act[(size_t)pair * ffn + f] = __float2half_rn(unit * up[0]);
        }
    }
}

// proj[pair][d] = act[pair] . Wd[e][d]
__global__ void __launch_bounds__(Q8_SIMT_WARPS * 32u)
q8_expert_down_kernel(const unsigned char *__restrict__ w_down, unsigned int hidden, unsigned int ffn,
                      const __half *__restrict__ act, const unsigned int *__restrict__ ids,
                      unsigned int experts, unsigned int tokens_max, const unsigned int *tokens_dev,
                      unsigned int used, float *__restrict__ proj)
{
    unsigned int tokens = tokens_max;
    if (tokens_dev != nullptr) {
        unsigned int live = *tokens_dev;
        tokens = live < tokens_max ? live : tokens_max;
    }
    unsigned int lane = threadIdx.x & 31u;
    unsigned int warp = threadIdx.x >> 5;
    unsigned long long stride = row_bytes(ffn);
    unsigned int d = blockIdx.x * Q8_SIMT_WARPS + warp;
    if (d >= hidden) {
        return;
    }
    for (unsigned int pair = blockIdx.y; pair < tokens * used; pair += gridDim.y) {
        unsigned int expert = ids[pair];
        if (expert >= experts) {
            continue;
        }
        const unsigned char *row = w_down + ((unsigned long long)expert * hidden + d) * stride;
        float sum[Q8_SIMT_TAKE];
        simt_row<__half>(row, ffn, act + (size_t)pair * ffn, ffn, 1u, sum);
        if (lane == 0u) {
            proj[(size_t)pair * hidden + d] = sum[0];
        }
    }
}

// out[t][d] = the ordered sum over ranks: rank 0 gives fmul(proj, p); each later rank adds
// fmul(proj, p) with a separate rounding of the product and of the sum.  A thread carries
// WIDTH neighbouring columns (WIDTH = 4: one 16-byte load of proj per rank); every column's
// chain of roundings is the one written above whatever the width.  The loads of up to eight
// ranks go out together before the chain of additions starts.
//
// `from` says where a pair's projection lies: in one array [tokens][used][hidden], or - expert
// parallel - in the array of the GPU that holds the pair's expert (experts dealt to `parts`
// GPUs as shard_rows deals rows: the first `extra` of them one expert more), at the row of
// the pair among all GPUs' pairs (first_pair + t * used + r).
template <typename YT, unsigned int WIDTH>
__global__ void q8_expert_sum_kernel(const __grid_constant__ ProjParts from, const float *prob,
                                     const unsigned int *ids, unsigned int tokens_max,
                                     const unsigned int *tokens_dev, unsigned int hidden,
                                     unsigned int experts, unsigned int used, YT *__restrict__ out)
{
    constexpr unsigned int kTogether = 8u;
    grid_dependency_wait();
    grid_launch_dependents();
    unsigned int tokens = tokens_max;
    if (tokens_dev != nullptr) {
        unsigned int live = *tokens_dev;
        tokens = live < tokens_max ? live : tokens_max;
    }
    // a block takes a part of a token's row, one step of its threads wide
    const unsigned int parts = (hidden + blockDim.x * WIDTH - 1u) / (blockDim.x * WIDTH);
    for (unsigned int item = blockIdx.x; item < tokens * parts; item += gridDim.x) {
        const unsigned int t = item / parts;
        const unsigned int d = ((item - t * parts) * blockDim.x + threadIdx.x) * WIDTH;
        if (d < hidden) {
            float sum[WIDTH];
#pragma unroll
            for (unsigned int i = 0; i < WIDTH; ++i) {
                sum[i] = 0.0f;
            }
            for (unsigned int r0 = 0; r0 < used; r0 += kTogether) {
                float value[kTogether][WIDTH];
                float p[kTogether];
#pragma unroll
                for (unsigned int q = 0; q < kTogether; ++q) {
                    const unsigned int r = r0 + q;
                    const unsigned int expert = r < used ? ids[(size_t)t * used + r] : 0xFFFFFFFFu;
                    // a selection outside the expert table has no probability and no projection
                    // (the product kernels leave it out): it adds nothing
                    p[q] = 0.0f;
#pragma unroll
                    for (unsigned int i = 0; i < WIDTH; ++i) {
                        value[q][i] = 0.0f;
                    }
                    if (expert < experts) {
                        p[q] = prob[(size_t)t * experts + expert];
                        const float *base = from.base[0];
                        if (from.parts > 1u) {
                            const unsigned int cut = from.extra * (from.share + 1u);
                            const unsigned int owner = expert < cut ? expert / (from.share + 1u)
                                                                    : from.extra + (expert - cut) / from.share;
                            base = from.base[owner];
                        }
                        const float *row = base + ((size_t)from.first_pair + (size_t)t * used + r) * hidden + d;
                        if (WIDTH == 4u) {
                            const float4 four = *reinterpret_cast<const float4 *>(row);
                            value[q][0] = four.x;
                            value[q][1 % WIDTH] = four.y;
                            value[q][2 % WIDTH] = four.z;
                            value[q][3 % WIDTH] = four.w;
                        } else {
#pragma unroll
                            for (unsigned int i = 0; i < WIDTH; ++i) {
                                value[q][i] = row[i];
                            }
                        }
                    }
                }
#pragma unroll
                for (unsigned int q = 0; q < kTogether; ++q) {
                    if (r0 + q < used) {
#pragma unroll
                        for (unsigned int i = 0; i < WIDTH; ++i) {
                            const float term = __fmul_rn(value[q][i], p[q]);
                            sum[i] = (r0 + q == 0u) ? term : __fadd_rn(sum[i], term);
                        }
                    }
                }
            }
#pragma unroll
            for (unsigned int i = 0; i < WIDTH; ++i) {
                store_out<YT>(out, (size_t)t * hidden + d + i, sum[i]);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------
// Launchers.
// ---------------------------------------------------------------------------------------
cudaError_t launch_dequant(cudaStream_t stream, const void *w, unsigned int k, unsigned int first_row,
                           unsigned int rows, void *out, bool overlap)
{
    unsigned long long blocks = (unsigned long long)rows * (k / Q8_BLOCK);
    if (blocks == 0ull) {
        return cudaSuccess;
    }
    const unsigned char *base = static_cast<const unsigned char *>(w) + row_bytes(k) * first_row;
    const unsigned long long pieces = blocks * 4ull;
    const int wide = (reinterpret_cast<uintptr_t>(out) & 15u) == 0u;
    // Four pieces per thread where that still gives every SM four blocks, and each block one run of the tensor:
    // 14336 x 4096 38.1 -> 32.9 us (5.5 TB/s), 20000 x 8192 104 -> 86.  (Blocks that come back for more, the
    // grid's width further on, keep as much in flight and take 39 us.)
    const unsigned long long many = (pieces + 256ull * Q8_DEQUANT_TOGETHER - 1ull) / (256ull * Q8_DEQUANT_TOGETHER);
    if (many >= 4ull * (unsigned long long)kSmCount) {
        const unsigned int grid = (unsigned int)(many < (1ull << 30) ? many : (1ull << 30));
        return launch_kernel_early(overlap, q8_dequant_kernel_many, grid, 256, 0, stream, base, blocks,
                                   static_cast<__half *>(out), wide);
    }
    const unsigned int grid = (unsigned int)((pieces + 255ull) / 256ull);
    return launch_kernel_early(overlap, q8_dequant_kernel, grid, 256, 0, stream, base, blocks, static_cast<__half *>(out), wide);
}

template <typename XT, typename YT>
static cudaError_t launch_gemv_simt_typed(cudaStream_t stream, const void *w, unsigned int n,
                                          unsigned int k, const void *x, unsigned int m,
                                          const unsigned int *m_dev, void *y, unsigned int epilogue)
{
    unsigned int want = (n + Q8_SIMT_WARPS - 1u) / Q8_SIMT_WARPS;
    unsigned int grid = want < kSmCount * 8u ? want : kSmCount * 8u;
    if (epilogue == kEpilogueStore) {
        return launch_kernel(q8_gemv_simt_kernel<XT, YT>, grid, Q8_SIMT_WARPS * 32u, 0, stream,
                             static_cast<const unsigned char *>(w), n, k, static_cast<const XT *>(x), m, m_dev,
                             static_cast<YT *>(y));
    }
    return launch_kernel(q8_gemv_simt_fused_kernel<XT, YT>, grid, Q8_SIMT_WARPS * 32u, 0, stream,
                         static_cast<const unsigned char *>(w), n, k, static_cast<const XT *>(x), m, m_dev,
                         static_cast<YT *>(y), epilogue);
}

cudaError_t launch_gemv_simt(cudaStream_t stream, const void *w, unsigned int n, unsigned int k,
                             const void *x, int x_bf16, unsigned int m, const unsigned int *m_dev,
                             void *y, int y_dtype, unsigned int epilogue, bool overlap)
{
    (void)overlap;
    if (n == 0u || m == 0u) {
        return cudaSuccess;
    }
    if ((epilogue == kEpilogueAdd && y_dtype != 0) || (epilogue == kEpilogueSwiglu && (n & 1u) != 0u)
        || epilogue > kEpilogueSwiglu) {
        return cudaErrorInvalidValue;
    }
#ifndef Q8_HOST_EMULATION
    if (warp_any_supports(w, Q8_TYPE_Q8_0, n, k, x, m)) {
        return launch_warp_any(stream, w, Q8_TYPE_Q8_0, n, k, x, x_bf16, m, m_dev, y, y_dtype, epilogue, overlap);
    }
#endif
#define Q8_CASE(XT, YD, YT)                                                                      \
    if (y_dtype == (YD)) {                                                                       \
        return launch_gemv_simt_typed<XT, YT>(stream, w, n, k, x, m, m_dev, y, epilogue);        \
    }
    if (x_bf16) {
        Q8_CASE(__nv_bfloat16, 0, float)
        Q8_CASE(__nv_bfloat16, 1, __half)
        Q8_CASE(__nv_bfloat16, 2, __nv_bfloat16)
    } else {
        Q8_CASE(__half, 0, float)
        Q8_CASE(__half, 1, __half)
        Q8_CASE(__half, 2, __nv_bfloat16)
    }
#undef Q8_CASE
    return cudaErrorInvalidValue;
}

cudaError_t launch_route(cudaStream_t stream, const void *x, const float *router, unsigned int tokens,
                         const unsigned int *tokens_dev, unsigned int hidden, unsigned int experts,
                         unsigned int used, float *prob, unsigned int *ids, unsigned int *status, bool overlap)
{
    if (tokens == 0u) {
        return cudaSuccess;
    }
#ifndef Q8_HOST_EMULATION
    if (route_tiles_fits(x, router, tokens, tokens_dev, hidden, experts)) {
        return launch_route_tiles(stream, x, router, tokens, hidden, experts, used, prob, ids, status, overlap);
    }
#else
    (void)status;
#endif
#ifdef Q8_HOST_EMULATION
    // a cluster of one block: it takes all experts
    const size_t emulated = (size_t)RouteShape<4u>::stride * hidden * sizeof(float);
    const unsigned int emulated_grid = (tokens + 3u) / 4u;
    return launch_kernel(q8_route_kernel, emulated_grid, Q8_ROUTE_THREADS, emulated, stream, static_cast<const __half *>(x),
                         router, tokens, tokens_dev, hidden, experts, used, prob, ids);
#else
    // Few tokens: two to a cluster of eight blocks, as long as the clusters have an SM per block (18 of them
    // are 144 blocks).  More: four to a cluster of eight, two blocks per SM (37 of them); then eight to a
    // cluster of four, which quarters the reads of the router and of the activations; eight tokens of a
    // row longer than 4096 no longer leave room for two blocks on an SM.  Latency bounds all three, so a
    // block has 16 warps of one or two experts each (measured against 8 warps of two or four; 128
    // experts, 2048 wide: 8 tokens 9.5 -> 7.2 us, 128 tokens 20.8 -> 13.0, 512 tokens 25.0 -> 22.6).
    // Few experts leave most warps of such a cluster without work, and every block of it reads the group's
    // activations: then a block takes all experts of four tokens by itself.  (Above 148 tokens q8_route.cu takes
    // most calls before they come here.)  (Clusters, and one block for all: 8
    // experts, 2048 wide, 512 tokens 15.4 us and 9.0, 4096 wide, 2048 tokens 160 and 24; 64 experts, 2048 wide, 512
    // tokens 17.2 and 29.3, 2048 tokens 64.1 and 57.2, 8192 wide, 300 tokens 74.3 and 53.2.)
    const bool few = tokens <= 36u;
    const bool alone = tokens > kSmCount && experts <= 64u && (experts <= 16u || hidden > 4096u || tokens > 1024u);
    const bool many = !few && !alone && tokens > kSmCount && hidden <= 4096u;
    const unsigned int group = few ? 2u : (many ? 8u : 4u);
    const unsigned int cluster = alone ? 1u : (many ? 4u : 8u);
    const unsigned int stride = few ? RouteShape<2u>::stride : (many ? RouteShape<8u>::stride : RouteShape<4u>::stride);
    const size_t smem = (size_t)stride * hidden * sizeof(float);
    if (smem > 200u * 1024u) {
        return cudaErrorInvalidValue;
    }
    unsigned int clusters = (tokens + group - 1u) / group;
    const unsigned int most = kSmCount * 4u / cluster;
    clusters = clusters < most ? clusters : most;
    static unsigned long long configured[3] = {0ull, 0ull, 0ull};
    void (*const kernels[3])(const __half *, const float *, unsigned int, const unsigned int *, unsigned int, unsigned int,
                             unsigned int, float *, unsigned int *) = {q8_route_kernel, q8_route_kernel_few,
                                                                       q8_route_kernel_many};
    const unsigned int which = few ? 1u : (many ? 2u : 0u);
    cudaError_t err = allow_shared_memory(kernels[which], 200u * 1024u, &configured[which]);
    if (err != cudaSuccess) {
        return err;
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(clusters * cluster, 1, 1);
    config.blockDim = dim3(Q8_ROUTE_GPU_THREADS, 1, 1);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attribute[2];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = cluster;
    attribute[0].val.clusterDim.y = 1;
    attribute[0].val.clusterDim.z = 1;
    attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attribute;
    config.numAttrs = overlap ? 2u : 1u;
    return cudaLaunchKernelEx(&config, kernels[which], static_cast<const __half *>(x), router, tokens, tokens_dev, hidden,
                              experts, used, prob, ids);
#endif
}

cudaError_t launch_expert_pairs_simt(cudaStream_t stream, const void *w_gate, const void *w_up,
                                     const void *w_down, unsigned int hidden, unsigned int ffn,
                                     const void *x, const unsigned int *ids, unsigned int experts,
                                     unsigned int tokens, const unsigned int *tokens_dev, unsigned int used,
                                     void *act, float *proj)
{
    unsigned int pairs = tokens * used;
    if (pairs == 0u) {
        return cudaSuccess;
    }
    unsigned int wave = pairs < 4096u ? pairs : 4096u;
    dim3 feed((ffn + Q8_SIMT_WARPS - 1u) / Q8_SIMT_WARPS, wave);
    dim3 down((hidden + Q8_SIMT_WARPS - 1u) / Q8_SIMT_WARPS, wave);
    cudaError_t err = launch_kernel(q8_expert_feed_kernel, feed, Q8_SIMT_WARPS * 32u, 0, stream,
                                    static_cast<const unsigned char *>(w_gate),
                                    static_cast<const unsigned char *>(w_up), hidden, ffn,
                                    static_cast<const __half *>(x), ids, experts, tokens, tokens_dev, used,
                                    static_cast<__half *>(act));
    if (err != cudaSuccess) {
        return err;
    }
    return launch_kernel(q8_expert_down_kernel, down, Q8_SIMT_WARPS * 32u, 0, stream,
                         static_cast<const unsigned char *>(w_down), hidden, ffn, static_cast<const __half *>(act),
                         ids, experts, tokens, tokens_dev, used, proj);
}

constexpr unsigned int kSumThreads = 64;

template <typename YT>
static cudaError_t expert_sum_launch(bool overlap, bool wide, cudaStream_t stream, const ProjParts &proj,
                                     const float *prob, const unsigned int *ids, unsigned int tokens,
                                     const unsigned int *tokens_dev, unsigned int hidden, unsigned int experts,
                                     unsigned int used, void *out)
{
    // A block per part of a token's row (see the kernel), sixteen blocks per SM at most.  Blocks of 64 threads, because the
    // down product before this leaves 6656 registers of an SM: the first blocks are there when it ends (routed experts, 512
    // tokens, 200.9 -> 199.6 us, 8 tokens 75.0 -> 73.7 against blocks of 256).
    const unsigned int step = kSumThreads * (wide ? 4u : 1u);
    const unsigned long long items = (unsigned long long)tokens * ((hidden + step - 1u) / step);
    const unsigned int grid = items < kSmCount * 16u ? (unsigned int)items : kSmCount * 16u;
    if (wide) {
        return launch_kernel_early(overlap, q8_expert_sum_kernel<YT, 4u>, grid, kSumThreads, 0, stream, proj, prob, ids, tokens, tokens_dev,
                             hidden, experts, used, static_cast<YT *>(out));
    }
    return launch_kernel_early(overlap, q8_expert_sum_kernel<YT, 1u>, grid, kSumThreads, 0, stream, proj, prob, ids, tokens, tokens_dev,
                         hidden, experts, used, static_cast<YT *>(out));
}

cudaError_t launch_expert_sum_parts(cudaStream_t stream, const ProjParts &proj, const float *prob,
                                    const unsigned int *ids, unsigned int tokens,
                                    const unsigned int *tokens_dev, unsigned int hidden, unsigned int experts,
                                    unsigned int used, void *out, int out_dtype, bool overlap)
{
    if (tokens == 0u) {
        return cudaSuccess;
    }
    // 16-byte loads of proj need rows of a multiple of four floats on a 16-byte boundary
    bool wide = (hidden % 4u) == 0u;
    for (unsigned int i = 0; i < (proj.parts > 1u ? proj.parts : 1u); ++i) {
        wide = wide && (reinterpret_cast<uintptr_t>(proj.base[i]) & 15u) == 0u;
    }
    if (out_dtype == 0) {
        return expert_sum_launch<float>(overlap, wide, stream, proj, prob, ids, tokens, tokens_dev, hidden, experts,
                                        used, out);
    }
    if (out_dtype == 1) {
        return expert_sum_launch<__half>(overlap, wide, stream, proj, prob, ids, tokens, tokens_dev, hidden, experts,
                                         used, out);
    }
    if (out_dtype == 2) {
        return expert_sum_launch<__nv_bfloat16>(overlap, wide, stream, proj, prob, ids, tokens, tokens_dev, hidden,
                                                experts, used, out);
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_expert_sum(cudaStream_t stream, const float *proj, const float *prob,
                              const unsigned int *ids, unsigned int tokens,
                              const unsigned int *tokens_dev, unsigned int hidden, unsigned int experts,
                              unsigned int used, void *out, int out_dtype, bool overlap)
{
    ProjParts one = {};
    one.base[0] = proj;
    one.parts = 1u;
    return launch_expert_sum_parts(stream, one, prob, ids, tokens, tokens_dev, hidden, experts, used, out,
                                   out_dtype, overlap);
}

} // namespace q8
