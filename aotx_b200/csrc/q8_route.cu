// The expert router on whole tiles of shared memory: logits of a group of tokens against all experts, the softmax, the
// experts in order.  Every float sum runs in the order of the reference kernel (cuda/model/experts.cu:10-75): 32
// chains of fused multiply-adds 32 positions apart, added in a tree of halves 16, 8, 4, 2, 1 apart.
//
// What bounds it: the operands' way from shared memory into registers and the order of the chains, 64 steps one after the
// other at 2048 wide; the float multiply-adds themselves (512 tokens, 128 experts, 2048 wide: 134 million) take 4.2 us on
// 128 SMs.  So:
//
//   * A cluster of up to eight blocks takes a group of 4, 8 or 16 tokens, each block 32 of the experts (a block by itself
//     16, where there are no more).  Rows of router and of x come by asynchronous copies of 128 positions into a
//     ring; nothing is converted or laid out on the way.  (Bulk copies of a row each, issued by the lanes of one
//     warp, take 80 cycles apiece: 8 tokens, 16 experts a block, 9.9 us against 6.9 by 16-byte copies.)
//   * A warp is two halves of 16 lanes, a lane two neighbouring chains.  A half takes TT tokens by ET experts, so a
//     step of 32 positions is ET + TT loads (router values as two floats, the same for both halves; x as two
//     halves) for 2 * ET * TT multiply-adds, which are issued in pairs (fma.rn.f32x2: each is the rounded
//     multiply-add it is alone).  Sixteen warps of half the tile are slower (18.4 us against 16.8 at 512 tokens).
//   * The tree's first four steps add lanes of a half; of the sums that two lanes exchange each keeps one half, so that
//     32 sums take 30 exchanges where one after the other took 128.
//   * Finished logits go to the shared memory of the block that chooses for the token, by stores that count themselves on
//     its barrier (st.async).
#include "q8_launch.h"
#include "q8_route.cuh"
#include "q8_warp_ptx.cuh"

#include <atomic>

namespace q8 {

constexpr uint32_t kRouteWarps = 8;
constexpr uint32_t kRouteThreads = kRouteWarps * 32u;
constexpr uint32_t kRouteStep = 32;                // positions
constexpr uint32_t kRouteChunk = 128;              // positions of a stage of the ring
constexpr uint32_t kRouteRowBytes = kRouteChunk * 4u;
// Rows of x of the two halves of a warp are neighbours and start 64 bytes apart modulo 128: a load of both meets 32 banks.
constexpr uint32_t kRouteXBytes = kRouteChunk * 2u + 64u;
constexpr uint32_t kRouteMaxStages = 32;
constexpr uint32_t kRouteBarBytes = 8u * kRouteMaxStages + 16u;
constexpr uint32_t kRouteFewExperts = 16;          // one set of them to a block, no cluster
constexpr uint32_t kRouteMostBytes = 200u * 1024u; // of shared memory, one block per SM
constexpr uint32_t kRouteHalfBytes = (228u * 1024u) / 2u - 1536u;    // two blocks

struct RouteArgs {
    const __half *x;
    const float *router;
    float *prob;
    unsigned int *ids;
    unsigned int *status;
    uint32_t tokens, hidden, experts, used;
    uint32_t stages;
};

__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

__device__ __forceinline__ uint64_t pair_of(float low, float high)
{
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(low), "f"(high));
    return d;
}

__device__ __forceinline__ float2 two_of(uint64_t pair)
{
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(pair));
    return v;
}

// Arrive on a barrier of this block when the copies that this thread has asked for are there.
__device__ __forceinline__ void copy_async_arrive(uint32_t bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

// `N` tokens and experts' pairs of chains of a half's 16 lanes, added over the lanes; what is left per lane, at
// index `at` of the N and after it: N / 16 sums, or one (of several lanes, `mine` says whose it is).
template <uint32_t N>
__device__ __forceinline__ void route_tree(uint64_t (&sum)[N], uint32_t lane, uint32_t &at, bool &mine)
{
    at = 0u;
    mine = true;
    uint32_t n = N;
#pragma unroll
    for (uint32_t step = 8u; step != 0u; step >>= 1) {
        const bool upper = (lane & step) != 0u;
        if (n > 1u) {
            n /= 2u;
#pragma unroll
            for (uint32_t i = 0; i < N / 2u; ++i) {
                if (i < n) {
                    const uint64_t give = upper ? sum[i] : sum[i + n];
                    const uint64_t keep = upper ? sum[i + n] : sum[i];
                    const float2 got = two_of(__shfl_xor_sync(0xFFFFFFFFu, give, step));
                    const float2 own = two_of(keep);
                    sum[i] = pair_of(own.x + got.x, own.y + got.y);
                }
            }
            at += upper ? n : 0u;
        } else {
            const float2 got = two_of(__shfl_xor_sync(0xFFFFFFFFu, sum[0], step));
            const float2 own = two_of(sum[0]);
            sum[0] = pair_of(own.x + got.x, own.y + got.y);
            mine = mine && !upper;
        }
    }
}

// TT tokens by ET experts per half of a warp; SET experts of a block, SET / ET warps side by side over them.
template <uint32_t TT, uint32_t ET, uint32_t SET>
struct RouteTile {
    static constexpr uint32_t across = SET / ET;                              // warps over the experts
    static constexpr uint32_t tokens = 2u * TT * (kRouteWarps / across);      // of a group
    static constexpr uint32_t stage_bytes = SET * kRouteRowBytes + tokens * kRouteXBytes;
    static constexpr uint32_t left = TT * ET >= 16u ? TT * ET / 16u : 1u;     // sums per lane after the tree
    static_assert(kRouteWarps % across == 0u, "whole warps over the tokens");
};

template <uint32_t TT, uint32_t ET, uint32_t SET>
__global__ void __launch_bounds__(kRouteThreads, 2)
q8_route_kernel_tiles(const RouteArgs args)
{
    using S = RouteTile<TT, ET, SET>;
    extern __shared__ __align__(128) unsigned char route_smem_[];
    __shared__ uint32_t abort_flag_;
    volatile uint32_t *abort_flag = &abort_flag_;
    const uint32_t ring = smem_u32(route_smem_);
    const uint32_t full = ring + args.stages * S::stage_bytes;
    const uint32_t gathered = full + 8u * kRouteMaxStages;
    float *const logits = reinterpret_cast<float *>(route_smem_ + args.stages * S::stage_bytes + kRouteBarBytes);
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t csize = cluster_nctarank();
    const uint32_t crank = cluster_ctarank();
    const uint32_t chunks = (args.hidden + kRouteChunk - 1u) / kRouteChunk;
    const uint32_t first_expert = crank * SET;

    grid_dependency_wait();
    grid_launch_dependents();
    const uint32_t t0 = blockIdx.x / csize * S::tokens;
    const uint32_t group = args.tokens - t0 < S::tokens ? args.tokens - t0 : S::tokens;
    const uint32_t chosen_here = group > crank ? (group - crank + csize - 1u) / csize : 0u;   // tokens crank, crank + csize, ..
    if (threadIdx.x == 0u) {
        for (uint32_t i = 0; i < args.stages; ++i) {
            mbar_init(full + 8u * i, kRouteThreads);
        }
        mbar_init(gathered, 1u);
        *abort_flag = 0u;
        mbar_init_fence();
        mbar_expect_tx(gathered, chosen_here * args.experts * 4u);
    }
    __syncthreads();
    if (csize > 1u) {
        // the barriers of every block are there before a logit is counted on them (waited for below)
        cluster_arrive_relaxed();
    }

    // Copies of the next chunk into its stage, 16 bytes per lane and neighbouring lanes neighbouring pieces: a warp takes a
    // row of the router, or two of x, at a time.  Rows past the last expert or token repeat the last one; their
    // sums are not used.
    uint32_t in_st = 0u, in_chunk = 0u;
    auto fetch = [&]() {
        const uint32_t left = args.hidden - in_chunk * kRouteChunk;
        const uint32_t to = ring + in_st * S::stage_bytes;
        if (lane * 4u < left) {
            const float *from = args.router + in_chunk * kRouteChunk + lane * 4u;
#pragma unroll
            for (uint32_t r = 0; r < SET; r += kRouteWarps) {
                const uint32_t e = first_expert + r + warp;
                copy_async_16(to + (r + warp) * kRouteRowBytes + lane * 16u,
                              from + (size_t)(e < args.experts ? e : args.experts - 1u) * args.hidden);
            }
        }
        const uint32_t piece = lane & 15u;
        if (piece * 8u < left) {
            const __half *from = args.x + (size_t)t0 * args.hidden + in_chunk * kRouteChunk + piece * 8u;
            for (uint32_t t = threadIdx.x / 16u; t < S::tokens; t += kRouteThreads / 16u) {
                copy_async_16(to + SET * kRouteRowBytes + t * kRouteXBytes + piece * 16u,
                              from + (size_t)(t < group ? t : group - 1u) * args.hidden);
            }
        }
        copy_async_arrive(full + 8u * in_st);
        in_st = in_st + 1u == args.stages ? 0u : in_st + 1u;
        ++in_chunk;
    };
    for (uint32_t i = 0; i < args.stages; ++i) {
        fetch();
    }

    const uint32_t part = lane & 15u;                                       // the lane's chains: 2 * part and the next
    const uint32_t expert0 = warp % S::across * ET;                         // of the block's
    const uint32_t token0 = warp / S::across * 2u * TT + (lane >> 4);       // and every second one after it
    uint64_t sum[TT * ET];
#pragma unroll
    for (uint32_t i = 0; i < TT * ET; ++i) {
        sum[i] = 0ull;
    }
    uint32_t st = 0u, ph = 0u;
    for (uint32_t chunk = 0; chunk < chunks; ++chunk) {
        // (where the wait runs out the sums are wrong, but every thread goes on to the same barriers)
        mbar_wait_hot(full + 8u * st, ph, abort_flag, args.status);
        __syncwarp();
        const uint32_t left = args.hidden - chunk * kRouteChunk;
        const uint32_t steps = (left < kRouteChunk ? left : kRouteChunk) / kRouteStep;
        const unsigned char *r_at = route_smem_ + st * S::stage_bytes + expert0 * kRouteRowBytes + part * 8u;
        const unsigned char *x_at = route_smem_ + st * S::stage_bytes + SET * kRouteRowBytes + token0 * kRouteXBytes + part * 4u;
#pragma unroll (TT * ET >= 32u ? 2 : 4)
        for (uint32_t step = 0; step < steps; ++step) {
            uint64_t r[ET];
            __half2 two[TT];
#pragma unroll
            for (uint32_t e = 0; e < ET; ++e) {
                r[e] = *reinterpret_cast<const uint64_t *>(r_at + step * (kRouteStep * 4u) + e * kRouteRowBytes);
            }
#pragma unroll
            for (uint32_t t = 0; t < TT; ++t) {
                two[t] = *reinterpret_cast<const __half2 *>(x_at + step * (kRouteStep * 2u) + 2u * t * kRouteXBytes);
            }
#pragma unroll
            for (uint32_t t = 0; t < TT; ++t) {
                const float2 xv = __half22float2(two[t]);
                const uint64_t xx = pair_of(xv.x, xv.y);
#pragma unroll
                for (uint32_t e = 0; e < ET; ++e) {
                    // the reference's own expression, which compiles to a fused multiply-add
                    sum[t * ET + e] = fma_pair(r[e], xx, sum[t * ET + e]);
                }
            }
        }
        if (chunk + args.stages < chunks) {
            __syncthreads();     // everyone has read the stage
            fetch();
        }
        st = st + 1u == args.stages ? 0u : st + 1u;
        ph ^= st == 0u ? 1u : 0u;
    }
    copy_async_wait_all();       // (there are none left unless a wait ran out)
    uint32_t at;
    bool mine;
    route_tree(sum, lane, at, mine);
    if (csize > 1u) {
        __syncwarp();
        cluster_wait_acquire();
    }
#pragma unroll
    for (uint32_t i = 0; i < S::left; ++i) {
        const uint32_t t = token0 + 2u * ((at + i) / ET);
        const uint32_t e = first_expert + expert0 + (at + i) % ET;
        if (mine && t < group && e < args.experts) {
            const float2 chains = two_of(sum[i]);
            const uint32_t slot = smem_u32(logits + (t / csize) * args.experts + e);
            store_counted(mapa_shared(slot, t % csize), chains.x + chains.y, mapa_shared(gathered, t % csize));
        }
    }
    // -------------------------------------------------------------------- a warp per token of this block
    if (warp >= chosen_here) {
        return;
    }
    if (!__all_sync(0xFFFFFFFFu, mbar_wait_counted(gathered, 0u, abort_flag, args.status))) {
        // Logits are missing, and may still be on their way into this block's shared memory: it stays until every
        // other thread of the cluster has ended (or come here).
        cluster_arrive_relaxed();
        cluster_wait_acquire();
        return;
    }
    for (uint32_t i = warp; i < chosen_here; i += kRouteWarps) {
        route_choose(logits + i * args.experts, t0 + crank + csize * i, args.experts, args.used, args.prob, args.ids);
    }
}

template <uint32_t TT, uint32_t ET, uint32_t SET>
static cudaError_t launch_route_sized(cudaStream_t stream, RouteArgs &args, bool deep, bool overlap)
{
    using S = RouteTile<TT, ET, SET>;
    static unsigned long long configured = 0ull;
    cudaError_t err = allow_shared_memory(q8_route_kernel_tiles<TT, ET, SET>, kRouteMostBytes, &configured);
    if (err != cudaSuccess) {
        return err;
    }
    const uint32_t cluster = (args.experts + SET - 1u) / SET;
    const uint32_t groups = (args.tokens + S::tokens - 1u) / S::tokens;
    const uint32_t chunks = (args.hidden + kRouteChunk - 1u) / kRouteChunk;
    const uint32_t logits = (S::tokens + cluster - 1u) / cluster * args.experts * 4u;
    const uint32_t most = deep ? kRouteMostBytes : kRouteHalfBytes;
    const uint32_t fits = (most - kRouteBarBytes - logits) / S::stage_bytes;
    args.stages = chunks < fits ? chunks : fits;
    args.stages = args.stages < kRouteMaxStages ? args.stages : kRouteMaxStages;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(groups * cluster, 1, 1);
    config.blockDim = dim3(kRouteThreads, 1, 1);
    config.dynamicSmemBytes = args.stages * S::stage_bytes + kRouteBarBytes + logits;
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
    return cudaLaunchKernelEx(&config, q8_route_kernel_tiles<TT, ET, SET>, args);
}

// How many clusters of `cluster` blocks run at the same time: low half a block per SM, high half two.  What a chip's
// parts have room for differs from one to the next, so it is asked for, once per device and size.
static uint32_t route_clusters(uint32_t cluster)
{
    static std::atomic<uint32_t> known[64][Q8_ROUTE_EXPERTS / 32u + 1u];
    static unsigned long long configured = 0ull;
    auto kernel = q8_route_kernel_tiles<4u, 8u, 32u>;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || allow_shared_memory(kernel, kRouteMostBytes, &configured) != cudaSuccess) {
        return 0u;
    }
    uint32_t at_once = known[device & 63][cluster].load(std::memory_order_relaxed);
    if (at_once == 0u) {
        cudaLaunchAttribute attribute[1];
        attribute[0].id = cudaLaunchAttributeClusterDimension;
        attribute[0].val.clusterDim.x = cluster;
        attribute[0].val.clusterDim.y = 1;
        attribute[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t config = {};
        config.gridDim = dim3(cluster, 1, 1);
        config.blockDim = dim3(kRouteThreads, 1, 1);
        config.attrs = attribute;
        config.numAttrs = 1u;
        int alone = 0, paired = 0;
        config.dynamicSmemBytes = kRouteMostBytes;
        cudaError_t err = cudaOccupancyMaxActiveClusters(&alone, kernel, &config);
        config.dynamicSmemBytes = kRouteHalfBytes;
        err = err == cudaSuccess ? cudaOccupancyMaxActiveClusters(&paired, kernel, &config) : err;
        if (err != cudaSuccess) {
            (void)cudaGetLastError();     // the launch does without
            return 0u;
        }
        at_once = (uint32_t)alone | ((uint32_t)paired << 16);
        known[device & 63][cluster].store(at_once, std::memory_order_relaxed);
    }
    return at_once;
}

// Only where the host knows the number of tokens: the tile of a group costs the same for one token as for all of them, and a
// launch for a maximum of which few are live was slower (us, other kernels and this one; maximum, live, experts x 2048: 512, 1,
// 128 14.5 and 16.6; 2048, 64, 8 7.4 and 15.0; 65536, 64, 256 23.8 and 56.4).
bool route_tiles_fits(const void *x, const float *router, unsigned int tokens, const unsigned int *tokens_dev,
                      unsigned int hidden, unsigned int experts)
{
    return tokens_dev == nullptr && route_tiles_pay(tokens, hidden, experts) && (hidden % kRouteStep) == 0u
        && (reinterpret_cast<uintptr_t>(x) & 15u) == 0u && (reinterpret_cast<uintptr_t>(router) & 15u) == 0u;
}

cudaError_t launch_route_tiles(cudaStream_t stream, const void *x, const float *router, unsigned int tokens,
                               unsigned int hidden, unsigned int experts, unsigned int used, float *prob, unsigned int *ids,
                               unsigned int *status, bool overlap)
{
    RouteArgs args = {};
    args.x = static_cast<const __half *>(x);
    args.router = router;
    args.prob = prob;
    args.ids = ids;
    args.status = status;
    args.tokens = tokens;
    args.hidden = hidden;
    args.experts = experts;
    args.used = used;
    const bool wide = experts > kRouteFewExperts;
    const uint32_t at_once = route_clusters(wide ? (experts + 31u) / 32u : 1u);
    const RoutePlan plan = route_plan(tokens, wide ? 4u : 8u, at_once & 0xFFFFu, at_once >> 16);
    if (wide) {
        return plan.group == 4u   ? launch_route_sized<1u, 8u, 32u>(stream, args, plan.deep, overlap)
               : plan.group == 8u ? launch_route_sized<2u, 8u, 32u>(stream, args, plan.deep, overlap)
                                  : launch_route_sized<4u, 8u, 32u>(stream, args, plan.deep, overlap);
    }
    return plan.group == 8u ? launch_route_sized<1u, 8u, 16u>(stream, args, plan.deep, overlap)
                            : launch_route_sized<2u, 8u, 16u>(stream, args, plan.deep, overlap);
}

} // namespace q8
