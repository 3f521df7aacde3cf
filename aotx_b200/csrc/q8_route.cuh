// What the router kernels share (q8_simt.cu, q8_route.cu): the host's rules between and for them, and the end of the router for
// one token, the softmax over its logits and the experts in order of probability.
#pragma once

#include "q8_common.cuh"

#include <math_constants.h>
#include <stdint.h>

namespace q8 {

#define Q8_ROUTE_EXPERTS 256u

// Whether the router runs on q8_route_kernel_tiles, for the number of tokens that it has.  Where the lines lie (us, the other
// kernels and this one, experts x width):
//   * Up to 148 tokens the others have an SM or more per token: 64 x 2048, 128 tokens 9.6 and 11.2; 149 14.0 and 11.2; 512 16.2
//     and 12.2; 32 x 1024, 128 tokens 6.6 and 7.2, 149 10.2 and 7.2; 256 x 4096, 400 tokens 74 and 49.  One line for all
//     numbers of experts, although 128 x 2048 have theirs below it: 128 tokens 12.9 and 11.3, 149 15.1 and 12.4, 256 18.3 and 12.4,
//     512 22.0 and 17.0, 2048 82 and 54.  (33 to 72 experts fill little more than half of their blocks: 65 to 72 of 1536 to 2048,
//     365 to 592 tokens, are a tenth slower at most, the same of 2560 or 4096 half the time of the others.)
//   * Few experts leave the tiles, 16 of them, without work, and one block of the others takes all of four tokens (two such
//     blocks to an SM: 1184 tokens at once).  16 x 2048, 300 tokens 7.9 and 8.2, 700 11.9 and 10.7, 2048 22 and 15; 16 x
//     4096, 700 18.2 and 18.5, 2048 35 and 24; 12 x 4096, 1184 tokens 1.2 times as long, 2400 the same; 8 x 4096, 1024 12.8 and
//     18.7, 2048 24 and 24; 2 x 6144, 593 2.2 times as long.
//   * The same block takes up to 64 experts where rows are long or tokens many (launch_route): up to 47 experts the tiles are
//     faster from its second turn on only.  17 x 8192, 149 to 592 tokens 26 and 38, 593 49 and 40; 32 x 8192 30 and 37, 593 59 and
//     40; 24 x 5120 or 6144, 149 to 592 tokens 1.3 times as long, 33 x 6144, 1500 1.1, 2048 0.9; 17 x 2048, 1184 tokens
//     1.13, 1500 0.9; 48 x 8192, 149 to 592 tokens 41 and 38.
__host__ __device__ inline bool route_tiles_pay(uint32_t tokens, uint32_t hidden, uint32_t experts)
{
    constexpr uint32_t kSms = 148u;
    if (experts <= 16u) {
        return experts > 12u && tokens > (hidden <= 2048u ? 4u : 8u) * kSms;
    }
    if (experts < 48u && (hidden > 4096u || tokens > 1024u)) {
        return tokens > (hidden <= 4096u ? 8u : hidden <= 6912u ? 12u : 4u) * kSms;
    }
    return tokens > kSms;
}

// How q8_route_kernel_tiles divides the tokens: rows of x to a group, and whether its rings are as deep as one block of an SM
// has room for, or half of that, for two.
struct RoutePlan {
    uint32_t group;
    bool deep;
};

// The fewest tokens to a group (`smallest`, doubled up to 16) with which all clusters run at the same time, a block per SM:
// `alone` is how many do, `paired` how many with two blocks to an SM.  Where not even groups of 16 do, groups of 8 if they
// run at the same time in pairs, else groups of 16.  (Clusters of five blocks and more leave SMs of each part of the chip
// over - 15 clusters of seven or eight, not 21 or 18 - and one cluster behind the others takes as long as all of them: 256 experts
// x 4096, 256 tokens, 16 clusters of groups of 16, 59 us alone, 49 in pairs, which share SMs while others have none; 32 clusters
// of groups of 8 in pairs 32.  A cluster more than run in pairs is still a second turn: 256 experts of up to 2048, 529 to
// 545 tokens, 1.1 times the other kernels' time, 560 0.9.)
__host__ __device__ inline RoutePlan route_plan(uint32_t tokens, uint32_t smallest, uint32_t alone, uint32_t paired)
{
    for (uint32_t group = smallest; group <= 16u; group *= 2u) {
        if ((tokens + group - 1u) / group <= alone) {
            return {group, true};
        }
    }
    return {(tokens + 7u) / 8u <= paired ? 8u : 16u, false};
}

// The largest value over the warp and the lowest index that has it.  Every value is a probability or -1, so
// their bits order them as signed integers do: two reductions in place of ten shuffles.
__device__ __forceinline__ void largest_first(float *best, float *best_at)
{
#ifdef Q8_HOST_EMULATION
    for (unsigned int step = 16u; step != 0u; step >>= 1) {
        const float other = __shfl_xor_sync(0xFFFFFFFFu, *best, step);
        const float other_at = __shfl_xor_sync(0xFFFFFFFFu, *best_at, step);
        if (other > *best || (other == *best && other_at < *best_at)) {
            *best = other;
            *best_at = other_at;
        }
    }
#else
    const int most = __reduce_max_sync(0xFFFFFFFFu, __float_as_int(*best));
    const unsigned int mine = __float_as_int(*best) == most ? (unsigned int)*best_at : 0xFFFFFFFFu;
    *best_at = (float)__reduce_min_sync(0xFFFFFFFFu, mine);
    *best = __int_as_float(most);
#endif
}

// By one warp.  Every sum runs in the reference kernel's order (cuda/model/experts.cu:10-75), so the probabilities are
// the same floats; equal ones come out the lower index first.
__device__ __forceinline__ void route_choose(const float *logits, unsigned int t, unsigned int experts, unsigned int used,
                                             float *__restrict__ prob, unsigned int *__restrict__ ids)
{
    constexpr unsigned int kPerLane = Q8_ROUTE_EXPERTS / 32u;
    const unsigned int lane = threadIdx.x & 31u;
    // lane holds experts lane, lane + 32, ..
    float value[kPerLane];
    float sum[kPerLane];
    float top = -CUDART_INF_F;
#pragma unroll
    for (unsigned int j = 0; j < kPerLane; ++j) {
        const unsigned int e = lane + 32u * j;
        value[j] = e < experts ? logits[e] : -CUDART_INF_F;
        top = fmaxf(top, value[j]);
    }
    for (unsigned int step = 16u; step != 0u; step >>= 1) {
        top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, step));
    }
#pragma unroll
    for (unsigned int j = 0; j < kPerLane; ++j) {
        value[j] = lane + 32u * j < experts ? expf(value[j] - top) : 0.0f;
        sum[j] = value[j];
    }
    // the reference's tree over 256 places: halves 128 apart, 64, 32, then within the warp
#pragma unroll
    for (unsigned int half = kPerLane / 2u; half != 0u; half >>= 1) {
#pragma unroll
        for (unsigned int j = 0; j < half; ++j) {
            sum[j] += sum[j + half];
        }
    }
    for (unsigned int step = 16u; step != 0u; step >>= 1) {
        sum[0] += __shfl_down_sync(0xFFFFFFFFu, sum[0], step);
    }
    // lane 0 holds the whole sum: hand it round (every other lane puts in a zero)
    float total = lane == 0u ? sum[0] : 0.0f;
    for (unsigned int step = 16u; step != 0u; step >>= 1) {
        total += __shfl_xor_sync(0xFFFFFFFFu, total, step);
    }
#pragma unroll
    for (unsigned int j = 0; j < kPerLane; ++j) {
        const unsigned int e = lane + 32u * j;
        value[j] /= total;
        if (e < experts) {
            prob[(size_t)t * experts + e] = value[j];
        } else {
            value[j] = -1.0f; // below every probability
        }
    }
    // the largest that is left, ties to the lower index, `used` times over
    for (unsigned int rank = 0; rank < used; ++rank) {
        float best = -1.0f;
        float best_at = (float)rank;   // an index as a float: exact, at most 255
#pragma unroll
        for (unsigned int j = 0; j < kPerLane; ++j) {
            if (value[j] > best) {
                best = value[j];
                best_at = (float)(lane + 32u * j);
            }
        }
        largest_first(&best, &best_at);
        const unsigned int chosen = (unsigned int)best_at;
#pragma unroll
        for (unsigned int j = 0; j < kPerLane; ++j) {
            if (lane + 32u * j == chosen) {
                value[j] = -1.0f;
            }
        }
        if (lane == 0u) {
            ids[(size_t)t * used + rank] = chosen;
        }
    }
}

} // namespace q8
