// The end of the expert router for one token: the softmax over its logits and the experts in order of probability.
// Shared by the router kernels (q8_simt.cu, q8_route.cu).
#pragma once

#include "q8_common.cuh"

#include <math_constants.h>
#include <stdint.h>

namespace q8 {

#define Q8_ROUTE_EXPERTS 256u

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
// of groups of 8 in pairs 32.)
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
