// Instructions of the kernels that multiply on the warp-level tensor path (q8_decode_warp.cu and
// its relatives), one small function each.
#pragma once

#include <stdint.h>

namespace q8 {

// D (16 x 8 floats) += A (16 x 16 halves) * B (16 x 8 halves).  Lane = 4 g + t holds of A the
// halves {2t, 2t+1} of rows g (a0) and g + 8 (a1) and {2t+8, 2t+9} of the same rows (a2, a3), of B
// the halves {2t, 2t+1} (b0) and {2t+8, 2t+9} (b1) of column g, of D the columns 2t, 2t+1 of rows
// g (d0, d1) and g + 8 (d2, d3).  Volatile: the hand-over of a stage counts on its place.
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Arrive on the cluster's barrier without ordering any memory access: tells the other blocks that
// this one has started.  (The releasing form waits for what the thread has in flight.)
__device__ __forceinline__ void cluster_arrive_relaxed()
{
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}

// The same with bfloat16 operands.
__device__ __forceinline__ void mma_16816_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// An ordinary thread's own copy of 16 bytes, global to shared; the copies before a commit form a
// group, and a wait leaves at most `LEFT` of the latest groups on their way.
__device__ __forceinline__ void copy_async_16(uint32_t dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void copy_async_commit()
{
    asm volatile("cp.async.commit_group;" ::: "memory");
}

template <int LEFT>
__device__ __forceinline__ void copy_async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

__device__ __forceinline__ void ld_shared_v2(uint32_t addr, uint32_t &a, uint32_t &b)
{
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(a), "=r"(b) : "r"(addr) : "memory");
}

__device__ __forceinline__ void st_shared_v2(uint32_t addr, uint32_t a, uint32_t b)
{
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}

} // namespace q8
