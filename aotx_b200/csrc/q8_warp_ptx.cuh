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

// All of this thread's copies, committed or not.
__device__ __forceinline__ void copy_async_wait_all()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// A barrier's memory may be used for something else, another barrier for instance.
__device__ __forceinline__ void mbar_inval(uint32_t bar)
{
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

// Ask for a line into L2.  It is a hint that reads nothing: a later write to the line is seen by later reads.
__device__ __forceinline__ void prefetch_l2(const void *at)
{
    asm volatile("prefetch.global.L2 [%0];" ::"l"(at) : "memory");
}

// An approximate reciprocal (within an ulp).
__device__ __forceinline__ float rcp_approx(float v)
{
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

// Add to a word with release at GPU scope: what this thread (and those it synchronised with) wrote before is there
// for who reads the word with acquire.
__device__ __forceinline__ void red_release_gpu_add(unsigned int *p, uint32_t v)
{
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ void ld_shared_v2(uint32_t addr, uint32_t &a, uint32_t &b)
{
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(a), "=r"(b) : "r"(addr) : "memory");
}

__device__ __forceinline__ void st_shared_v2(uint32_t addr, uint32_t a, uint32_t b)
{
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}

// 32 lanes x 16 columns: thread t of the warp writes lane (base lane + t).
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t *v)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
                 "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
                   "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
                 : "memory");
}

// ---- two blocks of a cluster on one tensor-core tile (cta_group::2) ---------------------------------
// The instructions below address both blocks: tensor memory columns and shared-memory offsets mean
// the same place in each of the two.

__device__ __forceinline__ void pair_tmem_alloc(uint32_t smem_result, uint32_t columns)
{
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_result), "r"(columns)
                 : "memory");
}

__device__ __forceinline__ void pair_tmem_relinquish()
{
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void pair_tmem_dealloc(uint32_t taddr, uint32_t columns)
{
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(columns) : "memory");
}

// D (256 x N: each block 128 rows) (+)= A (each block's 128 rows, in its own tensor memory) * B (each block N / 2
// columns, in its own shared memory), 16 deep.
__device__ __forceinline__ void pair_mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                                uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Arrive on the barrier at this offset in both blocks when every MMA this thread issued has finished.
__device__ __forceinline__ void pair_commit(uint32_t bar)
{
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
        ::"r"(bar), "h"((unsigned short)3)
        : "memory");
}

// A tensor copy into this block's shared memory that signals a barrier of either block of the pair (`bar`:
// an address of mapa_shared).
__device__ __forceinline__ void pair_tma_load_2d(uint32_t dst, const void *tmap, uint32_t bar, int c0, int c1)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"((uint64_t)tmap), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}

// Arrive on a barrier of either block (an address of mapa_shared).  Without cluster-scope release on purpose:
// what changes hands here is tensor memory, which tcgen05.wait and the tcgen05 fences order; a release
// at cluster scope holds the warp for 2400 cycles until its other memory operations are done.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

// A float into the shared memory of a block of the cluster, counted on that block's barrier `bar`
// (addresses of mapa_shared).
__device__ __forceinline__ void store_counted(uint32_t addr, float v, uint32_t bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(__float_as_uint(v)),
                 "r"(bar)
                 : "memory");
}

} // namespace q8
