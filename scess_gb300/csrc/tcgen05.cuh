// tcgen05 / TMEM / TMA / cluster helpers (inline PTX for sm_103a) shared by the
// tensor-core GEMMs: the split FP16 form (gemm_tc.cu) and the FP64 form on BF16
// slices (gemm_slice.cu).
#pragma once
#include <cuda.h>

#include <cstdint>

#include "mbarrier.cuh"

namespace scess {

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *tm, int x, int y,
                                            uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
      "%3}], [%4];" ::"r"(smem_u32(dst)),
      "l"((uint64_t)tm), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

// Two-SM (cluster pair) forms.  The pair's even CTA issues the MMAs; its
// shared-memory barriers count both CTAs' copies and both CTAs' drains.
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_id_x() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t nclusters_x() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%nclusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of the same shared-memory object in the pair's rank-0 CTA.
__device__ __forceinline__ uint32_t leader_addr(const void *p) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
  return r;
}
// TMA load into this CTA's shared memory whose completion is counted on a
// barrier of either CTA of the pair (cluster address).
__device__ __forceinline__ void tma_load_2d_pair(void *dst, const CUtensorMap *tm, int x, int y,
                                                 uint32_t bar_cluster) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], "
      "[%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"((uint64_t)tm), "r"(x), "r"(y), "r"(bar_cluster)
      : "memory");
}
// Arrival on a barrier of either CTA of the pair.  Release at CTA scope: it
// only has to follow this thread's completed TMEM loads (tcgen05.wait::ld);
// a cluster-scope release would also wait for the thread's earlier global
// stores to be acknowledged.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster) {
  asm volatile("mbarrier.arrive.release.cta.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster) : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Fire-and-forget FP32 reduction into global memory (an L2 atomic) of four
// consecutive floats at a 16-byte aligned address.
__device__ __forceinline__ void red_add_v4(float *p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c),
               "f"(d)
               : "memory");
}


// Shared-memory matrix descriptor of a K-major operand whose rows are SWZ
// bytes (one swizzle span: 128 or 64): 8-row core-matrix groups 8 x SWZ bytes
// apart (SBO), descriptor version 1 (sm_100 family), layout type 2
// (SWIZZLE_128B) or 4 (SWIZZLE_64B).  The leading byte offset is unused for
// swizzled K-major operands (one MMA's K = 16 x 16 bit = 32 B stays inside a row).
template <int SWZ>
__device__ __forceinline__ uint64_t sw_desc(uint32_t saddr) {
  static_assert(SWZ == 128 || SWZ == 64, "swizzle span");
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;                   // leading byte offset (unused)
  d |= (uint64_t)((8 * SWZ) >> 4) << 32;    // stride byte offset
  d |= (uint64_t)1 << 46;                   // version
  d |= (uint64_t)(SWZ == 128 ? 2 : 4) << 61;
  return d;
}

// Instruction descriptor of tcgen05.mma kind::f16: D=F32, A=B=BF16 (fmt 1) or
// F16 (fmt 0), both K-major; N>>3 at bits 17-22, M>>4 at bits 24-28.
__device__ __forceinline__ uint32_t idesc_f16kind(int M, int N, uint32_t ab_fmt) {
  return (1u << 4) | (ab_fmt << 7) | (ab_fmt << 10) | ((uint32_t)(N >> 3) << 17) |
         ((uint32_t)(M >> 4) << 24);
}

// One lane of a converged warp, the same at every call.  The issuing warp runs its loop
// with all lanes and issues under this predicate: what the loop computes is then uniform
// and stays in uniform registers.  With the loop inside `if (lane == 0)` every operand of
// every MMA is moved there one by one: beside four busy warps a scheduler that took 88
// cycles per MMA, more than an N = 128 MMA's 64, against 47 this way.
__device__ __forceinline__ bool elect_one() {
  uint32_t one;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(one));
  return one != 0;
}

// Operands by the low words of their descriptors (address field) and the high word they share.
__device__ __forceinline__ void mma_f16kind(uint32_t tmem_d, uint32_t alo, uint32_t blo, uint32_t hi,
                                            uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
      "mov.b64 a, {%1, %3};\n\t"
      "mov.b64 b, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p;\n\t}\n" ::"r"(tmem_d),
      "r"(alo), "r"(blo), "r"(hi), "r"(idesc), "r"(accum));
}

__device__ __forceinline__ void mma_commit(uint64_t *bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}

// M = 256 over the pair: A rows 0-127 from this CTA's shared memory, 128-255
// from the peer's at the same offset; B columns split likewise (N/2 each); D
// rows 0-127 in this SM's TMEM, 128-255 in the peer's.
__device__ __forceinline__ void mma2_f16kind(uint32_t tmem_d, uint32_t alo, uint32_t blo, uint32_t hi,
                                             uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
      "mov.b64 a, {%1, %3};\n\t"
      "mov.b64 b, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %4, p;\n\t}\n" ::"r"(tmem_d),
      "r"(alo), "r"(blo), "r"(hi), "r"(idesc), "r"(accum));
}
// Arrive on the barrier at this offset in both CTAs of the pair once the
// issued MMAs have completed.
__device__ __forceinline__ void mma2_commit_both(uint64_t *bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}
__device__ __forceinline__ void mma2_commit(uint64_t *bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}

// Asynchronous form: the 16 registers are valid after tmem_wait16 on them
// (the wait takes them as operands, so no use can be scheduled before it).
__device__ __forceinline__ void tmem_ld16_async(uint32_t taddr, uint32_t *r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// 16x256b shape, 4 repetitions: thread t gets TMEM lanes base + t/4 (r[4j],
// r[4j+1]) and base + 8 + t/4 (r[4j+2], r[4j+3]), columns 8j + 2 (t % 4) and
// the next, j = 0..3 (the accumulator fragment of an m16n8 tile per repetition).
__device__ __forceinline__ void tmem_ld16x256b_x4_async(uint32_t taddr, uint32_t *r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait16(uint32_t *r) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                 "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                 "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}

}  // namespace scess
