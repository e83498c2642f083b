// Asynchronous-copy helpers of the one-pass tiled step (lbm_tiled.cuh): 1-D
// bulk copies between global and this CTA's shared memory (cp.async.bulk),
// completion tracked by an mbarrier for loads and by the issuing thread's
// bulk async-group for stores.
#pragma once

#include "lbm_kernels.cuh"

namespace lbm {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Orders this thread's earlier generic-proxy accesses of shared memory before
// later async-proxy (bulk copy) writes to it.
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

// Global -> this CTA's shared memory, `bytes` a multiple of 16, both addresses
// 16-byte aligned; completion is signalled on `bar`.
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes,
                                              uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// Four bytes of global memory -> this CTA's shared memory, completed through
// word_copies_arrive.
__device__ __forceinline__ void word_copy_g2s(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src)
               : "memory");
}

// One arrival on `bar` (counted in its expected arrivals) once all earlier
// word copies of this thread have landed.
__device__ __forceinline__ void word_copies_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// Two runs of this CTA's shared memory -> global (the second one may be empty),
// sizes multiples of 16, addresses 16-byte aligned; tracked as one bulk
// async-group of the issuing thread, which this call commits.
__device__ __forceinline__ void bulk_store2_s2g(void* dst0, const void* src0, uint32_t bytes0,
                                                void* dst1, const void* src1, uint32_t bytes1) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst0),
               "r"(smem_u32(src0)), "r"(bytes0)
               : "memory");
  if (bytes1 > 0)
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst1),
                 "r"(smem_u32(src1)), "r"(bytes1)
                 : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// The issuing thread's bulk stores have finished reading shared memory.
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

// The issuing thread's bulk stores are complete.
__device__ __forceinline__ void bulk_wait_all() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

}  // namespace lbm
