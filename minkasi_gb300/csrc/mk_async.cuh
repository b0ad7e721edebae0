// Shared-memory mbarriers and 1-D bulk copies (cp.async.bulk) for sm_100+
// kernels: inline PTX, one CTA per cluster.  Every wait is bounded.
#pragma once
#include <stdint.h>

namespace mk {

// iterations of mbarrier.try_wait (each may suspend briefly) before a wait
// is declared timed out
constexpr uint32_t SPIN_LIMIT = 1u << 24;
// the same for the waits between the roles of a tensor-core kernel, after which
// its CTA stops and writes NaN (a compile-time constant: as a kernel argument it
// cost the sliced FP64 rotation 2 %)
#ifndef MK_ROLE_SPIN_LIMIT
#define MK_ROLE_SPIN_LIMIT SPIN_LIMIT
#endif
constexpr uint32_t ROLE_SPIN_LIMIT = MK_ROLE_SPIN_LIMIT;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

// makes initialised mbarriers visible to the async proxy (bulk copies)
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// bounded wait for the phase of the given parity; false on timeout
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
  for (uint32_t i = 0; i < SPIN_LIMIT; i++)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// arrive once and expect `bytes` of bulk-copy transactions on this phase
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

// plain arrive (release): this thread's earlier shared-memory reads are
// ordered before whoever completes a wait on the phase
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// global -> shared bulk copy completing on `bar`; both addresses 16-byte
// aligned, `bytes` a multiple of 16
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// 4-byte global -> shared asynchronous copy; when !valid nothing is read and
// the destination is zero-filled (src must still be a mapped address)
__device__ __forceinline__ void cp_async4_zfill(float *dst, const float *src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src),
               "r"(valid ? 4 : 0)
               : "memory");
}

// waits for all of this thread's cp.async copies
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// orders this thread's earlier generic-proxy shared-memory accesses before
// its later async-proxy ones (a bulk copy refilling a consumed stage)
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// L2 policy: lines brought in by these accesses are evicted first (streams
// that must not push a resident working set out of L2)
__device__ __forceinline__ uint64_t l2_evict_first_policy() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}

// bulk_g2s with an L2 cache policy
__device__ __forceinline__ void bulk_g2s_hint(void *dst, const void *src, uint32_t bytes, uint64_t *bar,
                                              uint64_t policy) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1], %2, [%3], %4;" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(policy)
      : "memory");
}

}  // namespace mk
