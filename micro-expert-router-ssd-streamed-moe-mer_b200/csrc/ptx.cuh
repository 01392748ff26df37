// Inline-PTX helpers shared by the kernel files: mbarriers with bounded waits, bulk async copies
// (1-D TMA), shared-memory loads on 32-bit shared addresses.
#pragma once

#include <stdint.h>

namespace {

constexpr uint32_t SPIN_LIMIT = 1u << 16;  // polls per bounded wait; a poll suspends for tens of microseconds

// Arrival counters between CTAs: what the CTA wrote before (a __syncthreads() in front) is visible to whoever acquires the count.
__device__ __forceinline__ uint32_t arrive_acq_rel(uint32_t *counter, uint32_t by = 1) {
  uint32_t v;
  asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(v) : "l"(counter), "r"(by) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t load_acquire(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Programmatic dependent launch: a kernel launched with the attribute starts while its predecessor runs and waits here, before
// it touches anything the predecessor reads or writes; without the attribute both are no-ops.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Whether the phase with this parity is complete; suspends for a while if not.
__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(addr), "r"(parity)
      : "memory");
  return ok != 0;
}
// The same without suspending.
__device__ __forceinline__ bool mbar_test(const uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: false when the phase did not complete within SPIN_LIMIT polls, or (with `abort`) once *abort is set.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, const volatile uint32_t *abort = nullptr) {
  const uint32_t addr = smem_u32(bar);
  for (uint32_t i = 0; i < SPIN_LIMIT; i++) {
    if (mbar_try(addr, parity)) return true;
    if (abort && *abort) return false;
  }
  return false;
}
// The same, bounded by time: for the way out after an error.
__device__ __forceinline__ void mbar_drain(uint64_t *bar, uint32_t parity, uint64_t ns) {
  const uint32_t addr = smem_u32(bar);
  const uint64_t since = global_ns();
  while (!mbar_try(addr, parity) && global_ns() - since < ns) {
  }
}
// Barriers that more than one CTA of a cluster signals or is signalled by.  An mbarrier operation without a scope orders memory within
// its own CTA only.  Where nothing but tensor memory crosses, the tcgen05 fences in front of the arrival and behind the wait order
// it, and the barrier operations are relaxed: an arrival that released the warp's memory at cluster scope would wait for all its
// stores (2048 tokens on 128 experts of 2048 x 768: 1140 us a pass as it is, 1661 so).
__device__ __forceinline__ void mbar_arrive_tmem(uint32_t bar) {  // an address in shared::cluster
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_wait_tmem(uint64_t *bar, uint32_t parity) {  // a tcgen05.fence::after_thread_sync follows
  const uint32_t addr = smem_u32(bar);
  for (uint32_t i = 0; i < SPIN_LIMIT; i++) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.relaxed.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
// Shared memory of the other CTA: bytes that its copies have counted here, or that the pair's MMAs have finished reading.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t *bar, uint32_t parity) {
  const uint32_t addr = smem_u32(bar);
  for (uint32_t i = 0; i < SPIN_LIMIT; i++) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// Shared-memory loads on 32-bit shared addresses (no generic-address arithmetic in the block loop).
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}

}  // namespace
