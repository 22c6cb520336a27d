// sweep_async.cuh -- shared-memory barriers, asynchronous copies and the
// per-step stage header used by the warp-specialised sweep kernels.
#pragma once

#include "sweep_common.cuh"

namespace msb {

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* b, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
// The barrier by its 32-bit shared-memory address (bar_...) or a pointer.
__device__ __forceinline__ void bar_arrive(uint32_t b) {
  asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.release.cta.shared::cta.b64 st, [%0];\n}" ::"r"(b) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) { bar_arrive(smem_u32(b)); }
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* b, uint32_t bytes) {
  asm volatile(
      "{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 st, [%0], %1;\n}" ::"r"(
          smem_u32(b)),
      "r"(bytes)
      : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// 16-byte asynchronous copy global -> shared (L2 only) and its groups.
__device__ __forceinline__ void cp_async16_s(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) { cp_async16_s(smem_u32(dst), src); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// L2 eviction policies (createpolicy) and the copies / stores that carry one.
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void cp_async16_hint(void* dst, const void* src, uint64_t pol) {
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "l"(pol)
               : "memory");
}
__device__ __forceinline__ void st_v2_hint(double* p, double a, double b, uint64_t pol) {
  asm volatile("st.global.L2::cache_hint.v2.f64 [%0], {%1, %2}, %3;" ::"l"(p), "d"(a), "d"(b), "l"(pol) : "memory");
}
__device__ __forceinline__ void st_f64_hint(double* p, double a, uint64_t pol) {
  asm volatile("st.global.L2::cache_hint.f64 [%0], %1, %2;" ::"l"(p), "d"(a), "l"(pol) : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// 1-D bulk copy global -> shared, completion counted on an mbarrier.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
// The same for shared memory: before a bulk copy writes where ordinary
// stores or cp.async wrote.
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Non-blocking test of a phase (test_wait never suspends the warp).
__device__ __forceinline__ bool bar_test(uint32_t b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(b), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_test_wait(uint64_t* b, uint32_t parity) { return bar_test(smem_u32(b), parity); }

// try_wait with a suspend-time hint: the warp sleeps in hardware until the
// phase completes or about `ns` nanoseconds pass (no busy polling).
__device__ __forceinline__ bool bar_try(uint32_t b, uint32_t parity, uint32_t ns) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(b), "r"(parity), "r"(ns)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* b, uint32_t parity, uint32_t ns) {
  return bar_try(smem_u32(b), parity, ns);
}

// Bounded wait on an mbarrier phase by a whole warp.  It does not give up
// when another CTA aborts: inside a CTA every phase that was started is
// completed (the loader finishes the stages it issued and then posts a stop),
// so only a time-out ends it early.
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity, const SyncArgs& s, int task) {
  if (mbar_test_wait(b, parity)) return true;  // already complete: no suspension
  if (mbar_try_wait(b, parity, 20000)) return true;
  const long long t0 = global_ns();
  for (;;) {
    if (mbar_try_wait(b, parity, 100000)) return true;
    if (global_ns() - t0 > s.timeout_ns) {
      if ((threadIdx.x & 31) == 0) raise_error(s.sync, MSB_ERR_TIMEOUT, task);
      return false;
    }
  }
}

// Per-step header written by the producer into each stage.
struct StepHdr {
  int task, s, oct, gp;
  int x0, x1, y0, y1, z0, z1;
  int flags, mat;  // mat: which matrix buffer holds this task's octant
  int stop, pad0, pad1, pad2;
};

}  // namespace msb
