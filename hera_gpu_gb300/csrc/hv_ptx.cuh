// hv_ptx.cuh -- PTX wrappers shared by the tensor-core kernels of
// libheravis.so: mbarriers and bounded waits, proxy and tcgen05 fences, MMA
// descriptors, commits and TMEM loads (sm_103a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace hv {

// Device error flag values (the host turns them into an hv_status).
constexpr int kErrTimeout = 1;
constexpr int kErrRange = 2;    // |U| beyond the exact range of rint_magic
constexpr int kErrLayout = 3;   // dynamic shared memory not 1024-byte aligned

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
// try_wait with a suspend-time hint: a waiting thread sleeps in hardware
// until the phase completes or the hint (ns) elapses, instead of polling
// the barrier through the shared-memory pipe.
constexpr uint32_t kSuspendHintNs = 20000;
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(kSuspendHintNs)
      : "memory");
  return ok != 0;
}

// the same, acquiring at cluster scope
__device__ __forceinline__ bool mbar_try_cluster(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(kSuspendHintNs)
      : "memory");
  return ok != 0;
}

// Single-thread bounded wait (kCl: acquire at cluster scope, for barriers
// that threads of other CTAs arrive on).
template <bool kCl = false>
__device__ __forceinline__ bool wait1(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                      int* gerr, unsigned long long limit_ns) {
  const unsigned long long t0 = global_ns();
  for (uint32_t i = 0;; ++i) {
    if (kCl ? mbar_try_cluster(bar, parity) : mbar_try(bar, parity)) return true;
    if ((i & 63) == 63) {
      if (*abort_flag) return false;
      if (global_ns() - t0 > limit_ns) {
        *abort_flag = 1;
        atomicExch(gerr, kErrTimeout);
        return false;
      }
    }
  }
}

// Whole-warp bounded wait; the outcome is uniform across the warp.
template <bool kCl = false>
__device__ __forceinline__ bool wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          int* gerr, unsigned long long limit_ns) {
  const unsigned long long t0 = global_ns();
  for (uint32_t i = 0;; ++i) {
    const bool done = kCl ? mbar_try_cluster(bar, parity) : mbar_try(bar, parity);
    if (__all_sync(0xffffffffu, done)) return true;
    if (i >= 2) __nanosleep(64);  // leave issue slots to the MMA warp
    if ((i & 63) == 63) {
      int give_up = 0;
      if ((threadIdx.x & 31) == 0) {
        if (*abort_flag) {
          give_up = 1;
        } else if (global_ns() - t0 > limit_ns) {
          *abort_flag = 1;
          atomicExch(gerr, kErrTimeout);
          give_up = 1;
        }
      }
      if (__shfl_sync(0xffffffffu, give_up, 0)) return false;
    }
  }
}

// Bounded wait used while shutting down: ignores the abort flag so that
// copies and MMAs already in flight still land before TMEM is released.
__device__ __forceinline__ void wait_drain(uint32_t bar, uint32_t parity, int* gerr,
                                           unsigned long long limit_ns) {
  const unsigned long long t0 = global_ns();
  for (uint32_t i = 0;; ++i) {
    if (mbar_try(bar, parity)) return;
    if ((i & 63) == 63 && global_ns() - t0 > limit_ns) {
      atomicExch(gerr, kErrTimeout);
      return;
    }
  }
}

__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Instruction descriptor: D F32, A and B K-major, M = 128, N = n; the A/B
// type code is 1 for BF16 (kind::f16) and 0 for FP16 (kind::f16) or E4M3
// (kind::f8f6f4).
__device__ __forceinline__ uint32_t idesc_mma(int n, bool negate_a, uint32_t ab_type) {
  uint32_t d = (1u << 4) | (ab_type << 7) | (ab_type << 10);
  d |= (uint32_t)(n >> 3) << 17;
  d |= (uint32_t)(128 >> 4) << 24;
  if (negate_a) d |= 1u << 13;
  return d;
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
      : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

}  // namespace hv
