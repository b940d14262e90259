// mbar.cuh -- shared-memory mbarrier helpers of the warp-specialized kernels.
#pragma once

#include <cuda_runtime.h>

#include "sht_internal.h"

namespace sht {

__device__ __forceinline__ unsigned smem_u32(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(void* mbar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mbar)), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try(void* mbar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(mbar)), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ void mbar_arrive(void* mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(mbar)) : "memory");
}

// one arrival on mbar by this thread once all its earlier cp.async copies have landed (the
// arrival is part of the barrier's expected count)
__device__ __forceinline__ void mbar_arrive_cp_async(void* mbar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(mbar)) : "memory");
}

// Wait for a phase, at most `limit` polls, giving up as well when another role raised the
// CTA's abort flag.  A wait that runs out raises the flag and stores SHT_ERR_TIMEOUT in the
// context's error word (host-mapped; every writer stores the same value).
__device__ __forceinline__ bool mbar_wait_bounded(void* mbar, unsigned parity, volatile int* abort, long long limit,
                                                  volatile int* err) {
  for (long long i = 0; i < limit; ++i) {
    if (mbar_try(mbar, parity)) return true;
    if (*abort) return false;
  }
  *abort = 1;
  *err = (int)SHT_ERR_TIMEOUT;
  __threadfence_system();
  return false;
}

// The same, each poll suspending the warp for up to a microsecond.
__device__ __forceinline__ bool mbar_wait_suspended(void* mbar, unsigned parity, volatile int* abort, long long limit,
                                                    volatile int* err) {
  for (long long i = 0; i < limit; ++i) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred P;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, P;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(mbar)), "r"(parity), "r"(1000)
        : "memory");
    if (ok) return true;
    if (*abort) return false;
  }
  *abort = 1;
  *err = (int)SHT_ERR_TIMEOUT;
  __threadfence_system();
  return false;
}

}  // namespace sht
