// Cluster launch control: a running CTA takes over the work of one that has not been launched yet.
//
// A kernel launched with one CTA per work item becomes persistent without giving up the hardware's
// scheduling: a CTA that is done with its item cancels the launch of a pending CTA and does that one's
// item as well.  Items therefore go to whatever SM is free, also when other streams hold some of them.
//
// `clc_try_cancel` is asynchronous: 16 bytes of answer arrive in shared memory and complete as many bytes
// on an mbarrier.  After an answer that cancelled nothing no further request may be made.
#pragma once
#include <stdint.h>

#include "ptx.cuh"

namespace cb {

__device__ __forceinline__ void clc_try_cancel(void* answer16, uint64_t* bar) {
  asm volatile(
      "clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
          smem_u32(answer16)),
      "r"(smem_u32(bar))
      : "memory");
}

// Block index (x) of the CTA whose launch was cancelled, or -1: none was left.
__device__ __forceinline__ int clc_cancelled_block(const void* answer16) {
  uint32_t ok, x;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      ".reg .b128 a;\n\t"
      "ld.shared.b128 a, [%2];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, a;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "mov.u32 %1, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, a;\n\t"
      "}\n"
      : "=r"(ok), "=r"(x)
      : "r"(smem_u32(answer16))
      : "memory");
  return ok != 0u ? static_cast<int>(x) : -1;
}

}  // namespace cb
