// Programmatic dependent launch: a kernel launched with the attribute may start while its
// predecessor in the stream is still running; it must execute `pdl_wait()` before it touches
// anything the predecessor wrote (the wait returns once the predecessor has completed and its
// writes are visible).  `pdl_launch_dependents()` lets the NEXT kernel of the stream be
// scheduled from that point on, so its launch latency and prologue overlap this kernel.
//
// What a kernel may do before and after the two:
//   * Every thread of a kernel launched this way calls pdl_wait() before it touches what an earlier kernel
//     writes, or writes what one reads, and before the kernel ends: its end then stands for the end of all
//     kernels before it.
//   * Release first, wait then (GEMM, attention; the row quantiser, an ordinary launch, only releases): the next
//     kernel may start before those further back have ended.  Right only because that kernel in its turn touches
//     nothing of theirs before its own wait.
//   * Wait first, release then (all kernels of the expert layer): the next kernel may rely, before its own wait,
//     on all that the releasing kernel's predecessors wrote.  The expert products do: they read the plan and
//     fetch weights first (early_b in gemm/gemm_sm100.cuh).  A kernel that is put before them keeps this order.
//   * A kernel that waits for another rank releases after that wait.  The next kernel may hold the shared memory
//     of every SM from its start on, and then the kernel that the other rank waits for, on another stream of
//     this one, would find no room while both wait.
// A released kernel's blocks occupy SMs while they wait: another stream's kernels get what is left until the
// kernel in front has ended.
//
// The reference chains its small expert-parallel kernels the same way
// (`cudaTriggerProgrammaticLaunchCompletion`: datasets/example079_deepep_jit_dispatch_notify/nv/
// empty_deepep_jit_dispatch_notify.cu:147; `cudaGridDependencySynchronize`:
// datasets/example081_deepep_jit_dispatch_copy_epilogue/nv/empty_deepep_jit_dispatch_copy_epilogue.cu:40;
// `kUsePDL`: datasets/example105_sglang_custom_allreduce_easy/empty_sglang_custom_allreduce_pull_easy.cu:105).
#pragma once
#include <cuda_runtime.h>

namespace cb {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launch with programmatic stream serialisation allowed (the kernel must call pdl_wait()).
template <class... KArgs, class... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                              cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

}  // namespace cb
