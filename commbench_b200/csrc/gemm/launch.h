// Kernel launch helper for the tcgen05 GEMM kernels: plain, as clusters of two
// CTAs (CTA pairs), and / or cooperative (rank emulation, where the CTAs of the
// virtual ranks wait on one another and must be co-resident).
//
// The reference launches its cluster kernels the same way (`cudaLaunchKernelEx`
// with a cluster dimension and a dynamic shared-memory attribute:
// datasets/example051_thunderkitten_ag_gemm_easy/nv/empty_thunderkitten_ag_gemm.cu:271-308).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace cb {

// Opt-in to `bytes` of dynamic shared memory, once per kernel and device: `done` is the kernel's own
// bit mask of devices (the attribute is idempotent, so a race only sets it twice).
inline cudaError_t allow_smem(const void* kernel, int bytes, std::atomic<uint64_t>& done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = dev < 64 ? 1ull << dev : 0ull;
  if ((done.load(std::memory_order_relaxed) & bit) != 0) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_relaxed);
  return e;
}

template <class... KArgs, class... Args>
inline cudaError_t launch_gemm_kernel_pdl(void (*kernel)(KArgs...), int grid, int threads, int smem,
                                          cudaStream_t st, int cluster, bool cooperative, bool pdl,
                                          Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  cfg.stream = st;
  cudaLaunchAttribute attr[3];
  unsigned n = 0;
  if (cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = static_cast<unsigned>(cluster);
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (cooperative) {
    attr[n].id = cudaLaunchAttributeCooperative;
    attr[n].val.cooperative = 1;
    ++n;
  }
  if (pdl) {  // the kernel must call pdl_wait()
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

template <class... KArgs, class... Args>
inline cudaError_t launch_gemm_kernel(void (*kernel)(KArgs...), int grid, int threads, int smem,
                                      cudaStream_t st, int cluster, bool cooperative,
                                      Args... args) {
  return launch_gemm_kernel_pdl(kernel, grid, threads, smem, st, cluster, cooperative, false,
                                args...);
}

}  // namespace cb
