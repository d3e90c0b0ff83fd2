// Kernel launches with programmatic dependent launch (sm_90 and later).
//
// Every kernel of this library starts with griddep_wait(), before its first
// access to memory that a kernel may have written, and every launch carries the
// programmatic stream serialization attribute.  What only the host writes, by
// copies that have completed when the entry point returns, may be read before
// it: the tables (c_tables, g_lane_tables; the 2D smoother's rows) and the
// coefficient (the kappa 3D smoother).  A kernel that came to write one of them
// would have to be followed by readers that wait first.  A kernel may then be launched, and its CTAs
// scheduled, while the previous kernel in the stream is still finishing;
// griddep_wait() returns once that grid has completed and its memory
// operations are visible.  Inside the CUDA graphs of the solvers the launch
// latency of each of the many small dependent kernels of a V-cycle (the
// coarse levels are latency-bound) overlaps its predecessor's tail.  Launched
// without the attribute, griddep_wait() returns at once.
#pragma once

#include <cuda_runtime.h>

#include <utility>

#ifndef TPS_PDL
#define TPS_PDL 1  // 0: plain stream-ordered launches (same kernels)
#endif
// 1: each CTA also allows the next kernel's launch right after its wait.
// Measured slower (CG 64^3 FP64 24.57 vs 23.16 ms, 16^3 FP32 1.78 vs 1.65
// ms): the waiting dependent CTAs take SM resources from the running grid.
#ifndef TPS_PDL_EARLY
#define TPS_PDL_EARLY 0
#endif

namespace tps {

__device__ __forceinline__ void griddep_wait()
{
#if defined(__CUDA_ARCH__)
  asm volatile("griddepcontrol.wait;" ::: "memory");
#if TPS_PDL_EARLY
  // the dependent grid may launch once every CTA of this grid has passed
  // here; its CTAs then wait in their own griddep_wait() for this grid's end
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#endif
#endif
}

// launch errors are recorded like those of <<< >>> launches and are read by
// the callers' cudaGetLastError()
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                              Args &&...args)
{
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = TPS_PDL;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

// the same for a grid that is one thread-block cluster
template <typename... KArgs, typename... Args>
inline cudaError_t launch_cluster(void (*kern)(KArgs...), unsigned ctas, dim3 block, size_t smem, cudaStream_t s,
                                  Args &&...args)
{
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = TPS_PDL;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = ctas;
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

}  // namespace tps

#define TPS_LAUNCH(kern, grid, block, smem, stream, ...) \
  ((void)::tps::launch_pdl(kern, grid, block, smem, stream, ##__VA_ARGS__))
