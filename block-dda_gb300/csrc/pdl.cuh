// Programmatic dependent launch: a kernel launched with launch_pdl may be put
// on the SMs while the kernel before it in the stream still runs, and waits at
// pdl_begin() until that one has finished and its writes are visible.  It hides
// the launch latency between the short kernels of an MVP and of a Krylov
// iteration (FP64 MVP N=64, L=2: 18.1 -> 16.0 us; f = 6 BiCGSTAB N=300, L=4:
// 2.26 -> 2.16 ms; 12 concurrent solves: 112.9 -> 108.2 ms).  A kernel may only be launched this way when pdl_begin() is
// the first thing it does: everything it reads or overwrites may belong to the
// kernel before.
#pragma once

#include <cuda_runtime.h>

namespace bdda {

__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

}  // namespace bdda
