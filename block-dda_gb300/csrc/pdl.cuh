// Programmatic dependent launch: a kernel launched with launch_pdl is set up
// while the kernel before it in the stream still runs, and waits at pdl_begin()
// until that one has finished and its writes are visible.  It hides the launch
// latency between the short kernels of an MVP and of a Krylov iteration (FP64
// MVP N=64, L=2: 18.1 -> 13.6 us; FP64 solve N=1024, L=2: 3.36 -> 3.14 ms).  A
// kernel may only be launched this way when pdl_begin() is the first thing it
// does: everything it reads or overwrites may belong to the kernel before.
//
// By default the next kernel's CTAs come when this one's have all ended.  A
// pdl_trigger() before that lets them take SMs as soon as all CTAs of this one
// run.  They fill the SMs that have room first and stay there while they wait,
// so a grid of about one wave ends up on some SMs twice and on others not at
// all: with triggers everywhere the FP32 MVP of a 24 x 24 x 243 box, L=1, took
// 100 us, without any 70 (88 before dependent launches), and one of 24 x 24 x
// 32, L=3, 27.8 and 21.3 (38).  It pays where a kernel's CTAs end raggedly and
// the next one has many waves (ypass_cols.cuh).
#pragma once

#include <cuda_runtime.h>

namespace bdda {

__device__ __forceinline__ void pdl_begin() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

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
