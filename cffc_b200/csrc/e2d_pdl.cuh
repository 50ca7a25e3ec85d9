// e2d_pdl.cuh — programmatic dependent launch for the chains of short kernels
// (ghost fill, stage, step bookkeeping): a kernel launched with launch_pdl may
// start while the one before it in the stream is still running, does what
// depends on nothing the stream computes (barriers, tensor copies of the
// geometry), and waits for the end of that kernel -- and with it of all
// earlier ones, as each of them waited the same way -- in pdl_wait before it
// reads or writes anything else.  Every kernel launched with launch_pdl calls
// pdl_wait in every thread that goes on; without the attribute both calls do
// nothing.  A kernel that never calls pdl_launch_next lets the next one start
// as its last CTAs end.
// What bounds the chains is the latency from one kernel's end to the next
// one's first result: 100 two-stage steps of 16 blocks of 32 x 32 (400 launches
// and 100 step ends) 2.88 -> 2.30 ms together with one bookkeeping kernel a step
// and graphs of four steps, 20 four-stage steps of 30 blocks of 37 x 29
// 2.65 -> 2.50 ms.
#pragma once
#include <cuda_runtime.h>

namespace e2d {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The next kernel in the stream may start (and wait) once every CTA of this
// one has said so or is done.
__device__ __forceinline__ void pdl_launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_pdl(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace e2d
