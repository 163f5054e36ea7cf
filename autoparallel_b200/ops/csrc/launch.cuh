// Launches that overlap with the end of the kernel before them on the stream (programmatic dependent launch).
//
// A kernel launched with ``launch_after`` may become resident while the kernel before it still runs; its threads pass ``after_previous`` - or
// ``wait_previous`` - only when that one has completed and its writes are visible.  So every kernel that is launched so calls one of them in every
// thread before it touches global memory, also where a thread has nothing to do, and lets the next kernel in (``let_next_in``) only after that:
// then at most two kernels of a stream overlap, and the earlier of them has seen everything before it complete.  A kernel that is launched in the
// ordinary way waits for all of its predecessor as ever, whether that one let it in or not.
//
// What such a kernel reads may still be written when it is resident already, so its loads carry no promise that data stays the same for the life of
// the kernel: no __restrict__ on its parameters, no __ldg, no ld.global.nc - with those the compiler may move a load above the wait.  Where a loop has to
// know that its stores do not touch what it loads, a function that is called behind the wait has the __restrict__ parameters, or the loads of several
// steps are written out before the stores.
//
// Worth it where kernels are short: without it the GPU starts the next kernel of a stream one to two microseconds after the end of the last, on
// a grid of 2.05 us (16 x 4096 x 4096, 8.8 us in a captured graph: 10.24 a launch, with it 8.6; 8 x 4096 x 4096 9.6 -> 7.4).
#pragma once
#include <cuda_runtime.h>

#include <utility>

// Whether the GEMMs are set to make room for communication kernels (gemm_tcgen05.cu).  Then no launch overlaps: the gap between two kernels is where a
// communication kernel becomes resident, and blocks that come early would take its place.
extern "C" int apb_gemm_makes_room();

namespace apb {

__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_in() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void after_previous() {
  wait_previous();
  let_next_in();
}

inline cudaLaunchAttribute overlap_attribute() {
  cudaLaunchAttribute a;
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  return a;
}

template <typename... P, typename... A>
inline cudaError_t launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchAttribute attr = overlap_attribute();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = apb_gemm_makes_room() ? 0 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace apb
