// What a CTA of a kernel takes of its SM: {threads, registers per thread, shared memory in bytes}, for the check that a communication
// kernel's CTA fits beside a GEMM CTA.
#pragma once
#include <cuda_runtime.h>

namespace apb {

// An SM's 64 K registers go to warps in units of 256, its 228 KB of shared memory to CTAs with 1 KB more than each asks for.
constexpr int SM_REGISTERS = 65536, SM_SMEM_BYTES = 233472, CTA_SMEM_RESERVED = 1024;
// Most that a communication kernel's CTA takes which is meant to become resident beside a GEMM CTA (gemm_core.cuh leaves that much): the
// all-gather and all-to-all of symm_comm.cu (512 threads of 64 registers) and the sums of dma_comm.cu.
constexpr int BESIDE_REGISTERS = SM_REGISTERS / 2, BESIDE_SMEM_BYTES = 512;

// Returns 0 or 4 (no such kernel on the current device).
inline int kernel_footprint(const void* kern, int threads, int dynamic_smem, int* out) {
  cudaFuncAttributes a;
  if (cudaFuncGetAttributes(&a, kern) != cudaSuccess) {
    cudaGetLastError();
    return 4;
  }
  out[0] = threads;
  out[1] = a.numRegs;
  out[2] = (int)a.sharedSizeBytes + dynamic_smem;
  return 0;
}

}  // namespace apb
