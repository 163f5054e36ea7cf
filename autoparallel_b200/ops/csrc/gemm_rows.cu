// bf16 products with a handful of rows, sm_100a: a projection of a few tokens (decoding).
//
//   C[M, N] = X[M, K] * W[N, K]^T, M <= 32, K % 8 == 0, fp32 sums; C bf16 or fp32
//
// Bound by reading W once.  The tensor-core kernel of gemm_split.cu spends half of such a launch outside that: TMEM allocation, barriers, tiles of
// 128 rows of which a few are used, fp32 tiles added up through a cluster.  Here a block owns 16 rows of W (columns of C), its sixteen warps
// take a sixteenth of K each, and W and X go from memory to registers in the fragments of mma.sync (m16n8k16, W as the 16-row operand): a thread
// loads 8 consecutive elements of a row, which are its share of two MMAs whose k is permuted alike for both operands.  The partial sums of the
// warps meet in shared memory, in warp order: the same result every time, and shorter chains of fp32 sums than the other kernel's.
// Split kernel -> this one, us: 1 x 4096 x 4096 10.7 -> 7.3 (4.6 TB/s with the launch), 16 x 4096 x 4096 10.3 -> 8.7, 8 x 2048 x 2048 7.3 -> 3.7,
// 8 x 256 x 256 3.9 -> 1.9, 1 x 32064 x 4096 51.6 -> 42.2.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "launch.cuh"

namespace apb {

constexpr int ROWS_WARPS = 16, ROWS_MAX = 32, ROWS_TILE = 16;

__device__ __forceinline__ uint4 ld_stream(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// MB: blocks of 8 rows of X; U: steps of 32 elements of K whose loads are under way together
template <int MB, int U, int MIN_BLOCKS>
__global__ void __launch_bounds__(32 * ROWS_WARPS, MIN_BLOCKS)
gemm_rows_kernel(const __nv_bfloat16* X, const __nv_bfloat16* W, void* C, int M, int N, int K, long long ldx,
                 long long ldw, long long ldc, int out_fp32) {
  after_previous();
  constexpr int TM = 8 * MB;
  __shared__ float part[ROWS_WARPS][TM * ROWS_TILE];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = (lane & 3) * 8;
  const int n0 = blockIdx.x * ROWS_TILE;
  const int steps = (K + 31) / 32, s0 = steps * warp / ROWS_WARPS, s1 = steps * (warp + 1) / ROWS_WARPS;
  const __nv_bfloat16* w[2];
  const __nv_bfloat16* x[MB];
  bool wk[2], xk[MB];  // rows outside the matrices load nothing
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    wk[i] = n0 + g + 8 * i < N;
    w[i] = W + (wk[i] ? n0 + g + 8 * i : 0) * ldw + c;
  }
#pragma unroll
  for (int i = 0; i < MB; ++i) {
    xk[i] = g + 8 * i < M;
    x[i] = X + (xk[i] ? g + 8 * i : 0) * ldx + c;
  }
  float acc[MB][4] = {};
  for (int s = s0; s < s1; s += U) {
    uint4 wv[U][2], xv[U][MB];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = (s + u) * 32;
      const bool in = s + u < s1 && k + c < K;  // (K % 8 == 0: eight elements are in or out together)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        wv[u][i] = make_uint4(0, 0, 0, 0);
        if (in && wk[i]) wv[u][i] = ld_stream(w[i] + k);
      }
#pragma unroll
      for (int i = 0; i < MB; ++i) {
        xv[u][i] = make_uint4(0, 0, 0, 0);
        if (in && xk[i]) xv[u][i] = __ldca(reinterpret_cast<const uint4*>(x[i] + k));
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint4 a = wv[u][0], b = wv[u][1];
#pragma unroll
      for (int m = 0; m < MB; ++m) {
        mma_bf16(acc[m], a.x, b.x, a.y, b.y, xv[u][m].x, xv[u][m].y);
        mma_bf16(acc[m], a.z, b.z, a.w, b.w, xv[u][m].z, xv[u][m].w);
      }
    }
  }
  const int m2 = (lane & 3) * 2;
#pragma unroll
  for (int m = 0; m < MB; ++m)
#pragma unroll
    for (int i = 0; i < 4; ++i) part[warp][(8 * m + m2 + (i & 1)) * ROWS_TILE + g + 8 * (i >> 1)] = acc[m][i];
  __syncthreads();
  for (int t = threadIdx.x; t < M * ROWS_TILE; t += 32 * ROWS_WARPS) {
    float v = 0.f;
#pragma unroll
    for (int i = 0; i < ROWS_WARPS; ++i) v += part[i][t];
    const int m = t / ROWS_TILE, n = n0 + t % ROWS_TILE;
    if (n < N) {
      if (out_fp32) reinterpret_cast<float*>(C)[m * ldc + n] = v;
      else reinterpret_cast<__nv_bfloat16*>(C)[m * ldc + n] = __float2bfloat16(v);
    }
  }
}

}  // namespace apb

using namespace apb;

// Whether the product is this kernel's: where it is no slower than the split kernel, both launched to overlap.  Fitted to 3478 sizes (1 to 32 rows,
// 64 <= N <= 32768, 64 <= K <= 14336): the mean loss against the better one of both is 0.2, 0.6 and 1.3 % with up to 8, 16 and 32 rows (as the line was
// drawn with launches that did not overlap: 4, 5 and 9 %, at worst a factor of four).  us in a captured graph, split / this one:
//   up to 8 rows  8 x 256 x 256 2.7 / 1.6, 8 x 4096 x 4096 10.7 / 7.4, 8 x 32064 x 4096 51 / 43.  Every round of the blocks that are resident together
//                 (two to an SM) costs as much as a launch, so that many columns need some K: 8 x 14336 x 256 5.4 / 6.3, x 1024 10.7 / 8.4.  With few
//                 columns and a long K there are too few blocks: 8 x 256 x 8192 4.9 / 6.6, 8 x 1024 x 8192 8.5 / 8.3, 1 x 512 x 8192 8.4 / 7.8.
//   up to 16      X comes from L2 once per 16 columns and is half of what a block reads: 16 x 2048 x 2048 6.1 / 4.1, 16 x 4096 x 4096 8.8 / 8.3, 16 x 512
//                 x 4096 4.2 / 5.3, 16 x 6144 x 512 5.8 / 4.8, 16 x 14336 x 512 7.2 / 8.8, x 1024 10.8 / 10.1, 16 x 4096 x 8192 15 / 16.
//   up to 32      32 x 1024 x 1024 4.1 / 3.4, 24 x 2048 x 2048 6.4 / 4.7, 32 x 4096 x 1024 6.0 / 5.8; 32 x 1024 x 2048 4.2 / 4.8, 32 x 4096 x 512 4.6 /
//                 5.3 (here it is one of the losses), 32 x 6144 x 256 4.0 / 6.4, 32 x 14336 x 256 5.5 / 11.6.
extern "C" int apb_gemm_rows_takes(int M, int N, int K, int num_sms) {
  if (M <= 0 || N <= 0 || K <= 0 || K % 8) return 0;
  const long long round = 2ll * ROWS_TILE * num_sms;  // columns of the blocks that are resident together
  const long long size = (long long)N * K, x = (long long)M * K;
  if (M <= 8) return K <= 6144 ? N <= 2 * round || N <= 32ll * K : N >= 512 && N <= round && x <= 65536;
  if (M <= 16) return K <= 3072 ? N <= (K >= 192 ? 2 : 1) * round || N <= 20ll * K : K <= 6144 && N >= 1024 && N <= round;
  return M <= ROWS_MAX && (size <= 8192 || (K >= 192 && x <= 49152 && size <= 2048 * 2048 && N <= 8ll * K));
}

// X, W: 16-byte bases and rows.  Returns 0, or an argument / launch error (nothing launched).
extern "C" int apb_gemm_rows(const void* X, const void* W, void* C, int M, int N, int K, long long ldx, long long ldw, long long ldc, int out_fp32,
                             int num_sms, cudaStream_t st) {
  if (M <= 0 || N <= 0) return 0;
  if (M > ROWS_MAX || K <= 0 || (K & 7) || (ldx & 7) || (ldw & 7) || ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(W)) & 15)) return 3;
  const unsigned grid = (unsigned)((N + ROWS_TILE - 1) / ROWS_TILE);
  auto launch = [&](auto kern) {
    launch_after(kern, grid, 32 * ROWS_WARPS, 0, st, (const __nv_bfloat16*)X, (const __nv_bfloat16*)W, C, M, N, K, ldx, ldw, ldc, out_fp32);
  };
  // Two blocks to an SM and three steps under way; where there is no second block and K is long enough for it, four (8 x 2048 x 2048 4.0 -> 3.7 us, 32
  // x 2048 x 2048 6.4 -> 5.3; 8 x 512 x 512 2.0 -> 2.2).
  const bool deep = grid <= (unsigned)num_sms && K >= 2048;
  if (M <= 8) deep ? launch(gemm_rows_kernel<1, 4, 1>) : launch(gemm_rows_kernel<1, 3, 2>);
  else if (M <= 16) launch(gemm_rows_kernel<2, 3, 2>);
  else deep ? launch(gemm_rows_kernel<4, 4, 1>) : launch(gemm_rows_kernel<4, 3, 2>);
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}
