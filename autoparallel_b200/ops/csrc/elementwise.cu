// Bandwidth-bound kernels of the transformer step for sm_100a: RMSNorm fwd/bwd, RoPE, SwiGLU
// fwd/bwd, cross-entropy fwd/bwd, dtype cast, embedding forward, multi-tensor AdamW.
// All use 16-byte vector accesses and fp32 math.  Kernels without anything to carry from one element to the next (casts, SwiGLU, RoPE, RMSNorm
// forward, AdamW) take one vector per thread and tensor, in blocks that end there: as many loads are under way as in loops over the tensor with 8
// blocks an SM, but the memory sees one front that moves through every tensor.  Loop -> so: casts to fp32 of 2^28 elements 333 -> 235 us, to bf16 252 ->
// 229; SwiGLU of 8192 x 14336 bf16 117 -> 100, its gradient 193 -> 170 (6.9 TB/s); AdamW over 218 M parameters 1067 -> 963.  Two and four vectors a thread
// are no faster there and slower in small tensors (SwiGLU gradient of 999 x 1408 2.7 / 3.2 / 3.7 us).
// They replace the ATen / Inductor-generated kernels the reference reaches for the same nodes
// (autoparallel/_testing/models/llama3.py:187-213, 355-356, 396-397).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "launch.cuh"
#include "ptx.cuh"

namespace apb {

template <typename T> struct Vec8;  // 8 elements
template <> struct Vec8<__nv_bfloat16> {
  uint4 raw;
  __device__ void load(const __nv_bfloat16* p) { raw = *reinterpret_cast<const uint4*>(p); }
  __device__ void store(__nv_bfloat16* p) const { *reinterpret_cast<uint4*>(p) = raw; }
  __device__ void to_float(float (&f)[8]) const {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 v = __bfloat1622float2(h[i]);
      f[2 * i] = v.x;
      f[2 * i + 1] = v.y;
    }
  }
  __device__ void from_float(const float (&f)[8]) {
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  }
};
template <> struct Vec8<float> {
  float4 a, b;
  __device__ void load(const float* p) {
    a = reinterpret_cast<const float4*>(p)[0];
    b = reinterpret_cast<const float4*>(p)[1];
  }
  __device__ void store(float* p) const {
    reinterpret_cast<float4*>(p)[0] = a;
    reinterpret_cast<float4*>(p)[1] = b;
  }
  __device__ void to_float(float (&f)[8]) const {
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  }
  __device__ void from_float(const float (&f)[8]) {
    a = make_float4(f[0], f[1], f[2], f[3]);
    b = make_float4(f[4], f[5], f[6], f[7]);
  }
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// block-wide sum; ``red`` is >= 32 floats of shared memory.  All threads get the result.
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float r = (l < nw) ? red[l] : 0.f;
  return warp_sum(r);
}
__device__ __forceinline__ float block_max(float v, float* red) {
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float r = (l < nw) ? red[l] : -INFINITY;
  return warp_max(r);
}

// ------------------------------------------------------------------------------------ RMSNorm
// Forward.  A group of ``TPR`` threads owns a row and keeps its NVEC x 8 elements per thread in registers between the
// sum of squares and the scaling, so x is read once.  TPR = 32: one warp per row, reduction by shuffles only, no
// block barrier; several rows per block keep enough loads in flight.  TPR = blockDim.x: a block takes a row at a time (see apb_rms_norm_fwd).
// D % 8 == 0 and D <= TPR * 8 * NVEC.
template <typename T, int NVEC, bool WARP_ROWS, bool IN_TURN>
__device__ __forceinline__ void rms_norm_fwd(const T* __restrict__ x, const T* __restrict__ w, T* __restrict__ y, float* __restrict__ rstd, long long rows,
                                             int D, float eps) {
  __shared__ float red[32];
  const int tpr = WARP_ROWS ? 32 : blockDim.x;
  const int t = WARP_ROWS ? (threadIdx.x & 31) : threadIdx.x;
  long long row = WARP_ROWS ? blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5) : blockIdx.x;
  if (row >= rows) return;
  do {
    const T* xr = x + row * D;
    T* yr = y + row * D;
    Vec8<T> v[NVEC];
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < NVEC; ++j) {
      const int c = (t + j * tpr) * 8;
      if (c < D) {
        v[j].load(xr + c);
        float f[8]; v[j].to_float(f);
#pragma unroll
        for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
      }
    }
    ss = WARP_ROWS ? warp_sum(ss) : block_sum(ss, red);
    const float r = rsqrtf(ss / D + eps);
    if (t == 0) rstd[row] = r;
#pragma unroll
    for (int j = 0; j < NVEC; ++j) {
      const int c = (t + j * tpr) * 8;
      if (c < D) {
        Vec8<T> wv; wv.load(w + c);
        float f[8], g[8]; v[j].to_float(f); wv.to_float(g);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = f[i] * r * g[i];
        Vec8<T> o; o.from_float(f); o.store(yr + c);
      }
    }
  } while (IN_TURN && (row += gridDim.x) < rows);  // (the same for the whole block)
}
template <typename T, int NVEC, bool WARP_ROWS, bool IN_TURN = false>
__global__ void rms_norm_fwd_kernel(const T* x, const T* w, T* y, float* rstd, long long rows, int D, float eps) {
  after_previous();
  rms_norm_fwd<T, NVEC, WARP_ROWS, IN_TURN>(x, w, y, rstd, rows, D, eps);
}

// block-wide sums of R values at once (one barrier pair for all of them); ``red`` holds 32 * R floats
template <int R>
__device__ __forceinline__ void block_sum_multi(float (&v)[R], float* red) {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int k = 0; k < R; ++k) v[k] = warp_sum(v[k]);
  __syncthreads();
  if (l == 0) {
#pragma unroll
    for (int k = 0; k < R; ++k) red[k * 32 + w] = v[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < R; ++k) v[k] = warp_sum(l < nw ? red[k * 32 + l] : 0.f);
}

// Where a backward block leaves its weight-gradient sums: its own row of fp32 partial sums, or (``shared`` > 0) added with
// atomics to one of ``shared`` rows that the caller zeroed.
struct RmsDw {
  float* base;
  long long D;
  int shared;
  __device__ __forceinline__ void put(int col, const float (&v)[8]) const {
    if (shared == 0) {
      float4* p = reinterpret_cast<float4*>(base + blockIdx.x * D + col);
      p[0] = make_float4(v[0], v[1], v[2], v[3]);
      p[1] = make_float4(v[4], v[5], v[6], v[7]);
    } else {
      float* p = base + (blockIdx.x % shared) * D + col;
#pragma unroll
      for (int i = 0; i < 8; ++i) atomicAdd(p + i, v[i]);
    }
  }
};

// Backward.  One persistent block per SM (a single wave).  Every iteration takes ROWS rows at once and the loads of
// the next iteration are issued before the current one is reduced and stored (two register sets that swap roles, so
// nothing is copied): the row loop is bound by memory bandwidth rather than by one load-reduce-store round trip per
// row.  The ROWS dot products share one block reduction.  Math per element: g*x once, then two fused multiply-adds
// (weight-gradient partial and dot product); the second pass forms dx = g*(r*w) - x*(r*r*mean) with two more.
// EXACT: D == blockDim.x * 8 * NVEC and rows % ROWS == 0, so no bounds predicate is needed anywhere.  Runs for fp32 rows that the
// ring of the form below does not hold.  (512, 1): without the one the compiler settles on 32 registers and spills the row;
// 16384 x 16384 fp32 2706 -> 1054 us.
// Requires D <= blockDim.x * 8 * RMS_BWD_MAX_VEC.
constexpr int RMS_BWD_MAX_VEC = 4;
template <typename T, int NVEC, int ROWS, bool EXACT>
__global__ void __launch_bounds__(512, 1) rms_norm_bwd_kernel(const T* dy, const T* x, const T* w, const float* rstd, T* dx, RmsDw dw, long long rows,
                                                             int D) {
  after_previous();
  __shared__ float red[32 * ROWS];
  float wreg[NVEC][8];
  float dwreg[NVEC][8];
  int col[NVEC];
#pragma unroll
  for (int j = 0; j < NVEC; ++j) {
    col[j] = (threadIdx.x + j * blockDim.x) * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      dwreg[j][i] = 0.f;
      wreg[j][i] = 0.f;
    }
    if (EXACT || col[j] < D) {
      Vec8<T> wv; wv.load(w + col[j]); wv.to_float(wreg[j]);
    }
  }
  const long long step = (long long)gridDim.x * ROWS;
  const float inv_d = 1.f / D;
  Vec8<T> xa[ROWS][NVEC], ga[ROWS][NVEC], xb[ROWS][NVEC], gb[ROWS][NVEC];
  float ra[ROWS], rb[ROWS];

  auto fetch = [&](Vec8<T> (&xs)[ROWS][NVEC], Vec8<T> (&gs)[ROWS][NVEC], float (&rs)[ROWS], long long row0) {
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const long long row = row0 + k;
      const bool row_ok = EXACT || row < rows;
      rs[k] = row_ok ? rstd[row] : 0.f;
      const T* xr = x + row * D;
      const T* gr = dy + row * D;
#pragma unroll
      for (int j = 0; j < NVEC; ++j) {
        if (row_ok && (EXACT || col[j] < D)) {
          xs[k][j].load(xr + col[j]);
          gs[k][j].load(gr + col[j]);
        }
      }
    }
  };
  auto process = [&](Vec8<T> (&xs)[ROWS][NVEC], Vec8<T> (&gs)[ROWS][NVEC], float (&rs)[ROWS], long long row0) {
    float dot[ROWS];
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      dot[k] = 0.f;
      const bool row_ok = EXACT || row0 + k < rows;
#pragma unroll
      for (int j = 0; j < NVEC; ++j) {
        if (row_ok && (EXACT || col[j] < D)) {
          float xf[8], gf[8]; xs[k][j].to_float(xf); gs[k][j].to_float(gf);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float gx = gf[i] * xf[i];
            dwreg[j][i] = fmaf(gx, rs[k], dwreg[j][i]);
            dot[k] = fmaf(gx, wreg[j][i], dot[k]);
          }
        }
      }
    }
    block_sum_multi<ROWS>(dot, red);
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const long long row = row0 + k;
      const bool row_ok = EXACT || row < rows;
      const float r = rs[k];
      const float c = r * r * r * dot[k] * inv_d;  // (sum g w x) * r is the dot product with x-hat; times r*r for the formula below
      T* dr = dx + row * D;
#pragma unroll
      for (int j = 0; j < NVEC; ++j) {
        if (row_ok && (EXACT || col[j] < D)) {
          float xf[8], gf[8], o[8]; xs[k][j].to_float(xf); gs[k][j].to_float(gf);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] = fmaf(gf[i], r * wreg[j][i], -xf[i] * c);
          Vec8<T> ov; ov.from_float(o); ov.store(dr + col[j]);
        }
      }
    }
  };

  long long row0 = (long long)blockIdx.x * ROWS;
  if (row0 < rows) fetch(xa, ga, ra, row0);
  while (row0 < rows) {
    if (row0 + step < rows) fetch(xb, gb, rb, row0 + step);
    process(xa, ga, ra, row0);
    row0 += step;
    if (row0 >= rows) break;
    if (row0 + step < rows) fetch(xa, ga, ra, row0 + step);
    process(xb, gb, rb, row0);
    row0 += step;
  }
#pragma unroll
  for (int j = 0; j < NVEC; ++j)
    if (EXACT || col[j] < D) dw.put(col[j], dwreg[j]);
}

// Backward, bulk-copy form (the one the launcher prefers).  Bound by memory: x and dy are read once, dx is written once.
// One row per step and block; the rows travel global -> shared memory as untiled bulk copies (``cp.async.bulk``,
// completion on an mbarrier) through a ring of RMS_STAGES stages, issued two steps ahead by one thread, so the prefetch
// costs no registers.  Blocks are small and several share an SM: while one waits at its barrier the others work (a single
// 512-thread block per SM taking four rows a step spent half its time in the reduction).  This kernel alone, before -> after: 8192 x 4096
// bf16 59 -> 33 us, 999 x 2048 20 -> 6, fp32 2047 x 2048 21 -> 10; with the weight gradient's column sums (before: a cleared row, atomics and a
// cast) 59 -> 36, 24 -> 11, 24 -> 14.
// One block barrier per step: the partial sums of consecutive steps sit in alternating slots, and a stage is refilled
// after the barrier of the following step, which every thread reaches only when it has read the stage for the last time.
// Waits are bounded: if a stage never arrives the block stops (its rows keep whatever dx held).
constexpr int RMS_STAGES = 3;
__host__ __device__ inline int rms_ring_bytes(int row_bytes) { return RMS_STAGES * 2 * row_bytes + 128; }
template <typename T, int NVEC, int THREADS>
__global__ void __launch_bounds__(THREADS, NVEC == 2 && THREADS == 512 ? 2 : 1) rms_norm_bwd_bulk_kernel(const T* dy, const T* x,
                                                                    const T* w, const float* rstd, T* dx, RmsDw dw, long long rows, int D) {
  extern __shared__ uint8_t rms_smem_raw[];
  __shared__ uint64_t bars[RMS_STAGES];
  __shared__ float red[2][THREADS / 32];
  __shared__ uint32_t abort_word;
  constexpr bool KEEP = sizeof(T) == 2;  // the row stays in registers between the two passes (fp32: read from shared memory again)
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(rms_smem_raw) + 127) & ~uintptr_t(127));
  const int row_bytes = D * (int)sizeof(T);
  volatile uint32_t* abort_flag = &abort_word;
  if (threadIdx.x == 0) {
    for (int s_ = 0; s_ < RMS_STAGES; ++s_) mbar_init(&bars[s_], 1);
    abort_word = 0;
    mbar_fence_init();
  }
  __syncthreads();
  after_previous();
  const long long step = gridDim.x, first = blockIdx.x;
  auto issue = [&](long long it) {  // one thread: start the copies of this block's step ``it``
    const long long row = first + it * step;
    if (row >= rows) return;
    const int st = (int)(it % RMS_STAGES);
    mbar_expect_tx(&bars[st], 2u * row_bytes);
    bulk_load(smem + (2 * st) * row_bytes, x + row * D, row_bytes, &bars[st]);
    bulk_load(smem + (2 * st + 1) * row_bytes, dy + row * D, row_bytes, &bars[st]);
  };
  if (threadIdx.x == 0)
    for (int it = 0; it < RMS_STAGES - 1; ++it) issue(it);

  Vec8<T> wv[NVEC];
  float dwreg[NVEC][8];
  int col[NVEC];
#pragma unroll
  for (int j = 0; j < NVEC; ++j) {
    col[j] = (threadIdx.x + j * THREADS) * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) dwreg[j][i] = 0.f;
    if (col[j] < D) wv[j].load(w + col[j]);
  }
  const float inv_d = 1.f / D;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  long long it = 0;
  float r_next = first < rows ? rstd[first] : 0.f;
  for (long long row = first; row < rows; row += step, ++it) {
    const int st = (int)(it % RMS_STAGES);
    const float r = r_next;
    if (row + step < rows) r_next = rstd[row + step];
    if (!mbar_wait(&bars[st], (uint32_t)((it / RMS_STAGES) & 1), abort_flag)) *abort_flag = 1;
    const T* xs = reinterpret_cast<const T*>(smem + (2 * st) * row_bytes);
    const T* gs = reinterpret_cast<const T*>(smem + (2 * st + 1) * row_bytes);
    Vec8<T> xk[KEEP ? NVEC : 1], gk[KEEP ? NVEC : 1];
    float dot = 0.f;
#pragma unroll
    for (int j = 0; j < NVEC; ++j) {
      if (col[j] < D) {
        Vec8<T>& xv = xk[KEEP ? j : 0];
        Vec8<T>& gv = gk[KEEP ? j : 0];
        xv.load(xs + col[j]);
        gv.load(gs + col[j]);
        float xf[8], gf[8], wf[8]; xv.to_float(xf); gv.to_float(gf); wv[j].to_float(wf);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float gx = gf[i] * xf[i];
          dwreg[j][i] = fmaf(gx, r, dwreg[j][i]);
          dot = fmaf(gx, wf[i], dot);
        }
      }
    }
    dot = warp_sum(dot);
    if (THREADS > 32) {
      if (lane == 0) red[it & 1][warp] = dot;
      __syncthreads();
      dot = 0.f;
#pragma unroll
      for (int k = 0; k < THREADS / 32; ++k) dot += red[it & 1][k];
    } else {
      __syncwarp();
    }
    if (*abort_flag) break;  // (set before the barrier, so every thread leaves here)
    if (threadIdx.x == 0) issue(it + RMS_STAGES - 1);
    const float c = r * r * r * dot * inv_d;
#pragma unroll
    for (int j = 0; j < NVEC; ++j) {
      if (col[j] < D) {
        Vec8<T>& xv = xk[KEEP ? j : 0];
        Vec8<T>& gv = gk[KEEP ? j : 0];
        if (!KEEP) {
          xv.load(xs + col[j]);
          gv.load(gs + col[j]);
        }
        float xf[8], gf[8], wf[8], o[8]; xv.to_float(xf); gv.to_float(gf); wv[j].to_float(wf);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = fmaf(gf[i], r * wf[i], -xf[i] * c);
        Vec8<T> ov; ov.from_float(o); ov.store(dx + row * D + col[j]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < NVEC; ++j)
    if (col[j] < D) dw.put(col[j], dwreg[j]);
}

// dw = column sums of the blocks' partial rows: 32 columns per block, 32 groups of partial rows
template <typename T>
__global__ void __launch_bounds__(1024) rms_dw_kernel(const float* part, T* dw, int nparts, int D) {
  after_previous();
  __shared__ float red[32][33];
  const int c = blockIdx.x * 32 + (threadIdx.x & 31), g = threadIdx.x >> 5;
  float s = 0.f;
  if (c < D) {
#pragma unroll 8
    for (int b = g; b < nparts; b += 32) s += part[(long long)b * D + c];
  }
  red[g][threadIdx.x & 31] = s;
  __syncthreads();
  s = warp_sum(red[threadIdx.x & 31][g]);
  const int co = blockIdx.x * 32 + g;
  if ((threadIdx.x & 31) == 0 && co < D) dw[co] = T(s);
}

// One vector of a thread: the ``vec``-th of ``n`` elements, or the end of them.
template <typename S, typename D>
__device__ __forceinline__ void cast_vec(const S* src, D* dst, long long n, long long vec) {
  const long long i = vec * 8;
  if (i + 8 <= n) {
    Vec8<S> v; v.load(src + i);
    float f[8]; v.to_float(f);
    Vec8<D> o; o.from_float(f); o.store(dst + i);
  } else {
    for (long long k = i; k < n; ++k) dst[k] = D(float(src[k]));
  }
}
template <typename S, typename D>
__global__ void __launch_bounds__(256) cast_kernel(const S* src, D* dst, long long n) {
  after_previous();
  cast_vec(src, dst, n, blockIdx.x * 256ll + threadIdx.x);
}

// Many small casts to bf16 in one launch: a block finds its tensor in the table that travels with the launch.  21 parameters of a debug-sized decoder:
// 21 launches of 1.7 us (and 7 us of host time each) -> one of 3.5.
constexpr int CAST_MANY = 48;
struct CastMany {
  const float* src[CAST_MANY];
  __nv_bfloat16* dst[CAST_MANY];
  long long n[CAST_MANY];
  int first[CAST_MANY];  // block of the tensor's first piece; INT_MAX past the last tensor
};
__global__ void __launch_bounds__(256) cast_many_kernel(const __grid_constant__ CastMany t) {
  after_previous();
  int lo = 0, hi = CAST_MANY;  // the last tensor that starts at or before this block
  while (hi - lo > 1) {
    const int mid = (lo + hi) / 2;
    if (t.first[mid] <= (int)blockIdx.x) lo = mid;
    else hi = mid;
  }
  cast_vec(t.src[lo], t.dst[lo], t.n[lo], ((int)blockIdx.x - t.first[lo]) * 256ll + threadIdx.x);
}

// ------------------------------------------------------------------------------------ RoPE
// x [B, S, H, D] with interleaved pairs; cos/sin fp32 [S, D/2].  One thread owns eight consecutive elements of a
// head (one 16-byte vector) at one position, in HEADS neighbouring heads: the 32 bytes of cos / sin it needs are read
// once for them (the tables would otherwise be twice the traffic of x itself).  Eight heads where that leaves the SMs 768 threads each, else
// four; all heads of a position in one thread -> 8 / 4 heads a thread: 8192 x 32 x 128 33.4 -> 25.3 / 27.7 us, 8192 x 8 x 128 8.3 -> 8.2 / 9.0,
// 8192 x 8 x 64 5.6 -> 5.5 / 4.2, 100 x 32 x 128 8.8 -> 3.6 / 2.7.
template <typename T, int HEADS>
__device__ __forceinline__ void rope(const T* __restrict__ x, const float* __restrict__ cs, const float* __restrict__ sn, T* __restrict__ y,
                                     long long total_pos_vec, int S, int H, int D, float sign) {
  const int vec_per_head = D / 8;
  const unsigned groups = (H + HEADS - 1) / HEADS;  // of heads; neighbouring blocks take the groups of the same positions
  const long long v = blockIdx.x / groups * 128ll + threadIdx.x;
  if (v >= total_pos_vec) return;
  const int dv = v % vec_per_head;
  const long long bs = v / vec_per_head;  // b * S + s
  const int s = bs % S;
  const float4 c = *reinterpret_cast<const float4*>(cs + (long long)s * (D / 2) + dv * 4);
  const float4 n = *reinterpret_cast<const float4*>(sn + (long long)s * (D / 2) + dv * 4);
  const float cc[4] = {c.x, c.y, c.z, c.w};
  const float nn[4] = {n.x * sign, n.y * sign, n.z * sign, n.w * sign};
  const long long base = (bs * H) * D + dv * 8;
  const int h0 = blockIdx.x % groups * HEADS, h1 = min(H, h0 + HEADS);
#pragma unroll
  for (int hg = 0; hg < HEADS; hg += 4) {  // four independent loads in flight
    Vec8<T> xv[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (h0 + hg + k < h1) xv[k].load(x + base + (long long)(h0 + hg + k) * D);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (h0 + hg + k >= h1) break;
      float f[8], o[8];
      xv[k].to_float(f);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        o[2 * i] = f[2 * i] * cc[i] - f[2 * i + 1] * nn[i];
        o[2 * i + 1] = f[2 * i] * nn[i] + f[2 * i + 1] * cc[i];
      }
      Vec8<T> ov; ov.from_float(o); ov.store(y + base + (long long)(h0 + hg + k) * D);
    }
  }
}
template <typename T, int HEADS>
__global__ void __launch_bounds__(128) rope_kernel(const T* x, const float* cs, const float* sn, T* y, long long total_pos_vec, int S, int H, int D,
                                                   float sign) {
  after_previous();
  rope<T, HEADS>(x, cs, sn, y, total_pos_vec, S, H, D, sign);
}

// ------------------------------------------------------------------------------------ SwiGLU
template <typename T>
__global__ void __launch_bounds__(256) swiglu_fwd_kernel(const T* a, const T* b, T* y, long long nvec) {
  after_previous();
  const long long v = blockIdx.x * 256ll + threadIdx.x;
  if (v >= nvec) return;
  Vec8<T> av, bv; av.load(a + v * 8); bv.load(b + v * 8);
  float fa[8], fb[8], o[8]; av.to_float(fa); bv.to_float(fb);
#pragma unroll
  for (int i = 0; i < 8; ++i) o[i] = fa[i] / (1.f + __expf(-fa[i])) * fb[i];
  Vec8<T> ov; ov.from_float(o); ov.store(y + v * 8);
}
template <typename T>
__global__ void __launch_bounds__(256) swiglu_bwd_kernel(const T* dy, const T* a, const T* b, T* da, T* db, long long nvec) {
  after_previous();
  const long long v = blockIdx.x * 256ll + threadIdx.x;
  if (v >= nvec) return;
  Vec8<T> gv, av, bv; gv.load(dy + v * 8); av.load(a + v * 8); bv.load(b + v * 8);
  float g[8], fa[8], fb[8], oa[8], ob[8]; gv.to_float(g); av.to_float(fa); bv.to_float(fb);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float sig = 1.f / (1.f + __expf(-fa[i]));
    const float silu = fa[i] * sig;
    oa[i] = g[i] * fb[i] * (sig * (1.f + fa[i] * (1.f - sig)));
    ob[i] = g[i] * silu;
  }
  Vec8<T> o1, o2; o1.from_float(oa); o2.from_float(ob); o1.store(da + v * 8); o2.store(db + v * 8);
}

// ------------------------------------------------------------------------------------ cross-entropy
// One block per row of V logits (V % 8 == 0).  Bound by memory: forward reads the logits once (online maximum and sum of
// exponentials; loss = lse - logit[label]), backward reads and writes them once.  Two independent loads per thread and step
// in most forms; four leave too much of a row to its end (``xent_fwd_threads`` has the times).
// The maximum moves once per step of all its vectors, not once per vector.
constexpr int XENT_UNROLL = 2;
template <typename T>
__global__ void __launch_bounds__(1024) xent_fwd_kernel(const T* logits, const long long* labels, float* loss, float* lse, int V) {
  after_previous();
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const T* lr = logits + row * V;
  float m = -INFINITY, s = 0.f;
  auto take = [&](const Vec8<T>* v, int n) {
    float f[XENT_UNROLL][8];
    float lm = -INFINITY;
#pragma unroll
    for (int k = 0; k < XENT_UNROLL; ++k) {
      if (k < n) {
        v[k].to_float(f[k]);
#pragma unroll
        for (int i = 0; i < 8; ++i) lm = fmaxf(lm, f[k][i]);
      }
    }
    const float nm = fmaxf(m, lm);
    const float ref = nm == -INFINITY ? 0.f : nm;  // (only -inf so far: every term is exp(-inf) = 0)
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < XENT_UNROLL; ++k) {
      if (k < n) {
#pragma unroll
        for (int i = 0; i < 8; ++i) acc += __expf(f[k][i] - ref);
      }
    }
    s = s * __expf(m - ref) + acc;
    m = nm;
  };
  const int step = blockDim.x * 8;
  int c = threadIdx.x * 8;
  for (; c + (XENT_UNROLL - 1) * step < V; c += XENT_UNROLL * step) {
    Vec8<T> v[XENT_UNROLL];
#pragma unroll
    for (int k = 0; k < XENT_UNROLL; ++k) v[k].load(lr + c + k * step);
    take(v, XENT_UNROLL);
  }
  if (c < V) {  // (at most one vector is left)
    Vec8<T> v; v.load(lr + c);
    take(&v, 1);
  }
  const float gm = block_max(m, red);
  s = (m == -INFINITY) ? 0.f : s * __expf(m - gm);
  s = block_sum(s, red);
  if (threadIdx.x == 0) {
    const float l = gm + __logf(s);
    lse[row] = l;
    loss[row] = l - float(lr[labels[row]]);
  }
}
template <typename T, bool PAIRS>
__global__ void __launch_bounds__(1024) xent_bwd_kernel(const float* dloss, const T* logits, const long long* labels, const float* lse,
                                                        T* dlogits, int V) {
  after_previous();
  const long long row = blockIdx.x;
  const T* lr = logits + row * V;
  T* dr = dlogits + row * V;
  const float l = lse[row], g = dloss[row];
  const int lab = (int)labels[row];
  auto put = [&](const Vec8<T>& v, int c) {
    float f[8]; v.to_float(f);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = (__expf(f[i] - l) - ((c + i) == lab ? 1.f : 0.f)) * g;
    Vec8<T> o; o.from_float(f); o.store(dr + c);
  };
  const int step = blockDim.x * 8;
  int c = threadIdx.x * 8;
  if (PAIRS) {
    for (; c + step < V; c += 2 * step) {
      Vec8<T> v[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) v[k].load(lr + c + k * step);
#pragma unroll
      for (int k = 0; k < 2; ++k) put(v[k], c + k * step);
    }
    if (c < V) {
      Vec8<T> v; v.load(lr + c);
      put(v, c);
    }
  } else {
#pragma unroll 1
    for (; c < V; c += step) {
      Vec8<T> v; v.load(lr + c);
      put(v, c);
    }
  }
}

// ------------------------------------------------------------------------------------ embedding forward
// out[token] = weight[ids[token]]: one block per token, 16-byte vectors (D % 8 == 0 for bf16, % 4 for fp32).
__device__ __forceinline__ void copy_row(const uint4* __restrict__ src, uint4* __restrict__ dst, int nvec) {
  for (int c = threadIdx.x; c < nvec; c += blockDim.x) dst[c] = src[c];
}
template <typename T>
__global__ void embedding_fwd_kernel(const T* weight, const long long* ids, T* out, int D, long long num_rows) {
  after_previous();
  const long long tok = blockIdx.x;
  long long r = ids[tok];
  r = r < 0 ? 0 : (r >= num_rows ? num_rows - 1 : r);  // (an id outside the table is the caller's bug; never read outside)
  copy_row(reinterpret_cast<const uint4*>(weight + r * D), reinterpret_cast<uint4*>(out + tok * D), D * (int)sizeof(T) / 16);
}

// ------------------------------------------------------------------------------------ AdamW
// Multi-tensor: a block takes ADAM_PART elements of a tensor, four a thread.  ``pieces`` lists {tensor, first part}: ``whole`` entries of ADAM_RUN parts each,
// then entries of one part, the ends of tensors and small ones (64 blocks for every tensor, however small: 2000 of 128 elements 134 us, so 4.5).
// Bound by memory, 28 or 30 bytes an element.  218 M elements: 65536 / 8192 / 4096 / 1024 to a block 1067 / 1003 / 992 / 963 us.  Where the parameter
// starts on a 16-byte boundary so do the other three (the optimizer sees to it); elsewhere elements are taken one by one.
struct AdamTensor {
  float* p;        // fp32 master / parameter
  const float* g;  // fp32 gradient
  float* m;
  float* v;
  __nv_bfloat16* p_lp;  // optional low-precision copy to emit (may be null)
  long long n;
};
constexpr int ADAM_PART = 1024, ADAM_RUN = 64;  // (optim.py makes the list by both)
// ``hyper`` (optional, device memory): {lr, bc1, bc2} read at run time instead of the launch arguments, so that a step
// captured in a CUDA graph follows the learning-rate schedule and the bias corrections of the step it is replayed for.
__global__ void __launch_bounds__(ADAM_PART / 4) adamw_kernel(const AdamTensor* tensors, const int2* pieces, int whole, float lr,
                             float beta1, float beta2, float eps, float wd, float bc1, float bc2, float grad_scale, const float* hyper) {
  after_previous();
  if (hyper != nullptr) {
    lr = hyper[0];
    bc1 = hyper[1];
    bc2 = hyper[2];
  }
  const int b = blockIdx.x, in_runs = whole * ADAM_RUN;
  const int2 piece = pieces[b < in_runs ? b / ADAM_RUN : whole + b - in_runs];
  const AdamTensor t = tensors[piece.x];
  const long long i = (piece.y + (b < in_runs ? b % ADAM_RUN : 0ll)) * ADAM_PART + threadIdx.x * 4;
  if (i >= t.n) return;
  if (i + 4 <= t.n && ((reinterpret_cast<uintptr_t>(t.p + i) & 15) == 0)) {
    float4 p = *reinterpret_cast<float4*>(t.p + i);
    const float4 g4 = *reinterpret_cast<const float4*>(t.g + i);
    float4 m = *reinterpret_cast<float4*>(t.m + i);
    float4 v = *reinterpret_cast<float4*>(t.v + i);
    float* pp = &p.x; const float* gg = &g4.x; float* mm = &m.x; float* vv = &v.x;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float g = gg[k] * grad_scale;
      mm[k] = beta1 * mm[k] + (1.f - beta1) * g;
      vv[k] = beta2 * vv[k] + (1.f - beta2) * g * g;
      const float mh = mm[k] / bc1;
      const float vh = vv[k] / bc2;
      pp[k] = pp[k] * (1.f - lr * wd) - lr * mh / (sqrtf(vh) + eps);
    }
    *reinterpret_cast<float4*>(t.p + i) = p;
    *reinterpret_cast<float4*>(t.m + i) = m;
    *reinterpret_cast<float4*>(t.v + i) = v;
    if (t.p_lp) {
      if ((reinterpret_cast<uintptr_t>(t.p_lp + i) & 7) == 0) {
        *reinterpret_cast<uint2*>(t.p_lp + i) = make_uint2(pack_bf16(p.x, p.y), pack_bf16(p.z, p.w));
      } else {
        t.p_lp[i] = __float2bfloat16(p.x); t.p_lp[i + 1] = __float2bfloat16(p.y);
        t.p_lp[i + 2] = __float2bfloat16(p.z); t.p_lp[i + 3] = __float2bfloat16(p.w);
      }
    }
  } else {
    for (long long k = i; k < min(i + 4, t.n); ++k) {
      const float g = t.g[k] * grad_scale;
      const float m = beta1 * t.m[k] + (1.f - beta1) * g;
      const float v = beta2 * t.v[k] + (1.f - beta2) * g * g;
      t.m[k] = m; t.v[k] = v;
      const float pn = t.p[k] * (1.f - lr * wd) - lr * (m / bc1) / (sqrtf(v / bc2) + eps);
      t.p[k] = pn;
      if (t.p_lp) t.p_lp[k] = __float2bfloat16(pn);
    }
  }
}

// Blocks of the backward launch: at most ``per_sm`` per SM and, below that, four rows each, so that few rows don't pay for
// more partial rows of dw than they have rows worth summing; but never fewer blocks than rows or SMs allow.
static inline int rms_grid(long long rows, int num_sms, int per_sm) {
  const long long cap = (long long)num_sms * per_sm, quarter = (rows + 3) / 4;
  long long g = quarter < cap ? quarter : cap;
  const long long least = rows < num_sms ? rows : num_sms;
  return (int)(g > least ? g : least);
}
// bulk form: rows short enough for three stages in shared memory
static inline bool rms_bulk(int D, int elem) { return rms_ring_bytes(D * elem) <= 200 * 1024; }
// Threads of a block of the bulk form: a warp per row up to D = 256, one vector per thread up to 256 threads, then two, then
// 512 threads.  Blocks per SM: what shared memory holds, up to 768 threads' worth of rows in flight (1024 for the widest).
struct RmsPlan {
  int threads, nvec, per_sm;
};
static inline RmsPlan rms_plan(int D, int elem) {
  const int vecs = D / 8;
  RmsPlan p;
  p.threads = vecs <= 32 ? 32 : vecs <= 64 ? 64 : vecs <= 128 ? 128 : vecs <= 512 ? 256 : 512;
  const int nv = (vecs + p.threads - 1) / p.threads;
  p.nvec = nv <= 2 ? nv : 4;
  const int by_smem = 220 * 1024 / (rms_ring_bytes(D * elem) + 2048);
  const int by_threads = p.threads == 32 ? 16 : p.threads == 512 ? (p.nvec == 2 ? 2 : 1) : 768 / p.threads;
  p.per_sm = by_smem < 1 ? 1 : by_smem < by_threads ? by_smem : by_threads;
  return p;
}

// Blocks where they add to shared rows: an atomic per column and block, so a block takes four rows, eight where the rows are
// long, unless that would leave more than three quarters of the SMs without any.
static inline int rms_grid_shared(long long rows, int D, int num_sms, int per_sm) {
  const long long cap = (long long)num_sms * per_sm, per_block = D < 2048 ? 4 : 8, least = rows < num_sms / 4 ? rows : num_sms / 4;
  const long long g = (rows + per_block - 1) / per_block;
  return (int)(g < least ? least : g < cap ? g : cap);
}

// Launches the row kernel; returns the number of partial rows of dw (its blocks, or ``shared``), < 0 on error.
template <typename T>
static inline int launch_rms_norm_bwd(const void* dy, const void* x, const void* w, const float* rstd, void* dx, float* dw_base,
                                      int shared, long long rows, int D, int num_sms, cudaStream_t st) {
  const RmsDw dw{dw_base, D, shared};
  if (rms_bulk(D, (int)sizeof(T))) {
    const int smem = rms_ring_bytes(D * (int)sizeof(T));
    const RmsPlan plan = rms_plan(D, (int)sizeof(T));
    const int grid = shared ? rms_grid_shared(rows, D, num_sms, plan.per_sm) : rms_grid(rows, num_sms, plan.per_sm);
#define APB_RMS_BULK(NV, TH)                                                                                             \
  if (plan.nvec == NV && plan.threads == TH) {                                                                           \
    auto kern = rms_norm_bwd_bulk_kernel<T, NV, TH>;                                                                     \
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -4;         \
    launch_after(kern, grid, TH, smem, st, (const T*)dy, (const T*)x, (const T*)w, rstd, (T*)dx, dw, rows, D);                     \
    return shared ? shared : grid;                                                                                       \
  }
    APB_RMS_BULK(1, 32)
    APB_RMS_BULK(1, 64)
    APB_RMS_BULK(1, 128)
    APB_RMS_BULK(1, 256)
    APB_RMS_BULK(2, 256)
    APB_RMS_BULK(2, 512)
    APB_RMS_BULK(4, 512)
#undef APB_RMS_BULK
  }
  // fp32 rows that the ring does not hold (D > 8512): a block of 512 threads keeps a row in registers
  if constexpr (sizeof(T) == 4) {
    const int grid = (int)(rows < num_sms ? rows : num_sms);
    auto kern = D == 512 * 8 * RMS_BWD_MAX_VEC ? rms_norm_bwd_kernel<T, RMS_BWD_MAX_VEC, 1, true> : rms_norm_bwd_kernel<T, RMS_BWD_MAX_VEC, 1, false>;
    launch_after(kern, grid, 512, 0, st, (const T*)dy, (const T*)x, (const T*)w, rstd, (T*)dx, dw, rows, D);
    return shared ? shared : grid;
  }
  return -3;
}

static inline unsigned blocks_for(long long items, int per_block) { return (unsigned)((items + per_block - 1) / per_block); }

// All kernels here read and write 16-byte vectors: the entries refuse (3) a base that is not on such a boundary.
template <typename... P>
static inline bool aligned16(P... p) {
  return ((reinterpret_cast<uintptr_t>(p) | ...) & 15) == 0;
}

}  // namespace apb

using namespace apb;
typedef __nv_bfloat16 bf16;

#define DISPATCH(is_bf16, ...)      \
  if (is_bf16) {                    \
    typedef bf16 T;                 \
    __VA_ARGS__;                    \
  } else {                          \
    typedef float T;                \
    __VA_ARGS__;                    \
  }

extern "C" {

int apb_rms_norm_fwd(const void* x, const void* w, void* y, float* rstd, long long rows, int D, float eps, int is_bf16,
                     cudaStream_t st) {
  if (!aligned16(x, w, y)) return 3;
  if (D % 8) return 3;
  if (rows == 0) return 0;
  if (D <= 32 * 8 * 4) {
    // one warp per row, eight rows per block
    const int nvec = (D + 255) / 256;
    const unsigned grid = blocks_for(rows, 8);
#define APB_RMS_FWD_W(NV) DISPATCH(is_bf16, launch_after(rms_norm_fwd_kernel<T, NV, true>, grid, 256, 0, st, (const T*)x, (const T*)w, (T*)y, rstd, rows, D, eps))
    if (nvec == 1) { APB_RMS_FWD_W(1); } else if (nvec == 2) { APB_RMS_FWD_W(2); } else { APB_RMS_FWD_W(4); }
#undef APB_RMS_FWD_W
  } else {
    // The threads of a row's block, and with them the order of its sum, follow from D alone: a row gives the same bits whatever other rows are in the
    // call (a rule by rows as well was faster, 64 x 4096 bf16 1.8 -> 1.6 us, 8192 x 1536 13.3 -> 11.3, but changed the bits and, with 16 squares to a
    // thread instead of 8, made the error of the sum 1 to 2 % larger).
    // Blocks end with their row, or, for bf16, take rows in turn, 8 (or 2048 threads) to an SM: row by row -> in turn 1024 x 1032 2.0 -> 2.3 us, 4096 x 1032
    // 7.1 -> 6.8, 32768 x 1032 43 -> 38, 1024 x 2048 3.1 -> 3.2, 4096 x 2048 8.6 -> 8.5, 512 x 2560 2.5 -> 2.3, 8192 x 3072 22.1 -> 18.6, x 4096 26.8 -> 25.6,
    // x 8192 49.3 -> 44.7; fp32 8192 x 2048 23.6 -> 29.4, x 4096 42.0 -> 52.7, x 8192 82.7 -> 87.9.
    int threads = 256;
    while (threads * 8 * 4 < D && threads < 1024) threads *= 2;
    const int nvec = (D + threads * 8 - 1) / (threads * 8);
    if (nvec > 4) return 3;
    unsigned grid = (unsigned)rows;
    const bool in_turn = is_bf16 && (D > 2048 || rows >= 4096);
    if (in_turn) {
      int dev = 0, sms = 148;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      const long long cap = (long long)sms * (threads >= 1024 ? 2 : threads >= 512 ? 4 : 8);
      if (rows > cap) grid = (unsigned)cap;
    }
#define APB_RMS_FWD_B(NV)                                                                                                                             \
  if (in_turn) launch_after(rms_norm_fwd_kernel<bf16, NV, false, true>, grid, threads, 0, st, (const bf16*)x, (const bf16*)w, (bf16*)y, rstd, rows, D, eps); \
  else DISPATCH(is_bf16, launch_after(rms_norm_fwd_kernel<T, NV, false>, grid, threads, 0, st, (const T*)x, (const T*)w, (T*)y, rstd, rows, D, eps))
    if (nvec == 1) { APB_RMS_FWD_B(1); } else if (nvec == 2) { APB_RMS_FWD_B(2); } else { APB_RMS_FWD_B(4); }
#undef APB_RMS_FWD_B
  }
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

// floats of workspace for apb_rms_norm_bwd: one partial row of dw per block (the form for wide fp32 rows has one block per SM, as
// the plan for such rows does)
long long apb_rms_norm_bwd_workspace(long long rows, int D, int is_bf16, int num_sms) {
  return (long long)rms_grid(rows, num_sms, rms_plan(D, is_bf16 ? 2 : 4).per_sm) * D;
}

int apb_rms_norm_bwd(const void* dy, const void* x, const void* w, const float* rstd, void* dx, void* dw, float* part,
                     long long rows, int D, int is_bf16, int num_sms, cudaStream_t st) {
  if (!aligned16(dy, x, w, dx, part)) return 3;
  if (D % 8) return 3;
  if (D > 512 * 8 * RMS_BWD_MAX_VEC) return 3;
  int n = 0;
  if (rows > 0) {
    DISPATCH(is_bf16, n = launch_rms_norm_bwd<T>(dy, x, w, rstd, dx, part, 0, rows, D, num_sms, st));
    if (n < 0) return -n;
  }
  DISPATCH(is_bf16, launch_after(rms_dw_kernel<T>, (D + 31) / 32, 1024, 0, st, part, (T*)dw, n, D));
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

int apb_cast(const void* src, void* dst, long long n, int src_bf16, int dst_bf16, int num_sms, cudaStream_t st) {
  if (!aligned16(src, dst)) return 3;
  if (n == 0) return 0;
  const unsigned grid = blocks_for((n + 7) / 8, 256);
  if (src_bf16 && !dst_bf16) launch_after(cast_kernel<bf16, float>, grid, 256, 0, st, (const bf16*)src, (float*)dst, n);
  else if (!src_bf16 && dst_bf16) launch_after(cast_kernel<float, bf16>, grid, 256, 0, st, (const float*)src, (bf16*)dst, n);
  else return 3;
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

// ``count`` fp32 tensors to bf16, CAST_MANY to a launch; 16-byte bases.  Returns 0, or an argument / launch error; ``launches`` are counted.
int apb_cast_many(const void* const* src, void* const* dst, const long long* n, int count, int* launches, cudaStream_t st) {
  for (int i = 0; i < count; ++i)
    if (!aligned16(src[i], dst[i]) || n[i] < 0 || n[i] > (1ll << 31)) return 3;
  *launches = 0;
  for (int i = 0; i < count;) {
    CastMany t;
    int used = 0;
    long long blocks = 0;
    for (; i < count && used < CAST_MANY; ++i) {
      const long long b = blocks_for(n[i], 2048);
      if (b == 0) continue;
      if (blocks + b > 0x3fffffff) break;
      t.src[used] = (const float*)src[i];
      t.dst[used] = (bf16*)dst[i];
      t.n[used] = n[i];
      t.first[used++] = (int)blocks;
      blocks += b;
    }
    if (used == 0) break;
    for (int k = used; k < CAST_MANY; ++k) t.first[k] = 0x7fffffff;
    launch_after(cast_many_kernel, (unsigned)blocks, 256, 0, st, t);
    ++*launches;
  }
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

int apb_rope(const void* x, const float* cs, const float* sn, void* y, long long B, int S, int H, int D, int conj,
             int is_bf16, int num_sms, cudaStream_t st) {
  if (!aligned16(x, cs, sn, y)) return 3;
  if (D % 8) return 3;
  const long long nvec = B * S * (D / 8);  // one thread per (position, 8-element group); the kernel walks the heads
  if (nvec == 0 || H == 0) return 0;
  const float sign = conj ? -1.f : 1.f;
  const int heads = nvec * ((H + 7) / 8) >= 768ll * num_sms ? 8 : 4;
  const unsigned grid = blocks_for(nvec, 128) * (unsigned)((H + heads - 1) / heads);
  if (heads == 8) {
    DISPATCH(is_bf16, launch_after(rope_kernel<T, 8>, grid, 128, 0, st, (const T*)x, cs, sn, (T*)y, nvec, S, H, D, sign));
  } else {
    DISPATCH(is_bf16, launch_after(rope_kernel<T, 4>, grid, 128, 0, st, (const T*)x, cs, sn, (T*)y, nvec, S, H, D, sign));
  }
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

int apb_swiglu_fwd(const void* a, const void* b, void* y, long long n, int is_bf16, int num_sms, cudaStream_t st) {
  if (!aligned16(a, b, y)) return 3;
  if (n % 8) return 3;
  if (n == 0) return 0;
  DISPATCH(is_bf16, launch_after(swiglu_fwd_kernel<T>, blocks_for(n / 8, 256), 256, 0, st, (const T*)a, (const T*)b, (T*)y, n / 8));
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

int apb_swiglu_bwd(const void* dy, const void* a, const void* b, void* da, void* db, long long n, int is_bf16, int num_sms,
                   cudaStream_t st) {
  if (!aligned16(dy, a, b, da, db)) return 3;
  if (n % 8) return 3;
  if (n == 0) return 0;
  DISPATCH(is_bf16, launch_after(swiglu_bwd_kernel<T>, blocks_for(n / 8, 256), 256, 0, st, (const T*)dy, (const T*)a, (const T*)b,
                                                                                       (T*)da, (T*)db, n / 8));
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

// Threads of a row's block.  Swept over 8 ... 256000 columns, 64 ... 8192 rows, both
// types, one, two and four vectors a step, 128 ... 1024 threads, against one vector a step and 256 threads (from 8192 columns on 1024).
// Forward: short rows waste large blocks on the reduction, long ones small blocks on latency; with at most two rows per SM the
// row itself is the latency.  8192 rows of bf16: 4096 columns 18.6 -> 15.4 us, 32064 132 -> 87, 128256 392 -> 314.
// Backward, bf16: two vectors a step (8192 x 32064 177 -> 158 us, 128256 646 -> 629).
// Backward, fp32: one, and not unrolled (8192 x 128256 1285 us; 1352 where the compiler unrolls the loop, 1346 with four).
static int xent_fwd_threads(long long rows, int V, bool is_bf16) {
  if (rows <= 2 * 148) return V <= 8192 ? 256 : V <= 16384 ? 512 : 1024;
  return V <= (is_bf16 ? 8192 : 4096) ? 128 : V < 36000 ? 256 : V < 140000 ? 512 : 1024;
}
static int xent_bwd_threads(int V, bool is_bf16) { return V < 8192 ? 256 : is_bf16 && V < 24000 ? 512 : 1024; }

int apb_xent_fwd(const void* logits, const long long* labels, float* loss, float* lse, long long rows, int V, int is_bf16,
                 cudaStream_t st) {
  if (!aligned16(logits)) return 3;
  if (V % 8) return 3;
  if (rows == 0) return 0;
  const int threads = xent_fwd_threads(rows, V, is_bf16);
  DISPATCH(is_bf16, launch_after(xent_fwd_kernel<T>, (unsigned)rows, threads, 0, st, (const T*)logits, labels, loss, lse, V));
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

int apb_xent_bwd(const float* dloss, const void* logits, const long long* labels, const float* lse, void* dlogits,
                 long long rows, int V, int is_bf16, cudaStream_t st) {
  if (!aligned16(logits, dlogits)) return 3;
  if (V % 8) return 3;
  if (rows == 0) return 0;
  const int threads = xent_bwd_threads(V, is_bf16);
  if (is_bf16) launch_after(xent_bwd_kernel<bf16, true>, (unsigned)rows, threads, 0, st, dloss, (const bf16*)logits, labels, lse, (bf16*)dlogits, V);
  else launch_after(xent_bwd_kernel<float, false>, (unsigned)rows, threads, 0, st, dloss, (const float*)logits, labels, lse, (float*)dlogits, V);
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

int apb_embedding_fwd(const void* weight, const long long* ids, void* out, long long tokens, int D, long long num_rows,
                      int is_bf16, cudaStream_t st) {
  if (!aligned16(weight, out)) return 3;
  if (tokens == 0) return 0;
  if ((D * (is_bf16 ? 2 : 4)) % 16) return 3;
  DISPATCH(is_bf16, launch_after(embedding_fwd_kernel<T>, (unsigned)tokens, 128, 0, st, (const T*)weight, ids, (T*)out, D, num_rows));
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

int apb_adamw(const void* tensors_dev, const void* pieces_dev, int num_pieces, int whole, float lr, float beta1, float beta2, float eps, float wd,
              float bc1, float bc2, float grad_scale, const float* hyper_dev, cudaStream_t st) {
  if (num_pieces == 0) return 0;
  launch_after(adamw_kernel, (unsigned)whole * ADAM_RUN + (unsigned)(num_pieces - whole), ADAM_PART / 4, 0, st, (const AdamTensor*)tensors_dev,
               (const int2*)pieces_dev, whole, lr, beta1, beta2, eps, wd, bc1, bc2, grad_scale, hyper_dev);
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

}  // extern "C"

// ------------------------------------------------------------------------------------------------
// Allocation-free RMSNorm backward (see apb_noalloc.h for the contract).
// ------------------------------------------------------------------------------------------------
#include <atomic>
#include <mutex>

#include "apb_noalloc.h"

// The weight-gradient accumulator.  In host code this name is only a handle for the runtime's
// symbol table, never a pointer a kernel could use: its device address is fetched once per device
// with cudaGetSymbolAddress below.
static __device__ __align__(256) float g_noalloc_dw_acc[APB_NOALLOC_MAX_D];

namespace {
constexpr int kMaxDevices = 64;
// The pointer is published with a release store after the SM count has been written, and read with
// an acquire load: a thread that sees the pointer also sees the count, without taking the mutex.
std::atomic<float*> g_noalloc_ptr[kMaxDevices] = {};
int g_noalloc_sms[kMaxDevices] = {};
std::mutex g_noalloc_mutex;

// One-time per-device set-up; the caller's current device is the one being set up.
int noalloc_setup(int dev) {
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (g_noalloc_ptr[dev].load(std::memory_order_acquire) != nullptr) return APB_NOALLOC_OK;
  float* p = nullptr;
  if (cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_noalloc_dw_acc) != cudaSuccess || p == nullptr) {
    (void)cudaGetLastError();
    return APB_NOALLOC_ERR_SETUP;
  }
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) {
    (void)cudaGetLastError();
    return APB_NOALLOC_ERR_SETUP;
  }
  g_noalloc_sms[dev] = sms;
  g_noalloc_ptr[dev].store(p, std::memory_order_release);
  return APB_NOALLOC_OK;
}
}  // namespace

extern "C" int apb_rms_norm_bwd_noalloc(const void* dy, const void* x, const void* w, const float* rstd, void* dx, void* dw,
                                        long long rows, int D, int is_bf16, cudaStream_t st) {
  if (D <= 0 || rows < 0 || (D % 8) != 0) return APB_NOALLOC_ERR_BAD_SHAPE;
  if (D > APB_NOALLOC_MAX_D) return APB_NOALLOC_ERR_TOO_LARGE;
  if (!aligned16(dy, x, w, dx, dw)) return APB_NOALLOC_ERR_ALIGNMENT;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return APB_NOALLOC_ERR_SETUP;
  float* acc = g_noalloc_ptr[dev].load(std::memory_order_acquire);
  if (acc == nullptr) {
    const int e = noalloc_setup(dev);
    if (e != APB_NOALLOC_OK) return e;
    acc = g_noalloc_ptr[dev].load(std::memory_order_acquire);
  }
  const int num_sms = g_noalloc_sms[dev];
  // The blocks share partial rows, one for sixteen of them as far as the array goes: all adding to one row would spend most of
  // the time on its D addresses (16384 x 256 bf16: 197 us with one row, 20.6 with 37).
  const int blocks = rms_grid_shared(rows, D, num_sms, rms_plan(D, is_bf16 ? 2 : 4).per_sm), most = APB_NOALLOC_MAX_D / D;
  const int shared = blocks < 80 ? 1 : (blocks / 16 < most ? blocks / 16 : most);
  // the array keeps the previous call's sums: start from zero
  if (cudaMemsetAsync(acc, 0, sizeof(float) * shared * D, st) != cudaSuccess) return APB_NOALLOC_ERR_LAUNCH;
  if (rows > 0) {
    int n;
    DISPATCH(is_bf16, n = launch_rms_norm_bwd<T>(dy, x, w, rstd, dx, acc, shared, rows, D, num_sms, st));
    if (n < 0) return APB_NOALLOC_ERR_BAD_SHAPE;
  }
  if (shared > 1) {
    DISPATCH(is_bf16, launch_after(rms_dw_kernel<T>, (D + 31) / 32, 1024, 0, st, acc, (T*)dw, shared, D));
  } else if (is_bf16) {
    launch_after(cast_kernel<float, bf16>, blocks_for(D / 8, 256), 256, 0, st, acc, (bf16*)dw, D);
  } else {
    if (cudaMemcpyAsync(dw, acc, sizeof(float) * D, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
      return APB_NOALLOC_ERR_LAUNCH;
  }
  return cudaGetLastError() == cudaSuccess ? APB_NOALLOC_OK : APB_NOALLOC_ERR_LAUNCH;
}

extern "C" const char* apb_noalloc_strerror(int code) {
  switch (code) {
    case APB_NOALLOC_OK: return "ok";
    case APB_NOALLOC_ERR_BAD_SHAPE: return "bad shape: D must be a positive multiple of 8 and rows >= 0";
    case APB_NOALLOC_ERR_LAUNCH: return "CUDA launch failed";
    case APB_NOALLOC_ERR_TOO_LARGE: return "D exceeds APB_NOALLOC_MAX_D (16384): the built-in scratch array is too small";
    case APB_NOALLOC_ERR_SETUP: return "could not obtain the device address of the built-in scratch array";
    case APB_NOALLOC_ERR_ALIGNMENT: return "dy, x, w, dx and dw must start on 16-byte boundaries";
    default: return "unknown error code";
  }
}
