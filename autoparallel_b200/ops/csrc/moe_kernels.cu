// Index kernels of the mixture-of-experts dispatch (capacity based, block local; semantics in ops/moe_ops.py):
//
//   moe_slots     arrival rank of every (token, choice) inside its expert, per token block, in token-major order
//                 -> row of the block's [E * C] buffer, or E * C for an assignment beyond the capacity
//   moe_scatter   buf[e, blk, c, :] = w[t, j] * src[t, :]            (buffer [E, nb, C, d]; every row is written here, the empty ones with zeros)
//   moe_gather    out[t, :] = sum_j w[t, j] * buf[slot[t, j], :]     (dropped assignments contribute nothing)
//   moe_gate_grad dw[t, j] = < buf[slot[t, j], :], g[t, :] >
//
// The counterpart in the reference is its one hand-written device kernel, the Triton permutation-index kernel of its
// DeepSeek-V3 test model (autoparallel/_testing/models/dsv3.py:62-91), which turns rank-major token order into expert-major
// order with per-expert padding; here the same job is a counting pass over static-capacity buffers.
//
// All four are bound by memory or latency; they exist so that the dispatch is a few launches instead of a few dozen index
// kernels, and so that no intermediate [T * k, d] tensor is materialised.
//
// Rows travel as 16-byte vectors, or element by element where a row is not a whole number of them or a base is not
// aligned.  Times below: 8192 tokens, top-8 of 64 experts, capacity 1280, d = 2048, bf16 (one B200, before -> after).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "launch.cuh"

namespace apb {

// Slots: latency bound.  The arrival rank of an assignment is the number of earlier ones of its token block with the same
// expert.  The assignments of a block are cut into chunks, one CTA each: the first kernel counts every chunk's experts,
// the second adds up the counts of the chunks before its own and ranks its assignments round by round.
// 170 -> 7.4 us (one CTA walked the block in rounds of 1024 before).
constexpr int SLOT_THREADS = 512;

__global__ void __launch_bounds__(SLOT_THREADS) moe_count_kernel(const long long* gate_idx, int* counts, int per_block, int chunk, int nchunks,
                                                                 int E) {
  after_previous();
  extern __shared__ int smem_i[];
  const int blk = blockIdx.x / nchunks, ch = blockIdx.x % nchunks;
  for (int e = threadIdx.x; e < E; e += blockDim.x) smem_i[e] = 0;
  __syncthreads();
  const long long* in = gate_idx + (long long)blk * per_block;
  const int end = (int)min((long long)per_block, ((long long)ch + 1) * chunk);
  for (int i = ch * chunk + threadIdx.x; i < end; i += blockDim.x) {
    const long long e = in[i];
    if (e >= 0 && e < E) atomicAdd(smem_i + e, 1);
  }
  __syncthreads();
  int* out = counts + (long long)blockIdx.x * E;
  for (int e = threadIdx.x; e < E; e += blockDim.x) out[e] = smem_i[e];
}

// Shared memory: base[E] (assignments of each expert seen so far) and wcnt[warps][E] (those of each warp in this round).
__global__ void __launch_bounds__(SLOT_THREADS) moe_slots_kernel(const long long* gate_idx, long long* slot, const int* counts, int per_block,
                                                                 int chunk, int nchunks, int E, int C) {
  after_previous();
  extern __shared__ int smem_i[];
  const int blk = blockIdx.x / nchunks, ch = blockIdx.x % nchunks;
  int* base = smem_i;
  int* wcnt = smem_i + E;
  const int nwarps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long* in = gate_idx + (long long)blk * per_block;
  long long* out = slot + (long long)blk * per_block;
  for (int i = threadIdx.x; i < E * (nwarps + 1); i += blockDim.x) smem_i[i] = 0;
  __syncthreads();
  if (ch > 0) {  // chunks before this one: threads share the chunks of an expert
    const int* cnt = counts + (long long)blk * nchunks * E;
    const int groups = max(1, (int)blockDim.x / E);
    for (int x = threadIdx.x; x < E * groups; x += blockDim.x) {
      const int e = x % E;
      int s = 0;
#pragma unroll 4
      for (int c = x / E; c < ch; c += groups) s += cnt[(long long)c * E + e];
      atomicAdd(base + e, s);
    }
    __syncthreads();
  }
  const int end = (int)min((long long)per_block, ((long long)ch + 1) * chunk);
  for (int start = ch * chunk; start < end; start += blockDim.x) {
    const int i = start + threadIdx.x;
    const bool valid = i < end;
    const long long raw = valid ? in[i] : -1;
    const bool ok = raw >= 0 && raw < E;
    const int e = (int)raw;
    const unsigned active = __ballot_sync(0xffffffffu, ok);
    int lane_rank = 0;
    if (ok) {
      const unsigned same = __match_any_sync(active, e);
      lane_rank = __popc(same & ((1u << lane) - 1u));
      if (lane_rank == 0) wcnt[warp * E + e] = __popc(same);
    }
    __syncthreads();
    if (ok) {
      int pos = base[e] + lane_rank;
      for (int w = 0; w < warp; ++w) pos += wcnt[w * E + e];
      out[i] = pos < C ? (long long)e * C + pos : (long long)E * C;
    } else if (valid) {
      out[i] = (long long)E * C;
    }
    if (start + (int)blockDim.x >= end) break;  // (uniform)
    __syncthreads();
    for (int x = threadIdx.x; x < E; x += blockDim.x) {
      int s = 0;
      for (int w = 0; w < nwarps; ++w) {
        s += wcnt[w * E + x];
        wcnt[w * E + x] = 0;
      }
      base[x] += s;
    }
    __syncthreads();
  }
}

template <typename T>
__device__ __forceinline__ float to_f(T v);
template <>
__device__ __forceinline__ float to_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T>
__device__ __forceinline__ T from_f(float v);
template <>
__device__ __forceinline__ float from_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16(v); }

// W consecutive elements of a row: one 16-byte vector, or one element
template <typename T, int W>
struct alignas(W == 1 ? sizeof(T) : 16) Pack {
  T v[W];
};

// the gate weight in the operand's precision (as the reference formula applies it); stored as fp32 or bf16
template <typename T>
__device__ __forceinline__ float gate_weight(const void* w, long long a, int w_bf16) {
  const float f = w_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(w)[a]) : reinterpret_cast<const float*>(w)[a];
  return to_f<T>(from_f<T>(f));
}

// row of buf [E, nb, C, d] addressed by (slot in the block's [E * C] buffer, block); -1 when the assignment was dropped
__device__ __forceinline__ long long buf_row(long long s, int blk, int E, int C, int nb) {
  if (s < 0 || s >= (long long)E * C) return -1;
  if ((long long)E * C <= 0x7fffffffll) {  // 32-bit division
    const int e = (int)s / C;
    return ((long long)e * nb + blk) * C + ((int)s - e * C);
  }
  const long long e = s / C, c = s % C;
  return (e * nb + blk) * C + c;
}

// token block of assignment ``a`` (64-bit divisions only where there is more than one block)
__device__ __forceinline__ int block_of(long long a, int k, long long tokens_per_block, int nb) { return nb == 1 ? 0 : (int)(a / k / tokens_per_block); }

// Scatter: every buffer row is written exactly once, with its assignment's weighted token or with zeros, so the buffer is
// not zero-filled first.  ``inv`` names the assignment of a row; rows that none names hold whatever the memory held, so a
// row's entry counts only if that assignment's slot leads back to the row.  Where several do, the last of them has the row, as if they were stored in
// order: whoever takes a later one out of the entry puts it back, so that of all that name the row none but the last is left, in whatever order
// the threads come.
// 136 -> 69 us (zero fill and 2-byte copies before).
__global__ void moe_inverse_kernel(const long long* slot, long long* inv, long long n, int k, long long tokens_per_block, int E, int C, int nb) {
  after_previous();
  const long long a = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= n) return;
  auto row_of = [&](long long i) { return buf_row(slot[i], block_of(i, k, tokens_per_block, nb), E, C, nb); };
  const long long row = row_of(a);
  if (row < 0) return;
  unsigned long long* entry = reinterpret_cast<unsigned long long*>(inv) + row;
  for (long long put = a;;) {  // (``put`` grows: it ends)
    const long long was = (long long)atomicExch(entry, (unsigned long long)put);
    if (was <= put || was >= n || row_of(was) != row) break;
    put = was;  // a later assignment of the row: back with it
  }
}

// The words of a Pack: the bf16 values of a vector that waits for its turn stay in 4 registers (as values they take 8).
template <typename T, int W>
struct RawOf { typedef uint4 type; };
template <typename T>
struct RawOf<T, 1> { typedef T type; };
template <typename T, int W>
using Raw = typename RawOf<T, W>::type;
template <typename T, int W>
__device__ __forceinline__ Pack<T, W> weighted(const Raw<T, W>& raw, float wt) {
  Pack<T, W> out;
  const Pack<T, W> in = *reinterpret_cast<const Pack<T, W>*>(&raw);
#pragma unroll
  for (int c = 0; c < W; ++c) out.v[c] = from_f<T>(to_f<T>(in.v[c]) * wt);
  return out;
}

// 16-byte vectors may be stored to leave L2 first
template <bool STREAM, typename T, int W>
__device__ __forceinline__ void put(T* p, const Pack<T, W>& v) {
  if constexpr (STREAM && W > 1) __stcs(reinterpret_cast<uint4*>(p), *reinterpret_cast<const uint4*>(&v));
  else *reinterpret_cast<Pack<T, W>*>(p) = v;
}

// one warp per buffer row.  STREAM (buffers of more than half of L2): the rows leave L2 first, which keeps the tokens in it; they were read from memory
// three times over.  64 x 1280 x 2048, 8192 tokens 71.7 -> 65.1 us, 32 x 1280 x 1024 19.3 -> 18.0; 8 x 2560 x 128 7.5 -> 7.7.
template <typename T, int W, bool STREAM>
__global__ void __launch_bounds__(256, 8) moe_scatter_kernel(const T* src, const long long* slot, const void* w, int w_bf16, const long long* inv, T* buf,
                                                          long long n, int k, long long tokens_per_block, int d, long long rows, int E, int C, int nb) {
  after_previous();
  const long long row = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const long long a = inv[row];
  T* y = buf + row * d;
  const bool named = a >= 0 && a < n;
  const long long to = named ? slot[a] : -1;
  const float wt = named ? gate_weight<T>(w, a, w_bf16) : 0.f;  // (under way with the slot)
  if (!named || buf_row(to, block_of(a, k, tokens_per_block, nb), E, C, nb) != row) {
    const Pack<T, W> zero{};
    for (int i = lane * W; i < d; i += 32 * W) put<STREAM>(y + i, zero);
    return;
  }
  const T* x = src + a / k * d;
#pragma unroll 1
  for (int i = lane * W; i < d; i += 4 * 32 * W) {  // four loads under way
    Raw<T, W> v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (i + q * 32 * W < d) v[q] = *reinterpret_cast<const Raw<T, W>*>(x + i + q * 32 * W);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (i + q * 32 * W < d) put<STREAM>(y + i + q * 32 * W, weighted<T, W>(v[q], wt));
  }
}

// Gather: bound by reading k rows per token.  One warp per token and share of its columns: the lanes work out the rows and weights of up to
// 32 choices at once and pass them round by shuffles, and the loads of eight choices are under way together for every 512 bytes of the
// result, without a branch (a dropped choice loads nothing and adds zero).  Blocks of 256 threads that shared rows and weights of one
// token through shared memory spent most of their life waiting for the slots, and 2-byte values in registers cost as much as the loads:
// 97 -> 65 us; 32768 tokens 370 -> 230.  (Before that: 371 us, one row address per element.)
constexpr int GATHER_K = 8;
// acc += wt * v, element by element
__device__ __forceinline__ void add_weighted(float (&acc)[8], float wt, const Pack<__nv_bfloat16, 8>& v) {
  const uint4 r = *reinterpret_cast<const uint4*>(&v);
  const uint32_t x[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    acc[2 * i] += wt * __uint_as_float(x[i] << 16);
    acc[2 * i + 1] += wt * __uint_as_float(x[i] & 0xffff0000u);
  }
}
template <typename T, int W>
__device__ __forceinline__ void add_weighted(float (&acc)[W], float wt, const Pack<T, W>& v) {
#pragma unroll
  for (int c = 0; c < W; ++c) acc[c] += wt * to_f<T>(v.v[c]);
}
// MIN_BLOCKS: 8 hold the kernel to 64 registers (80 without), a third more loads under way: 8192 tokens 62.5 -> 53.6 us (5.6 TB/s), 1000 10.9 -> 8.7;
// where the launch does not fill the SMs it is the latency of one token that counts, 333 tokens 3.6 -> 4.3.
template <typename T, int W, int MIN_BLOCKS>
__global__ void __launch_bounds__(128, MIN_BLOCKS) moe_gather_kernel(const T* buf, const long long* slot, const void* w, int w_bf16, T* out,
                                                         long long Tn, int k, long long tokens_per_block, int d, int E, int C, int nb) {
  after_previous();
  const long long t = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (t >= Tn) return;  // (a whole warp)
  const int blk = (int)(t / tokens_per_block);
  const T* my_row = nullptr;  // of choice ``lane``; null where it was dropped
  float my_wt = 0.f;
  auto choice = [&](int j) {
    const long long row = j < k ? buf_row(slot[t * k + j], blk, E, C, nb) : -1;
    my_row = row >= 0 ? buf + row * d : nullptr;
    my_wt = row >= 0 ? gate_weight<T>(w, t * k + j, w_bf16) : 0.f;
  };
  choice(lane);
#pragma unroll 1
  for (int col = ((int)blockIdx.y * 32 + lane) * W; col - lane * W < d; col += (int)gridDim.y * 32 * W) {
    float acc[W] = {};
#pragma unroll 1
    for (int j0 = 0; j0 < k; j0 += GATHER_K) {
      if (k > 32 && j0 % 32 == 0) choice(j0 + lane);
      Pack<T, W> in[GATHER_K];
#pragma unroll
      for (int j = 0; j < GATHER_K; ++j) {
        const T* x = reinterpret_cast<const T*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(my_row), (j0 + j) & 31));
        in[j] = Pack<T, W>{};  // (a dropped choice adds zero times zero, which changes no sum)
        if (x != nullptr && col < d) in[j] = *reinterpret_cast<const Pack<T, W>*>(x + col);
      }
#pragma unroll
      for (int j = 0; j < GATHER_K; ++j) add_weighted(acc, __shfl_sync(0xffffffffu, my_wt, (j0 + j) & 31), in[j]);
    }
    if (col < d) {
      Pack<T, W> o;
#pragma unroll
      for (int c = 0; c < W; ++c) o.v[c] = from_f<T>(acc[c]);
      *reinterpret_cast<Pack<T, W>*>(out + t * d + col) = o;
    }
  }
}

// one warp per assignment; the choices of a token sit in one block, so its gradient row comes from cache after the first
// 118 -> 61 us (2-byte loads before)
template <typename T, int W>
__global__ void __launch_bounds__(256) moe_gate_grad_kernel(const T* buf, const long long* slot, const T* g, float* dw, long long n, int k,
                                                            long long tokens_per_block, int d, int E, int C, int nb) {
  after_previous();
  const long long a = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (a >= n) return;
  const long long t = a / k;
  const long long row = buf_row(slot[a], (int)(t / tokens_per_block), E, C, nb);
  float acc = 0.f;
  if (row >= 0) {
    const T* x = buf + row * d;
    const T* y = g + t * d;
#pragma unroll 4
    for (int i = lane * W; i < d; i += 32 * W) {
      const Pack<T, W> xv = *reinterpret_cast<const Pack<T, W>*>(x + i);
      const Pack<T, W> yv = *reinterpret_cast<const Pack<T, W>*>(y + i);
#pragma unroll
      for (int c = 0; c < W; ++c) acc += to_f<T>(xv.v[c]) * to_f<T>(yv.v[c]);
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) dw[a] = acc;
}

}  // namespace apb

using namespace apb;

static int launch_status() { return (int)cudaGetLastError(); }

static int slot_threads(int per_block) { return per_block >= SLOT_THREADS ? SLOT_THREADS : ((per_block + 31) / 32) * 32; }

// assignments per CTA: one round, more once that would be over two CTAs per SM (the prefix of every CTA reads all earlier counts).
// Up to two rounds stay with one CTA: a second round costs less than the count kernel's launch (1024 assignments: 4.2 us against 6.3).
static int slot_chunk(int num_blocks, int per_block, int num_sms) {
  const int threads = slot_threads(per_block);
  if (per_block <= 2 * threads) return per_block;
  const long long rounds = ((long long)num_blocks * per_block + 2ll * num_sms * threads - 1) / (2ll * num_sms * threads);
  const long long chunk = rounds * threads;
  return chunk < per_block ? (int)chunk : per_block;
}

// Largest expert count the slot kernel takes for ``per_block`` assignments per token block (48 KB of static-limit shared memory).
extern "C" int apb_moe_slots_max_experts(int per_block) { return (48 * 1024 / 4) / ((slot_threads(per_block) >> 5) + 1); }

// ints of workspace for apb_moe_slots; 0 for the sizes that it refuses
extern "C" long long apb_moe_slots_workspace(int num_blocks, int per_block, int E, int num_sms) {
  if (num_blocks <= 0 || per_block <= 0 || E <= 0) return 0;
  const int chunk = slot_chunk(num_blocks, per_block, num_sms);
  return (long long)num_blocks * ((per_block + chunk - 1) / chunk) * E;
}

extern "C" int apb_moe_slots(const long long* gate_idx, long long* slot, int* counts, int num_blocks, int per_block, int E, int C,
                             int num_sms, cudaStream_t st) {
  if (num_blocks <= 0 || per_block <= 0 || E <= 0 || C <= 0) return (int)cudaErrorInvalidValue;
  if (E > apb_moe_slots_max_experts(per_block)) return (int)cudaErrorInvalidValue;
  const int threads = slot_threads(per_block);
  const int chunk = slot_chunk(num_blocks, per_block, num_sms);
  const int nchunks = (per_block + chunk - 1) / chunk;
  const unsigned grid = (unsigned)((long long)nchunks * num_blocks);
  if (nchunks > 1) launch_after(moe_count_kernel, grid, threads, (size_t)E * sizeof(int), st, gate_idx, counts, per_block, chunk, nchunks, E);
  const size_t smem = (size_t)E * ((threads >> 5) + 1) * sizeof(int);
  launch_after(moe_slots_kernel, grid, threads, smem, st, gate_idx, slot, counts, per_block, chunk, nchunks, E, C);
  return launch_status();
}

static bool vec_rows(int d, int elem_bytes, const void* p, const void* q) {
  return (d * (long long)elem_bytes) % 16 == 0 && ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(q)) & 15) == 0;
}

#define APB_MOE_DISPATCH(is_bf16, vec, ...)                   \
  if (is_bf16) {                                              \
    typedef __nv_bfloat16 T;                                  \
    if (vec) { constexpr int W = 8; __VA_ARGS__; }            \
    else { constexpr int W = 1; __VA_ARGS__; }                \
  } else {                                                    \
    typedef float T;                                          \
    if (vec) { constexpr int W = 4; __VA_ARGS__; }            \
    else { constexpr int W = 1; __VA_ARGS__; }                \
  }

// ``inv``: E * nb * C int64 of workspace; every element of buf is written
extern "C" int apb_moe_scatter(const void* src, const long long* slot, const void* w, int w_bf16, long long* inv, void* buf, long long T_, int k,
                               int d, int E, int C, int nb, int is_bf16, cudaStream_t st) {
  if (T_ <= 0 || k <= 0 || d <= 0 || nb <= 0 || T_ % nb) return (int)cudaErrorInvalidValue;
  const long long n = T_ * k, rows = (long long)E * nb * C;
  if (rows <= 0) return 0;
  const long long tpb = T_ / nb;
  launch_after(moe_inverse_kernel, (unsigned)((n + 255) / 256), 256, 0, st, slot, inv, n, k, tpb, E, C, nb);
  const bool stream = rows * d * (is_bf16 ? 2 : 4) > 64000000ll;
  APB_MOE_DISPATCH(is_bf16, vec_rows(d, sizeof(T), src, buf), {
    auto kern = stream ? moe_scatter_kernel<T, W, true> : moe_scatter_kernel<T, W, false>;
    launch_after(kern, (unsigned)((rows + 7) / 8), 256, 0, st, (const T*)src, slot, w, w_bf16, inv, (T*)buf, n, k, tpb, d, rows, E, C, nb);
  });
  return launch_status();
}

extern "C" int apb_moe_gather(const void* buf, const long long* slot, const void* w, int w_bf16, void* out, long long T_, int k, int d, int E,
                              int C, int nb, int is_bf16, int num_sms, cudaStream_t st) {
  if (T_ <= 0 || k <= 0 || d <= 0 || nb <= 0 || T_ % nb) return (int)cudaErrorInvalidValue;
  const long long tpb = T_ / nb;
  APB_MOE_DISPATCH(is_bf16, vec_rows(d, sizeof(T), buf, out), {
    // the columns of a token are shared by warps until there are 64 for every SM; each has at least one 512-byte piece
    const int pieces = (d + 32 * W - 1) / (32 * W);
    const long long want = (64ll * num_sms + T_ - 1) / T_;
    const dim3 grid((unsigned)((T_ + 3) / 4), (unsigned)(want < pieces ? want : pieces));
    auto kern = (long long)grid.x * grid.y >= 6ll * num_sms ? moe_gather_kernel<T, W, 8> : moe_gather_kernel<T, W, 1>;
    launch_after(kern, grid, 128, 0, st, (const T*)buf, slot, w, w_bf16, (T*)out, T_, k, tpb, d, E, C, nb);
  });
  return launch_status();
}

extern "C" int apb_moe_gate_grad(const void* buf, const long long* slot, const void* g, float* dw, long long T_, int k, int d, int E,
                                 int C, int nb, int is_bf16, cudaStream_t st) {
  if (T_ <= 0 || k <= 0 || d <= 0 || nb <= 0 || T_ % nb) return (int)cudaErrorInvalidValue;
  const long long n = T_ * k;
  APB_MOE_DISPATCH(is_bf16, vec_rows(d, sizeof(T), buf, g),
                   launch_after(moe_gate_grad_kernel<T, W>, (unsigned)((n + 7) / 8), 256, 0, st, (const T*)buf, slot, (const T*)g, dw, n, k, T_ / nb, d, E,
                                                                                       C, nb));
  return launch_status();
}
