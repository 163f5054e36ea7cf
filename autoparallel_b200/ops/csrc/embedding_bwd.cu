// Embedding table gradient for sm_100a: out[v, :] = sum of dy[t, :] over the tokens with ids[t] == v, zero rows included.
//
// Bound by memory: the table gradient is written once in its own type and dy is read once.  The tokens are grouped by row
// first, so that every output row is summed in fp32 registers and stored once - no fp32 table, no zero fill of it, no
// second pass that converts it, no atomics on row data.  8192 tokens of 4096 bf16, 128256 rows (1.05 GB written):
// 278 us for the three kernels (246 of them the rows); the fp32 zero fill + atomics + cast that they replace took 841 us.
//
//   emb_group_kernel    one cluster of 8 CTAs: counts per row (one atomic per warp and distinct id), segment starts, token
//                       list sorted by row.  A cluster because its barrier orders the phases inside one launch; 8192
//                       threads take a usual batch in one or two steps.
//   emb_partial_kernel  rows with more than EMB_CHUNK tokens (frequent words, padding): one fp32 partial row per chunk, so
//                       that no block walks a long list alone.
//   emb_rows_kernel     every row: zeros, the sum of its tokens, or the sum of its chunks.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ptx.cuh"

namespace apb {

constexpr int EMB_CHUNK = 32;
constexpr int EMB_CTAS = 8, EMB_GROUP_THREADS = 1024;
constexpr int EMB_ROWS = 8;  // most rows of one block of emb_rows_kernel

// Workspace (32-bit words), carved from one allocation of the caller.
struct EmbWs {
  int* count;    // [V] tokens of the row
  int* start;    // [V] first entry of the row in perm
  int* chunk0;   // [V] first chunk of the row (rows with more than EMB_CHUNK tokens)
  int* perm;     // [T] tokens grouped by row
  int* rank;     // [T] arrival number of the token inside its row
  int2* desc;    // [max_chunks] {first entry in perm, tokens}
  int* ctr;      // [2] entries and chunks handed out so far
  float* part;   // [max_chunks, D]
};

__host__ __device__ inline long long emb_max_chunks(long long T) { return T / EMB_CHUNK + T / (EMB_CHUNK + 1); }
static inline long long emb_round4(long long n) { return (n + 3) & ~3ll; }

__global__ void __cluster_dims__(EMB_CTAS, 1, 1) __launch_bounds__(EMB_GROUP_THREADS)
emb_group_kernel(const long long* __restrict__ ids, EmbWs ws, int T, long long V) {
  const int tid = blockIdx.x * EMB_GROUP_THREADS + threadIdx.x, lane = threadIdx.x & 31;
  constexpr int nt = EMB_CTAS * EMB_GROUP_THREADS;
  for (long long v = tid; v < V; v += nt) ws.count[v] = 0;
  if (tid < 2) ws.ctr[tid] = 0;
  auto sync = [] {  // every phase reads what other CTAs of the cluster wrote in the one before
    __threadfence();
    cluster_arrive();
    cluster_wait();
  };
  sync();
  for (int t0 = tid - lane; t0 < T; t0 += nt) {  // (whole warps stay together for the match)
    const int t = t0 + lane;
    const long long v = t < T ? ids[t] : -1;
    const bool ok = v >= 0 && v < V;
    const unsigned active = __ballot_sync(0xffffffffu, ok);
    if (ok) {
      const unsigned same = __match_any_sync(active, v);
      const int leader = __ffs(same) - 1;
      int base = 0;
      if (lane == leader) base = atomicAdd(ws.count + v, __popc(same));
      base = __shfl_sync(same, base, leader);
      ws.rank[t] = base + __popc(same & ((1u << lane) - 1u));
    }
  }
  sync();
  // the first token of every row takes the row's entries: one atomic per warp on each of the two counters
  for (int t0 = tid - lane; t0 < T; t0 += nt) {
    const int t = t0 + lane;
    const long long v = t < T ? ids[t] : -1;
    const bool first = v >= 0 && v < V && ws.rank[t] == 0;  // (rank: written by this very thread)
    const int c = first ? __ldcg(ws.count + v) : 0;
    const int n = c > EMB_CHUNK ? (c + EMB_CHUNK - 1) / EMB_CHUNK : 0;
    int cs = c, ns = n;  // inclusive sums over the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, cs, o), y = __shfl_up_sync(0xffffffffu, ns, o);
      if (lane >= o) {
        cs += x;
        ns += y;
      }
    }
    int cb = 0, nb = 0;
    if (lane == 31) {
      cb = cs > 0 ? atomicAdd(ws.ctr, cs) : 0;
      nb = ns > 0 ? atomicAdd(ws.ctr + 1, ns) : 0;
    }
    const int s = __shfl_sync(0xffffffffu, cb, 31) + cs - c, b = __shfl_sync(0xffffffffu, nb, 31) + ns - n;
    if (first) ws.start[v] = s;
    if (n > 0) {
      ws.chunk0[v] = b;
      for (int i = 0; i < n; ++i) ws.desc[b + i] = make_int2(s + i * EMB_CHUNK, min(EMB_CHUNK, c - i * EMB_CHUNK));
    }
  }
  sync();
  for (int t = tid; t < T; t += nt) {
    const long long v = ids[t];
    if (v >= 0 && v < V) ws.perm[__ldcg(ws.start + v) + ws.rank[t]] = t;
  }
}

// W consecutive elements: 16 bytes, or one element where rows are not whole 16-byte vectors
template <typename T, int W> struct EmbVec;
template <> struct EmbVec<__nv_bfloat16, 8> {
  uint4 r;
  __device__ void load(const __nv_bfloat16* p) { r = __ldg(reinterpret_cast<const uint4*>(p)); }
  __device__ void add_to(float (&a)[8]) const {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(h[i]);
      a[2 * i] += f.x;
      a[2 * i + 1] += f.y;
    }
  }
  static __device__ void store(__nv_bfloat16* p, const float (&a)[8]) {
    *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16(a[0], a[1]), pack_bf16(a[2], a[3]), pack_bf16(a[4], a[5]), pack_bf16(a[6], a[7]));
  }
};
template <> struct EmbVec<float, 4> {
  float4 r;
  __device__ void load(const float* p) { r = __ldg(reinterpret_cast<const float4*>(p)); }
  __device__ void add_to(float (&a)[4]) const { a[0] += r.x; a[1] += r.y; a[2] += r.z; a[3] += r.w; }
  static __device__ void store(float* p, const float (&a)[4]) { *reinterpret_cast<float4*>(p) = make_float4(a[0], a[1], a[2], a[3]); }
};
template <> struct EmbVec<__nv_bfloat16, 1> {
  float r;
  __device__ void load(const __nv_bfloat16* p) { r = __bfloat162float(*p); }
  __device__ void add_to(float (&a)[1]) const { a[0] += r; }
  static __device__ void store(__nv_bfloat16* p, const float (&a)[1]) { *p = __float2bfloat16(a[0]); }
};
template <> struct EmbVec<float, 1> {
  float r;
  __device__ void load(const float* p) { r = *p; }
  __device__ void add_to(float (&a)[1]) const { a[0] += r; }
  static __device__ void store(float* p, const float (&a)[1]) { *p = a[0]; }
};

// acc += rows list[0 .. n) of dy at column ``col``; eight loads in flight
template <typename T, int W>
__device__ __forceinline__ void emb_sum(const T* __restrict__ dy, const int* list, int n, long long D, int col, float (&acc)[W]) {
  int i = 0;
  for (; i + 8 <= n; i += 8) {
    EmbVec<T, W> v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k].load(dy + list[i + k] * D + col);
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k].add_to(acc);
  }
  for (; i < n; ++i) {
    EmbVec<T, W> v;
    v.load(dy + list[i] * D + col);
    v.add_to(acc);
  }
}

template <typename T, int W>
__global__ void __launch_bounds__(128) emb_partial_kernel(const T* __restrict__ dy, EmbWs ws, int D) {
  __shared__ int list[EMB_CHUNK];
  if ((int)blockIdx.x >= ws.ctr[1]) return;
  const int2 d = ws.desc[blockIdx.x];
  if ((int)threadIdx.x < d.y) list[threadIdx.x] = ws.perm[d.x + threadIdx.x];
  __syncthreads();
  for (int col = (blockIdx.y * 128 + threadIdx.x) * W; col < D; col += gridDim.y * 128 * W) {
    float acc[W] = {};
    emb_sum<T, W>(dy, list, d.y, D, col, acc);
#pragma unroll
    for (int k = 0; k < W; ++k) ws.part[(long long)blockIdx.x * D + col + k] = acc[k];
  }
}

// ``tx`` threads (a power of two, 32..256) walk a row, 256 / tx rows at a time; the block owns ``R`` consecutive rows
template <typename T, int W>
__global__ void __launch_bounds__(256) emb_rows_kernel(const T* __restrict__ dy, EmbWs ws, T* __restrict__ out, long long V, int D,
                                                       int R, int tx) {
  __shared__ int cnt[EMB_ROWS], from[EMB_ROWS];
  const long long row0 = (long long)blockIdx.x * R;
  const int nrows = (int)min((long long)R, V - row0);
  if ((int)threadIdx.x < nrows) {
    const int c = ws.count[row0 + threadIdx.x];
    cnt[threadIdx.x] = c;
    from[threadIdx.x] = c == 0 ? 0 : (c > EMB_CHUNK ? ws.chunk0 : ws.start)[row0 + threadIdx.x];
  }
  __syncthreads();
  for (int r = threadIdx.x / tx; r < nrows; r += 256 / tx) {
    T* dst = out + (row0 + r) * D;
    const int c = cnt[r];
    for (int col = (threadIdx.x & (tx - 1)) * W; col < D; col += tx * W) {
      float acc[W] = {};
      if (c > EMB_CHUNK) {
        const float* p = ws.part + (long long)from[r] * D + col;
        const int n = (c + EMB_CHUNK - 1) / EMB_CHUNK;
#pragma unroll 4
        for (int i = 0; i < n; ++i)
#pragma unroll
          for (int k = 0; k < W; ++k) acc[k] += p[(long long)i * D + k];
      } else if (c > 0) {
        emb_sum<T, W>(dy, ws.perm + from[r], c, D, col, acc);
      }
      EmbVec<T, W>::store(dst + col, acc);
    }
  }
}

template <typename T, int W>
static void emb_launch(const void* dy, const EmbWs& ws, void* out, long long T_, long long V, int D, int num_sms, cudaStream_t st) {
  const long long chunks = emb_max_chunks(T_);
  const int nvec = D / W;
  if (chunks > 0) {
    const int split = (nvec + 127) / 128;
    emb_partial_kernel<T, W><<<dim3((unsigned)chunks, (unsigned)(split < 16 ? split : 16)), 128, 0, st>>>((const T*)dy, ws, D);
  }
  int tx = 32;
  while (tx < nvec && tx < 256) tx *= 2;
  // rows per block: eight where the table is long (one 64-KB store stream per block), fewer where it would leave SMs idle,
  // but never fewer than the block takes at a time
  const long long want = V / ((long long)num_sms * 8);
  int R = (int)(want < 1 ? 1 : (want > EMB_ROWS ? EMB_ROWS : want));
  if (R < 256 / tx) R = 256 / tx;
  emb_rows_kernel<T, W><<<(unsigned)((V + R - 1) / R), 256, 0, st>>>((const T*)dy, ws, (T*)out, V, D, R, tx);
}

static long long emb_carve(EmbWs* ws, void* base, long long T, long long V, int D) {
  int* p = reinterpret_cast<int*>(base);
  long long off = 0;
  auto take = [&](long long words) {
    int* r = p + off;
    off += emb_round4(words);
    return r;
  };
  const long long chunks = emb_max_chunks(T);
  ws->part = reinterpret_cast<float*>(take(chunks * D));
  ws->desc = reinterpret_cast<int2*>(take(2 * chunks));
  ws->ctr = take(2);
  ws->count = take(V);
  ws->start = take(V);
  ws->chunk0 = take(V);
  ws->perm = take(T);
  ws->rank = take(T);
  return off * 4;
}

}  // namespace apb

using namespace apb;

extern "C" long long apb_embedding_bwd_workspace(long long tokens, long long num_rows, int D) {
  EmbWs ws;
  return emb_carve(&ws, nullptr, tokens, num_rows, D);
}

// dy [tokens, D], out [num_rows, D] of the same type (every element is written); ids outside the table are skipped.
extern "C" int apb_embedding_bwd(const void* dy, const long long* ids, void* out, void* workspace, long long tokens, long long num_rows,
                                 int D, int is_bf16, int num_sms, cudaStream_t st) {
  if (num_rows <= 0 || D <= 0) return 0;
  if (tokens >= (1ll << 30) || num_rows >= (1ll << 31)) return 3;
  EmbWs ws;
  emb_carve(&ws, workspace, tokens, num_rows, D);
  emb_group_kernel<<<EMB_CTAS, EMB_GROUP_THREADS, 0, st>>>(ids, ws, (int)tokens, num_rows);
  const int w = is_bf16 ? 8 : 4;
  const bool vec = D % w == 0 && ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  if (is_bf16) {
    if (vec) emb_launch<__nv_bfloat16, 8>(dy, ws, out, tokens, num_rows, D, num_sms, st);
    else emb_launch<__nv_bfloat16, 1>(dy, ws, out, tokens, num_rows, D, num_sms, st);
  } else {
    if (vec) emb_launch<float, 4>(dy, ws, out, tokens, num_rows, D, num_sms, st);
    else emb_launch<float, 1>(dy, ws, out, tokens, num_rows, D, num_sms, st);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}
