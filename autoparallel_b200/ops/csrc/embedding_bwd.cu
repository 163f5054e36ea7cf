// Embedding table gradient for sm_100a: out[v, :] = sum of dy[t, :] over the tokens with ids[t] == v, zero rows included.
//
// Two forms; ``apb_embedding_bwd_sorts`` says which one runs.
//
// Sorted, bound by memory: the table gradient is written once in its own type and dy is read once.  The tokens are grouped by row
// first, so that every output row is summed in fp32 registers and stored once - no fp32 table, no second
// pass that converts it, no atomics on row data.
//
//   emb_group_kernel    one cluster of 8 CTAs: counts per row (one atomic per warp and distinct id), segment starts, token
//                       list sorted by row.  A cluster because its barrier orders the phases inside one launch; 8192
//                       threads take a usual batch in one or two steps.
//   emb_partial_kernel  rows with more than EMB_CHUNK tokens (frequent words, padding): one fp32 partial row per chunk, so
//                       that no block walks a long list alone.  Of rows with more than EMB_DIRECT chunks the last block of a group adds
//                       the group up, and the last group the row.
//   emb_rows_kernel     every other row: zeros, the sum of its tokens, or of its chunks.
//
// Where the table has far more rows than there are tokens (``emb_zeros_first``), the whole of it is filled with zeros beside the grouping,
// by the SMs that the cluster leaves idle, and the last kernel is
//
//   emb_tokens_kernel   only the rows that have tokens.
//
// Atomic: an fp32 table of zeros, one block per token, for bf16 a conversion.  Better where the table is small or the rows are
// short (the grouping is a chain of latencies that a small table does not pay for), and for most fp32 tables, which the atomics
// fill in place.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "launch.cuh"
#include "ptx.cuh"

extern "C" int apb_cast(const void* src, void* dst, long long n, int src_bf16, int dst_bf16, int num_sms, cudaStream_t st);  // elementwise.cu

namespace apb {

constexpr int EMB_CHUNK = 32;
constexpr int EMB_DIRECT = 32;  // most chunks of a row that emb_rows_kernel adds up
constexpr int EMB_GROUP = 16;   // chunks of a longer one that are added up by one block
constexpr int EMB_CTAS = 8, EMB_GROUP_THREADS = 1024;
constexpr int EMB_ZERO_VECS = 2048;  // 16-byte vectors of zeros that a block fills
constexpr int EMB_ROWS = 8;  // most rows of one block of emb_rows_kernel

// Workspace (32-bit words), carved from one allocation of the caller.
struct EmbWs {
  int* count;    // [V] tokens of the row
  int* start;    // [V] first entry of the row in perm
  int* chunk0;   // [V] first chunk of the row (rows with more than EMB_CHUNK tokens)
  int* perm;     // [T] tokens grouped by row
  int* rank;     // [T] arrival number of the token inside its row
  int4* desc;    // [max_chunks] {first entry in perm, tokens, row, number of the chunk in the row}
  int* ctr;      // [2] entries and chunks handed out so far
  int* done;     // [2, max_chunks, column slices] finished chunks of the group that starts here, finished groups of the row
  float* part;   // [max_chunks, D]
};

__host__ __device__ inline long long emb_max_longs(long long T) { return T / (EMB_CHUNK + 1); }
__host__ __device__ inline long long emb_max_chunks(long long T) { return T / EMB_CHUNK + emb_max_longs(T); }
static inline long long emb_round4(long long n) { return (n + 3) & ~3ll; }

// Blocks of the clusters after the first fill EMB_ZERO_VECS of the ``nzero`` vectors of ``zeros`` each.
__global__ void __cluster_dims__(EMB_CTAS, 1, 1) __launch_bounds__(EMB_GROUP_THREADS)
emb_group_kernel(const long long* ids, EmbWs ws, int T, long long V, long long ndone, uint4* zeros, long long nzero) {
  after_previous();
  if (blockIdx.x >= EMB_CTAS) {
    const long long i = (long long)(blockIdx.x - EMB_CTAS) * EMB_ZERO_VECS + threadIdx.x;
#pragma unroll
    for (int k = 0; k < EMB_ZERO_VECS; k += EMB_GROUP_THREADS)
      if (i + k < nzero) zeros[i + k] = make_uint4(0, 0, 0, 0);
    return;
  }
  const int tid = blockIdx.x * EMB_GROUP_THREADS + threadIdx.x, lane = threadIdx.x & 31;
  constexpr int nt = EMB_CTAS * EMB_GROUP_THREADS;
  for (long long v = tid; v < V; v += nt) ws.count[v] = 0;
  for (long long i = tid; i < ndone; i += nt) ws.done[i] = 0;
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
      for (int i = 0; i < n; ++i) ws.desc[b + i] = make_int4(s + i * EMB_CHUNK, min(EMB_CHUNK, c - i * EMB_CHUNK), (int)v, i);
    }
  }
  sync();
  for (int t = tid; t < T; t += nt) {
    const long long v = ids[t];
    if (v >= 0 && v < V) ws.perm[__ldcg(ws.start + v) + ws.rank[t]] = t;
  }
}

// W consecutive elements: 16 bytes, or one element where rows are not whole 16-byte vectors.  A row of dy is read once: past L1 (through it 32768
// tokens by Zipf's law, 8192 x 4096 bf16 154 -> 163 us).
template <typename T, int W> struct EmbVec;
template <> struct EmbVec<__nv_bfloat16, 8> {
  uint4 r;
  __device__ void load(const __nv_bfloat16* p) { r = __ldcg(reinterpret_cast<const uint4*>(p)); }
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
  __device__ void load(const float* p) { r = __ldcg(reinterpret_cast<const float4*>(p)); }
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

// acc += n partial rows that lie ``stride`` floats apart, written by other blocks of this launch
template <int W>
__device__ __forceinline__ void emb_part_sum(const float* p, int n, long long stride, float (&acc)[W]) {
#pragma unroll 8
  for (int i = 0; i < n; ++i, p += stride) {
    if constexpr (W == 1) {
      acc[0] += __ldcg(p);
    } else {
#pragma unroll
      for (int k = 0; k < W / 4; ++k) {
        const float4 x = __ldcg(reinterpret_cast<const float4*>(p) + k);
        acc[4 * k] += x.x; acc[4 * k + 1] += x.y; acc[4 * k + 2] += x.z; acc[4 * k + 3] += x.w;
      }
    }
  }
}

// What the block has written is visible to the one that finds itself the last of ``n``; true there, in all threads.
__device__ __forceinline__ bool emb_last(int* counter, int n) {
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(counter, 1) == n - 1;
  __syncthreads();
  __threadfence();
  return last != 0;
}

// A block takes a slice of the columns of one chunk.  In rows of many chunks the blocks that finish last add up, in the order of the
// chunks and in two steps: one block of the kernel below that added all chunks of a row took 2.9 ms for 131072 tokens of one row,
// D = 4096.  Rows of up to 32 chunks are left to that kernel, which adds them beside the stores of the table's other rows: 8192 tokens by
// Zipf's law, 128256 x 4096, 222 us with the sums here, 228 with a launch of their own, 206 so.
template <typename T, int W>
__global__ void __launch_bounds__(128) emb_partial_kernel(const T* dy, EmbWs ws, T* out, long long max_chunks, int D) {
  after_previous();
  __shared__ int list[EMB_CHUNK];
  const int b = blockIdx.x, slices = gridDim.y, step = slices * 128 * W, col0 = (blockIdx.y * 128 + threadIdx.x) * W;
  if (b >= ws.ctr[1]) return;
  const int4 d = ws.desc[b];
  const int n = (ws.count[d.z] + EMB_CHUNK - 1) / EMB_CHUNK;  // chunks of the row
  if ((int)threadIdx.x < d.y) list[threadIdx.x] = ws.perm[d.x + threadIdx.x];
  __syncthreads();
  for (int col = col0; col < D; col += step) {
    float acc[W] = {};
    emb_sum<T, W>(dy, list, d.y, D, col, acc);
#pragma unroll
    for (int k = 0; k < W; ++k) ws.part[(long long)b * D + col + k] = acc[k];
  }
  if (n <= EMB_DIRECT) return;
  const int g = d.w / EMB_GROUP, row0 = b - d.w, first = row0 + g * EMB_GROUP, members = min(EMB_GROUP, n - g * EMB_GROUP);
  if (!emb_last(ws.done + (long long)first * slices + blockIdx.y, members)) return;
  for (int col = col0; col < D; col += step) {
    float acc[W] = {};
    emb_part_sum<W>(ws.part + (long long)first * D + col, members, D, acc);
#pragma unroll  // (the group's first row takes the sum: nobody else reads these columns of it any more)
    for (int k = 0; k < W; ++k) ws.part[(long long)first * D + col + k] = acc[k];
  }
  const int groups = (n + EMB_GROUP - 1) / EMB_GROUP;
  if (!emb_last(ws.done + (max_chunks + row0) * slices + blockIdx.y, groups)) return;
  for (int col = col0; col < D; col += step) {
    float acc[W] = {};
    emb_part_sum<W>(ws.part + (long long)row0 * D + col, groups, (long long)EMB_GROUP * D, acc);
    EmbVec<T, W>::store(out + (long long)d.z * D + col, acc);
  }
}

// Columns of one row with ``c`` tokens; ``from``: its first entry in perm, or its first chunk.
template <typename T, int W>
__device__ __forceinline__ void emb_row(const T* __restrict__ dy, const EmbWs& ws, T* dst, int c, int from, int D, int col, int step) {
  for (; col < D; col += step) {
    float acc[W] = {};
    if (c > EMB_CHUNK) {
      const float* p = ws.part + (long long)from * D + col;
      const int n = (c + EMB_CHUNK - 1) / EMB_CHUNK;
#pragma unroll 4
      for (int i = 0; i < n; ++i)
#pragma unroll
        for (int k = 0; k < W; ++k) acc[k] += p[(long long)i * D + k];
    } else if (c > 0) {
      emb_sum<T, W>(dy, ws.perm + from, c, D, col, acc);
    }
    EmbVec<T, W>::store(dst + col, acc);
  }
}

// The first token of every row stores it; ``tx`` threads to a token, as below.
template <typename T, int W>
__global__ void __launch_bounds__(256) emb_tokens_kernel(const T* dy, const long long* ids, EmbWs ws, T* out,
                                                         int tokens, long long V, int D, int tx) {
  after_previous();
  const int t = blockIdx.x * (256 / tx) + threadIdx.x / tx;
  if (t >= tokens) return;
  const long long v = ids[t];
  if (v < 0 || v >= V || ws.rank[t] != 0) return;
  const int c = ws.count[v];
  if (c > EMB_CHUNK * EMB_DIRECT) return;
  emb_row<T, W>(dy, ws, out + v * D, c, (c > EMB_CHUNK ? ws.chunk0 : ws.start)[v], D, (threadIdx.x & (tx - 1)) * W, tx * W);
}

// ``tx`` threads (a power of two, 32..256) walk a row, 256 / tx rows at a time; the block owns ``R`` consecutive rows
template <typename T, int W>
__global__ void __launch_bounds__(256) emb_rows_kernel(const T* dy, EmbWs ws, T* out, long long V, int D,
                                                       int R, int tx) {
  after_previous();
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
    const int c = cnt[r];
    if (c > EMB_CHUNK * EMB_DIRECT) continue;
    emb_row<T, W>(dy, ws, out + (row0 + r) * D, c, from[r], D, (threadIdx.x & (tx - 1)) * W, tx * W);
  }
}

// The other form: an fp32 table of zeros, one block per token that adds its row with atomics (a bf16 table is converted after).
// ``U`` elements of a thread are loaded before the token's id is there: one in rows of up to 256, four in longer ones.
template <typename T, int U>
__global__ void __launch_bounds__(256) emb_atomic_kernel(const T* dy, const long long* ids, float* out,
                                                         long long V, int D) {
  after_previous();
  const long long tok = blockIdx.x;
  const long long r = ids[tok];
  const bool ok = (unsigned long long)r < (unsigned long long)V;
  const T* src = dy + tok * D;
  if constexpr (U == 1) {  // (the loop below with one element makes a block half as long again: 524288 x 64 276 -> 390 us)
    for (int c = threadIdx.x; c < D; c += blockDim.x) {
      const float x = float(src[c]);
      if (ok) atomicAdd(out + r * D + c, x);
    }
  } else {
    for (int c = threadIdx.x; c < D; c += 256 * U) {
      float x[U];
#pragma unroll
      for (int k = 0; k < U; ++k)
        if (c + k * 256 < D) x[k] = float(src[c + k * 256]);
      if (ok) {
#pragma unroll
        for (int k = 0; k < U; ++k)
          if (c + k * 256 < D) atomicAdd(out + r * D + c + k * 256, x[k]);
      }
    }
  }
}

template <typename T>
static void emb_atomic(const void* dy, const long long* ids, float* out, long long tokens, long long V, int D, cudaStream_t st) {
  if (D <= 256) launch_after(emb_atomic_kernel<T, 1>, (unsigned)tokens, 256, 0, st, (const T*)dy, ids, out, V, D);
  else launch_after(emb_atomic_kernel<T, 4>, (unsigned)tokens, 256, 0, st, (const T*)dy, ids, out, V, D);
}

// (a memset of the same bytes takes 1 to 3 us more)
__global__ void __launch_bounds__(256) emb_zero_kernel(float4* p, long long n) {
  after_previous();
  const long long i = (long long)blockIdx.x * 1024 + threadIdx.x;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (i + k * 256 < n) p[i + k * 256] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// column slices of emb_partial_kernel, ``w`` elements per thread
static int emb_slices(int D, int w) {
  const int n = (D / w + 127) / 128;
  return n < 16 ? n : 16;
}

// Zeros first, beside the grouping (a chain of latencies on eight SMs, 20 us and more), in blocks that end with their 32 KB: those write 7.3 TB/s,
// blocks that stay and take many pieces 6.2, emb_rows_kernel 7.8 in rows of 8 KB and 5.8 in shorter ones.  The rows that have tokens are written
// twice, so the line lies where a table has four times as many rows as there are tokens, ten times in rows of more than 4 KB.  bf16, ids by Zipf's law /
// at random, rows first -> zeros first: 128256 x 1024, 8000 tokens 85 / 78 -> 66 / 57 us, x 2048 127 / 125 -> 110 / 105, x 4096 210 / 195 -> 194 /
// 186, 16000 tokens 221 / 215 -> 211 / 224; 32000 x 2048, 8000 tokens 57 / 52 -> 51 / 46, 16000 73 / 66 -> 72 / 72; 32000 x 4096, 2000 tokens 74 /
// 63 -> 67 / 51, 8000 85 / 77 -> 89 / 79; 8000 x 2048, 2000 tokens 27 / 24 -> 23 / 21, 4000 26 / 25 -> 27 / 24.
static bool emb_zeros_first(long long tokens, long long V, long long row_bytes) {
  return tokens > 0 && tokens <= V / (row_bytes > 4096 ? 10 : 4);  // (without tokens emb_rows_kernel writes the zeros)
}

template <typename T, int W>
static void emb_launch(const void* dy, const long long* ids, const EmbWs& ws, void* out, long long T_, long long V, int D, int num_sms,
                       cudaStream_t st) {
  const int nvec = D / W, slices = emb_slices(D, W);
  const long long chunks = emb_max_chunks(T_);
  const bool zeros_first = W > 1 && emb_zeros_first(T_, V, (long long)D * sizeof(T));
  const long long fill = (long long)EMB_CTAS * EMB_ZERO_VECS;  // vectors of a cluster
  const unsigned clusters = 1 + (zeros_first ? (unsigned)((V * nvec + fill - 1) / fill) : 0u);
  launch_after(emb_group_kernel, EMB_CTAS * clusters, EMB_GROUP_THREADS, 0, st, ids, ws, (int)T_, V, 2 * chunks * slices, reinterpret_cast<uint4*>(out),
                                                                       V * nvec);
  if (emb_max_longs(T_) > 0)
    launch_after(emb_partial_kernel<T, W>, dim3((unsigned)chunks, (unsigned)slices), 128, 0, st, (const T*)dy, ws, (T*)out, chunks, D);
  int tx = 32;
  while (tx < nvec && tx < 256) tx *= 2;
  if constexpr (W > 1) {
    if (zeros_first) {
      const int per = 256 / tx;
      launch_after(emb_tokens_kernel<T, W>, (unsigned)((T_ + per - 1) / per), 256, 0, st, (const T*)dy, ids, ws, (T*)out, (int)T_, V, D, tx);
      return;
    }
  }
  // rows per block: eight where the table is long (one 64-KB store stream per block), fewer where it would leave SMs idle,
  // but never fewer than the block takes at a time
  const long long want = V / ((long long)num_sms * 8);
  int R = (int)(want < 1 ? 1 : (want > EMB_ROWS ? EMB_ROWS : want));
  if (R < 256 / tx) R = 256 / tx;
  launch_after(emb_rows_kernel<T, W>, (unsigned)((V + R - 1) / R), 256, 0, st, (const T*)dy, ws, (T*)out, V, D, R, tx);
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
  ws->desc = reinterpret_cast<int4*>(take(4 * chunks));
  ws->done = take(2 * chunks * emb_slices(D, 1));  // (the most of all forms)
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

// Estimates of both forms in microseconds, fitted to 405 sizes (1 ... 524288 tokens, 2 ... 1000000 rows of 16 ... 4096) in both types with
// ids at random, by Zipf's law, half of them and all of them the same: bytes of the table and atomics, or the grouping and one
// read of dy.  Sorting has to promise a tenth.  bf16, 8192 tokens at random, sorted / atomic: 32000 x 64 24.7 / 16.5 us, 8192 x 1024
// 24.7 / 24.7, 32000 x 4096 82 / 263, 128256 x 4096 201 / 806; fp32: 128256 x 1024 123 / 92, 1024 x 4096 53 / 68.  Rows that are no whole vectors are slow to gather:
// in fp32 nothing is left to gain.  Where it sorts, that was the slower form by more than 3 % in 8 of 3240 timings.
extern "C" int apb_embedding_bwd_sorts(long long tokens, long long num_rows, int D, int is_bf16) {
  const double T = (double)tokens, V = (double)num_rows, td = T * D, vd = V * D;
  const bool vec = D % (is_bf16 ? 8 : 4) == 0;
  double atomic, sorted;
  if (is_bf16) {
    atomic = 7 + vd * 10 / 4.2e6 + (td / 0.7e6 > 6.3e-4 * T ? td / 0.7e6 : 6.3e-4 * T);
    sorted = 31 + (vec ? 5.6e-4 : 7.0e-4) * T + 1.0e-4 * V + vd * 2 / 4.3e6 + (vec ? 2.0e-7 : 6.0e-7) * td;
  } else {
    if (!vec) return 0;
    atomic = 3 + vd * 4 / 5.4e6 + (td / 0.6e6 > 6.0e-4 * T ? td / 0.6e6 : 6.0e-4 * T);
    sorted = 23 + 5.5e-4 * T + 1.2e-4 * V + vd * 4 / 5.6e6 + 2.3e-7 * td;
  }
  if (T >= 16 * V) sorted += 18;  // most lists are long, and summed in two steps
  return sorted < 0.9 * atomic;
}

// kernels that a call launches
extern "C" int apb_embedding_bwd_launches(long long tokens, long long num_rows, int D, int is_bf16) {
  if (num_rows <= 0 || D <= 0) return 0;
  if (apb_embedding_bwd_sorts(tokens, num_rows, D, is_bf16)) return emb_max_longs(tokens) > 0 ? 3 : 2;
  return (num_rows * D % 4 == 0) + (tokens > 0) + (is_bf16 != 0);
}

// bytes of workspace
extern "C" long long apb_embedding_bwd_workspace(long long tokens, long long num_rows, int D, int is_bf16) {
  if (!apb_embedding_bwd_sorts(tokens, num_rows, D, is_bf16)) return is_bf16 ? num_rows * D * 4 : 0;
  EmbWs ws;
  return emb_carve(&ws, nullptr, tokens, num_rows, D);
}

// dy [tokens, D], out [num_rows, D] of the same type (every element is written); ids outside the table are skipped.
extern "C" int apb_embedding_bwd(const void* dy, const long long* ids, void* out, void* workspace, long long tokens, long long num_rows,
                                 int D, int is_bf16, int num_sms, cudaStream_t st) {
  if (num_rows <= 0 || D <= 0) return 0;
  if (!apb_embedding_bwd_sorts(tokens, num_rows, D, is_bf16)) {
    if (tokens >= (1ll << 31) || (is_bf16 && (reinterpret_cast<uintptr_t>(out) & 15))) return 3;
    float* acc = reinterpret_cast<float*>(is_bf16 ? workspace : out);
    const long long n = num_rows * D;
    if (n % 4 == 0 && (reinterpret_cast<uintptr_t>(acc) & 15) == 0) launch_after(emb_zero_kernel, (unsigned)((n / 4 + 1023) / 1024), 256, 0, st, reinterpret_cast<float4*>(acc), n / 4);
    else if (cudaMemsetAsync(acc, 0, sizeof(float) * n, st) != cudaSuccess) return 4;
    if (tokens > 0) {
      if (is_bf16) emb_atomic<__nv_bfloat16>(dy, ids, acc, tokens, num_rows, D, st);
      else emb_atomic<float>(dy, ids, acc, tokens, num_rows, D, st);
    }
    if (is_bf16) return apb_cast(acc, out, num_rows * D, 0, 1, num_sms, st);
    return cudaGetLastError() == cudaSuccess ? 0 : 4;
  }
  if (tokens >= (1ll << 30) || num_rows >= (1ll << 31)) return 3;
  EmbWs ws;
  emb_carve(&ws, workspace, tokens, num_rows, D);
  const int w = is_bf16 ? 8 : 4;
  const bool vec = D % w == 0 && ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  if (is_bf16) {
    if (vec) emb_launch<__nv_bfloat16, 8>(dy, ids, ws, out, tokens, num_rows, D, num_sms, st);
    else emb_launch<__nv_bfloat16, 1>(dy, ids, ws, out, tokens, num_rows, D, num_sms, st);
  } else {
    if (vec) emb_launch<float, 4>(dy, ids, ws, out, tokens, num_rows, D, num_sms, st);
    else emb_launch<float, 1>(dy, ids, ws, out, tokens, num_rows, D, num_sms, st);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}
