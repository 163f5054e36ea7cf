// Python bindings: torch tensors in, raw-pointer launchers (extern "C", defined in the .cu files)
// out.  All launches go to the current CUDA stream of the tensor's device.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>
#include <torch/library.h>

#include <array>
#include <atomic>
#include <cstdint>
#include <map>
#include <mutex>
#include <string>
#include <vector>

extern "C" {
int apb_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc,
                  int a_mn_major, int b_mn_major, int out_fp32, uint32_t* status, int num_sms, cudaStream_t stream);
int apb_gemm_grouped_bf16(const void* A, const void* B, void* C, int G, int M, int N, int K, int a_mn_major, int b_mn_major,
                          int out_fp32, uint32_t* status, int num_sms, cudaStream_t stream);
int apb_gemm_split(const void* A, const void* B, void* C, int G, int M, int N, int K, long long lda, long long ldb, long long ldc,
                   int a_mn, int b_mn, int out_fp32, int bn, int s, uint32_t* status, cudaStream_t stream);
void apb_gemm_split_choice(int G, int M, int N, int K, int num_sms, int reserved, int* bn, int* s);
void apb_gemm_set_pair_mode(int on);
int apb_gemm_get_pair_mode();
int apb_gemm_yield_request(int pairs, cudaStream_t stream);
int apb_gemm_yield_outstanding();
void apb_gemm_set_dynamic_tiles(int on);
int apb_gemm_get_dynamic_tiles();
void apb_gemm_set_pair_stages(int n);
int apb_gemm_get_pair_stages();
void apb_gemm_set_reserved_sms(int n);
int apb_gemm_get_reserved_sms();
int apb_gemm_fused_ctas(int fuse, int M, int N, int comm_ctas, int num_sms);
int apb_rms_norm_fwd(const void* x, const void* w, void* y, float* rstd, long long rows, int D, float eps, int is_bf16,
                     cudaStream_t st);
long long apb_rms_norm_bwd_workspace(long long rows, int D, int is_bf16, int num_sms);
int apb_rms_norm_bwd(const void* dy, const void* x, const void* w, const float* rstd, void* dx, void* dw, float* part,
                     long long rows, int D, int is_bf16, int num_sms, cudaStream_t st);
int apb_cast(const void* src, void* dst, long long n, int src_bf16, int dst_bf16, int num_sms, cudaStream_t st);
int apb_cast_many(const void* const* src, void* const* dst, const long long* n, int count, int* launches, cudaStream_t st);
int apb_rope(const void* x, const float* cs, const float* sn, void* y, long long B, int S, int H, int D, int conj, int is_bf16,
             int num_sms, cudaStream_t st);
int apb_swiglu_fwd(const void* a, const void* b, void* y, long long n, int is_bf16, int num_sms, cudaStream_t st);
int apb_swiglu_bwd(const void* dy, const void* a, const void* b, void* da, void* db, long long n, int is_bf16, int num_sms,
                   cudaStream_t st);
int apb_xent_fwd(const void* logits, const long long* labels, float* loss, float* lse, long long rows, int V, int is_bf16,
                 cudaStream_t st);
int apb_xent_bwd(const float* dloss, const void* logits, const long long* labels, const float* lse, void* dlogits,
                 long long rows, int V, int is_bf16, cudaStream_t st);
int apb_embedding_bwd_sorts(long long tokens, long long num_rows, int D, int is_bf16);
int apb_embedding_bwd_launches(long long tokens, long long num_rows, int D, int is_bf16);
long long apb_embedding_bwd_workspace(long long tokens, long long num_rows, int D, int is_bf16);
int apb_embedding_bwd(const void* dy, const long long* ids, void* out, void* workspace, long long tokens, long long num_rows, int D,
                      int is_bf16, int num_sms, cudaStream_t st);
int apb_embedding_fwd(const void* weight, const long long* ids, void* out, long long tokens, int D, long long num_rows,
                      int is_bf16, cudaStream_t st);
int apb_moe_slots_max_experts(int per_block);
long long apb_moe_slots_workspace(int num_blocks, int per_block, int E, int num_sms);
int apb_moe_slots(const long long* gate_idx, long long* slot, int* counts, int num_blocks, int per_block, int E, int C, int num_sms,
                  cudaStream_t st);
int apb_moe_scatter(const void* src, const long long* slot, const void* w, int w_bf16, long long* inv, void* buf, long long T, int k, int d,
                    int E, int C, int nb, int is_bf16, cudaStream_t st);
int apb_moe_gather(const void* buf, const long long* slot, const void* w, int w_bf16, void* out, long long T, int k, int d, int E, int C,
                   int nb, int is_bf16, int num_sms, cudaStream_t st);
int apb_moe_gate_grad(const void* buf, const long long* slot, const void* g, float* dw, long long T, int k, int d, int E, int C, int nb,
                      int is_bf16, cudaStream_t st);
int apb_symm_header_bytes();
int apb_symm_wait_probe(const uint32_t* flag, unsigned target, unsigned limit_ms, uint32_t* status, cudaStream_t st);
int apb_symm_collective(int mode, const unsigned long long* peer_ptrs, int rank, int n, unsigned epoch, const void* src,
                        void* dst, long long outer, long long inner_bytes, int elem_kind, float scale, long long stage_capacity,
                        uint32_t* status, int num_ctas, unsigned target0, unsigned target1, unsigned long long multicast_base, cudaStream_t st);
int apb_gemm_fused(int fuse, const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                   long long ldc, int a_mn_major, int b_mn_major, int out_fp32, const unsigned long long* peer_ptrs, int rank,
                   int n, unsigned epoch, int rows_per_shard, const void* shard_src, void* gbuf, long long shard_bytes,
                   uint32_t* landed, unsigned landed_target, int rows_per_rank, float scale, long long stage_capacity,
                   const unsigned* targets, int comm_ctas, uint32_t* status, int num_sms, cudaStream_t stream);
int apb_dma_flag_bytes();
int apb_dma_ring_max();
int apb_dma_barrier(const unsigned long long* flags, int rank, int n, unsigned epoch, uint32_t* status, cudaStream_t st);
int apb_dma_all_gather(void* dst, const unsigned long long* bases, long long offset, long long outer, long long inner_bytes,
                       int rank, int n, cudaStream_t st);
int apb_dma_rs_push(const void* src, const unsigned long long* bases, const unsigned long long* flags, long long stage_offset,
                    long long slot_bytes, long long chunk_bytes, int entry, int ring, unsigned seq, int rank, int n,
                    uint32_t* status, cudaStream_t st);
int apb_dma_rs_sum(const void* src, void* dst, const unsigned long long* bases, const unsigned long long* flags,
                   long long stage_offset, long long slot_bytes, long long chunk_bytes, int entry, unsigned seq, float scale,
                   int rank, int n, int num_ctas, uint32_t* status, cudaStream_t st);
int apb_attention_fwd(const void* q, const void* k, const void* v, void* out, float* lse, int B, int S, int Sk, int H, int Hkv,
                      int D, int causal, float scale, uint32_t* status, cudaStream_t stream);
int apb_gemm_footprint(int i, int* out);
int apb_gemm_split_footprint(int i, int* out);
int apb_symm_footprint(int mode, int* out);
int apb_dma_sum_footprint(int n, int* out);
int apb_adamw(const void* tensors_dev, const void* pieces_dev, int num_pieces, int whole, float lr, float beta1, float beta2, float eps,
              float wd, float bc1, float bc2, float grad_scale, const float* hyper_dev, cudaStream_t st);
}

namespace {

int num_sms() { return at::cuda::getCurrentDeviceProperties()->multiProcessorCount; }
cudaStream_t stream() { return at::cuda::getCurrentCUDAStream().stream(); }

void check(int err, const char* what) {
  TORCH_CHECK(err == 0, what, " failed with code ", err,
              err == 3 ? " (unsupported shape / alignment)" : err == 4 ? " (launch error)" : "");
}

bool is_bf16(const at::Tensor& t) {
  TORCH_CHECK(t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kFloat, "expected bf16 or fp32, got ",
              t.scalar_type());
  return t.scalar_type() == at::kBFloat16;
}

// C[M,N] = opA * opB.  a: [M,K] (or [K,M] if a_mn_major); b: [N,K] (or [K,N] if b_mn_major).
void gemm(const at::Tensor& a, const at::Tensor& b, at::Tensor& c, bool a_mn_major, bool b_mn_major, at::Tensor& status) {
  c10::cuda::CUDAGuard g(a.device());
  TORCH_CHECK(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16, "gemm: bf16 operands required");
  TORCH_CHECK(a.dim() == 2 && b.dim() == 2 && c.dim() == 2 && a.stride(1) == 1 && b.stride(1) == 1 && c.stride(1) == 1,
              "gemm: 2-d row-major operands required");
  const int M = c.size(0), N = c.size(1);
  const int K = a_mn_major ? a.size(0) : a.size(1);
  TORCH_CHECK((a_mn_major ? a.size(1) : a.size(0)) == M, "gemm: A shape mismatch");
  TORCH_CHECK((b_mn_major ? b.size(1) : b.size(0)) == N && (b_mn_major ? b.size(0) : b.size(1)) == K, "gemm: B shape mismatch");
  const bool out_fp32 = c.scalar_type() == at::kFloat;
  TORCH_CHECK(out_fp32 || c.scalar_type() == at::kBFloat16, "gemm: output must be bf16 or fp32");
  check(apb_gemm_bf16(a.data_ptr(), b.data_ptr(), c.data_ptr(), M, N, K, a.stride(0), b.stride(0), c.stride(0), a_mn_major,
                      b_mn_major, out_fp32, reinterpret_cast<uint32_t*>(status.data_ptr()), num_sms(), stream()),
        "apb_gemm_bf16");
}

// c[g] = opA[g] * opB[g]; a: [G,M,K] (or [G,K,M] if a_mn_major); b: [G,N,K] (or [G,K,N]); c: [G,M,N]; all contiguous.
void gemm_grouped(const at::Tensor& a, const at::Tensor& b, at::Tensor& c, bool a_mn_major, bool b_mn_major, at::Tensor& status) {
  c10::cuda::CUDAGuard g(a.device());
  TORCH_CHECK(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16, "gemm_grouped: bf16 operands required");
  TORCH_CHECK(a.dim() == 3 && b.dim() == 3 && c.dim() == 3 && a.is_contiguous() && b.is_contiguous() && c.is_contiguous(),
              "gemm_grouped: contiguous 3-d operands required");
  const int G = c.size(0), M = c.size(1), N = c.size(2);
  const int K = a_mn_major ? a.size(1) : a.size(2);
  TORCH_CHECK(a.size(0) == G && b.size(0) == G && (a_mn_major ? a.size(2) : a.size(1)) == M, "gemm_grouped: A shape mismatch");
  TORCH_CHECK((b_mn_major ? b.size(2) : b.size(1)) == N && (b_mn_major ? b.size(1) : b.size(2)) == K, "gemm_grouped: B shape mismatch");
  const bool out_fp32 = c.scalar_type() == at::kFloat;
  TORCH_CHECK(out_fp32 || c.scalar_type() == at::kBFloat16, "gemm_grouped: output must be bf16 or fp32");
  check(apb_gemm_grouped_bf16(a.data_ptr(), b.data_ptr(), c.data_ptr(), G, M, N, K, a_mn_major, b_mn_major, out_fp32,
                              reinterpret_cast<uint32_t*>(status.data_ptr()), num_sms(), stream()),
        "apb_gemm_grouped_bf16");
}

// The cluster split-k kernel (gemm_split.cu) with an explicit tile width and slice count; 2-d operands as in ``gemm`` or
// contiguous 3-d stacks as in ``gemm_grouped``.
void gemm_split(const at::Tensor& a, const at::Tensor& b, at::Tensor& c, bool a_mn_major, bool b_mn_major, int64_t bn, int64_t slices,
                at::Tensor& status) {
  c10::cuda::CUDAGuard g(a.device());
  const int64_t d = c.dim();
  TORCH_CHECK(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16 && (d == 2 || d == 3) && a.dim() == d && b.dim() == d &&
                  a.stride(-1) == 1 && b.stride(-1) == 1 && c.stride(-1) == 1,
              "gemm_split: bf16 row-major operands, 2-d or 3-d");
  TORCH_CHECK(d == 2 || (a.is_contiguous() && b.is_contiguous() && c.is_contiguous() && a.size(0) == c.size(0) && b.size(0) == c.size(0)),
              "gemm_split: contiguous stacks required");
  const int M = c.size(-2), N = c.size(-1);
  const int K = a_mn_major ? a.size(-2) : a.size(-1);
  TORCH_CHECK((a_mn_major ? a.size(-1) : a.size(-2)) == M && (b_mn_major ? b.size(-1) : b.size(-2)) == N &&
                  (b_mn_major ? b.size(-2) : b.size(-1)) == K,
              "gemm_split: shape mismatch");
  const bool out_fp32 = c.scalar_type() == at::kFloat;
  TORCH_CHECK(out_fp32 || c.scalar_type() == at::kBFloat16, "gemm_split: output must be bf16 or fp32");
  check(apb_gemm_split(a.data_ptr(), b.data_ptr(), c.data_ptr(), d == 3 ? (int)c.size(0) : 0, M, N, K, a.stride(-2), b.stride(-2),
                       c.stride(-2), a_mn_major, b_mn_major, out_fp32, (int)bn, (int)slices,
                       reinterpret_cast<uint32_t*>(status.data_ptr()), stream()),
        "apb_gemm_split");
}

// q [B,S,H,D], k / v [B,Sk,Hkv,D] -> out [B,S,H,D] bf16, lse [B,H,S] fp32.  Returns false (nothing launched) for
// shapes the kernel does not cover.
bool attention_fwd(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, at::Tensor& out, at::Tensor& lse, bool causal,
                   double scale, at::Tensor& status) {
  c10::cuda::CUDAGuard g(q.device());
  TORCH_CHECK(q.scalar_type() == at::kBFloat16 && k.scalar_type() == at::kBFloat16 && v.scalar_type() == at::kBFloat16 &&
                  out.scalar_type() == at::kBFloat16 && lse.scalar_type() == at::kFloat,
              "attention_fwd: bf16 q / k / v / out and fp32 lse required");
  TORCH_CHECK(q.dim() == 4 && k.dim() == 4 && v.dim() == 4 && q.is_contiguous() && k.is_contiguous() && v.is_contiguous() &&
                  out.is_contiguous() && lse.is_contiguous(),
              "attention_fwd: contiguous [B, S, H, D] tensors required");
  TORCH_CHECK(k.sizes() == v.sizes() && k.size(0) == q.size(0) && k.size(3) == q.size(3) && out.sizes() == q.sizes() &&
                  lse.numel() == q.size(0) * q.size(1) * q.size(2),
              "attention_fwd: shape mismatch");
  const int err = apb_attention_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr<float>(), q.size(0),
                                    q.size(1), k.size(1), q.size(2), k.size(2), q.size(3), causal, (float)scale,
                                    reinterpret_cast<uint32_t*>(status.data_ptr()), stream());
  if (err == 3) return false;
  check(err, "apb_attention_fwd");
  return true;
}

void rms_norm_fwd(const at::Tensor& x, const at::Tensor& w, at::Tensor& y, at::Tensor& rstd, double eps) {
  c10::cuda::CUDAGuard g(x.device());
  const int D = x.size(-1);
  check(apb_rms_norm_fwd(x.data_ptr(), w.data_ptr(), y.data_ptr(), rstd.data_ptr<float>(), x.numel() / D, D, (float)eps,
                         is_bf16(x), stream()),
        "apb_rms_norm_fwd");
}

void rms_norm_bwd(const at::Tensor& dy, const at::Tensor& x, const at::Tensor& w, const at::Tensor& rstd, at::Tensor& dx,
                  at::Tensor& dw) {
  c10::cuda::CUDAGuard g(x.device());
  const int D = x.size(-1);
  const int64_t rows = x.numel() / D;
  const bool bf16 = is_bf16(x);
  at::Tensor part = at::empty({(int64_t)apb_rms_norm_bwd_workspace(rows, D, bf16, num_sms())}, rstd.options());  // partial sums of dw
  check(apb_rms_norm_bwd(dy.data_ptr(), x.data_ptr(), w.data_ptr(), rstd.data_ptr<float>(), dx.data_ptr(), dw.data_ptr(),
                         part.data_ptr<float>(), rows, D, bf16, num_sms(), stream()),
        "apb_rms_norm_bwd");
}

void cast(const at::Tensor& src, at::Tensor& dst) {
  c10::cuda::CUDAGuard g(src.device());
  check(apb_cast(src.data_ptr(), dst.data_ptr(), src.numel(), is_bf16(src), is_bf16(dst), num_sms(), stream()), "apb_cast");
}

void rope(const at::Tensor& x, const at::Tensor& cs, const at::Tensor& sn, at::Tensor& y, bool conj) {
  c10::cuda::CUDAGuard g(x.device());
  check(apb_rope(x.data_ptr(), cs.data_ptr<float>(), sn.data_ptr<float>(), y.data_ptr(), x.size(0), x.size(1), x.size(2),
                 x.size(3), conj, is_bf16(x), num_sms(), stream()),
        "apb_rope");
}

void swiglu_fwd(const at::Tensor& a, const at::Tensor& b, at::Tensor& y) {
  c10::cuda::CUDAGuard g(a.device());
  check(apb_swiglu_fwd(a.data_ptr(), b.data_ptr(), y.data_ptr(), a.numel(), is_bf16(a), num_sms(), stream()), "apb_swiglu_fwd");
}

void swiglu_bwd(const at::Tensor& dy, const at::Tensor& a, const at::Tensor& b, at::Tensor& da, at::Tensor& db) {
  c10::cuda::CUDAGuard g(a.device());
  check(apb_swiglu_bwd(dy.data_ptr(), a.data_ptr(), b.data_ptr(), da.data_ptr(), db.data_ptr(), a.numel(), is_bf16(a), num_sms(),
                       stream()),
        "apb_swiglu_bwd");
}

void xent_fwd(const at::Tensor& logits, const at::Tensor& labels, at::Tensor& loss, at::Tensor& lse) {
  c10::cuda::CUDAGuard g(logits.device());
  const int V = logits.size(-1);
  check(apb_xent_fwd(logits.data_ptr(), (const long long*)labels.data_ptr<int64_t>(), loss.data_ptr<float>(),
                     lse.data_ptr<float>(), logits.numel() / V, V, is_bf16(logits), stream()),
        "apb_xent_fwd");
}

void xent_bwd(const at::Tensor& dloss, const at::Tensor& logits, const at::Tensor& labels, const at::Tensor& lse,
              at::Tensor& dlogits) {
  c10::cuda::CUDAGuard g(logits.device());
  const int V = logits.size(-1);
  check(apb_xent_bwd(dloss.data_ptr<float>(), logits.data_ptr(), (const long long*)labels.data_ptr<int64_t>(),
                     lse.data_ptr<float>(), dlogits.data_ptr(), logits.numel() / V, V, is_bf16(logits), stream()),
        "apb_xent_bwd");
}

void embedding_fwd(const at::Tensor& weight, const at::Tensor& ids, at::Tensor& out) {
  c10::cuda::CUDAGuard g(weight.device());
  TORCH_CHECK(weight.dim() == 2 && weight.is_contiguous() && ids.scalar_type() == at::kLong && ids.is_contiguous() && out.is_contiguous(),
              "embedding_fwd: contiguous [V, D] table, int64 ids");
  check(apb_embedding_fwd(weight.data_ptr(), reinterpret_cast<const long long*>(ids.data_ptr()), out.data_ptr(), ids.numel(),
                          (int)weight.size(1), weight.size(0), is_bf16(weight), stream()),
        "apb_embedding_fwd");
}

// out [num_rows, D] of dy's dtype receives every row (zeros where no token names it).  Returns the number of kernels launched.
int64_t embedding_bwd(const at::Tensor& dy, const at::Tensor& ids, at::Tensor& out) {
  c10::cuda::CUDAGuard g(dy.device());
  const int64_t D = dy.size(-1), rows = out.size(0);
  TORCH_CHECK(dy.is_contiguous() && ids.is_contiguous() && out.is_contiguous() && out.dim() == 2 && out.size(1) == D &&
                  out.scalar_type() == dy.scalar_type() && ids.numel() * D == dy.numel(),
              "embedding_bwd: dy [..., D], ids [...], out [num_rows, D] of dy's dtype, all contiguous");
  const bool bf16 = is_bf16(dy);
  at::Tensor ws = at::empty({(int64_t)apb_embedding_bwd_workspace(ids.numel(), rows, (int)D, bf16)}, dy.options().dtype(at::kByte));
  check(apb_embedding_bwd(dy.data_ptr(), (const long long*)ids.data_ptr<int64_t>(), out.data_ptr(), ws.data_ptr(), ids.numel(), rows,
                          (int)D, bf16, num_sms(), stream()),
        "apb_embedding_bwd");
  return apb_embedding_bwd_launches(ids.numel(), rows, (int)D, bf16);
}

// Mixture-of-experts dispatch (ops/moe_ops.py): gate_idx / slot [T, k] int64, w [T, k] fp32 or bf16, buf [E, nb, C, d], src / out / g [T, d].
static void moe_check(const at::Tensor& x, const char* what) {
  TORCH_CHECK(x.is_cuda() && x.is_contiguous(), what, ": contiguous CUDA tensor expected");
}

int64_t moe_slots_max_experts(int64_t per_block) { return apb_moe_slots_max_experts((int)std::min<int64_t>(per_block, 1 << 30)); }

// Returns the number of kernels launched.
int64_t moe_slots(const at::Tensor& gate_idx, at::Tensor& slot, int64_t E, int64_t C, int64_t nb) {
  c10::cuda::CUDAGuard g(gate_idx.device());
  moe_check(gate_idx, "moe_slots");
  moe_check(slot, "moe_slots");
  TORCH_CHECK(gate_idx.scalar_type() == at::kLong && slot.scalar_type() == at::kLong && gate_idx.dim() == 2 &&
                  gate_idx.numel() == slot.numel() && nb > 0 && gate_idx.size(0) % nb == 0,
              "moe_slots: int64 [T, k] with T a multiple of the block count");
  const int64_t per_block = gate_idx.size(0) / nb * gate_idx.size(1);
  const int64_t words = apb_moe_slots_workspace((int)nb, (int)per_block, (int)E, num_sms());  // counts of every chunk
  at::Tensor counts = at::empty({words}, gate_idx.options().dtype(at::kInt));
  check(apb_moe_slots((const long long*)gate_idx.data_ptr<int64_t>(), (long long*)slot.data_ptr<int64_t>(), counts.data_ptr<int>(), (int)nb,
                      (int)per_block, (int)E, (int)C, num_sms(), stream()),
        "apb_moe_slots");
  return words > nb * E ? 2 : 1;  // (one chunk per block needs no counts)
}

// gate weights: fp32 or bf16, used in the operand's precision
bool gate_is_bf16(const at::Tensor& w, const at::Tensor& slot, const char* what) {
  TORCH_CHECK((w.scalar_type() == at::kFloat || w.scalar_type() == at::kBFloat16) && w.numel() == slot.numel(), what,
              ": fp32 or bf16 gate weights [T, k] expected");
  return w.scalar_type() == at::kBFloat16;
}

void moe_scatter(const at::Tensor& src, const at::Tensor& slot, const at::Tensor& w, at::Tensor& buf, int64_t E, int64_t C, int64_t nb) {
  c10::cuda::CUDAGuard g(src.device());
  moe_check(src, "moe_scatter"); moe_check(slot, "moe_scatter"); moe_check(w, "moe_scatter"); moe_check(buf, "moe_scatter");
  TORCH_CHECK(src.dim() == 2 && slot.dim() == 2 && slot.scalar_type() == at::kLong && slot.size(0) == src.size(0) &&
                  buf.scalar_type() == src.scalar_type() && buf.numel() == E * nb * C * src.size(1),
              "moe_scatter: src [T, d], slot [T, k] int64, buf [E, nb, C, d] of src's dtype");
  at::Tensor inv = at::empty({E * nb * C}, slot.options());
  check(apb_moe_scatter(src.data_ptr(), (const long long*)slot.data_ptr<int64_t>(), w.data_ptr(), gate_is_bf16(w, slot, "moe_scatter"),
                        (long long*)inv.data_ptr<int64_t>(), buf.data_ptr(), src.size(0), (int)slot.size(1), (int)src.size(1), (int)E, (int)C,
                        (int)nb, is_bf16(src), stream()),
        "apb_moe_scatter");
}

void moe_gather(const at::Tensor& buf, const at::Tensor& slot, const at::Tensor& w, at::Tensor& out) {
  c10::cuda::CUDAGuard g(buf.device());
  moe_check(buf, "moe_gather"); moe_check(slot, "moe_gather"); moe_check(w, "moe_gather"); moe_check(out, "moe_gather");
  TORCH_CHECK(buf.dim() == 4 && slot.dim() == 2 && slot.scalar_type() == at::kLong && out.dim() == 2 && out.size(0) == slot.size(0) &&
                  out.size(1) == buf.size(3) && out.scalar_type() == buf.scalar_type(),
              "moe_gather: buf [E, nb, C, d], slot [T, k] int64, out [T, d] of buf's dtype");
  check(apb_moe_gather(buf.data_ptr(), (const long long*)slot.data_ptr<int64_t>(), w.data_ptr(), gate_is_bf16(w, slot, "moe_gather"),
                       out.data_ptr(), slot.size(0), (int)slot.size(1), (int)buf.size(3), (int)buf.size(0), (int)buf.size(2),
                       (int)buf.size(1), is_bf16(buf), num_sms(), stream()),
        "apb_moe_gather");
}

void moe_gate_grad(const at::Tensor& buf, const at::Tensor& slot, const at::Tensor& g_, at::Tensor& dw) {
  c10::cuda::CUDAGuard g(buf.device());
  moe_check(buf, "moe_gate_grad"); moe_check(slot, "moe_gate_grad"); moe_check(g_, "moe_gate_grad"); moe_check(dw, "moe_gate_grad");
  TORCH_CHECK(buf.dim() == 4 && slot.dim() == 2 && slot.scalar_type() == at::kLong && g_.dim() == 2 && g_.size(0) == slot.size(0) &&
                  g_.size(1) == buf.size(3) && g_.scalar_type() == buf.scalar_type() && dw.scalar_type() == at::kFloat &&
                  dw.numel() == slot.numel(),
              "moe_gate_grad: buf [E, nb, C, d], slot [T, k] int64, g [T, d] of buf's dtype, dw [T, k] fp32");
  check(apb_moe_gate_grad(buf.data_ptr(), (const long long*)slot.data_ptr<int64_t>(), g_.data_ptr(), dw.data_ptr<float>(), slot.size(0),
                          (int)slot.size(1), (int)buf.size(3), (int)buf.size(0), (int)buf.size(2), (int)buf.size(1), is_bf16(buf), stream()),
        "apb_moe_gate_grad");
}

void adamw(const at::Tensor& table, const at::Tensor& pieces, int64_t whole, double lr, double b1, double b2, double eps,
           double wd, double bc1, double bc2, double grad_scale, const c10::optional<at::Tensor>& hyper) {
  c10::cuda::CUDAGuard g(table.device());
  const float* hp = nullptr;
  if (hyper.has_value()) {
    TORCH_CHECK(hyper->scalar_type() == at::kFloat && hyper->numel() >= 3 && hyper->is_cuda(), "adamw: hyper = fp32 [3] on the device");
    hp = hyper->data_ptr<float>();
  }
  TORCH_CHECK(pieces.dim() == 2 && pieces.size(1) == 2 && pieces.scalar_type() == at::kInt && whole >= 0 && whole <= pieces.size(0),
              "adamw: pieces = int32 [n, 2], the first ``whole`` of them whole runs");
  check(apb_adamw(table.data_ptr(), pieces.data_ptr(), (int)pieces.size(0), (int)whole, (float)lr, (float)b1, (float)b2, (float)eps, (float)wd,
                  (float)bc1, (float)bc2, (float)grad_scale, hp, stream()),
        "apb_adamw");
}

// ------------------------------------------------------------------ whole operators: checks, allocation and launch in one call
// What ops/cuda_impl.py asks for first; an empty result means "not this kernel's form" and is answered there.

// Dense and on the 16-byte base that the kernels' vector and bulk accesses need: contiguous() returns a dense view at an odd
// offset as it is.
at::Tensor dense(const at::Tensor& t) {
  at::Tensor d = t.contiguous();
  return reinterpret_cast<uintptr_t>(d.data_ptr()) % 16 == 0 ? d : d.clone(at::MemoryFormat::Contiguous);
}

// [rows, last] with unit inner stride, rows of 16 bytes and an aligned base, as TMA needs it
at::Tensor as2d(const at::Tensor& t) {
  // (a single row is reshaped too: contiguous() does not look at its stride, which TMA does; the reshape makes it the width)
  at::Tensor m = t.dim() == 2 && t.size(0) > 1 && t.size(1) > 0 ? t : t.reshape({-1, t.size(-1)});
  if (m.stride(1) != 1 || m.stride(0) % 8 != 0 || reinterpret_cast<uintptr_t>(m.data_ptr()) % 16 != 0) m = dense(m);
  return m;
}

c10::optional<at::Tensor> gemm_new(const at::Tensor& a, const at::Tensor& b, bool a_mn, bool b_mn, bool out_fp32, at::Tensor& status) {
  if (a.scalar_type() != at::kBFloat16 || b.scalar_type() != at::kBFloat16) return c10::nullopt;
  at::Tensor a2 = as2d(a), b2 = as2d(b);
  const int64_t M = a2.size(a_mn ? 1 : 0), N = b2.size(b_mn ? 1 : 0);
  if (a2.size(1) % 8 || b2.size(1) % 8 || N % 8) return c10::nullopt;
  at::Tensor c = at::empty({M, N}, a2.options().dtype(out_fp32 ? at::kFloat : at::kBFloat16));
  gemm(a2, b2, c, a_mn, b_mn, status);
  return c;
}

// a[..., K] x (b[N, K] or b[K, N]) -> [..., N]
c10::optional<at::Tensor> mm_nd(const at::Tensor& a, const at::Tensor& b, bool trans_b, bool out_fp32, at::Tensor& status) {
  auto c = gemm_new(a, b, false, !trans_b, out_fp32, status);
  if (!c.has_value() || a.dim() == 2) return c;
  auto shape = a.sizes().vec();
  shape.back() = c->size(1);
  return c->view(shape);
}

std::tuple<at::Tensor, at::Tensor> rms_norm_new(const at::Tensor& x_, const at::Tensor& w, double eps) {
  at::Tensor x = dense(x_), y = at::empty_like(x);
  at::Tensor rstd = at::empty(x.sizes().slice(0, x.dim() - 1), x.options().dtype(at::kFloat));
  rms_norm_fwd(x, dense(w.to(x.scalar_type())), y, rstd, eps);
  return {y, rstd};
}

std::tuple<at::Tensor, at::Tensor> rms_norm_bwd_new(const at::Tensor& dy_, const at::Tensor& x_, const at::Tensor& w, const at::Tensor& rstd) {
  at::Tensor dy = dense(dy_), x = dense(x_), dx = at::empty_like(x), dw = at::empty_like(w, x.scalar_type());
  rms_norm_bwd(dy, x, dense(w.to(x.scalar_type())), rstd.contiguous(), dx, dw);
  return {dx, dw.to(w.scalar_type())};
}

at::Tensor rope_new(const at::Tensor& x_, const at::Tensor& cs, const at::Tensor& sn, bool conj) {
  at::Tensor x = dense(x_), y = at::empty_like(x);
  rope(x, dense(cs.to(at::kFloat)), dense(sn.to(at::kFloat)), y, conj);
  return y;
}

at::Tensor swiglu_new(const at::Tensor& a_, const at::Tensor& b_) {
  at::Tensor a = dense(a_), b = dense(b_), y = at::empty_like(a);
  swiglu_fwd(a, b, y);
  return y;
}

std::tuple<at::Tensor, at::Tensor> swiglu_bwd_new(const at::Tensor& dy_, const at::Tensor& a_, const at::Tensor& b_) {
  at::Tensor dy = dense(dy_), a = dense(a_), b = dense(b_), da = at::empty_like(a), db = at::empty_like(b);
  swiglu_bwd(dy, a, b, da, db);
  return {da, db};
}

// fp32 <-> bf16 copy of a contiguous, aligned tensor
c10::optional<at::Tensor> cast_new(const at::Tensor& x, bool to_bf16) {
  if (x.scalar_type() != (to_bf16 ? at::kFloat : at::kBFloat16) || !x.is_contiguous() || reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 != 0)
    return c10::nullopt;
  at::Tensor out = at::empty_like(x, to_bf16 ? at::kBFloat16 : at::kFloat);
  cast(x, out);
  return out;
}

int64_t symm_header_bytes() { return apb_symm_header_bytes(); }

// Bounded wait on a device flag (int32 tensor, element 0) that the caller may or may not ever raise.
void symm_wait_probe(const at::Tensor& flag, int64_t target, int64_t limit_ms, at::Tensor& status) {
  c10::cuda::CUDAGuard g(flag.device());
  TORCH_CHECK(flag.scalar_type() == at::kInt && flag.numel() >= 1, "symm_wait_probe: int32 flag tensor required");
  check(apb_symm_wait_probe(reinterpret_cast<const uint32_t*>(flag.data_ptr()), (unsigned)target, (unsigned)limit_ms,
                            reinterpret_cast<uint32_t*>(status.data_ptr()), stream()),
        "apb_symm_wait_probe");
}

// One collective on a symmetric workspace (see symm_comm.cu).  src/dst are ordinary device tensors.
void symm_collective(int64_t mode, const std::vector<int64_t>& peer_ptrs, int64_t rank, int64_t epoch, const at::Tensor& src,
                     at::Tensor& dst, int64_t outer, int64_t inner_bytes, int64_t elem_kind, double scale,
                     int64_t stage_capacity, at::Tensor& status, int64_t num_ctas, int64_t target0, int64_t target1,
                     int64_t multicast_base) {
  c10::cuda::CUDAGuard g(src.device());
  std::vector<unsigned long long> ptrs(peer_ptrs.begin(), peer_ptrs.end());
  check(apb_symm_collective((int)mode, ptrs.data(), (int)rank, (int)ptrs.size(), (unsigned)epoch, src.data_ptr(), dst.data_ptr(),
                            outer, inner_bytes, (int)elem_kind, (float)scale, stage_capacity,
                            reinterpret_cast<uint32_t*>(status.data_ptr()), (int)num_ctas, (unsigned)target0, (unsigned)target1,
                            (unsigned long long)multicast_base, stream()),
        "apb_symm_collective");
}

// GEMM fused with a collective (see gemm_fused.cu).  a/b follow the conventions of ``gemm``; for the
// gather modes the gathered operand passed here is the local full-size buffer ``gbuf``.
void gemm_fused(int64_t fuse, const at::Tensor& a, const at::Tensor& b, at::Tensor& c, bool a_mn_major, bool b_mn_major,
                const std::vector<int64_t>& peer_ptrs, int64_t rank, int64_t epoch, int64_t rows_per_shard,
                const at::Tensor& shard_src, const at::Tensor& landed, int64_t landed_target, int64_t rows_per_rank,
                double scale, int64_t stage_capacity, const std::vector<int64_t>& targets, int64_t comm_ctas,
                at::Tensor& status) {
  c10::cuda::CUDAGuard g(a.device());
  TORCH_CHECK(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16, "gemm_fused: bf16 operands required");
  TORCH_CHECK(a.dim() == 2 && b.dim() == 2 && a.stride(1) == 1 && b.stride(1) == 1 && c.is_contiguous(), "gemm_fused: layout");
  const int K = a_mn_major ? a.size(0) : a.size(1);
  const int M = a_mn_major ? a.size(1) : a.size(0);
  const int N = b_mn_major ? b.size(1) : b.size(0);
  TORCH_CHECK((b_mn_major ? b.size(0) : b.size(1)) == K, "gemm_fused: contraction mismatch");
  const bool out_fp32 = c.scalar_type() == at::kFloat;
  std::vector<unsigned long long> ptrs(peer_ptrs.begin(), peer_ptrs.end());
  unsigned tg[3] = {(unsigned)targets[0], (unsigned)targets[1], (unsigned)targets[2]};
  void* gbuf = fuse == 1 ? a.data_ptr() : b.data_ptr();
  check(apb_gemm_fused((int)fuse, a.data_ptr(), b.data_ptr(), c.data_ptr(), M, N, K, a.stride(0), b.stride(0),
                       c.dim() == 2 ? c.stride(0) : N, a_mn_major, b_mn_major, out_fp32, ptrs.data(), (int)rank, (int)ptrs.size(),
                       (unsigned)epoch, (int)rows_per_shard, shard_src.data_ptr(), gbuf,
                       (long long)shard_src.numel() * shard_src.element_size(),
                       reinterpret_cast<uint32_t*>(landed.data_ptr()), (unsigned)landed_target, (int)rows_per_rank, (float)scale,
                       stage_capacity, tg, (int)comm_ctas, reinterpret_cast<uint32_t*>(status.data_ptr()), num_sms(), stream()),
        "apb_gemm_fused");
}

// ------------------------------------------------------------------ copy-engine collectives (dma_comm.cu)
std::vector<unsigned long long> u64(const std::vector<int64_t>& v) { return std::vector<unsigned long long>(v.begin(), v.end()); }

void dma_barrier(const std::vector<int64_t>& flags, int64_t rank, int64_t epoch, at::Tensor& status) {
  c10::cuda::CUDAGuard g(status.device());
  auto f = u64(flags);
  check(apb_dma_barrier(f.data(), (int)rank, (int)f.size(), (unsigned)epoch, reinterpret_cast<uint32_t*>(status.data_ptr()), stream()),
        "apb_dma_barrier");
}

void dma_all_gather(at::Tensor& dst, const std::vector<int64_t>& bases, int64_t offset, int64_t outer, int64_t inner_bytes,
                    int64_t rank) {
  c10::cuda::CUDAGuard g(dst.device());
  auto b = u64(bases);
  TORCH_CHECK(dst.is_contiguous() && (int64_t)dst.nbytes() == outer * inner_bytes * (int64_t)b.size(), "dma_all_gather: output size");
  check(apb_dma_all_gather(dst.data_ptr(), b.data(), offset, outer, inner_bytes, (int)rank, (int)b.size(), stream()),
        "apb_dma_all_gather");
}

void dma_rs_push(const at::Tensor& src, const std::vector<int64_t>& bases, const std::vector<int64_t>& flags, int64_t stage_offset,
                 int64_t slot_bytes, int64_t entry, int64_t ring, int64_t seq, int64_t rank, at::Tensor& status) {
  c10::cuda::CUDAGuard g(src.device());
  auto b = u64(bases), f = u64(flags);
  TORCH_CHECK(src.is_contiguous() && src.nbytes() % b.size() == 0, "dma_rs_push: contiguous input of n equal chunks");
  check(apb_dma_rs_push(src.data_ptr(), b.data(), f.data(), stage_offset, slot_bytes, (long long)(src.nbytes() / b.size()), (int)entry,
                        (int)ring, (unsigned)seq, (int)rank, (int)b.size(), reinterpret_cast<uint32_t*>(status.data_ptr()), stream()),
        "apb_dma_rs_push");
}

void dma_rs_sum(const at::Tensor& src, at::Tensor& dst, const std::vector<int64_t>& bases, const std::vector<int64_t>& flags,
                int64_t stage_offset, int64_t slot_bytes, int64_t entry, int64_t seq, double scale, int64_t rank, int64_t num_ctas,
                at::Tensor& status) {
  c10::cuda::CUDAGuard g(src.device());
  auto b = u64(bases), f = u64(flags);
  TORCH_CHECK(src.scalar_type() == at::kFloat && dst.scalar_type() == at::kFloat && src.is_contiguous() && dst.is_contiguous(),
              "dma_rs_sum: contiguous fp32 tensors");
  TORCH_CHECK(dst.nbytes() * b.size() == src.nbytes(), "dma_rs_sum: output is one of n equal chunks");
  check(apb_dma_rs_sum(src.data_ptr(), dst.data_ptr(), b.data(), f.data(), stage_offset, slot_bytes, (long long)dst.nbytes(), (int)entry,
                       (unsigned)seq, (float)scale, (int)rank, (int)b.size(), (int)num_ctas,
                       reinterpret_cast<uint32_t*>(status.data_ptr()), stream()),
        "apb_dma_rs_sum");
}

// (threads, registers per thread, bytes of shared memory) of a CTA of every kernel of a kind: "gemm", "split", and the communication kernels
// that are meant to become resident beside one of those, "beside".
std::map<std::string, std::vector<std::array<int, 3>>> kernel_footprints() {
  std::map<std::string, std::vector<std::array<int, 3>>> all;
  auto add = [&](const char* kind, int (*of)(int, int*), int i) {
    std::array<int, 3> out;
    const int err = of(i, out.data());
    if (err < 0) return false;
    check(err, "kernel_footprint");
    all[kind].push_back(out);
    return true;
  };
  for (int i = 0; add("gemm", apb_gemm_footprint, i); ++i) {}
  for (int i = 0; add("split", apb_gemm_split_footprint, i); ++i) {}
  for (int mode : {0, 2}) add("beside", apb_symm_footprint, mode);  // (the reduce-scatter keeps the loads from all peers in registers)
  for (int n = 2; add("beside", apb_dma_sum_footprint, n); ++n) {}
  return all;
}

// ------------------------------------------------------------------ the operators' CUDA entries
// Registered over the Python entries once the extension is loaded, so that an operator call - from a graph, from the autograd engine's
// threads - runs no Python on its way to the kernel: 6 to 9 us of host time per call, and the interpreter's lock.  Every function takes the
// forms that its counterpart in ops/cuda_impl.py gives to this extension, under the same conditions; all others, what the flags there
// ask for, and every call of an operator for which register_cuda_impl has installed another function go to the table of ops/library.py.
enum Entry : int {
  MM_ND, MM_WGRAD, GROUPED_MM, GROUPED_MM_WGRAD, DTYPE_CAST, RMS_NORM, RMS_NORM_BWD, ROPE, SWIGLU, SWIGLU_BWD, CROSS_ENTROPY, CROSS_ENTROPY_BWD,
  EMBEDDING, EMBEDDING_BWD, MOE_SLOTS, MOE_SCATTER, MOE_GATHER, MOE_GATE_GRAD, CAST_MANY, NUM_ENTRIES
};
constexpr const char* ENTRY_NAMES[NUM_ENTRIES] = {
    "mm_nd", "mm_wgrad", "grouped_mm", "grouped_mm_wgrad", "dtype_cast", "rms_norm", "rms_norm_bwd", "rope", "swiglu", "swiglu_bwd", "cross_entropy",
    "cross_entropy_bwd", "embedding", "embedding_bwd", "moe_slots", "moe_scatter", "moe_gather", "moe_gate_grad", "cast_many"};
struct Native {
  py::object table;  // operator name -> Python function, as it is at the time of a call
  py::object status_buffer;
  std::atomic<uint32_t> installed{0};  // bit per entry: the table's function is not the one of ops/cuda_impl.py
  bool diag_library_gemm = false, moe_kernels = true;
  std::atomic<bool> shadows{false};  // low-precision copies of parameters may exist: casts ask Python for them
  std::atomic<int64_t> launches{0};
};
Native& native() {
  static Native* n = new Native;  // (never destroyed: its Python object must not outlive the interpreter's end)
  return *n;
}

bool ours(Entry e) { return (native().installed.load(std::memory_order_relaxed) >> e & 1u) == 0; }

template <typename R, typename... A>
R in_python(Entry e, const A&... args) {
  py::gil_scoped_acquire gil;
  return py::cast<R>(native().table[ENTRY_NAMES[e]](args...));
}
py::object py_dtype(at::ScalarType t) { return py::reinterpret_borrow<py::object>(reinterpret_cast<PyObject*>(torch::getTHPDtype(t))); }

// The word that bounded waits report to, one per device: made by Python at the first use on a device and shared with it.
at::Tensor& status_of(const at::Tensor& t) {
  static auto& words = *new std::array<at::Tensor, 64>;  // (never destroyed, like Native)
  static std::array<std::atomic<bool>, 64> known{};
  static std::mutex m;
  const int dev = t.get_device();
  TORCH_CHECK(dev >= 0 && dev < 64, "unexpected device index ", dev);
  if (!known[dev].load(std::memory_order_acquire)) {
    at::Tensor w = [&]() {
      py::gil_scoped_acquire gil;
      return py::cast<at::Tensor>(native().status_buffer(t.device()));
    }();
    std::lock_guard<std::mutex> g(m);
    if (!known[dev].load(std::memory_order_relaxed)) {
      words[dev] = w;
      known[dev].store(true, std::memory_order_release);
    }
  }
  return words[dev];
}
void count(int64_t n = 1) { native().launches.fetch_add(n, std::memory_order_relaxed); }
bool float_or_bf16(at::ScalarType t) { return t == at::kBFloat16 || t == at::kFloat; }

using at::Tensor;
using Two = std::tuple<Tensor, Tensor>;

Tensor op_mm_nd(const Tensor& a, const Tensor& b, bool trans_b, at::ScalarType dtype) {
  if (ours(MM_ND) && float_or_bf16(dtype) && !native().diag_library_gemm) {
    auto c = mm_nd(a, b, trans_b, dtype == at::kFloat, status_of(a));
    if (c.has_value()) {
      count();
      return *c;
    }
  }
  py::gil_scoped_acquire gil;
  return in_python<Tensor>(MM_ND, a, b, trans_b, py_dtype(dtype));
}
Tensor op_mm_wgrad(const Tensor& a, const Tensor& b, at::ScalarType dtype) {
  if (ours(MM_WGRAD) && float_or_bf16(dtype) && !native().diag_library_gemm) {
    auto c = gemm_new(a, b, true, true, dtype == at::kFloat, status_of(a));
    if (c.has_value()) {
      count();
      return *c;
    }
  }
  py::gil_scoped_acquire gil;
  return in_python<Tensor>(MM_WGRAD, a, b, py_dtype(dtype));
}
bool grouped_ok(const Tensor& a, const Tensor& b, at::ScalarType dtype) {
  return a.dim() == 3 && b.dim() == 3 && a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16 && a.size(2) % 8 == 0 &&
         b.size(2) % 8 == 0 && float_or_bf16(dtype);
}
Tensor op_grouped_mm(const Tensor& a, const Tensor& b, bool trans_b, at::ScalarType dtype) {
  if (ours(GROUPED_MM) && grouped_ok(a, b, dtype) && b.size(trans_b ? 1 : 2) % 8 == 0) {
    Tensor c = at::empty({a.size(0), a.size(1), b.size(trans_b ? 1 : 2)}, a.options().dtype(dtype));
    gemm_grouped(dense(a), dense(b), c, false, !trans_b, status_of(a));
    count();
    return c;
  }
  py::gil_scoped_acquire gil;
  return in_python<Tensor>(GROUPED_MM, a, b, trans_b, py_dtype(dtype));
}
Tensor op_grouped_wgrad(const Tensor& a, const Tensor& b, at::ScalarType dtype) {
  if (ours(GROUPED_MM_WGRAD) && grouped_ok(a, b, dtype)) {
    Tensor c = at::empty({a.size(0), a.size(2), b.size(2)}, a.options().dtype(dtype));
    gemm_grouped(dense(a), dense(b), c, true, true, status_of(a));
    count();
    return c;
  }
  py::gil_scoped_acquire gil;
  return in_python<Tensor>(GROUPED_MM_WGRAD, a, b, py_dtype(dtype));
}
Tensor op_cast(const Tensor& x, at::ScalarType dtype) {
  if (x.scalar_type() == dtype && ours(DTYPE_CAST)) return x;
  if (ours(DTYPE_CAST) && !native().shadows.load(std::memory_order_relaxed) &&
      (dtype == at::kBFloat16 || (dtype == at::kFloat && x.scalar_type() == at::kBFloat16))) {
    auto y = cast_new(x, dtype == at::kBFloat16);
    if (y.has_value()) {
      count();
      return *y;
    }
  }
  py::gil_scoped_acquire gil;
  return in_python<Tensor>(DTYPE_CAST, x, py_dtype(dtype));
}
// dtype_cast of every tensor; those that its kernel would take are cast together.
std::vector<Tensor> op_cast_many(at::TensorList xs, at::ScalarType dtype) {
  if (!ours(CAST_MANY)) {
    py::gil_scoped_acquire gil;
    return in_python<std::vector<Tensor>>(CAST_MANY, xs.vec(), py_dtype(dtype));
  }
  const bool together = dtype == at::kBFloat16 && ours(DTYPE_CAST) && !native().shadows.load(std::memory_order_relaxed);
  std::vector<Tensor> out;
  std::vector<const void*> src;
  std::vector<void*> dst;
  std::vector<long long> n;
  out.reserve(xs.size());
  for (const Tensor& x : xs) {
    if (!together || x.scalar_type() != at::kFloat || x.get_device() != xs[0].get_device() || !x.is_contiguous() ||
        reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 != 0 || x.numel() > (int64_t(1) << 31)) {
      out.push_back(op_cast(x, dtype));
      continue;
    }
    out.push_back(at::empty(x.sizes(), x.options().dtype(at::kBFloat16)));
    src.push_back(x.data_ptr());
    dst.push_back(out.back().data_ptr());
    n.push_back(x.numel());
  }
  if (!src.empty()) {
    c10::cuda::CUDAGuard g(xs[0].device());
    int launches = 0;
    check(apb_cast_many(src.data(), dst.data(), n.data(), (int)src.size(), &launches, stream()), "apb_cast_many");
    count(launches);
  }
  return out;
}
Two op_rms_norm(const Tensor& x, const Tensor& w, double eps) {
  if (!ours(RMS_NORM)) return in_python<Two>(RMS_NORM, x, w, eps);
  count();
  return rms_norm_new(x, w, eps);
}
Two op_rms_norm_bwd(const Tensor& dy, const Tensor& x, const Tensor& w, const Tensor& rstd) {
  if (!ours(RMS_NORM_BWD)) return in_python<Two>(RMS_NORM_BWD, dy, x, w, rstd);
  count(2);
  return rms_norm_bwd_new(dy, x, w, rstd);
}
Tensor op_rope(const Tensor& x, const Tensor& cos, const Tensor& sin, bool conj) {
  if (!ours(ROPE)) return in_python<Tensor>(ROPE, x, cos, sin, conj);
  count();
  return rope_new(x, cos, sin, conj);
}
Tensor op_swiglu(const Tensor& a, const Tensor& b) {
  if (!ours(SWIGLU)) return in_python<Tensor>(SWIGLU, a, b);
  count();
  return swiglu_new(a, b);
}
Two op_swiglu_bwd(const Tensor& dy, const Tensor& a, const Tensor& b) {
  if (!ours(SWIGLU_BWD)) return in_python<Two>(SWIGLU_BWD, dy, a, b);
  count();
  return swiglu_bwd_new(dy, a, b);
}
Two op_xent(const Tensor& logits_, const Tensor& labels) {
  if (!ours(CROSS_ENTROPY)) return in_python<Two>(CROSS_ENTROPY, logits_, labels);
  Tensor logits = dense(logits_);
  const auto shape = logits.sizes().slice(0, logits.dim() - 1);
  Tensor loss = at::empty(shape, logits.options().dtype(at::kFloat)), lse = at::empty(shape, loss.options());
  xent_fwd(logits, labels.contiguous(), loss, lse);
  count();
  return {loss, lse};
}
Tensor op_xent_bwd(const Tensor& dloss, const Tensor& logits_, const Tensor& labels, const Tensor& lse) {
  if (!ours(CROSS_ENTROPY_BWD)) return in_python<Tensor>(CROSS_ENTROPY_BWD, dloss, logits_, labels, lse);
  Tensor logits = dense(logits_), out = at::empty_like(logits);
  xent_bwd(dloss.to(at::kFloat).contiguous(), logits, labels.contiguous(), lse.contiguous(), out);
  count();
  return out;
}
Tensor op_embedding(const Tensor& weight, const Tensor& ids) {
  if (ours(EMBEDDING) && weight.dim() == 2 && float_or_bf16(weight.scalar_type()) && weight.size(1) * weight.element_size() % 16 == 0 &&
      ids.scalar_type() == at::kLong) {
    auto shape = ids.sizes().vec();
    shape.push_back(weight.size(1));
    Tensor out = at::empty(shape, weight.options());
    embedding_fwd(dense(weight), ids.contiguous(), out);
    count();
    return out;
  }
  py::gil_scoped_acquire gil;
  return in_python<Tensor>(EMBEDDING, weight, ids);
}
Tensor op_embedding_bwd(const Tensor& dy_, const Tensor& ids, int64_t rows) {
  if (!ours(EMBEDDING_BWD)) return in_python<Tensor>(EMBEDDING_BWD, dy_, ids, rows);
  Tensor dy = dy_.contiguous(), out = at::empty({rows, dy.size(-1)}, dy.options());
  count(embedding_bwd(dy, ids.contiguous(), out));
  return out;
}

bool moe_ok(std::initializer_list<const Tensor*> ts) {
  if (!native().moe_kernels) return false;
  for (const Tensor* t : ts)
    if (!t->is_cuda()) return false;
  return true;
}
Tensor gate_weights(const Tensor& w, at::ScalarType dtype) { return (float_or_bf16(w.scalar_type()) ? w : w.to(dtype)).contiguous(); }
Tensor op_moe_slots(const Tensor& idx, int64_t E, int64_t C, int64_t nb) {
  if (ours(MOE_SLOTS) && moe_ok({&idx}) && idx.scalar_type() == at::kLong && idx.dim() == 2 && nb > 0 && idx.size(0) > 0 && idx.size(0) % nb == 0 &&
      E <= moe_slots_max_experts(idx.size(0) / nb * idx.size(1)) && E * C < (int64_t(1) << 31)) {
    Tensor slot = at::empty_like(idx, at::MemoryFormat::Contiguous);
    count(moe_slots(idx.contiguous(), slot, E, C, nb));
    return slot;
  }
  return in_python<Tensor>(MOE_SLOTS, idx, E, C, nb);
}
Tensor op_moe_scatter(const Tensor& src, const Tensor& slot, const Tensor& w, int64_t E, int64_t C, int64_t nb) {
  if (ours(MOE_SCATTER) && moe_ok({&src, &slot, &w}) && float_or_bf16(src.scalar_type()) && src.dim() == 2 && nb > 0 && src.size(0) > 0 &&
      src.size(0) % nb == 0) {
    Tensor buf = at::empty({E, nb, C, src.size(1)}, src.options());
    moe_scatter(src.contiguous(), slot.contiguous(), gate_weights(w, src.scalar_type()), buf, E, C, nb);
    count(2);
    return buf;
  }
  return in_python<Tensor>(MOE_SCATTER, src, slot, w, E, C, nb);
}
Tensor op_moe_gather(const Tensor& buf, const Tensor& slot, const Tensor& w) {
  if (ours(MOE_GATHER) && moe_ok({&buf, &slot, &w}) && float_or_bf16(buf.scalar_type()) && buf.dim() == 4 && buf.size(1) > 0 &&
      slot.dim() == 2 && slot.size(0) > 0 && slot.size(0) % buf.size(1) == 0) {
    Tensor out = at::empty({slot.size(0), buf.size(3)}, buf.options());
    moe_gather(buf.contiguous(), slot.contiguous(), gate_weights(w, buf.scalar_type()), out);
    count();
    return out;
  }
  return in_python<Tensor>(MOE_GATHER, buf, slot, w);
}
Tensor op_moe_gate_grad(const Tensor& buf, const Tensor& slot, const Tensor& g) {
  if (ours(MOE_GATE_GRAD) && moe_ok({&buf, &slot, &g}) && float_or_bf16(buf.scalar_type()) && buf.dim() == 4 &&
      g.scalar_type() == buf.scalar_type() && buf.size(1) > 0 && slot.dim() == 2 && slot.size(0) > 0 && slot.size(0) % buf.size(1) == 0) {
    Tensor dw = at::empty(slot.sizes(), buf.options().dtype(at::kFloat));
    moe_gate_grad(buf.contiguous(), slot.contiguous(), g.contiguous(), dw);
    count();
    return dw;
  }
  return in_python<Tensor>(MOE_GATE_GRAD, buf, slot, g);
}

// What register_cuda_impl installed for ``name``: ``on`` if it is not the function that the native entry stands for.
void native_installed(const std::string& name, bool on) {
  for (int e = 0; e < NUM_ENTRIES; ++e)
    if (name == ENTRY_NAMES[e]) {
      if (on) native().installed.fetch_or(1u << e, std::memory_order_relaxed);
      else native().installed.fetch_and(~(1u << e), std::memory_order_relaxed);
    }
}

// Once per process, after the Python functions are known.  The dispatcher warns when a kernel takes another's place, which here is meant.
void register_native(py::dict table, py::object status_buffer, bool diag_library_gemm, bool moe_kernels) {
  static torch::Library* lib = nullptr;
  if (lib != nullptr) return;
  native().table = std::move(table);
  native().status_buffer = std::move(status_buffer);
  native().diag_library_gemm = diag_library_gemm;
  native().moe_kernels = moe_kernels;
  struct Quiet : c10::WarningHandler {
    void process(const c10::Warning&) override {}
  } quiet;
  c10::WarningUtils::WarningHandlerGuard guard(&quiet);
  lib = new torch::Library(torch::Library::IMPL, "apb200", c10::DispatchKey::CUDA, __FILE__, __LINE__);
  lib->impl(ENTRY_NAMES[MM_ND], op_mm_nd);
  lib->impl(ENTRY_NAMES[MM_WGRAD], op_mm_wgrad);
  lib->impl(ENTRY_NAMES[GROUPED_MM], op_grouped_mm);
  lib->impl(ENTRY_NAMES[GROUPED_MM_WGRAD], op_grouped_wgrad);
  lib->impl(ENTRY_NAMES[DTYPE_CAST], op_cast);
  lib->impl(ENTRY_NAMES[RMS_NORM], op_rms_norm);
  lib->impl(ENTRY_NAMES[RMS_NORM_BWD], op_rms_norm_bwd);
  lib->impl(ENTRY_NAMES[ROPE], op_rope);
  lib->impl(ENTRY_NAMES[SWIGLU], op_swiglu);
  lib->impl(ENTRY_NAMES[SWIGLU_BWD], op_swiglu_bwd);
  lib->impl(ENTRY_NAMES[CROSS_ENTROPY], op_xent);
  lib->impl(ENTRY_NAMES[CROSS_ENTROPY_BWD], op_xent_bwd);
  lib->impl(ENTRY_NAMES[EMBEDDING], op_embedding);
  lib->impl(ENTRY_NAMES[EMBEDDING_BWD], op_embedding_bwd);
  lib->impl(ENTRY_NAMES[MOE_SLOTS], op_moe_slots);
  lib->impl(ENTRY_NAMES[MOE_SCATTER], op_moe_scatter);
  lib->impl(ENTRY_NAMES[MOE_GATHER], op_moe_gather);
  lib->impl(ENTRY_NAMES[MOE_GATE_GRAD], op_moe_gate_grad);
  lib->impl(ENTRY_NAMES[CAST_MANY], op_cast_many);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("kernel_footprints", &kernel_footprints);
  m.def("register_native", &register_native);
  m.def("native_installed", &native_installed);
  m.def("native_launches", []() { return native().launches.load(std::memory_order_relaxed); });
  m.def("native_shadows", [](bool on) { native().shadows.store(on, std::memory_order_relaxed); });
  m.def("dma_flag_bytes", []() { return (int64_t)apb_dma_flag_bytes(); });
  m.def("dma_ring_max", []() { return (int64_t)apb_dma_ring_max(); });
  m.def("dma_barrier", &dma_barrier);
  m.def("dma_all_gather", &dma_all_gather);
  m.def("dma_rs_push", &dma_rs_push);
  m.def("dma_rs_sum", &dma_rs_sum);
  m.def("gemm", &gemm);
  m.def("gemm_grouped", &gemm_grouped);
  m.def("gemm_split", &gemm_split);
  m.def("gemm_split_choice", [](int64_t groups, int64_t M, int64_t N, int64_t K) {  // groups 0: a plain product
    int bn = 0, s = 0;
    apb_gemm_split_choice((int)groups, (int)M, (int)N, (int)K, num_sms(), apb_gemm_get_reserved_sms(), &bn, &s);
    return std::make_tuple((int64_t)bn, (int64_t)s);
  });
  m.def("gemm_set_pair_mode", [](bool on) { apb_gemm_set_pair_mode(on ? 1 : 0); });
  m.def("gemm_yield_request", [](int64_t pairs) { check(apb_gemm_yield_request((int)pairs, stream()), "apb_gemm_yield_request"); });
  m.def("gemm_yield_outstanding", []() { return (int64_t)apb_gemm_yield_outstanding(); });
  m.def("gemm_set_dynamic_tiles", [](bool on) { apb_gemm_set_dynamic_tiles(on ? 1 : 0); });
  m.def("gemm_get_dynamic_tiles", []() { return apb_gemm_get_dynamic_tiles() != 0; });
  m.def("gemm_set_pair_stages", [](int64_t n) { apb_gemm_set_pair_stages((int)n); });
  m.def("gemm_get_pair_stages", []() { return (int64_t)apb_gemm_get_pair_stages(); });
  m.def("gemm_set_reserved_sms", [](int64_t n) { apb_gemm_set_reserved_sms((int)n); });
  m.def("gemm_get_reserved_sms", []() { return (int64_t)apb_gemm_get_reserved_sms(); });
  m.def("gemm_get_pair_mode", []() { return apb_gemm_get_pair_mode() != 0; });
  m.def("attention_fwd", &attention_fwd);
  m.def("mm", &gemm_new);
  m.def("mm_nd", &mm_nd);
  m.def("rms_norm", &rms_norm_new);
  m.def("rms_norm_bwd", &rms_norm_bwd_new);
  m.def("rope", &rope_new);
  m.def("swiglu", &swiglu_new);
  m.def("swiglu_bwd", &swiglu_bwd_new);
  m.def("cast", &cast_new);
  m.def("xent_fwd", &xent_fwd);
  m.def("xent_bwd", &xent_bwd);
  m.def("embedding_bwd", &embedding_bwd);
  m.def("embedding_bwd_sorts", [](int64_t tokens, int64_t rows, int64_t D, bool bf16) { return apb_embedding_bwd_sorts(tokens, rows, (int)D, bf16) != 0; });
  m.def("embedding_fwd", &embedding_fwd);
  m.def("adamw", &adamw);
  m.def("moe_slots_max_experts", &moe_slots_max_experts);
  m.def("moe_slots", &moe_slots);
  m.def("moe_scatter", &moe_scatter);
  m.def("moe_gather", &moe_gather);
  m.def("moe_gate_grad", &moe_gate_grad);
  m.def("symm_header_bytes", &symm_header_bytes);
  m.def("symm_wait_probe", &symm_wait_probe);
  m.def("symm_collective", &symm_collective);
  m.def("gemm_fused", &gemm_fused);
  m.def("gemm_fused_ctas", [](int64_t fuse, int64_t M, int64_t N, int64_t comm_ctas) {
    return (int64_t)apb_gemm_fused_ctas((int)fuse, (int)M, (int)N, (int)comm_ctas, num_sms());
  });
}
