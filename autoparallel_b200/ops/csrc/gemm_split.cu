// bf16 GEMM for shapes with few output tiles, sm_100a: one 128 x BN tile per thread-block cluster, the contraction split
// over the cluster's CTAs.
//
//   C[M,N] = opA * opB, operands and layouts as in gemm_tcgen05.cu; grouped form: G stacked problems of one shape
//
// The persistent kernels give every CTA (pair) whole tiles of 128 or 256 x 256, so a product with fewer tiles than SMs
// leaves most of the chip idle: 16 x 4096 x 4096 ran on 16 SMs, a router's weight gradient (64 x 2048, contracted over
// 8192 tokens) on 8, each waiting for its own serial chain of loads.  Here BN (64, 128, 256) and the number of k-slices S
// (1..8) are picked so that tiles x S fills the SMs.  Every CTA of a cluster accumulates its k-slice in TMEM, writes the
// fp32 tile to its own shared memory (the load stages are free by then), and after one cluster barrier each CTA adds up
// its share of the tile's rows from all S shared memories, in slice order, and stores it: no workspace, no atomics, no
// second launch, the same result every time.
//
// A cluster of one CTA has nothing to add and stores its tile from TMEM (store_tile).
//
//   warp 0: TMA producer | warp 1: TMEM owner + MMA issuer | warps 2..9 (64 columns: 2..5): TMEM -> shared memory (or C) | all: sum and store
// Persistent kernels -> this one, us: 16 x 4096 x 4096 27 -> 10.4, 16 x 4096 x 14336 84 -> 23.5, 64 x 2048 x 2048 15.6 -> 6.6, 64 x 2048 x 8192 46 -> 11.5,
// 512 x 256 x 256 5.8 -> 4.9, 160 x 8192 x 8192 45 -> 37; 1221 products in profiles/gemm_split_estimate_sweep.txt.
#include "gemm_core.cuh"

#include <mutex>

namespace apb {

constexpr int SPLIT_MAX = 8;  // portable cluster size
constexpr int SPLIT_STAGE_TOTAL = 196608;  // 8 x 24 KB, 6 x 32 KB or 4 x 48 KB: deep enough for one CTA to hide the load latency
constexpr int SPLIT_THREADS = GEMM_PLAIN_THREADS;
constexpr int SPLIT_SMEM_BYTES = SPLIT_STAGE_TOTAL + 1024 + 256;

__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

template <bool A_MN, bool B_MN, int BN_T, bool GROUPED>
__global__ void __launch_bounds__(SPLIT_THREADS, GEMM_MIN_CTAS)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmParams p) {
  constexpr int B_BYTES = BN_T * BK * 2;
  constexpr int ST = SPLIT_STAGE_TOTAL / (A_STAGE_BYTES + B_BYTES);
  constexpr int HALVES = BN_T >= 128 ? EPI_WARPS / 4 : 1, COLS = BN_T / HALVES;  // warps per lane quarter, and their columns: blocks of 64
  constexpr int LD = BN_T + 4;  // floats per row of the fp32 tile: rows start 16 bytes apart modulo the banks
  static_assert(BM * LD * 4 <= SPLIT_STAGE_TOTAL, "the fp32 tile reuses the stages");
  static_assert((2 * ST + 1) * 8 + 8 <= 256, "barrier block");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + ST * A_STAGE_BYTES;
  float* tile = reinterpret_cast<float*>(smem);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + SPLIT_STAGE_TOTAL);
  uint64_t* empty = full + ST;
  uint64_t* tmem_full = empty + ST;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_full + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int S = (int)cluster_size(), slice = (int)cluster_ctarank();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per_group = p.num_m_tiles * p.num_n_tiles;
  const int t = blockIdx.x / S;
  const int grp = GROUPED ? t / per_group : 0;
  int tm, tn;
  tile_coords(GROUPED ? t - grp * per_group : t, p.num_m_tiles, p.num_n_tiles, tm, tn);
  const int m0 = tm * BM, n0 = tn * BN_T;
  const int rows = min(BM, p.M - m0);  // of the tile that are inside the matrix
  const bool solo = S == 1 && p.vec_store;
  const int num_kb = (p.K + BK - 1) / BK;
  const int kb0 = (int)((long long)num_kb * slice / S), kb1 = (int)((long long)num_kb * (slice + 1) / S);  // S <= num_kb: never empty

  // The producer goes on as soon as it has set up the barriers; the others wait for them and for the TMEM columns, whose allocation
  // (half a microsecond) the first loads hide.
  uint32_t tmem_base = 0;
  if (warp == 0) {
    if (elect_one()) {
      for (int s = 0; s < ST; ++s) {
        mbar_init(&full[s], 1);
        mbar_init(&empty[s], 1);
      }
      mbar_init(tmem_full, 1);
      *abort_flag = 0;
      mbar_fence_init();
    }
    __syncwarp();
    named_arrive(1, SPLIT_THREADS);
    wait_previous();
  } else {
    if (warp == 1) {
      tmem_alloc(tmem_slot, BN_T);
      tmem_relinquish();
    } else if (warp == 2 && lane == 0) {
      tma_prefetch_desc(&tmA);
      tma_prefetch_desc(&tmB);
    }
    tc_fence_before();
    named_sync(1, SPLIT_THREADS);
    tc_fence_after();
    tmem_base = *tmem_slot;
    wait_previous();
  }
  auto fail = [&](uint32_t code) {
    atomicCAS(p.status, 0u, code);
    *abort_flag = 1;
  };

  // One elected thread per role, the stages unrolled, so that the barriers, the shared-memory addresses and the descriptors of a
  // stage are constants added to a base: issue is what bounded a k-block before (293 ns at any tile width, with lane 0 chosen by a
  // comparison and descriptors built from scratch; now 115 at 64 columns, 148 at 128, 277 - the tensor core's time - at 256).
  if (warp == 0) {
    if (elect_one()) {
      bool ok = true;
      uint32_t phase = 1;
      for (int kb = kb0; kb < kb1 && ok; kb += ST, phase ^= 1) {
#pragma unroll
        for (int stage = 0; stage < ST; ++stage) {
          if (kb + stage >= kb1) break;
          if (!mbar_wait(&empty[stage], phase, abort_flag)) {
            fail(ST_TIMEOUT_EMPTY);
            ok = false;
            break;
          }
          auto load = [&](uint8_t* dst, const CUtensorMap* m, int x, int y) {
            if (GROUPED) tma_load_3d(dst, m, &full[stage], x, y, grp);
            else tma_load_2d(dst, m, &full[stage], x, y);
          };
          mbar_expect_tx(&full[stage], A_STAGE_BYTES + B_BYTES);
          uint8_t* a_dst = sA + stage * A_STAGE_BYTES;
          uint8_t* b_dst = sB + stage * B_BYTES;
          const int k0 = (kb + stage) * BK;
          if (!A_MN) {
            load(a_dst, &tmA, k0, m0);
          } else {
#pragma unroll
            for (int c = 0; c < BM / 64; ++c) load(a_dst + c * CHUNK_BYTES, &tmA, m0 + c * 64, k0);
          }
          if (!B_MN) {
            load(b_dst, &tmB, k0, n0);
          } else {
#pragma unroll
            for (int c = 0; c < BN_T / 64; ++c) load(b_dst + c * CHUNK_BYTES, &tmB, n0 + c * 64, k0);
          }
        }
      }
      let_next_in();
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(BM, BN_T, A_MN ? 1u : 0u, B_MN ? 1u : 0u);
      const uint64_t a_desc = make_smem_desc(smem_u32(sA), A_MN ? CHUNK_BYTES : 16, 1024);
      const uint64_t b_desc = make_smem_desc(smem_u32(sB), B_MN ? CHUNK_BYTES : 16, 1024);
      bool ok = true;
      uint32_t phase = 0, accumulate = 0;
      for (int kb = kb0; kb < kb1 && ok; kb += ST, phase ^= 1) {
#pragma unroll
        for (int stage = 0; stage < ST; ++stage) {
          if (kb + stage >= kb1) break;
          if (!mbar_wait(&full[stage], phase, abort_flag)) {
            fail(ST_TIMEOUT_FULL);
            ok = false;
            break;
          }
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            umma_f16(tmem_base, a_desc + desc_offset(stage * A_STAGE_BYTES + k * (A_MN ? UMMA_K * 128 : UMMA_K * 2)),
                     b_desc + desc_offset(stage * B_BYTES + k * (B_MN ? UMMA_K * 128 : UMMA_K * 2)), idesc, k > 0 ? 1u : accumulate);
            accumulate = 1;
          }
          umma_commit(&empty[stage]);
        }
      }
      if (ok) umma_commit(tmem_full);
    }
    __syncwarp();
  } else if (warp < 2 + 4 * HALVES) {
    const int q = warp & 3;  // TMEM lane quarter this warp may read
    const int col0 = ((warp - 2) >> 2) * COLS;  // first of its columns
    // (the TMEM loads are warp-wide: the warp goes on together or not at all)
    if (!__all_sync(0xffffffffu, mbar_wait(tmem_full, 0, abort_flag))) {
      fail(ST_TIMEOUT_TMEM_FULL);
    } else if (solo) {
      tc_fence_after();
      uint8_t* stg = smem + (warp - 2) * STORE_BYTES;
      const uint32_t taddr = tmem_base + (uint32_t(q * 32) << 16) + col0;
      const long long c_off = GROUPED ? (long long)grp * p.M * p.ldc : 0;
      auto nothing = []() {};
      if (p.out_fp32) store_tile<true>(reinterpret_cast<float*>(p.C) + c_off, p.ldc, stg, taddr, m0 + q * 32, n0 + col0, COLS, p.M, p.N, lane, nothing);
      else store_tile<false>(reinterpret_cast<__nv_bfloat16*>(p.C) + c_off, p.ldc, stg, taddr, m0 + q * 32, n0 + col0, COLS, p.M, p.N, lane, nothing);
    } else if (q * 32 < rows) {
      tc_fence_after();
      float* row = tile + (q * 32 + lane) * LD + col0;
#pragma unroll (COLS > 64 ? 2 : 4)  // (the registers of four loads are more than a communication kernel's CTA leaves)
      for (int c = 0; c < COLS / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32(tmem_base + (uint32_t(q * 32) << 16) + col0 + c * 32, r);
        tmem_ld_wait_for(r);
#pragma unroll
        for (int i = 0; i < 8; ++i)
          reinterpret_cast<uint4*>(row + c * 32)[i] = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
      }
    }
  }
  if (solo) {  // nothing to add up: the warps have stored the tile from TMEM
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
      tc_fence_after();
      tmem_dealloc(tmem_base, BN_T);
    }
    return;
  }
  tc_fence_before();
  __syncwarp();
  cluster_arrive();  // (also orders the threads of a cluster of one CTA)
  cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, BN_T);
  }

  // The sum: four columns per thread and row, the rows of a thread a whole stride apart, two at a time so that their loads are under way
  // together (the other CTAs' shared memory gives 16 bytes a cycle and SM, with a round trip of hundreds of cycles).  The loops stay small on
  // purpose: eight rows at a time, unrolled, were slower in every product (64 x 1408 x 2048 6.9 us against 5.8): the code is fetched once
  // per launch.  128 x 128 tiles in two slices: sum and store 2.8 -> 1.6 us, in one 2.8 + 0.8 -> 1.2 (TMEM to C).
  if (*abort_flag == 0) {
    constexpr int VPR = BN_T / 4, RSTEP = SPLIT_THREADS / VPR;  // threads per row, rows per pass of the CTA
    static_assert(RSTEP * VPR == SPLIT_THREADS, "whole rows");
    const int c = (threadIdx.x % VPR) * 4, col = n0 + c, step = S * RSTEP;
    const bool whole = (p.ldc & 3) == 0 && col + 4 <= p.N;
    const int esz = p.out_fp32 ? 4 : 2;
    const uint32_t src0 = smem_u32(tile) + c * 4;
    uint8_t* dst0 = reinterpret_cast<uint8_t*>(p.C) + ((GROUPED ? (long long)grp * p.M * p.ldc : 0) + (long long)m0 * p.ldc + col) * esz;
    const long long ld_bytes = p.ldc * esz;
    auto add = [](float4& a, const float4& x) { a.x += x.x; a.y += x.y; a.z += x.z; a.w += x.w; };
    auto store = [&](int r, const float4& v) {
      uint8_t* dst = dst0 + r * ld_bytes;
      if (whole) {
        if (p.out_fp32) *reinterpret_cast<float4*>(dst) = v;
        else *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
      } else {
        const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (col + i >= p.N) break;
          if (p.out_fp32) reinterpret_cast<float*>(dst)[i] = f[i];
          else reinterpret_cast<__nv_bfloat16*>(dst)[i] = __float2bfloat16(f[i]);
        }
      }
    };
#pragma unroll 1
    for (int r = slice * RSTEP + threadIdx.x / VPR; r < rows && col < p.N; r += 2 * step) {
      const uint32_t src = src0 + r * (LD * 4);
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
      if (r + step < rows) {
#pragma unroll 2
        for (int s = 0; s < S; ++s) {
          const uint32_t from = map_to_cta(src, (uint32_t)s);
          const float4 x = ld_cluster_f4(from), y = ld_cluster_f4(from + step * (LD * 4));
          add(a, x);
          add(b, y);
        }
        store(r + step, b);
      } else {
#pragma unroll 4
        for (int s = 0; s < S; ++s) add(a, ld_cluster_f4(map_to_cta(src, (uint32_t)s)));
      }
      store(r, a);
    }
  }
  __syncwarp();
  cluster_arrive_relaxed();  // no CTA leaves while another may still read its tile
  cluster_wait();
}

}  // namespace apb

using namespace apb;

typedef void (*SplitKernel)(CUtensorMap, CUtensorMap, GemmParams);

template <int BN_T, bool GROUPED>
static SplitKernel split_kernel_of(int a_mn, int b_mn) {
  if (!a_mn && !b_mn) return gemm_split_kernel<false, false, BN_T, GROUPED>;
  if (!a_mn) return gemm_split_kernel<false, true, BN_T, GROUPED>;
  if (!b_mn) return gemm_split_kernel<true, false, BN_T, GROUPED>;
  return gemm_split_kernel<true, true, BN_T, GROUPED>;
}

template <bool GROUPED>
static SplitKernel split_kernel_of(int bn, int a_mn, int b_mn) {
  return bn == 64 ? split_kernel_of<64, GROUPED>(a_mn, b_mn) : bn == 128 ? split_kernel_of<128, GROUPED>(a_mn, b_mn)
                                                                         : split_kernel_of<256, GROUPED>(a_mn, b_mn);
}

// Tile width and slice count for a product, or bn = 0 where the persistent kernels are expected to be faster.
//
// Only forms whose clusters are all resident at once: in a second wave every tile pays its fixed part again.  Left out as well, because the
// sweeps showed the estimates to flatter them: forms with no more CTAs than the persistent kernels would use (twice as many where the contraction
// has one or two blocks), slices of a single block, whole contractions in 256-wide tiles, and in 64-wide ones on most of the chip.
//
// Two sets of estimates (SplitCosts, microseconds on one B200).  FITTED, to a sweep of 1221 products with every form that fits, 1 <= M <= 4096,
// 64 <= N, K <= 8192, all layouts (profiles/gemm_split_estimate_sweep.txt), picks the form for contractions of more than 16 blocks.  EARLIER,
// fitted to the kernels before their single-thread roles were elected, bounds the length of a slice's chain of fp32 sums: the tensor cores'
// rounding error grows in proportion to it, 2.1 times at twice the length (fp32 results, 64 x 1 in place of 128 x 2, 1160 <= K <= 2800), and
// without the bound one product in a hundred got a longer chain than it had, up to twice.  Contractions of up to 16 blocks (K <= 1024) keep the
// form that EARLIER gives them: FITTED would gain 0.1 to 0.4 us each, most of it by fewer slices.
// On the products of the sweep with K > 1024 the forms picked take 2.4 % more than the best one in the geometric mean (without the bound 2.3,
// by EARLIER alone 7.4).
struct SplitPlan {
  int bn, s;
};
extern "C" int apb_gemm_resident_pairs(int num_sms);

static SplitKernel split_kernel_any() { return gemm_split_kernel<false, false, 64, false>; }

// CTAs of clusters of 1 ... SPLIT_MAX that are resident at once on the current device (one CTA per SM; the partial ends of the GPCs are
// lost); asked once per device.
static void ask_slots(int* slots, int num_sms) {
  SplitKernel kern = split_kernel_any();
  const bool opted_in = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SPLIT_SMEM_BYTES) == cudaSuccess;
  for (int s = 1; s <= SPLIT_MAX; ++s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(num_sms / s * s));
    cfg.blockDim = dim3(SPLIT_THREADS);
    cfg.dynamicSmemBytes = SPLIT_SMEM_BYTES;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)s;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (!opted_in || cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      n = num_sms / s / 2;
    }
    slots[s] = n * s;
  }
}
static const int* split_slots(int num_sms) {
  constexpr int DEVICES = 64;
  static int slots[DEVICES][SPLIT_MAX + 1];
  static std::once_flag asked[DEVICES];
  static const int none[SPLIT_MAX + 1] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= DEVICES) return none;  // (the persistent kernels)
  std::call_once(asked[dev], ask_slots, slots[dev], num_sms);
  return slots[dev];
}

// What a form is expected to take: a fixed part (launch, prologue, the way out of TMEM), then the longest of a chain of k-blocks, the operand
// traffic out of L2 and the operands out of memory (less while few bytes are in flight; the sweep's operands were partly in L2, which its rates
// include), a round trip more where the chain is longer than the stages, then what comes through the other CTAs' shared memory.
struct SplitCosts {
  double pair_launch, pair_wave, pair_kb, single_launch, single_wave, single_kb, margin;  // the persistent kernels, and what a form has to beat
  double per_kb[3], one_slice[3], more_slices[3];                                          // by tile width: 64, 128, 256
  double l2, memory, memory_per_mb;                                                        // bytes per us; the last per megabyte in flight
  double long_chain, sum_width, sum_byte, sum_slice;                                       // us; per slice and 64 columns, per byte, per slice
};
constexpr SplitCosts EARLIER = {5.5, 0.5, 0.38, 5.5, 0.5, 0.35, 0.95,
                                {0.27, 0.20, 0.27}, {5.6, 7.0, 9.0}, {5.6, 7.0, 9.0},
                                9.5e6, 6.5e6, 0.62e6,
                                0.0, 0.05, 0.0, 0.0};
constexpr SplitCosts FITTED = {3.35, 0.49, 0.45, 3.2, 0.87, 0.33, 1.0,
                               {0.23, 0.26, 0.39}, {3.5, 4.0, 4.0}, {4.1, 4.1, 3.8},
                               14.7e6, 8.6e6, 0.684e6,
                               0.31, 0.0, 1 / 18.7e3, 0.034};

// The fastest form by ``costs`` with at most ``max_chain`` k-blocks to a slice; the persistent kernels have them all.
static SplitPlan split_pick(const SplitCosts& costs, int max_chain, int G, int M, int N, int K, int num_sms, int reserved) {
  const long long g = G > 0 ? G : 1;
  const long long m_tiles = (M + BM - 1) / BM;
  const int usable = num_sms - reserved > 0 ? num_sms - reserved : 1;
  SplitPlan best{0, 0};
  if (g * m_tiles * ((N + 255) / 256) > usable) return best;  // no width fits in one wave
  const int kb = (K + BK - 1) / BK;
  const bool pair = pair_shape(M, N, K);
  const long long tiles = g * (pair ? (M + 2 * BM - 1) / (2 * BM) : m_tiles) * ((N + BN - 1) / BN);
  int units = pair ? apb_gemm_resident_pairs(num_sms) - reserved / 2 : usable;  // as the launches have it
  if (units < 1) units = 1;
  const double waves = (double)((tiles + units - 1) / units);
  const double now = pair ? costs.pair_launch + waves * (costs.pair_wave + costs.pair_kb * kb)
                          : costs.single_launch + waves * (costs.single_wave + costs.single_kb * kb);
  const long long ctas = (tiles < units ? tiles : units) * (pair ? 2 : 1) * (kb <= 2 ? 2 : 1);
  const double operands = 2.0 * g * ((double)M * K + (double)N * K);
  const int* slots = split_slots(num_sms);
  double t_best = kb <= max_chain ? costs.margin * now : 1e30;
  for (int w = 0; w < 3; ++w) {
    const int bn = 64 << w;
    const int stages = SPLIT_STAGE_TOTAL / (A_STAGE_BYTES + bn * BK * 2);
    const long long t = g * m_tiles * ((N + bn - 1) / bn);
    const double rows = M < BM ? M : BM, cols = N < bn ? N : bn, kb_bytes = 128.0 * (rows + cols);
    for (int s = 1; s <= SPLIT_MAX && s <= kb; ++s) {
      if (t * s > usable) break;
      if (t * s > slots[s] || t * s <= ctas) continue;
      if (s > 1 ? kb < 2 * s : bn == 256 || (bn == 64 && t > 100)) continue;
      const int chain = (kb + s - 1) / s;
      if (chain > max_chain) continue;
      double flow = costs.per_kb[w] * chain;
      const double l2 = (double)t * kb * kb_bytes / costs.l2;
      if (l2 > flow) flow = l2;
      // megabytes in flight: the stages of all CTAs, rows and columns outside the matrices not counted
      const double grows = costs.memory_per_mb * 0.1875 * t * s * kb_bytes / (128.0 * (BM + bn));
      const double from_memory = operands / (grows < costs.memory ? grows : costs.memory);
      if (from_memory > flow) flow = from_memory;
      double est = (s > 1 ? costs.more_slices[w] : costs.one_slice[w]) + flow + (chain > stages ? costs.long_chain : 0.0);
      if (s > 1) est += costs.sum_width * s * bn / 64 + costs.sum_byte * 4.0 * rows * cols * (s - 1) / s + costs.sum_slice * s;
      if (est < t_best) {
        t_best = est;
        best = SplitPlan{bn, s};
      }
    }
  }
  return best;
}

static SplitPlan split_plan(int G, int M, int N, int K, int num_sms, int reserved) {
  const int kb = (K + BK - 1) / BK;
  const SplitPlan earlier = split_pick(EARLIER, kb, G, M, N, K, num_sms, reserved);
  if (kb <= 16) return earlier;
  return split_pick(FITTED, earlier.bn ? (kb + earlier.s - 1) / earlier.s : kb, G, M, N, K, num_sms, reserved);
}

// The rule above: tile width and slices, 0 and 0 where the persistent kernels run.
extern "C" void apb_gemm_split_choice(int G, int M, int N, int K, int num_sms, int reserved, int* bn, int* s) {
  const SplitPlan plan = split_plan(G, M, N, K, num_sms, reserved);
  *bn = plan.bn;
  *s = plan.s;
}

// One launch with the given tile width (64, 128, 256) and number of k-slices (1..8, at most one per 64 of K).  G > 0: grouped,
// dense stacks (lda / ldb / ldc ignored).  Returns 0, or an argument / driver error (nothing launched).
extern "C" int apb_gemm_split(const void* A, const void* B, void* C, int G, int M, int N, int K, long long lda, long long ldb, long long ldc,
                              int a_mn, int b_mn, int out_fp32, int bn, int s, uint32_t* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (bn != 64 && bn != 128 && bn != 256) return 3;
  if (s < 1 || s > SPLIT_MAX || s > (K + BK - 1) / BK) return 3;
  const bool grouped = G > 0;
  if (grouped) {
    lda = a_mn ? M : K;
    ldb = b_mn ? N : K;
    ldc = N;
  }
  if ((lda & 7) || (ldb & 7) ||
      ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) & 15))
    return 3;  // 16-byte bases and rows for TMA and for the vector stores
  CUtensorMap tmA, tmB;
  int e;
  if (grouped) {
    e = !a_mn ? make_map_3d(&tmA, A, (uint64_t)K, (uint64_t)M, (uint64_t)G, (uint64_t)lda, BM)
              : make_map_3d(&tmA, A, (uint64_t)M, (uint64_t)K, (uint64_t)G, (uint64_t)lda, BK);
    if (e) return e;
    e = !b_mn ? make_map_3d(&tmB, B, (uint64_t)K, (uint64_t)N, (uint64_t)G, (uint64_t)ldb, bn)
              : make_map_3d(&tmB, B, (uint64_t)N, (uint64_t)K, (uint64_t)G, (uint64_t)ldb, BK);
  } else {
    e = !a_mn ? make_map(&tmA, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda, BM) : make_map(&tmA, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, BK);
    if (e) return e;
    e = !b_mn ? make_map(&tmB, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, bn) : make_map(&tmB, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, BK);
  }
  if (e) return e;
  GemmParams p;
  p.M = M; p.N = N; p.K = K; p.C = C; p.ldc = ldc; p.out_fp32 = out_fp32;
  p.num_m_tiles = (M + BM - 1) / BM;
  p.num_n_tiles = (N + bn - 1) / bn;
  p.status = status;
  p.groups = grouped ? G : 1;
  p.vec_store = ldc % (out_fp32 ? 4 : 8) == 0 && N % (out_fp32 ? 4 : 8) == 0;
  const long long ctas = (long long)p.num_m_tiles * p.num_n_tiles * p.groups * s;
  if (ctas > 0x7fffffffll / s) return 3;
  SplitKernel kern = grouped ? split_kernel_of<true>(bn, a_mn, b_mn) : split_kernel_of<false>(bn, a_mn, b_mn);
  // (the attribute belongs to the current device's instance of the kernel)
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SPLIT_SMEM_BYTES) != cudaSuccess) return 4;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(SPLIT_THREADS);
  cfg.dynamicSmemBytes = SPLIT_SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = (unsigned)s;
  attrs[0].val.clusterDim.y = 1;
  attrs[0].val.clusterDim.z = 1;
  attrs[1] = overlap_attribute();
  cfg.attrs = attrs;
  cfg.numAttrs = apb_gemm_makes_room() ? 1 : 2;
  return cudaLaunchKernelEx(&cfg, kern, tmA, tmB, p) == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : 4;
}

// The rule above and its launch: 0 = launched, -1 = the caller's kernels are the better choice (nothing launched), > 0 = error.
extern "C" int apb_gemm_split_auto(const void* A, const void* B, void* C, int G, int M, int N, int K, long long lda, long long ldb,
                                   long long ldc, int a_mn, int b_mn, int out_fp32, uint32_t* status, int num_sms, int reserved,
                                   cudaStream_t stream) {
  const SplitPlan plan = split_plan(G, M, N, K, num_sms, reserved);
  if (plan.bn == 0) return -1;
  return apb_gemm_split(A, B, C, G, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_fp32, plan.bn, plan.s, status, stream);
}

// Footprint of the ``i``-th kernel of this file; -1 past the last.
extern "C" int apb_gemm_split_footprint(int i, int* out) {
  if (i < 0 || i >= 24) return -1;
  const int bn = 64 << (i % 3), a_mn = i / 3 & 1, b_mn = i / 6 & 1;
  const SplitKernel kern = i < 12 ? split_kernel_of<false>(bn, a_mn, b_mn) : split_kernel_of<true>(bn, a_mn, b_mn);
  return kernel_footprint((const void*)kern, SPLIT_THREADS, SPLIT_SMEM_BYTES, out);
}
