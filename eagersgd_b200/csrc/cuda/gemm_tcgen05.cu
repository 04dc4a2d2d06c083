// bf16 GEMM on tcgen05 / TMEM / TMA for sm_100a:  C[M,N] = op(A) * op(B)^T
//
// Operands may be K-major (rows contiguous along K) or MN-major (stored [K][MN]);
// the latter is what weight-gradient GEMMs over NHWC activations need, where K is
// the pixel dimension.  Split-K with partial sums added by TMA reductions covers their
// few-tiles / long-K shape.  Used for dense layers, 1x1 convolutions (NHWC makes
// them plain GEMMs) and the LSTM projections; the reference reaches cuBLAS / cuDNN
// through TensorFlow for the same ops (official/resnet/resnet_model.py:97-101,552)
// and has a naive CPU GEMM (deep500 .../cpp/utility/gemm.hpp:9-64), the oracle.
// The pipeline itself (producer / MMA / epilogue warps) lives in umma_pipeline.cuh.
#include <cuda_runtime.h>
#include <stdint.h>
#include "launch.cuh"
#include "tensormap.cuh"
#include "umma_pipeline.cuh"
#include "umma_split.cuh"

using namespace umma;
using esgd::sm_count;

namespace {

template <int BN_, bool A_MN_, bool B_MN_, bool kPair_ = false, int kTwoPanels_ = 1>
struct GemmProblem {
  static constexpr int BN = BN_;
  static constexpr bool A_MN = A_MN_, B_MN = B_MN_, kZeroStages = false, kHalo = false, kPair = kPair_;
  static constexpr int kTwoPanels = kTwoPanels_;
  CUtensorMap tmA, tmB, tmC, tmR;   // tmC: bf16 panels of 64 columns or fp32 ones of 32; tmR: optional residual
  int M, N, K;
  int m_tiles, n_tiles, splits, kb_total, kb_per_split;
  int fixed_n;        // every CTA keeps one column range (needed for the per-CTA statistics flush)
  int res_kb;         // > 0: all k-blocks of B for the CTA's column range stay in shared memory
  static constexpr int ksteps = BK / 16, n_mma = BN_;

  struct Tile { int kb0, kb1, n0, m0; };

  __device__ __forceinline__ bool tile(int it, Tile& t) const {
    // a pair walks over tiles of 256 rows; m_tiles counts those
    const int worker = kPair ? blockIdx.x / 2 : blockIdx.x, workers = kPair ? gridDim.x / 2 : gridDim.x;
    int m_idx, n_idx, split = 0;
    if (fixed_n) {
      n_idx = worker % n_tiles;
      m_idx = worker / n_tiles + it * (workers / n_tiles);
      if (m_idx >= m_tiles) return false;
    } else {
      const int id = worker + it * workers;
      if (id >= m_tiles * n_tiles * splits) return false;
      split = id / (m_tiles * n_tiles);
      const int rem = id % (m_tiles * n_tiles);
      m_idx = rem / n_tiles;
      n_idx = rem % n_tiles;
    }
    place(kPair ? 2 * m_idx + (int)(blockIdx.x & 1) : m_idx, n_idx, t);
    t.kb0 = split * kb_per_split;
    t.kb1 = min(t.kb0 + kb_per_split, kb_total);
    return true;
  }
  __device__ __forceinline__ void place(int m_idx, int n_idx, Tile& t) const {
    t.m0 = m_idx * BM;
    t.n0 = n_idx * BN;
  }
  using Step = int;            // the k-block's number
  __device__ __forceinline__ Step begin(const Tile& t) const { return t.kb0; }
  __device__ __forceinline__ void advance(Step& kb) const { ++kb; }
  __device__ __forceinline__ void load_a(const Tile& t, int kb, uint8_t* a, uint64_t* bar) const {
    const int k0 = kb * BK;
    if (A_MN) {
#pragma unroll
      for (int i = 0; i < BM / 64; ++i) tma_load_2d(a + i * 8192, &tmA, bar, t.m0 + 64 * i, k0);
    } else {
      tma_load_2d(a, &tmA, bar, k0, t.m0);
    }
  }
  __device__ __forceinline__ void load_b(const Tile& t, int kb, uint8_t* b, uint64_t* bar) const {
    const int k0 = kb * BK;
    if (B_MN) {
#pragma unroll
      for (int i = 0; i < BN / 64; ++i) tma_load_2d(b + i * 8192, &tmB, bar, t.n0 + 64 * i, k0);
    } else {
      tma_load_2d(b, &tmB, bar, k0, t.n0);
    }
  }
  // pair: this CTA's rows of A and its half of the columns of B
  __device__ __forceinline__ void load(const Tile& t, int kb, uint8_t* a, uint8_t* b, uint32_t leader_bar) const {
    const int k0 = kb * BK, n0 = t.n0 + (int)(blockIdx.x & 1) * (BN / 2);
    if (A_MN) {
#pragma unroll
      for (int i = 0; i < BM / 64; ++i) tma_load_2d_pair(a + i * 8192, &tmA, leader_bar, t.m0 + 64 * i, k0);
    } else {
      tma_load_2d_pair(a, &tmA, leader_bar, k0, t.m0);
    }
    if (B_MN) {
#pragma unroll
      for (int i = 0; i < BN / 128; ++i) tma_load_2d_pair(b + i * 8192, &tmB, leader_bar, n0 + 64 * i, k0);
    } else {
      tma_load_2d_pair(b, &tmB, leader_bar, k0, n0);
    }
  }
  __device__ __forceinline__ void load(const Tile& t, int kb, uint8_t* a, uint8_t* b, uint64_t* bar) const {
    load_a(t, kb, a, bar);
    load_b(t, kb, b, bar);
  }
  __device__ __forceinline__ void store_panel(const Tile& t, int panel, const void* smem) const {
    if (!kPair || t.m0 < M) tma_store_2d(&tmC, smem, t.n0 + panel * 64, t.m0);
  }
  __device__ __forceinline__ int out_row(int row) const { return row; }
  __device__ __forceinline__ int valid_prefix(const Tile& t) const { return min(BM, M - t.m0); }
  __device__ __forceinline__ int64_t first_row(const Tile& t) const { return t.m0; }
  __device__ __forceinline__ void load_res_panel(const Tile& t, int panel, void* smem, uint64_t* bar) const {
    tma_load_2d(smem, &tmR, bar, t.n0 + panel * 64, t.m0);
  }
  __device__ __forceinline__ void store_f32(const Tile& t, int col, const void* smem, bool add) const {
    if (kPair && t.m0 >= M) return;              // the second half of the last tile
    if (add) tma_reduce_2d(&tmC, smem, col, t.m0);
    else tma_store_2d(&tmC, smem, col, t.m0);
  }
};

template <class P, bool kBn>
__global__ void __launch_bounds__(NUM_THREADS, 1) gemm_kernel(const __grid_constant__ P prob, const Epilogue ep) {
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&prob.tmA);
    tma_prefetch_desc(&prob.tmB);
  }
  run<P, kBn>(prob, ep);
}

template <class P, int S>
__global__ void __launch_bounds__(SPLIT_THREADS, 1) gemm_split_kernel(const __grid_constant__ P prob, const Epilogue ep, const SplitOut so) {
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&prob.tmA);
    tma_prefetch_desc(&prob.tmB);
  }
  run_split<P, S>(prob, ep, so);
}

struct GemmArgs {
  const void *A, *B;
  void* C;
  int M, N, K, lda, ldb, ldc, out_mode, splits;
};

// Whether B stays in shared memory: its whole K extent fits beside the A stages (max_kb k-blocks of it) and every CTA has several tiles
// of one column range to amortise the load over.
template <int BN>
bool b_resident(const GemmArgs& g, int max_kb, int sms) {
  const int m_tiles = (g.M + BM - 1) / BM, n_tiles = (g.N + BN - 1) / BN;
  return resident_enabled() && g.splits <= 1 && (g.K + BK - 1) / BK <= max_kb && n_tiles <= sms / 2 && m_tiles >= 2 * (sms / n_tiles);
}

template <int BN, bool A_MN, bool B_MN, bool kBn = false, bool kPair = false, bool kResPanels = false>
int launch(const GemmArgs& g, Epilogue ep, cudaStream_t stream) {
  using P = GemmProblem<BN, A_MN, B_MN, kPair, kResPanels ? 2 : 1>;
  static esgd::SmemAllowed allowed{0};
  if (const int e = esgd::allow_smem(gemm_kernel<P, kBn>, Cfg<BN>::SMEM_BYTES, allowed)) return e;
  P p;
  uint64_t dims[2], strides[1];
  uint32_t box[2];
  if (A_MN) { dims[0] = (uint64_t)g.M; dims[1] = (uint64_t)g.K; box[0] = 64; box[1] = 64; }
  else { dims[0] = (uint64_t)g.K; dims[1] = (uint64_t)g.M; box[0] = 64; box[1] = 128; }
  strides[0] = (uint64_t)g.lda * 2;
  int r = esgd::make_tensormap_bf16(&p.tmA, g.A, 2, dims, strides, box, nullptr);
  if (r != 0) return 1000 + r;
  if (B_MN) { dims[0] = (uint64_t)g.N; dims[1] = (uint64_t)g.K; box[0] = 64; box[1] = 64; }
  else { dims[0] = (uint64_t)g.K; dims[1] = (uint64_t)g.N; box[0] = 64; box[1] = (uint32_t)(kPair ? BN / 2 : BN); }
  strides[0] = (uint64_t)g.ldb * 2;
  r = esgd::make_tensormap_bf16(&p.tmB, g.B, 2, dims, strides, box, nullptr);
  if (r != 0) return 2000 + r;
  if (g.out_mode == OUT_BF16) {
    dims[0] = (uint64_t)g.N; dims[1] = (uint64_t)g.M; box[0] = 64; box[1] = 128;
    strides[0] = (uint64_t)g.ldc * 2;
    r = esgd::make_tensormap_bf16(&p.tmC, g.C, 2, dims, strides, box, nullptr);
    if (r != 0) return 3000 + r;
  } else {
    dims[0] = (uint64_t)g.N; dims[1] = (uint64_t)g.M; box[0] = 32; box[1] = 128;
    strides[0] = (uint64_t)g.ldc * 4;
    r = esgd::make_tensormap_f32(&p.tmC, g.C, 2, dims, strides, box, nullptr);
    if (r != 0) return 3000 + r;
  }
  p.tmR = p.tmC;
  if (ep.residual != nullptr) {
    dims[0] = (uint64_t)g.N; dims[1] = (uint64_t)g.M; box[0] = 64; box[1] = 128;
    strides[0] = (uint64_t)ep.ldr * 2;
    r = esgd::make_tensormap_bf16(&p.tmR, ep.residual, 2, dims, strides, box, nullptr);
    if (r != 0) return 4000 + r;
  }
  p.M = g.M; p.N = g.N; p.K = g.K;
  constexpr int kRows = kPair ? 2 * BM : BM;
  p.m_tiles = (g.M + kRows - 1) / kRows;
  p.n_tiles = (g.N + BN - 1) / BN;
  p.kb_total = (g.K + BK - 1) / BK;
  int splits = g.splits < 1 ? 1 : g.splits;
  if (splits > p.kb_total) splits = p.kb_total;
  p.kb_per_split = (p.kb_total + splits - 1) / splits;
  p.splits = (p.kb_total + p.kb_per_split - 1) / p.kb_per_split;  // no empty split
  if (p.splits > 1 && g.out_mode != OUT_F32_ADD) return -2;
  if constexpr (BN == 64 && !A_MN && !kBn && !kPair) {
    const int tiles = p.m_tiles * p.n_tiles, split = split_ctas((int64_t)p.m_tiles * p.n_tiles, p.kb_total, sm_count());
    if (split > 1 && g.out_mode == OUT_BF16 && ep.col_sum == nullptr && ep.bias_kind == BIAS_F32 && g.N % 8 == 0) {
      p.res_kb = p.fixed_n = 0;
      const SplitOut so{(__nv_bfloat16*)g.C, g.ldc, p.n_tiles, p.kb_total, (p.kb_total + split - 1) / split};
      if (split == 2) return launch_split<2>(gemm_split_kernel<P, 2>, tiles, stream, p, ep, so);
      if (split == 4) return launch_split<4>(gemm_split_kernel<P, 4>, tiles, stream, p, ep, so);
      return launch_split<8>(gemm_split_kernel<P, 8>, tiles, stream, p, ep, so);
    }
  }
  ep.res_bytes = PANEL_BYTES;
  const int sms = kPair ? sm_count() / 2 : sm_count();         // workers: CTAs, or pairs of them
  int grid;
  const int max_kb = kResPanels ? 2 : kBn && ep.residual != nullptr ? Cfg<BN>::MAX_RES_KB2 : Cfg<BN>::MAX_RES_KB;
  const bool resident = !kPair && p.splits == 1 && b_resident<BN>(g, max_kb, sms);
  p.res_kb = resident ? p.kb_total : 0;
  p.fixed_n = (ep.col_sum != nullptr || resident) ? 1 : 0;
  if (p.fixed_n) {
    if (p.splits != 1 || p.n_tiles > sms) return -3;
    const int total = p.m_tiles * p.n_tiles;
    grid = (sms / p.n_tiles) * p.n_tiles;
    if (grid > total) grid = total;
  } else {
    const int total = p.m_tiles * p.n_tiles * p.splits;
    grid = total < sms ? total : sms;
  }
  return esgd::launch<kPair ? 2 : 1>(gemm_kernel<P, kBn>, dim3(kPair ? 2 * grid : grid), NUM_THREADS, Cfg<BN>::SMEM_BYTES, stream, p, ep);
}

// Pairs of CTAs: 256 x 256 tiles that read each operand once for both (32 KB a k-block and CTA instead of 48, five stages
// deep instead of three).
bool pair_applicable(int64_t M, int64_t N, int64_t K, int sms) { return M > BM && N > BM && K > 4 * BK && (N + 255) / 256 <= sms / 2; }

template <int BN>
int launch_major(int a_mn, int b_mn, const GemmArgs& g, const Epilogue& ep, cudaStream_t s) {
  if (!a_mn && !b_mn) return launch<BN, false, false>(g, ep, s);
  if (!a_mn && b_mn) return launch<BN, false, true>(g, ep, s);
  if (a_mn && b_mn) return launch<BN, true, true>(g, ep, s);
  return launch<BN, true, false>(g, ep, s);
}

}  // namespace

extern "C" {

int esgd_sm_count() { return sm_count(); }

// C[M,N] = A * B^T (+bias, ReLU, column statistics).  A is [M][K] (a_mn=0, row stride lda)
// or stored [K][M] (a_mn=1); B is [N][K] (b_mn=0, row stride ldb) or stored [K][N] (b_mn=1).
// out_mode: 0 bf16, 1 fp32, 2 fp32, added to C by TMA reductions (split-K; C zeroed by the caller or an accumulator).
// Requirements: 16-byte aligned bases, lda/ldb/ldc multiples of 8; N need not be.
// relu: bit 0 ReLU, bit 1 the bias is bf16.  scale (optional, with an fp32 bias, both 16-byte aligned): the product's
// columns are multiplied by it before the bias is added.
// col_sum / col_sqsum (bf16 output only) accumulate into caller-zeroed fp32 arrays of N.
// residual (bf16 output only): a bf16 [M][N] tensor with row stride ldr (multiple of 8), added before rounding.
int esgd_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc, int a_mn,
                   int b_mn, int out_mode, const float* scale, const float* bias, int relu, int splits, float* col_sum,
                   float* col_sqsum, const void* residual, int ldr, int* error_flag, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || (lda % 8) || (ldb % 8) || (ldc % 8)) return -1;
  if (ldc < N) return -1;
  if (col_sum != nullptr && out_mode != OUT_BF16) return -4;
  if (residual != nullptr && (out_mode != OUT_BF16 || (ldr % 8) || ((uintptr_t)residual & 15))) return -5;
  if ((uintptr_t)C & 15) return -6;
  if (scale != nullptr && (bias == nullptr || (relu & 2) || (((uintptr_t)scale | (uintptr_t)bias) & 15))) return -7;
  GemmArgs g{A, B, C, M, N, K, lda, ldb, ldc, out_mode, splits};
  Epilogue ep;
  ep.out_mode = out_mode; ep.relu = relu & 1; ep.n_total = N; ep.scale = scale; ep.bias = bias;
  ep.bias_kind = relu & 2 ? BIAS_BF16 : (((uintptr_t)bias & 15) ? BIAS_F32_UNALIGNED : BIAS_F32);
  ep.col_sum = col_sum; ep.col_sqsum = col_sqsum; ep.error_flag = error_flag;
  ep.tx_bytes = 0; ep.tx_bytes_a = 0;
  ep.residual = residual; ep.ldr = ldr;
  cudaStream_t s = (cudaStream_t)stream;
  const int BN = tile_columns(N, (M + BM - 1) / BM * (splits > 1 ? splits : 1), sm_count());
  if (BN == 64) return launch_major<64>(a_mn, b_mn, g, ep, s);
  if (BN == 128) return launch_major<128>(a_mn, b_mn, g, ep, s);
  if (pair_applicable(M, N, K, sm_count())) {
    if (!a_mn && !b_mn) return launch<256, false, false, false, true>(g, ep, s);
    if (!a_mn && b_mn) return launch<256, false, true, false, true>(g, ep, s);
    if (a_mn && b_mn) return launch<256, true, true, false, true>(g, ep, s);
  }
  // Residual panels in buffers of their own, where resident B leaves room for the whole A of a tile beside them: K of 64 and 128
  // (392000 x 256 x 64 83.9 -> 81.7 us, 98000 x 512 x 128 48.6 -> 46.9; 24500 x 1024 x 256 would lose A stages, 30.7 -> 32.2).  A kernel
  // of its own: as a run-time choice it spills registers in the others.
  if (residual != nullptr && !a_mn && !b_mn && splits <= 1 && b_resident<256>(g, 2, sm_count()))
    return launch<256, false, false, false, false, true>(g, ep, s);
  return launch_major<256>(a_mn, b_mn, g, ep, s);
}

// Split-K factor of a weight gradient, [cout][cin] sums over `pixels`, as esgd_gemm_bf16 will launch it: the one with the least work in
// whole rounds of the SMs (or pairs of them) and sums that meet in L2.  Cycles: 250, 300, 600 for a k-block of a tile of 64, 128, 256
// columns, 450 for a pair's; 1000 a tile; 1600 bytes of sums.  One more split than fits a round costs a whole round: with "as many as
// fill the SMs", rounded up, 50176 x 1024 x 256 took 19 splits and 36.3 us, 18 take 27.5; 12544 x 2048 x 512 5 and 32.8, 4 24.4;
// 3136 x 2048 x 512 5 and 16.3, 2 10.4.  Over 45 shapes of 784 to 802816 pixels the choice is within 5 % of the best (0.5 % on average).
int esgd_gemm_wgrad_splits(int64_t pixels, int64_t cout, int64_t cin, int sms) {
  const int64_t blocks = (pixels + BK - 1) / BK, bank = cout * cin * 4, most = blocks < sms ? blocks : sms;
  int64_t best = 0, chosen = 1;
  for (int64_t s = 1; s <= most; ++s) {
    const int64_t per = (blocks + s - 1) / s, splits = (blocks + per - 1) / per;
    if (splits != s) continue;                                  // the same launch as a smaller number
    const int bn = tile_columns((int)cin, (int)((cout + BM - 1) / BM * s), sms);
    const bool pair = bn == 256 && pair_applicable(cout, cin, pixels, sms);
    const int64_t rows = pair ? 2 * BM : BM, workers = pair ? sms / 2 : sms;
    const int64_t rounds = ((cout + rows - 1) / rows * ((cin + bn - 1) / bn) * s + workers - 1) / workers;
    const int64_t cost = rounds * (per * (pair ? 450 : bn == 64 ? 250 : bn == 128 ? 300 : 600) + 1000) + s * bank / 1600;
    if (s > 1 && cost >= best) continue;
    best = cost;
    chosen = s;
  }
  return (int)chosen;
}

// Data gradient of a 1x1 convolution behind a batch norm: dx [M][N] = dy [M][K] * w [K][N] (+ residual), see bn_grad.h.
// -100: not a shape for it.
int esgd_gemm_bn_dgrad(const void* dy, const void* w, void* dx, int M, int N, int K, const void* residual, const esgd_bn_grad* bn,
                       int* error_flag, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || N % 8 || K % 8 || ((uintptr_t)dx & 15) || ((uintptr_t)residual & 15)) return -1;
  GemmArgs g{dy, w, dx, M, N, K, K, N, N, OUT_BF16, 1};
  Epilogue ep;
  ep.out_mode = OUT_BF16; ep.relu = 0; ep.n_total = N; ep.scale = nullptr; ep.bias = nullptr; ep.bias_kind = BIAS_F32;
  ep.col_sum = nullptr; ep.col_sqsum = nullptr; ep.error_flag = error_flag;
  ep.tx_bytes = 0; ep.tx_bytes_a = 0;
  ep.residual = residual; ep.ldr = N;
  if (!set_bn_grad(ep, bn)) return -100;
  cudaStream_t s = (cudaStream_t)stream;
  const int BN = tile_columns(N, (M + BM - 1) / BM, sm_count());
  if (BN == 64) return launch<64, false, true, true>(g, ep, s);
  if (BN == 128) return launch<128, false, true, true>(g, ep, s);
  return launch<256, false, true, true>(g, ep, s);
}

}  // extern "C"
