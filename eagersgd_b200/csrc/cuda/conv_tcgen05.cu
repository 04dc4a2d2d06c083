// Implicit-GEMM convolution (forward and data gradient) for NHWC bf16 on sm_100a.
//
//   y[n, p, q, k] = sum_{r, s, c} x[n, p*stride + r - pad, q*stride + s - pad, c] * w[k, r, s, c]
//
// GEMM view: M = output pixels, N = Cout, K = R*S*Cin.  One k-block is one filter
// tap (r, s) and 64 input channels: the A tile is fetched by ONE 4-D TMA load over
// the NHWC tensor — a box of BW x BH x BI output pixels shifted by the tap, with the
// hardware zero-filling everything outside the image (that is the padding) and
// element strides 2 for strided convolutions — and lands in shared memory already in
// the 128-byte-swizzled K-major layout tcgen05.mma reads.  Weights are used in their
// channels_last storage [Cout][R][S][Cin], which is the K-major B matrix as is.  The
// output tile goes back with a 4-D TMA store (clipped at the image edge) and the
// batch-norm statistics of the stored values are taken in the epilogue.
//
// The data gradient of a stride-1 convolution is the same kernel run on dy with the
// filter rotated by 180 degrees and its channel axes swapped.  The reference gets
// these ops from cuDNN through TensorFlow (official/resnet/resnet_model.py:97-101);
// its CPU restatements are deep500 .../cpp/utility/crosscorrelation.hpp:14-129 and
// conv_op.cpp:291-321.
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>
#include "launch.cuh"
#include "tensormap.cuh"
#include "umma_pipeline.cuh"
#include "umma_split.cuh"

using namespace umma;
using esgd::sm_count;

namespace {

// The filter bank of a problem, read by TMA as stored ([K][R][S][C], channels_last).  Forward: the rows of a k-block's
// B tile are output channels and its 64 columns the input channels of one tap (K-major).  Data gradient
// (kTransposed): rows are the 64 reduced output channels, columns the input channels (MN-major), and the taps of
// the problem are taps (r0 + r * dr, s0 + s * ds) of the stored filter -- rotated by 180 degrees, or the subset that
// meets one output parity of a strided convolution -- so that no rotated copy of the weights is ever made.
// Channel counts that are no multiple of 64 are zero-filled by TMA on both operands.
struct FilterTaps { int r0, dr, s0, ds; };

// A k-block: 64 channels of one tap, taps before channels.
struct TapStep { int r, s, cb; };
__device__ __forceinline__ void next_tap(TapStep& k, int cblks, int S) {
  if (++k.cb < cblks) return;
  k.cb = 0;
  if (++k.s < S) return;
  k.s = 0;
  ++k.r;
}

template <int BN, bool kTransposed>
__device__ __forceinline__ void load_filter_tap(const CUtensorMap* tm, const FilterTaps& f, int r, int s, int cb, int n0,
                                                uint8_t* b, uint64_t* bar) {
  const int rw = f.r0 + r * f.dr, sw = f.s0 + s * f.ds;
  if (kTransposed) {
#pragma unroll
    for (int i = 0; i < BN / 64; ++i) tma_load_4d(b + i * 8192, tm, bar, n0 + 64 * i, sw, rw, cb * 64);
  } else {
    tma_load_4d(b, tm, bar, cb * 64, sw, rw, n0);
  }
}

template <int BN_, bool kT, bool kPair_>
struct ConvProblem {
  static constexpr int BN = BN_;
  static constexpr bool A_MN = false, B_MN = kT, kZeroStages = false, kHalo = false, kPair = kPair_;
  static constexpr int kTwoPanels = 0;
  CUtensorMap tmX, tmW, tmY, tmR;   // tmR: optional residual, same geometry as the output
  int N, Ho, Wo, Cout;
  int R, S, stride, pad;
  FilterTaps taps;
  int cblks;                 // 64-channel blocks of the reduction
  int ksteps, n_mma;         // 16-channel steps of a block that hold anything; columns the MMA computes
  int BW, BH, BI;            // output-pixel box of a tile (BW*BH*BI <= 128)
  int w_tiles, h_tiles, i_tiles, n_tiles;
  int fixed_n;
  int res_kb;                // > 0: the whole filter bank of the CTA's channel range stays in shared memory

  struct Tile { int kb0, kb1, n0, w0, h0, i0; };

  __device__ __forceinline__ bool tile(int it, Tile& t) const {
    // a pair takes two boxes at a time (the last one may be past the last image: loaded as zeros, not stored)
    const int boxes = w_tiles * h_tiles * i_tiles, m_tiles = kPair ? (boxes + 1) / 2 : boxes;
    const int worker = kPair ? blockIdx.x / 2 : blockIdx.x, workers = kPair ? gridDim.x / 2 : gridDim.x;
    int m_idx, n_idx;
    if (fixed_n) {
      n_idx = worker % n_tiles;
      m_idx = worker / n_tiles + it * (workers / n_tiles);
      if (m_idx >= m_tiles) return false;
    } else {
      const int id = worker + it * workers;
      if (id >= m_tiles * n_tiles) return false;
      m_idx = id / n_tiles;
      n_idx = id % n_tiles;
    }
    if (kPair) m_idx = 2 * m_idx + (int)(blockIdx.x & 1);
    place(m_idx, n_idx, t);
    return true;
  }
  __device__ __forceinline__ void place(int m_idx, int n_idx, Tile& t) const {
    t.w0 = (m_idx % w_tiles) * BW;
    t.h0 = ((m_idx / w_tiles) % h_tiles) * BH;
    t.i0 = (m_idx / (w_tiles * h_tiles)) * BI;
    t.n0 = n_idx * BN;
    t.kb0 = 0;
    t.kb1 = R * S * cblks;
  }
  using Step = TapStep;
  __device__ __forceinline__ Step begin(const Tile& t) const {
    if (t.kb0 == 0) return Step{0, 0, 0};
    const int tap = t.kb0 / cblks;
    return Step{tap / S, tap % S, t.kb0 - tap * cblks};
  }
  __device__ __forceinline__ void advance(Step& k) const { next_tap(k, cblks, S); }
  __device__ __forceinline__ void load_a(const Tile& t, const Step& k, uint8_t* a, uint64_t* bar) const {
    tma_load_4d(a, &tmX, bar, k.cb * 64, t.w0 * stride + k.s - pad, t.h0 * stride + k.r - pad, t.i0);
  }
  __device__ __forceinline__ void load_b(const Tile& t, const Step& k, uint8_t* b, uint64_t* bar) const {
    load_filter_tap<BN, kT>(&tmW, taps, k.r, k.s, k.cb, t.n0, b, bar);
  }
  __device__ __forceinline__ void load(const Tile& t, const Step& k, uint8_t* a, uint8_t* b, uint64_t* bar) const {
    load_a(t, k, a, bar);
    load_b(t, k, b, bar);
  }
  // pair: this CTA's box and its half of the output channels' filters
  __device__ __forceinline__ void load(const Tile& t, const Step& k, uint8_t* a, uint8_t* b, uint32_t leader_bar) const {
    const int rw = taps.r0 + k.r * taps.dr, sw = taps.s0 + k.s * taps.ds, n0 = t.n0 + (int)(blockIdx.x & 1) * (BN / 2);
    tma_load_4d_pair(a, &tmX, leader_bar, k.cb * 64, t.w0 * stride + k.s - pad, t.h0 * stride + k.r - pad, t.i0);
    if (kT) {
#pragma unroll
      for (int i = 0; i < BN / 128; ++i) tma_load_4d_pair(b + i * 8192, &tmW, leader_bar, n0 + 64 * i, sw, rw, k.cb * 64);
    } else {
      tma_load_4d_pair(b, &tmW, leader_bar, k.cb * 64, sw, rw, n0);
    }
  }
  __device__ __forceinline__ void store_panel(const Tile& t, int panel, const void* smem) const {
    if (!kPair || t.i0 < N) tma_store_4d(&tmY, smem, t.n0 + panel * 64, t.w0, t.h0, t.i0);
  }
  // A box is part of one row (BH = BI = 1), whole rows of one image (BH divides Ho) or whole images: consecutive pixels.
  __device__ __forceinline__ int valid_prefix(const Tile& t) const {
    if (kPair && t.i0 >= N) return 0;
    return BI > 1 ? min(BI, N - t.i0) * BW * BH : min(BW, Wo - t.w0) * BH;
  }
  __device__ __forceinline__ int64_t first_row(const Tile& t) const { return ((int64_t)t.i0 * Ho + t.h0) * Wo + t.w0; }
  __device__ __forceinline__ void store_f32(const Tile&, int, const void*, bool) const {}
  __device__ __forceinline__ void load_res_panel(const Tile& t, int panel, void* smem, uint64_t* bar) const {
    tma_load_4d(smem, &tmR, bar, t.n0 + panel * 64, t.w0, t.h0, t.i0);
  }
  __device__ __forceinline__ int out_row(int row) const { return row; }
};

// Stride-1 convolution whose taps are shifted views of one input box per 64-channel block (halo mode of the
// pipeline).  A tile is BH full output rows of one image; GEMM row m stands for the pixel (m / PW, m % PW) of
// the box pitch PW = Wo + S - 1, so the S - 1 margin columns of every row (and the rows past BH * PW) compute
// values that are dropped: out_row() gives a GEMM row its place in the dense [BH][Wo] tile that is stored.
template <int BN_, bool kT, bool kPair_>
struct ConvHaloProblem {
  static constexpr int BN = BN_;
  static_assert(!kPair_ || BN_ == 128, "a CTA's half of a pair's filters is one block of 64 channels");
  static constexpr bool A_MN = false, B_MN = kT, kZeroStages = false, kHalo = true, kPair = kPair_;
  static constexpr int kTwoPanels = 0;
  CUtensorMap tmX, tmW, tmY, tmR;   // tmR: optional residual, same geometry as the output
  int N, Ho, Wo, Cout;
  int R, S, pad;
  FilterTaps taps;
  int cblks;                 // 64-channel blocks of the reduction
  int ksteps, n_mma;
  int BH, PW;                // output rows per tile, pixel pitch of the input box
  int h_tiles, n_tiles;
  int res_kb;                // > 0: the filter bank of the CTA's channel range is resident

  struct Tile { int kb0, kb1, n0, h0, i0; };

  __device__ __forceinline__ bool tile(int it, Tile& t) const {
    // a pair takes two boxes at a time (the last one may be past the last image: loaded as zeros, not stored)
    const int boxes = h_tiles * N, worker = kPair ? blockIdx.x / 2 : blockIdx.x, workers = kPair ? gridDim.x / 2 : gridDim.x;
    const int n_idx = worker % n_tiles;
    int m_idx = worker / n_tiles + it * (workers / n_tiles);
    if (m_idx >= (kPair ? (boxes + 1) / 2 : boxes)) return false;
    if (kPair) m_idx = 2 * m_idx + (int)(blockIdx.x & 1);
    t.h0 = (m_idx % h_tiles) * BH;
    t.i0 = m_idx / h_tiles;
    t.n0 = n_idx * BN;
    t.kb0 = 0;
    t.kb1 = R * S * cblks;
    return true;
  }
  __device__ __forceinline__ void load_halo(const Tile& t, int cb, void* smem, uint64_t* bar) const {
    if (kPair) tma_load_4d_pair(smem, &tmX, leader_addr(bar), cb * 64, -pad, t.h0 - pad, t.i0);
    else tma_load_4d(smem, &tmX, bar, cb * 64, -pad, t.h0 - pad, t.i0);
  }
  using Step = TapStep;
  __device__ __forceinline__ Step begin(const Tile&) const { return Step{0, 0, 0}; }
  __device__ __forceinline__ void advance(Step& k) const { next_tap(k, cblks, S); }
  __device__ __forceinline__ void load_b(const Tile& t, const Step& k, uint8_t* b, uint64_t* bar) const {
    if (kPair) {               // this CTA's half of the output channels' filters
      const int rw = taps.r0 + k.r * taps.dr, sw = taps.s0 + k.s * taps.ds, n0 = t.n0 + (int)(blockIdx.x & 1) * (BN / 2);
      if (kT) tma_load_4d_pair(b, &tmW, leader_addr(bar), n0, sw, rw, k.cb * 64);
      else tma_load_4d_pair(b, &tmW, leader_addr(bar), k.cb * 64, sw, rw, n0);
    } else {
      load_filter_tap<BN, kT>(&tmW, taps, k.r, k.s, k.cb, t.n0, b, bar);
    }
  }
  __device__ __forceinline__ void load_a(const Tile&, const Step&, uint8_t*, uint64_t*) const {}
  __device__ __forceinline__ void load(const Tile&, const Step&, uint8_t*, uint8_t*, uint64_t*) const {}
  __device__ __forceinline__ void store_panel(const Tile& t, int panel, const void* smem) const {
    if (!kPair || t.i0 < N) tma_store_4d(&tmY, smem, t.n0 + panel * 64, 0, t.h0, t.i0);
  }
  __device__ __forceinline__ int out_row(int row) const {
    const int hl = row / PW, wl = row - hl * PW;
    return (hl < BH && wl < Wo) ? hl * Wo + wl : -1;
  }
  __device__ __forceinline__ int valid_prefix(const Tile& t) const { return kPair && t.i0 >= N ? 0 : BH * Wo; }
  __device__ __forceinline__ int64_t first_row(const Tile& t) const { return ((int64_t)t.i0 * Ho + t.h0) * Wo; }
  __device__ __forceinline__ void store_f32(const Tile&, int, const void*, bool) const {}
  __device__ __forceinline__ void load_res_panel(const Tile& t, int panel, void* smem, uint64_t* bar) const {
    tma_load_4d(smem, &tmR, bar, t.n0 + panel * 64, 0, t.h0, t.i0);
  }
};


// Weight gradient:  dw[k, r, s, c] = sum over output pixels of dy[pixel, k] * x[pixel shifted by tap (r, s), c].
// GEMM view per tap: M = Cout, N = Cin, K = pixels.  Both operands are "MN-major" (the pixel dimension is the
// row of the NHWC storage): a k-block is a box of up to 64 output pixels, loaded once from dy (two 64-channel
// atoms for the 128 MMA rows) and once from x at the tap's offset (zero-filled outside the image, element
// strides for stride 2).  Boxes smaller than 64 pixels leave the tail rows of the stage at their initial
// zeros.  Work is split over taps, channel tiles and pixel ranges (split-K) and meets in TMA reductions.
template <int BN_>
struct ConvWgradProblem {
  static constexpr int BN = BN_;
  static constexpr bool A_MN = true, B_MN = true, kZeroStages = true, kPair = false;
  static constexpr int kTwoPanels = 0;
  CUtensorMap tmDY, tmX, tmDW;
  int N, Ho, Wo, Cout, Cin;
  int R, S, stride, pad;
  int BW, BH, BI, w_tiles, h_tiles, i_tiles;
  int m_tiles, n_tiles, splits, boxes_total, boxes_per_split;
  static constexpr int res_kb = 0;   // both operands change with every k-block
  static constexpr int ksteps = BK / 16;
  int n_mma;

  struct Tile { int kb0, kb1, n0, m0, tap; };

  __device__ __forceinline__ bool tile(int it, Tile& t) const {
    const int taps = R * S;
    const int per_split = taps * m_tiles * n_tiles;
    const int id = blockIdx.x + it * gridDim.x;
    if (id >= per_split * splits) return false;
    const int split = id / per_split;       // neighbouring CTAs share a pixel range: the boxes are reused out of L2
    int rem = id - split * per_split;
    t.tap = rem % taps; rem /= taps;
    t.n0 = (rem % n_tiles) * BN;
    t.m0 = (rem / n_tiles) * BM;
    t.kb0 = split * boxes_per_split;
    t.kb1 = min(t.kb0 + boxes_per_split, boxes_total);
    return true;
  }
  struct Step { int r, s, w0, h0, i0; };     // the tile's tap; a box of pixels
  __device__ __forceinline__ Step begin(const Tile& t) const {
    const int r = t.tap / S;
    return Step{r, t.tap - r * S, (t.kb0 % w_tiles) * BW, ((t.kb0 / w_tiles) % h_tiles) * BH, (t.kb0 / (w_tiles * h_tiles)) * BI};
  }
  __device__ __forceinline__ void advance(Step& k) const {
    if ((k.w0 += BW) < w_tiles * BW) return;
    k.w0 = 0;
    if ((k.h0 += BH) < h_tiles * BH) return;
    k.h0 = 0;
    k.i0 += BI;
  }
  __device__ __forceinline__ void load(const Tile& t, const Step& k, uint8_t* a, uint8_t* b, uint64_t* bar) const {
    const int r = k.r, s = k.s, w0 = k.w0, h0 = k.h0, i0 = k.i0;
#pragma unroll
    for (int i = 0; i < BM / 64; ++i) tma_load_4d(a + i * 8192, &tmDY, bar, t.m0 + 64 * i, w0, h0, i0);
#pragma unroll
    for (int i = 0; i < BN / 64; ++i)
      tma_load_4d(b + i * 8192, &tmX, bar, t.n0 + 64 * i, w0 * stride + s - pad, h0 * stride + r - pad, i0);
  }
  __device__ __forceinline__ void load_a(const Tile&, const Step&, uint8_t*, uint64_t*) const {}
  __device__ __forceinline__ void load_b(const Tile&, const Step&, uint8_t*, uint64_t*) const {}
  __device__ __forceinline__ void store_panel(const Tile&, int, const void*) const {}
  __device__ __forceinline__ int valid_prefix(const Tile& t) const { return min(BM, Cout - t.m0); }
  __device__ __forceinline__ int64_t first_row(const Tile& t) const { return t.m0; }
  __device__ __forceinline__ void load_res_panel(const Tile&, int, void*, uint64_t*) const {}
  __device__ __forceinline__ int out_row(int row) const { return row; }
  static constexpr bool kHalo = false;
  __device__ __forceinline__ void store_f32(const Tile& t, int col, const void* smem, bool) const {
    tma_reduce_3d(&tmDW, smem, col, t.tap, t.m0);
  }
};

template <class P, bool kBn>
__global__ void __launch_bounds__(NUM_THREADS, 1) conv_kernel(const __grid_constant__ P prob, const Epilogue ep) {
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&prob.tmX);
    tma_prefetch_desc(&prob.tmW);
    tma_prefetch_desc(&prob.tmY);
  }
  run<P, kBn>(prob, ep);
}

template <class P, int S>
__global__ void __launch_bounds__(SPLIT_THREADS, 1) conv_split_kernel(const __grid_constant__ P prob, const Epilogue ep, const SplitOut so) {
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&prob.tmX);
    tma_prefetch_desc(&prob.tmW);
  }
  run_split<P, S>(prob, ep, so);
}

template <class P>
__global__ void __launch_bounds__(NUM_THREADS, 1) conv_wgrad_kernel(const __grid_constant__ P prob, const Epilogue ep) {
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&prob.tmX);
    tma_prefetch_desc(&prob.tmDY);
  }
  run(prob, ep);
}

struct ConvArgs {
  const void *x, *w;
  void* y;
  int N, H, W, Cin, Cout, R, S, stride, pad;
  int out_h = 0, out_w = 0;                 // output extent override (0: from the usual formula)
  int64_t ys_w = 0, ys_h = 0, ys_n = 0;     // output strides in elements (0: dense NHWC)
  FilterTaps taps = {0, 1, 0, 1};           // taps of the stored filter that the problem uses
  int fR = 0, fS = 0;                       // extent of the stored filter
};

// Tensor map over the stored filter bank [K][fR][fS][C]; forward: K = a.Cout, C = a.Cin, data gradient the other way.
template <int BN, bool kT, bool kPair = false>
int filter_map(CUtensorMap* tm, const ConvArgs& a) {
  const int C = kT ? a.Cout : a.Cin, K = kT ? a.Cin : a.Cout;
  uint64_t dims[4] = {(uint64_t)C, (uint64_t)a.fS, (uint64_t)a.fR, (uint64_t)K};
  uint64_t strides[3] = {(uint64_t)C * 2, (uint64_t)a.fS * C * 2, (uint64_t)a.fR * a.fS * C * 2};
  uint32_t box[4] = {64, 1, 1, kT ? 64u : (uint32_t)(kPair ? BN / 2 : BN)};
  return esgd::make_tensormap_bf16(tm, a.w, 4, dims, strides, box, nullptr);
}
inline int ksteps_of(int c) { return c >= 64 ? BK / 16 : (c + 15) / 16; }
// narrow layers: the MMA computes no more columns than there are (the epilogue drops the rest either way)
inline int mma_columns(int n, int bn) { return n >= bn ? bn : (n + 15) / 16 * 16; }

// Boxes of output pixels: whole rows when they fit, as many rows / images as 128 GEMM rows allow.
struct PixelBoxes { int BW, BH, BI, w_tiles, h_tiles, i_tiles; };
inline PixelBoxes pixel_boxes(int N, int Ho, int Wo) {
  PixelBoxes b = {128, 1, 1, 0, 0, 0};
  if (Wo < 128) {
    b.BW = Wo;
    for (int d = 1; d <= 128 / b.BW && d <= Ho; ++d) if (Ho % d == 0) b.BH = d;       // largest divisor of Ho that fits
    if (b.BH == Ho) {
      b.BI = 128 / (b.BW * b.BH);
      if (b.BI > N) b.BI = N;
      if (b.BI < 1) b.BI = 1;
    }
  }
  b.w_tiles = (Wo + b.BW - 1) / b.BW;
  b.h_tiles = (Ho + b.BH - 1) / b.BH;
  b.i_tiles = (N + b.BI - 1) / b.BI;
  return b;
}

// split: CTAs that share the reduction of a tile (64 columns), 1 for the pipeline.
template <int BN, bool kT, bool kBn, bool kPair = false>
int launch(const ConvArgs& a, Epilogue ep, cudaStream_t stream, int split = 1) {
  using P = ConvProblem<BN, kT, kPair>;
  static esgd::SmemAllowed allowed{0};
  if (const int e = esgd::allow_smem(conv_kernel<P, kBn>, Cfg<BN>::SMEM_BYTES, allowed)) return e;
  P p;
  p.N = a.N; p.Cout = a.Cout; p.R = a.R; p.S = a.S; p.stride = a.stride; p.pad = a.pad;
  p.Ho = a.out_h ? a.out_h : (a.H + 2 * a.pad - a.R) / a.stride + 1;
  p.Wo = a.out_w ? a.out_w : (a.W + 2 * a.pad - a.S) / a.stride + 1;
  p.cblks = (a.Cin + 63) / 64;
  p.ksteps = ksteps_of(a.Cin);
  p.n_mma = mma_columns(a.Cout, BN);
  p.taps = a.taps;
  const PixelBoxes b = pixel_boxes(a.N, p.Ho, p.Wo);
  p.BW = b.BW; p.BH = b.BH; p.BI = b.BI; p.w_tiles = b.w_tiles; p.h_tiles = b.h_tiles; p.i_tiles = b.i_tiles;
  p.n_tiles = (a.Cout + BN - 1) / BN;
  {
    // input: dims (C, W, H, N); box in INPUT elements = output box * stride (element strides pick every stride-th)
    uint64_t dims[4] = {(uint64_t)a.Cin, (uint64_t)a.W, (uint64_t)a.H, (uint64_t)a.N};
    uint64_t strides[3] = {(uint64_t)a.Cin * 2, (uint64_t)a.W * a.Cin * 2, (uint64_t)a.H * a.W * a.Cin * 2};
    uint32_t box[4] = {64, (uint32_t)(p.BW * a.stride), (uint32_t)(p.BH * a.stride), (uint32_t)p.BI};
    uint32_t es[4] = {1, (uint32_t)a.stride, (uint32_t)a.stride, 1};
    if (box[1] > 256 || box[2] > 256) return -5;
    int r = esgd::make_tensormap_bf16(&p.tmX, a.x, 4, dims, strides, box, es);
    if (r != 0) return 1000 + r;
  }
  {
    int r = filter_map<BN, kT, kPair>(&p.tmW, a);
    if (r != 0) return 2000 + r;
  }
  {
    uint64_t dims[4] = {(uint64_t)a.Cout, (uint64_t)p.Wo, (uint64_t)p.Ho, (uint64_t)a.N};
    uint64_t strides[3] = {(uint64_t)a.Cout * 2, (uint64_t)p.Wo * a.Cout * 2, (uint64_t)p.Ho * p.Wo * a.Cout * 2};
    if (a.ys_w) { strides[0] = (uint64_t)a.ys_w * 2; strides[1] = (uint64_t)a.ys_h * 2; strides[2] = (uint64_t)a.ys_n * 2; }
    uint32_t box[4] = {64, (uint32_t)p.BW, (uint32_t)p.BH, (uint32_t)p.BI};
    int r = esgd::make_tensormap_bf16(&p.tmY, a.y, 4, dims, strides, box, nullptr);
    if (r == 0 && ep.residual != nullptr) r = esgd::make_tensormap_bf16(&p.tmR, ep.residual, 4, dims, strides, box, nullptr);
    if (r != 0) return 3000 + r;
    ep.res_bytes = (uint32_t)(p.BW * p.BH * p.BI * 128);
  }
  if constexpr (BN == 64 && !kBn && !kPair) {
    if (split > 1) {
      const int tiles = p.w_tiles * p.h_tiles * p.i_tiles * p.n_tiles, blocks = a.R * a.S * p.cblks;
      ep.tx_bytes = (uint32_t)(p.BW * p.BH * p.BI * 128 + Cfg<BN>::B_STAGE_BYTES);
      p.res_kb = p.fixed_n = 0;
      const SplitOut so{(__nv_bfloat16*)a.y, a.Cout, p.n_tiles, blocks, (blocks + split - 1) / split};
      if (split == 2) return launch_split<2>(conv_split_kernel<P, 2>, tiles, stream, p, ep, so);
      if (split == 4) return launch_split<4>(conv_split_kernel<P, 4>, tiles, stream, p, ep, so);
      return launch_split<8>(conv_split_kernel<P, 8>, tiles, stream, p, ep, so);
    }
  }
  const int sms = kPair ? sm_count() / 2 : sm_count();           // workers: CTAs, or pairs of them
  const int boxes = p.w_tiles * p.h_tiles * p.i_tiles, total = (kPair ? (boxes + 1) / 2 : boxes) * p.n_tiles;
  int grid;
  // the filter bank of the CTA's channel range stays in shared memory when it fits beside four input stages
  const int kb_total = a.R * a.S * p.cblks;
  const bool resident = !kPair && resident_enabled() && kb_total <= Cfg<BN>::MAX_RES_KB && p.n_tiles <= sms / 2 &&
                        total / p.n_tiles >= 2 * (sms / p.n_tiles);
  p.res_kb = resident ? kb_total : 0;
  p.fixed_n = (ep.col_sum != nullptr || resident) ? 1 : 0;
  if (p.fixed_n) {
    if (p.n_tiles > sms) return -3;
    grid = (sms / p.n_tiles) * p.n_tiles;
    if (grid > total) grid = total;
  } else {
    grid = total < sms ? total : sms;
  }
  ep.tx_bytes_a = (uint32_t)(p.BW * p.BH * p.BI * 128);
  ep.tx_bytes = ep.tx_bytes_a + (uint32_t)Cfg<BN>::B_STAGE_BYTES;
  return esgd::launch<kPair ? 2 : 1>(conv_kernel<P, kBn>, dim3(kPair ? 2 * grid : grid), NUM_THREADS, Cfg<BN>::SMEM_BYTES, stream, p, ep);
}

// Halo mode applies to stride-1 convolutions with full-width tiles: the box (output rows + filter margin, full
// width + margin, 64 channels) and the rows its most shifted view reaches must fit in one HALO_BYTES slot.
bool halo_applicable(const ConvArgs& a, int Ho, int Wo, int* bh_out) {
  if (a.stride != 1 || a.R * a.S < 2 || a.out_h || a.out_w || a.ys_w) return false;
  const char* e = getenv("ESGD_CONV_HALO");
  if (e != nullptr && e[0] == '0') return false;
  const int PW = Wo + a.S - 1;
  if (PW > 128 || PW != a.W + 2 * a.pad || Ho + a.R - 1 != a.H + 2 * a.pad) return false;
  int bh = 0;
  for (int d = 1; d * PW <= BM && d <= Ho; ++d) if (Ho % d == 0) bh = d;
  if (bh == 0) return false;
  if (bh * Wo < 64) return false;                                   // too few real rows per tile: keep multi-image tiles
  const int view_rows = (a.R - 1) * PW + (a.S - 1) + BM;            // rows the last tap's view may touch
  if (view_rows * 128 > HALO_BYTES || (bh + a.R - 1) * PW * 128 > HALO_BYTES) return false;
  *bh_out = bh;
  return true;
}

// Pairs of CTAs: each holds half of the filters of a k-block, so they cross L2 -> SM and shared memory half as often; a CTA's half is
// one block of 64 channels.  28 x 28 x 128, one CTA and pairs: 11.6 and 11.6 us for 11 images, 12.6 and 11.5 for 22, 21.9 and 18.8 for
// 64, 31.6 and 26.8 for 125, 63.5 and 52.2 for 256.
bool halo_pairs(const ConvArgs& a, int BN) { return BN == 128 && a.Cin % 64 == 0 && a.Cout == 128; }

template <int BN, bool kT, bool kBn, bool kPair = false>
int launch_halo(const ConvArgs& a, Epilogue ep, int bh, cudaStream_t stream) {
  using P = ConvHaloProblem<BN, kT, kPair>;
  static esgd::SmemAllowed allowed{0};
  if (const int e = esgd::allow_smem(conv_kernel<P, kBn>, Cfg<BN>::SMEM_BYTES, allowed)) return e;
  P p;
  p.N = a.N; p.Cout = a.Cout; p.R = a.R; p.S = a.S; p.pad = a.pad;
  p.Ho = a.H + 2 * a.pad - a.R + 1;
  p.Wo = a.W + 2 * a.pad - a.S + 1;
  p.cblks = (a.Cin + 63) / 64;
  p.ksteps = ksteps_of(a.Cin);
  p.n_mma = mma_columns(a.Cout, BN);
  p.taps = a.taps;
  p.BH = bh;
  p.PW = p.Wo + a.S - 1;
  p.h_tiles = p.Ho / bh;
  p.n_tiles = (a.Cout + BN - 1) / BN;
  {
    uint64_t dims[4] = {(uint64_t)a.Cin, (uint64_t)a.W, (uint64_t)a.H, (uint64_t)a.N};
    uint64_t strides[3] = {(uint64_t)a.Cin * 2, (uint64_t)a.W * a.Cin * 2, (uint64_t)a.H * a.W * a.Cin * 2};
    uint32_t box[4] = {64, (uint32_t)p.PW, (uint32_t)(bh + a.R - 1), 1};
    int r = esgd::make_tensormap_bf16(&p.tmX, a.x, 4, dims, strides, box, nullptr);
    if (r != 0) return 1000 + r;
  }
  {
    int r = filter_map<BN, kT, kPair>(&p.tmW, a);
    if (r != 0) return 2000 + r;
  }
  {
    uint64_t dims[4] = {(uint64_t)a.Cout, (uint64_t)p.Wo, (uint64_t)p.Ho, (uint64_t)a.N};
    uint64_t strides[3] = {(uint64_t)a.Cout * 2, (uint64_t)p.Wo * a.Cout * 2, (uint64_t)p.Ho * p.Wo * a.Cout * 2};
    uint32_t box[4] = {64, (uint32_t)p.Wo, (uint32_t)bh, 1};
    int r = esgd::make_tensormap_bf16(&p.tmY, a.y, 4, dims, strides, box, nullptr);
    if (r == 0 && ep.residual != nullptr) r = esgd::make_tensormap_bf16(&p.tmR, ep.residual, 4, dims, strides, box, nullptr);
    if (r != 0) return 3000 + r;
    ep.res_bytes = (uint32_t)(p.Wo * bh * 128);
  }
  const int sms = kPair ? sm_count() / 2 : sm_count();           // workers: CTAs, or pairs of them
  if (p.n_tiles > sms) return -3;
  const int kb_total = a.R * a.S * p.cblks;
  // resident filter bank: beside two input boxes
  p.res_kb = (!kPair && kb_total * Cfg<BN>::B_STAGE_BYTES + 2 * HALO_BYTES <= Cfg<BN>::STAGE_AREA) ? kb_total : 0;
  const int boxes = p.h_tiles * a.N, total = (kPair ? (boxes + 1) / 2 : boxes) * p.n_tiles;
  int grid = (sms / p.n_tiles) * p.n_tiles;
  if (grid > total) grid = total;
  ep.tx_bytes_a = (uint32_t)(p.PW * (bh + a.R - 1) * 128);
  ep.tx_bytes = 0;
  return esgd::launch<kPair ? 2 : 1>(conv_kernel<P, kBn>, dim3(kPair ? 2 * grid : grid), NUM_THREADS, Cfg<BN>::SMEM_BYTES, stream, p, ep);
}

template <int BN>
int launch_wgrad(const ConvArgs& a, const void* dy, float* dw, int* error_flag, cudaStream_t stream) {
  using P = ConvWgradProblem<BN>;
  static esgd::SmemAllowed allowed{0};
  if (const int e = esgd::allow_smem(conv_wgrad_kernel<P>, Cfg<BN>::SMEM_BYTES, allowed)) return e;
  P p;
  p.N = a.N; p.Cout = a.Cout; p.Cin = a.Cin; p.R = a.R; p.S = a.S; p.stride = a.stride; p.pad = a.pad;
  p.Ho = (a.H + 2 * a.pad - a.R) / a.stride + 1;
  p.Wo = (a.W + 2 * a.pad - a.S) / a.stride + 1;
  // pixel box of at most 64 rows (one k-block)
  if (p.Wo >= 64) { p.BW = 64; p.BH = 1; }
  else {
    p.BW = p.Wo;
    p.BH = 1;
    for (int d = 1; d <= 64 / p.BW && d <= p.Ho; ++d) if (p.Ho % d == 0) p.BH = d;
  }
  p.BI = 1;
  p.w_tiles = (p.Wo + p.BW - 1) / p.BW;
  p.h_tiles = (p.Ho + p.BH - 1) / p.BH;
  p.i_tiles = a.N;
  p.boxes_total = p.w_tiles * p.h_tiles * p.i_tiles;
  p.n_mma = mma_columns(a.Cin, BN);
  p.m_tiles = (a.Cout + BM - 1) / BM;
  p.n_tiles = (a.Cin + BN - 1) / BN;
  const int sms = sm_count();
  const int base_tiles = a.R * a.S * p.m_tiles * p.n_tiles;
  // As many splits as one wave of CTAs takes: every split adds a whole filter bank of partial sums, and one more than fits costs a
  // wave (rounded up, in one or two waves by the size of the bank, and this way, stride 2: 256 x 56 x 56 x 128 82 and 68 us, 256 x 28 x
  // 28 x 256 125 and 96, 64 images of these 33 and 25, 256 x 14 x 14 x 512 74 and 59).
  int splits = sms / base_tiles;
  if (splits < 1) splits = 1;
  if (splits > p.boxes_total) splits = p.boxes_total;
  p.boxes_per_split = (p.boxes_total + splits - 1) / splits;
  p.splits = (p.boxes_total + p.boxes_per_split - 1) / p.boxes_per_split;
  {
    uint64_t dims[3] = {(uint64_t)a.Cin, (uint64_t)a.R * a.S, (uint64_t)a.Cout};
    uint64_t strides[2] = {(uint64_t)a.Cin * 4, (uint64_t)a.R * a.S * a.Cin * 4};
    uint32_t box[3] = {32, 1, 128};
    int r = esgd::make_tensormap_f32(&p.tmDW, dw, 3, dims, strides, box, nullptr);
    if (r != 0) return 3000 + r;
  }
  {
    uint64_t dims[4] = {(uint64_t)a.Cout, (uint64_t)p.Wo, (uint64_t)p.Ho, (uint64_t)a.N};
    uint64_t strides[3] = {(uint64_t)a.Cout * 2, (uint64_t)p.Wo * a.Cout * 2, (uint64_t)p.Ho * p.Wo * a.Cout * 2};
    uint32_t box[4] = {64, (uint32_t)p.BW, (uint32_t)p.BH, 1};
    int r = esgd::make_tensormap_bf16(&p.tmDY, dy, 4, dims, strides, box, nullptr);
    if (r != 0) return 1000 + r;
  }
  {
    uint64_t dims[4] = {(uint64_t)a.Cin, (uint64_t)a.W, (uint64_t)a.H, (uint64_t)a.N};
    uint64_t strides[3] = {(uint64_t)a.Cin * 2, (uint64_t)a.W * a.Cin * 2, (uint64_t)a.H * a.W * a.Cin * 2};
    uint32_t box[4] = {64, (uint32_t)(p.BW * a.stride), (uint32_t)(p.BH * a.stride), 1};
    uint32_t es[4] = {1, (uint32_t)a.stride, (uint32_t)a.stride, 1};
    int r = esgd::make_tensormap_bf16(&p.tmX, a.x, 4, dims, strides, box, es);
    if (r != 0) return 2000 + r;
  }
  Epilogue ep;
  ep.out_mode = OUT_F32_ADD; ep.relu = 0; ep.n_total = a.Cin; ep.scale = nullptr; ep.bias = nullptr; ep.bias_kind = BIAS_F32; ep.res_bytes = 0;
  ep.col_sum = nullptr; ep.col_sqsum = nullptr; ep.error_flag = error_flag;
  ep.tx_bytes = (uint32_t)(p.BW * p.BH * 128 * (BM / 64 + BN / 64));
  ep.tx_bytes_a = 0; ep.residual = nullptr; ep.ldr = 0;
  const int total = base_tiles * p.splits;
  const int grid = total < sms ? total : sms;
  return esgd::launch(conv_wgrad_kernel<P>, dim3(grid), NUM_THREADS, Cfg<BN>::SMEM_BYTES, stream, p, ep);
}

Epilogue epilogue_for(int n, int relu, float* col_sum, float* col_sqsum, int* error_flag) {
  Epilogue ep;
  ep.out_mode = OUT_BF16; ep.relu = relu; ep.n_total = n; ep.scale = nullptr; ep.bias = nullptr; ep.bias_kind = BIAS_F32; ep.res_bytes = 0;
  ep.col_sum = col_sum; ep.col_sqsum = col_sqsum; ep.error_flag = error_flag;
  ep.tx_bytes = 0; ep.tx_bytes_a = 0; ep.residual = nullptr; ep.ldr = n;
  return ep;
}

// Columns of a tile (shared with the plan query below).
int tile_width(const ConvArgs& a, int Ho, int Wo) {
  return tile_columns(a.Cout, (int)(((int64_t)a.N * Ho * Wo + BM - 1) / BM), sm_count());
}

// Tiles of 64 columns that launch() will make of the output.
int64_t conv_tiles(const ConvArgs& a, int Ho, int Wo) {
  const PixelBoxes b = pixel_boxes(a.N, Ho, Wo);
  return (int64_t)b.w_tiles * b.h_tiles * b.i_tiles * ((a.Cout + 63) / 64);
}

template <bool kT, bool kBn = false>
int dispatch(const ConvArgs& a, const Epilogue& ep, cudaStream_t s) {
  const int Ho = a.out_h ? a.out_h : (a.H + 2 * a.pad - a.R) / a.stride + 1, Wo = a.out_w ? a.out_w : (a.W + 2 * a.pad - a.S) / a.stride + 1;
  const int BN = tile_width(a, Ho, Wo);
  if (!kBn && BN == 64 && ep.col_sum == nullptr && !a.ys_w && a.Cin % 64 == 0) {
    const int split = split_ctas(conv_tiles(a, Ho, Wo), a.R * a.S * (a.Cin / 64), sm_count());
    if (split > 1) return launch<64, kT, false>(a, ep, s, split);
  }
  int bh = 0;
  if (a.Cout <= 128 && halo_applicable(a, (a.H + 2 * a.pad - a.R) / a.stride + 1, (a.W + 2 * a.pad - a.S) / a.stride + 1, &bh))
    return BN == 64                   ? launch_halo<64, kT, kBn>(a, ep, bh, s)
           : halo_pairs(a, BN)        ? launch_halo<128, kT, kBn, true>(a, ep, bh, s)
                                      : launch_halo<128, kT, kBn>(a, ep, bh, s);
  if (BN == 64) return launch<64, kT, kBn>(a, ep, s);
  if (BN == 128) return launch<128, kT, kBn>(a, ep, s);
  // Pairs of CTAs (256-column tiles read each operand once for two boxes of pixels) where the reduction is full blocks:
  // 256 channels at 14 x 14 and 512 at 7 x 7, batch 256: 79 -> 65 us
  if (a.Cin % 64 == 0 && a.Cout >= 256 && a.R * a.S * (a.Cin / 64) > 4 && a.Cout <= sm_count() / 2 * 256)
    return launch<256, kT, kBn, true>(a, ep, s);
  return launch<256, kT, kBn>(a, ep, s);
}

}  // namespace

extern "C" {

// dw: fp32 [Cout][R][S][Cin], zeroed by the caller (split-K partial sums are added by TMA reductions).
// x: [N,H,W,Cin] bf16, dy: [N,Ho,Wo,Cout] bf16.  Cin % 8 == 0, Cout % 8 == 0.
int esgd_conv2d_wgrad(const void* x, const void* dy, float* dw, int N, int H, int W, int Cin, int Cout, int R, int S,
                      int stride, int pad, int* error_flag, void* stream) {
  if (Cin % 8 || Cout % 8 || stride < 1 || stride > 2) return -1;
  ConvArgs a{x, nullptr, nullptr, N, H, W, Cin, Cout, R, S, stride, pad};
  cudaStream_t s = (cudaStream_t)stream;
  const int BN = Cin <= 64 ? 64 : (Cin <= 128 ? 128 : 256);
  if (BN == 64) return launch_wgrad<64>(a, dy, dw, error_flag, s);
  if (BN == 128) return launch_wgrad<128>(a, dy, dw, error_flag, s);
  return launch_wgrad<256>(a, dy, dw, error_flag, s);
}

// x: [N,H,W,Cin] bf16, w: [Cout,R,S,Cin] bf16, y: [N,Ho,Wo,Cout] bf16.  Cin % 8 == 0, Cout % 8 == 0.
// y = act(scale * conv + bias + residual), each part optional (scale needs a bias; all 16-byte aligned; residual like y).
// col_sum / col_sqsum (optional, caller-zeroed fp32[Cout]) receive the statistics of the stored y.
int esgd_conv2d_fwd(const void* x, const void* w, void* y, int N, int H, int W, int Cin, int Cout, int R, int S,
                    int stride, int pad, const float* scale, const float* bias, const void* residual, int relu, float* col_sum,
                    float* col_sqsum, int* error_flag, void* stream) {
  if (Cin % 8 || Cout % 8 || stride < 1 || stride > 2) return -1;
  if ((scale != nullptr && bias == nullptr) || (((uintptr_t)scale | (uintptr_t)bias | (uintptr_t)residual) & 15)) return -7;
  ConvArgs a{x, w, y, N, H, W, Cin, Cout, R, S, stride, pad};
  a.fR = R; a.fS = S;
  Epilogue ep = epilogue_for(Cout, relu, col_sum, col_sqsum, error_flag);
  ep.scale = scale; ep.bias = bias; ep.residual = residual;
  return dispatch<false>(a, ep, (cudaStream_t)stream);
}

// Data gradient on the weights as stored: dy [N,Ho,Wo,Cout], w [Cout,R,S,Cin], dx [N,H,W,Cin] (dense NHWC); residual
// (optional, stride 1, like dx) is added before the rounding.  bn (optional, stride 1): see bn_grad.h; -100 for channels it
// does not take.
// Stride 1: one launch, any R x S with padding up to min(R, S) - 1.  Stride 2: 3x3 filters with padding 1 on even H and W;
// each output parity (h % 2, w % 2) meets 1, 2, 2 or 4 of the nine taps and is a dense stride-1 problem written
// into its interleaved pixels of dx (dx[2i + p] uses the filter rows r with (p + 1 - r) even).
int esgd_conv2d_dgrad(const void* dy, const void* w, void* dx, int N, int H, int W, int Cin, int Cout, int R, int S,
                      int stride, int pad, const void* residual, const esgd_bn_grad* bn, int* error_flag, void* stream) {
  if (Cin % 8 || Cout % 8 || ((uintptr_t)residual & 15)) return -1;
  if ((residual != nullptr || bn != nullptr) && stride != 1) return -2;
  Epilogue ep = epilogue_for(Cin, 0, nullptr, nullptr, error_flag);
  ep.residual = residual;
  if (!set_bn_grad(ep, bn)) return -100;
  cudaStream_t s = (cudaStream_t)stream;
  if (stride == 1) {
    if (pad > R - 1 || pad > S - 1 || R != S) return -1;
    ConvArgs a{dy, w, dx, N, H + 2 * pad - R + 1, W + 2 * pad - S + 1, Cout, Cin, R, S, 1, R - 1 - pad};
    a.fR = R; a.fS = S;
    a.taps = FilterTaps{R - 1, -1, S - 1, -1};
    return bn != nullptr ? dispatch<true, true>(a, ep, s) : dispatch<true>(a, ep, s);
  }
  if (stride != 2 || R != 3 || S != 3 || pad != 1 || H % 2 || W % 2) return -1;
  for (int ph = 0; ph < 2; ++ph)
    for (int pw = 0; pw < 2; ++pw) {
      ConvArgs a{dy, w, (char*)dx + ((int64_t)ph * W + pw) * Cin * 2, N, H / 2, W / 2, Cout, Cin, 1 + ph, 1 + pw, 1, 0};
      a.out_h = H / 2; a.out_w = W / 2;
      a.ys_w = 2 * (int64_t)Cin; a.ys_h = 2 * (int64_t)W * Cin; a.ys_n = (int64_t)H * W * Cin;
      a.fR = a.fS = 3;
      a.taps = FilterTaps{ph ? 2 : 1, -2, pw ? 2 : 1, -2};
      int rc = dispatch<true>(a, ep, s);
      if (rc != 0) return rc;
    }
  return 0;
}

// Host arithmetic of the halo-mode forward / data-gradient launch, without launching (no device needed).
// out[0..10]: applicable (0/1), BH, PW, BN, resident filter k-blocks (0: streamed), input-box slots, filter stages,
// bytes of one input box, bytes the most shifted view reaches, stage area used, stage area there is.
void esgd_conv2d_halo_plan(int N, int H, int W, int Cin, int Cout, int R, int S, int stride, int pad, int* out) {
  for (int i = 0; i < 11; ++i) out[i] = 0;
  if (Cin % 8 || Cout % 8) return;
  ConvArgs a{nullptr, nullptr, nullptr, N, H, W, Cin, Cout, R, S, stride, pad};
  const int BN = stride == 1 ? tile_width(a, H + 2 * pad - R + 1, W + 2 * pad - S + 1) : 0;
  int bh = 0;
  if (Cout > 128 || stride != 1 || !halo_applicable(a, H + 2 * pad - R + 1, W + 2 * pad - S + 1, &bh)) return;
  const int PW = W + 2 * pad;
  const bool pairs = halo_pairs(a, BN);
  const int b_stage = pairs ? BN * 64 : BN * 128, stage_area = BN == 64 ? Cfg<64>::STAGE_AREA : Cfg<128>::STAGE_AREA;
  const int kb_total = R * S * ((Cin + 63) / 64);
  const int res_kb = (!pairs && kb_total * b_stage + 2 * HALO_BYTES <= stage_area) ? kb_total : 0;
  const int nhalo = res_kb > 0 ? 2 : MAX_HALOS;
  int nstages = 1;
  if (res_kb == 0) {
    nstages = (stage_area - nhalo * HALO_BYTES) / b_stage;
    if (nstages > 8) nstages = 8;
  }
  out[0] = 1; out[1] = bh; out[2] = PW; out[3] = BN; out[4] = res_kb; out[5] = nhalo; out[6] = nstages;
  out[7] = PW * (bh + R - 1) * 128;
  out[8] = ((R - 1) * PW + (S - 1) + BM) * 128;
  out[9] = nhalo * HALO_BYTES + (res_kb > 0 ? res_kb : nstages) * b_stage;
  out[10] = stage_area;
}

}  // extern "C"
