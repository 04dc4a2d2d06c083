// Softmax cross-entropy (forward + backward in one pass), 3x3/2 max pooling and
// global average pooling for NHWC bf16 activations.
//
// Reference semantics: sparse softmax cross-entropy averaged over the batch
// (official/resnet/resnet_run_loop_solo_imagenet_300.py:321-322; CPU restatements
// deep500 .../cpp/operators/softmax_op.cpp:53-96, python/softmax_crossentropy_op.py:11-49),
// max_pooling2d 3x3 stride 2 'SAME' and reduce_mean over H,W (resnet_model.py:521-549;
// maxpool_op.cpp, globalaveragepool_op.cpp).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>
#include "launch.cuh"

namespace {

using esgd::pdl_enter;

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16(v); }

__device__ __forceinline__ float block_reduce(float v, bool is_max, float* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    float other = __shfl_xor_sync(0xffffffffu, v, o);
    v = is_max ? fmaxf(v, other) : v + other;
  }
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  float r = sh[0];
  for (int w = 1; w < nw; ++w) r = is_max ? fmaxf(r, sh[w]) : r + sh[w];
  __syncthreads();
  return r;
}

// One block per sample.  loss_sum accumulates sum_i loss_i * inv_batch; dlogits = (softmax - onehot) * grad_scale.
// A label outside [0, classes) is never used as an index: that sample gets zero loss and a zero gradient row.
template <typename T>
__global__ void __launch_bounds__(256) softmax_ce_kernel(const T* __restrict__ logits, const int64_t* __restrict__ labels,
                                                         int classes, int ld, float inv_batch, float grad_scale,
                                                         float* __restrict__ loss_sum, float* __restrict__ per_sample,
                                                         T* __restrict__ dlogits) {
  pdl_enter();
  __shared__ float sh[8];
  const int row = blockIdx.x;
  const T* x = logits + (size_t)row * ld;
  float mx = -FLT_MAX;
  for (int c = threadIdx.x; c < classes; c += blockDim.x) mx = fmaxf(mx, to_f(x[c]));
  mx = block_reduce(mx, true, sh);
  float se = 0.0f;
  for (int c = threadIdx.x; c < classes; c += blockDim.x) se += __expf(to_f(x[c]) - mx);
  se = block_reduce(se, false, sh);
  const int64_t raw_label = labels[row];
  const bool valid = raw_label >= 0 && raw_label < (int64_t)classes;
  const int label = valid ? (int)raw_label : 0;
  const float lse = mx + __logf(se);
  if (threadIdx.x == 0) {
    float li = valid ? lse - to_f(x[label]) : 0.0f;
    if (per_sample != nullptr) per_sample[row] = li;
    atomicAdd(loss_sum, li * inv_batch);
  }
  if (dlogits != nullptr) {
    T* d = dlogits + (size_t)row * ld;
    const float inv_se = 1.0f / se;
    for (int c = threadIdx.x; c < classes; c += blockDim.x) {
      float p = __expf(to_f(x[c]) - mx) * inv_se;
      d[c] = from_f<T>(valid ? (p - (c == label ? 1.0f : 0.0f)) * grad_scale : 0.0f);
    }
  }
}

// ---- max pool 3x3 stride 2 pad 1, NHWC, vectors of 8 channels -----------------
__device__ __forceinline__ void ld8(const __nv_bfloat16* p, float v[8]) {
  uint4 raw = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float2 f = __bfloat1622float2(h[q]);
    v[2 * q] = f.x;
    v[2 * q + 1] = f.y;
  }
}
__device__ __forceinline__ void st8(__nv_bfloat16* p, const float v[8]) {
  uint4 raw;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
  for (int q = 0; q < 4; ++q) h[q] = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
  *reinterpret_cast<uint4*>(p) = raw;
}

// One output row of an image per block (the only divisions left are by the row's own extent).  Bound by instructions as long
// as every element was converted, compared and selected in fp32: 256 x 112 x 112 x 64, 224 -> 135 us (219 -> 111 without idx).
__global__ void __launch_bounds__(256) maxpool_fwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                          __nv_bfloat16* __restrict__ y, uint8_t* __restrict__ idx,
                                                          int N, int H, int W, int C, int OH, int OW) {
  pdl_enter();
  const int G = C / 8;
  for (int row = blockIdx.x; row < N * OH; row += gridDim.x) {
    const int n = row / OH, oh = row - n * OH;
    const int64_t out0 = (int64_t)row * OW * G;
    for (int i = threadIdx.x; i < OW * G; i += blockDim.x) {
      const int ow = i / G, g = i - ow * G;
      uint4 raw[9];
#pragma unroll
      for (int t = 0; t < 9; ++t) {                 // every load before the first use
        const int h = oh * 2 - 1 + t / 3, w = ow * 2 - 1 + t % 3;
        if (h >= 0 && h < H && w >= 0 && w < W)
          raw[t] = __ldg(reinterpret_cast<const uint4*>(x + (((int64_t)n * H + h) * W + w) * C + g * 8));
      }
      // Two channels per instruction, in bf16 (a maximum is exact): the largest first, then the first tap that equals it.
      __align__(16) __nv_bfloat162 m[4];
      uint32_t first[4] = {0, 0, 0, 0};
#pragma unroll
      for (int q = 0; q < 4; ++q) m[q] = __floats2bfloat162_rn(-INFINITY, -INFINITY);
#pragma unroll
      for (int t = 0; t < 9; ++t) {
        const int h = oh * 2 - 1 + t / 3, w = ow * 2 - 1 + t % 3;
        if (h < 0 || h >= H || w < 0 || w >= W) continue;
        const __nv_bfloat162* hv = reinterpret_cast<const __nv_bfloat162*>(&raw[t]);
#pragma unroll
        for (int q = 0; q < 4; ++q) m[q] = __hmax2(m[q], hv[q]);
      }
      *reinterpret_cast<uint4*>(y + (out0 + i) * 8) = *reinterpret_cast<const uint4*>(m);
      if (idx == nullptr) continue;
#pragma unroll
      for (int t = 8; t >= 0; --t) {
        const int h = oh * 2 - 1 + t / 3, w = ow * 2 - 1 + t % 3;
        if (h < 0 || h >= H || w < 0 || w >= W) continue;
        const __nv_bfloat162* hv = reinterpret_cast<const __nv_bfloat162*>(&raw[t]);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t same = __heq2_mask(hv[q], m[q]);
          first[q] = (first[q] & ~same) | (same & (uint32_t)(t * 0x00010001));
        }
      }
      // a byte per channel out of each half
      *reinterpret_cast<uint2*>(idx + (out0 + i) * 8) = make_uint2(__byte_perm(first[0], first[1], 0x6420), __byte_perm(first[2], first[3], 0x6420));
    }
  }
}

// Gather form: an input pixel receives dy of every window whose recorded arg-max it is.  A thread makes the 2 x 2 pixels
// (2k, 2j) .. (2k+1, 2j+1), which meet the windows (k, j) .. (k+1, j+1) and no others: four windows are read for four
// pixels, where a thread per pixel read nine.
__global__ void __launch_bounds__(256) maxpool_bwd_kernel(const uint8_t* __restrict__ idx,
                                                          const __nv_bfloat16* __restrict__ dy,
                                                          __nv_bfloat16* __restrict__ dx, int N, int H, int W, int C,
                                                          int OH, int OW) {
  pdl_enter();
  const int G = C / 8, HP = (H + 1) / 2, WP = (W + 1) / 2;
  for (int row = blockIdx.x; row < N * HP; row += gridDim.x) {
    const int n = row / HP, k = row - n * HP;
    for (int i = threadIdx.x; i < WP * G; i += blockDim.x) {
      const int j = i / G, g = i - j * G;
      uint2 pk[4];
      uint4 dv[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const int oh = k + (a >> 1), ow = j + (a & 1);
        pk[a] = make_uint2(0xffffffffu, 0xffffffffu);          // no position: a window outside the output
        dv[a] = make_uint4(0, 0, 0, 0);
        if (oh < OH && ow < OW) {
          const int64_t o = (((int64_t)n * OH + oh) * OW + ow) * C + g * 8;
          pk[a] = __ldg(reinterpret_cast<const uint2*>(idx + o));
          dv[a] = __ldg(reinterpret_cast<const uint4*>(dy + o));
        }
      }
      float acc[4][8];
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[p][q] = 0.0f;
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const __nv_bfloat162* hv = reinterpret_cast<const __nv_bfloat162*>(&dv[a]);
        float d[8];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float2 f = __bfloat1622float2(hv[q]);
          d[2 * q] = f.x; d[2 * q + 1] = f.y;
        }
#pragma unroll
        for (int p = 0; p < 4; ++p) {                          // pixel (2k + p/2, 2j + p%2) inside window (k + a/2, j + a%2)
          const int r = 1 + (p >> 1) - 2 * (a >> 1), c = 1 + (p & 1) - 2 * (a & 1);
          if (r < 0 || c < 0) continue;                        // (compile time)
          const uint32_t pos = (uint32_t)(r * 3 + c);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const uint32_t word = q < 4 ? pk[a].x : pk[a].y;
            if (((word >> ((q & 3) * 8)) & 0xffu) == pos) acc[p][q] += d[q];
          }
        }
      }
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const int h = 2 * k + (p >> 1), w = 2 * j + (p & 1);
        if (h < H && w < W) st8(dx + (((int64_t)n * H + h) * W + w) * C + g * 8, acc[p]);
      }
    }
  }
}

// ---- 2x spatial subsampling (the gather in front of a strided 1x1 convolution) ---------
__global__ void __launch_bounds__(256) subsample2_fwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                             __nv_bfloat16* __restrict__ y, int N, int H, int W,
                                                             int C, int OH, int OW) {
  pdl_enter();
  const int G = C / 8;
  const int64_t total = (int64_t)N * OH * OW * G;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int g = (int)(i % G);
    int64_t t = i / G;
    const int ow = (int)(t % OW); t /= OW;
    const int oh = (int)(t % OH);
    const int n = (int)(t / OH);
    *reinterpret_cast<uint4*>(y + i * 8) =
        *reinterpret_cast<const uint4*>(x + (((int64_t)n * H + oh * 2) * W + ow * 2) * C + g * 8);
  }
}
__global__ void __launch_bounds__(256) subsample2_bwd_kernel(const __nv_bfloat16* __restrict__ dy,
                                                             __nv_bfloat16* __restrict__ dx, int N, int H, int W,
                                                             int C, int OH, int OW) {
  pdl_enter();
  const int G = C / 8;
  const int64_t total = (int64_t)N * H * W * G;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int g = (int)(i % G);
    int64_t t = i / G;
    const int w = (int)(t % W); t /= W;
    const int h = (int)(t % H);
    const int n = (int)(t / H);
    uint4 v = make_uint4(0, 0, 0, 0);
    if (!(h & 1) && !(w & 1))
      v = *reinterpret_cast<const uint4*>(dy + (((int64_t)n * OH + h / 2) * OW + w / 2) * C + g * 8);
    *reinterpret_cast<uint4*>(dx + i * 8) = v;
  }
}

// ---- global average pool: [N, HW, C] -> [N, C] -----------------------------------
// A block covers up to 16 channel groups of one image with 16 or more pixels at a time.
__global__ void __launch_bounds__(256) avgpool_fwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                          __nv_bfloat16* __restrict__ y, int N, int HW, int C, int cg) {
  pdl_enter();
  __shared__ float part[256 * 9];
  const int G = C / 8, n = blockIdx.x, gl = threadIdx.x % cg, rl = threadIdx.x / cg, rows = 256 / cg;
  const int g = blockIdx.y * cg + gl;
  float a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (g < G) {
    for (int p = rl; p < HW; p += rows) {
      float v[8];
      ld8(x + ((int64_t)n * HW + p) * C + g * 8, v);
#pragma unroll
      for (int q = 0; q < 8; ++q) a[q] += v[q];
    }
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) part[threadIdx.x * 9 + q] = a[q];
  __syncthreads();
  if (rl == 0 && g < G) {
    const float inv = 1.0f / (float)HW;
    for (int r = 1; r < rows; ++r)
#pragma unroll
      for (int q = 0; q < 8; ++q) a[q] += part[(r * cg + gl) * 9 + q];
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q] *= inv;
    st8(y + ((int64_t)n * G + g) * 8, a);
  }
}

__global__ void __launch_bounds__(256) avgpool_bwd_kernel(const __nv_bfloat16* __restrict__ dy,
                                                          __nv_bfloat16* __restrict__ dx, int N, int HW, int C) {
  pdl_enter();
  const int G = C / 8;
  const int64_t total = (int64_t)N * HW * G;
  const float inv = 1.0f / (float)HW;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int g = (int)(i % G);
    const int n = (int)(i / ((int64_t)HW * G));
    float v[8];
    ld8(dy + ((int64_t)n * G + g) * 8, v);
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] *= inv;
    st8(dx + i * 8, v);
  }
}

// im2col for convolutions with very few input channels (the 7x7 / 2 stem on RGB images): the sizes that stem_tcgen05.cu
// does not take (other filters, other widths).
// Column layout per output pixel: R segments of SEG = roundup8(S*C) elements; segment r holds the
// S*C input values of filter row r — in NHWC they are contiguous in memory — followed by zeros, and the
// row is zero-padded to Kpad (a multiple of 64, so the product runs as a tensor-core GEMM).
// One thread per (pixel, segment): no divisions per element, 16-byte stores.
template <int MAXSEG>
__global__ void __launch_bounds__(256) im2col_small_c_kernel(const __nv_bfloat16* __restrict__ x,
                                                             __nv_bfloat16* __restrict__ col, int N, int H, int W,
                                                             int C, int R, int S, int stride, int pad, int Ho, int Wo,
                                                             int seg, int Kpad) {
  pdl_enter();
  const int segs = Kpad / seg;              // R real segments + zero segments
  const int64_t total = (int64_t)N * Ho * Wo * segs;
  const int sc = S * C;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(i % segs);
    int64_t t = i / segs;
    const int q = (int)(t % Wo); t /= Wo;
    const int p = (int)(t % Ho);
    const int n = (int)(t / Ho);
    __align__(16) __nv_bfloat16 v[MAXSEG];
#pragma unroll
    for (int j = 0; j < MAXSEG; ++j) v[j] = __float2bfloat16(0.0f);
    const int h = p * stride + r - pad;
    if (r < R && h >= 0 && h < H) {
      const int w0 = q * stride - pad;
      const __nv_bfloat16* src = x + (((int64_t)n * H + h) * W + w0) * C;
      const int lo = w0 < 0 ? -w0 * C : 0;                       // first valid element of the segment
      const int hi = (w0 + S > W) ? (W - w0) * C : sc;           // one past the last valid element
#pragma unroll
      for (int j = 0; j < MAXSEG; ++j)
        if (j >= lo && j < hi) v[j] = src[j];
    }
    __nv_bfloat16* dst = col + (t * 0 + (((int64_t)n * Ho + p) * Wo + q)) * Kpad + (int64_t)r * seg;
    for (int j = 0; j < seg; j += 8) *reinterpret_cast<uint4*>(dst + j) = *reinterpret_cast<const uint4*>(v + j);
  }
}

// The same columns, one output row of the image per block: the R input rows that the row's windows touch are
// staged in shared memory with 16-byte loads between zero guards (the horizontal padding), and every thread
// assembles 16-byte chunks of the column matrix from them with funnel shifts (a window starts on an even byte,
// not on a word).  Elements of a segment beyond S*C carry the neighbouring pixels instead of zeros; they meet
// zero weights.  Writes are the only large traffic (N*Ho*Wo*Kpad*2 bytes) and they are fully coalesced.
constexpr int kImLeftGuard = 32, kImRightGuard = 64;
__global__ void __launch_bounds__(256) im2col_rows_kernel(const __nv_bfloat16* __restrict__ x,
                                                          __nv_bfloat16* __restrict__ col, int N, int H, int W, int C,
                                                          int R, int S, int stride, int pad, int Ho, int Wo, int seg,
                                                          int Kpad) {
  pdl_enter();
  extern __shared__ __align__(16) uint8_t im_rows[];
  const int rowbytes = W * C * 2;
  const int pitch = kImLeftGuard + rowbytes + kImRightGuard;
  const int n = blockIdx.x / Ho, p = blockIdx.x % Ho;
  for (int r = 0; r < R; ++r) {
    const int h = p * stride + r - pad;
    const uint8_t* src = reinterpret_cast<const uint8_t*>(x) + ((int64_t)n * H + h) * rowbytes;
    for (int i = threadIdx.x; i < pitch / 16; i += blockDim.x) {
      const int byte = i * 16 - kImLeftGuard;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (h >= 0 && h < H && byte >= 0 && byte < rowbytes) v = __ldg(reinterpret_cast<const uint4*>(src + byte));
      *reinterpret_cast<uint4*>(im_rows + r * pitch + i * 16) = v;
    }
  }
  __syncthreads();
  const int chunks_per_seg = seg / 8, chunks_per_pixel = Kpad / 8;
  __nv_bfloat16* dst_row = col + ((int64_t)n * Ho + p) * Wo * Kpad;
  for (int ci = threadIdx.x; ci < Wo * chunks_per_pixel; ci += blockDim.x) {
    const int q = ci / chunks_per_pixel, k8 = ci - q * chunks_per_pixel;
    const int r = k8 / chunks_per_seg, c = k8 - r * chunks_per_seg;
    uint4 out = make_uint4(0, 0, 0, 0);
    if (r < R) {
      const int off = kImLeftGuard + ((q * stride - pad) * C + 8 * c) * 2;
      const uint32_t* wp = reinterpret_cast<const uint32_t*>(im_rows + r * pitch + (off & ~3));
      const int sh = (off & 3) * 8;
      const uint32_t w0 = wp[0], w1 = wp[1], w2 = wp[2], w3 = wp[3], w4 = wp[4];
      out.x = __funnelshift_r(w0, w1, sh);
      out.y = __funnelshift_r(w1, w2, sh);
      out.z = __funnelshift_r(w2, w3, sh);
      out.w = __funnelshift_r(w3, w4, sh);
    }
    *reinterpret_cast<uint4*>(dst_row + (int64_t)ci * 8) = out;
  }
}

// Stem filters [Cout][R][S][C] -> the column layout above ([Cout][Kpad], segments of `seg`, zeros elsewhere).
__global__ void __launch_bounds__(256) stem_pack_kernel(const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ out,
                                                        int Cout, int R, int sc, int seg, int Kpad) {
  pdl_enter();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= Cout * Kpad) return;
  const int co = i / Kpad, k = i - co * Kpad, r = k / seg, j = k - r * seg;
  out[i] = r < R && j < sc ? w[(co * R + r) * sc + j] : __float2bfloat16(0.0f);
}
// The way back for the filter gradient: fp32 columns -> bf16 filters (dw) or added to an fp32 accumulator (acc).
__global__ void __launch_bounds__(256) stem_unpack_kernel(const float* __restrict__ col, __nv_bfloat16* dw, float* acc, int Cout,
                                                          int R, int sc, int seg, int Kpad) {
  pdl_enter();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= Cout * R * sc) return;
  const int co = i / (R * sc), k = i - co * R * sc, r = k / sc, j = k - r * sc;
  const float v = col[(int64_t)co * Kpad + r * seg + j];
  if (acc != nullptr) acc[i] += v;
  else dw[i] = __float2bfloat16(v);
}

// Gradient of a dense layer's fp32 output: bf16 copy with the row padded to np columns (zeros), and its column sums in the
// same pass (dy is read once).  A thread keeps four columns and walks down the rows of its block; a grid has 65,535 blocks
// of rows, and beyond a million rows they go round.
constexpr int kCastRows = 16;      // rows of a block: short enough that a small batch is not one serial chain of loads
__global__ void __launch_bounds__(256) cast_colsum_kernel(const float* __restrict__ dy, int64_t ld, int M, int N, int np,
                                                          __nv_bfloat16* __restrict__ out, float* __restrict__ colsum, int vec) {
  pdl_enter();
  const int c = (blockIdx.x * 256 + threadIdx.x) * 4;
  if (c >= np) return;
  float s[4] = {0, 0, 0, 0};
  for (int64_t r0 = (int64_t)blockIdx.y * kCastRows; r0 < M; r0 += (int64_t)gridDim.y * kCastRows) {
    const int r1 = (int)min((int64_t)M, r0 + kCastRows);
#pragma unroll 8
    for (int r = (int)r0; r < r1; ++r) {
      float v[4];
      if (vec && c + 4 <= N) {
        const float4 f = __ldcs(reinterpret_cast<const float4*>(dy + r * ld + c));
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = c + q < N ? dy[r * ld + c + q] : 0.0f;
      }
      __nv_bfloat162 h[2] = {__floats2bfloat162_rn(v[0], v[1]), __floats2bfloat162_rn(v[2], v[3])};
      *reinterpret_cast<uint2*>(out + (int64_t)r * np + c) = *reinterpret_cast<const uint2*>(h);
#pragma unroll
      for (int q = 0; q < 4; ++q) s[q] += v[q];
    }
  }
  if (colsum != nullptr) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (c + q < N) atomicAdd(colsum + c + q, s[q]);
  }
}

int grid_for(int64_t items) {
  int64_t b = (items + 255) / 256;
  const int64_t cap = (int64_t)esgd::sm_count() * 16;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace

extern "C" {

// loss_sum (one float) must be zeroed by the caller.
int esgd_softmax_ce(const void* logits, int is_bf16, const int64_t* labels, int batch, int classes, int ld,
                    float grad_scale, float* loss_sum, float* per_sample, void* dlogits, void* stream) {
  if (is_bf16)
    return esgd::launch(softmax_ce_kernel<__nv_bfloat16>, dim3(batch), 256, 0, stream, (const __nv_bfloat16*)logits, labels, classes, ld,
                        1.0f / batch, grad_scale, loss_sum, per_sample, (__nv_bfloat16*)dlogits);
  return esgd::launch(softmax_ce_kernel<float>, dim3(batch), 256, 0, stream, (const float*)logits, labels, classes, ld, 1.0f / batch,
                      grad_scale, loss_sum, per_sample, (float*)dlogits);
}

// idx (optional, one byte per output element) records the arg-max for the backward pass.
int esgd_maxpool3x3s2_fwd(const void* x, void* y, void* idx, int N, int H, int W, int C, void* stream) {
  if (C % 8) return -1;
  if (N == 0) return 0;                                // a grid of no blocks is an error
  const int OH = (H + 1) / 2, OW = (W + 1) / 2;
  return esgd::launch(maxpool_fwd_kernel, dim3(N * OH), 256, 0, stream,
                      (const __nv_bfloat16*)x, (__nv_bfloat16*)y, (uint8_t*)idx, N, H, W, C, OH, OW);
}

int esgd_maxpool3x3s2_bwd(const void* idx, const void* dy, void* dx, int N, int H, int W, int C, void* stream) {
  if (C % 8) return -1;
  if (N == 0) return 0;
  const int OH = (H + 1) / 2, OW = (W + 1) / 2;
  return esgd::launch(maxpool_bwd_kernel, dim3(N * ((H + 1) / 2)), 256, 0, stream, (const uint8_t*)idx,
                      (const __nv_bfloat16*)dy, (__nv_bfloat16*)dx, N, H, W, C, OH, OW);
}

// y[n, oh, ow, :] = x[n, 2*oh, 2*ow, :]   (OH = ceil(H/2), OW = ceil(W/2))
int esgd_subsample2_fwd(const void* x, void* y, int N, int H, int W, int C, void* stream) {
  if (C % 8) return -1;
  const int OH = (H + 1) / 2, OW = (W + 1) / 2;
  return esgd::launch(subsample2_fwd_kernel, dim3(grid_for((int64_t)N * OH * OW * (C / 8))), 256, 0, stream,
                      (const __nv_bfloat16*)x, (__nv_bfloat16*)y, N, H, W, C, OH, OW);
}
int esgd_subsample2_bwd(const void* dy, void* dx, int N, int H, int W, int C, void* stream) {
  if (C % 8) return -1;
  const int OH = (H + 1) / 2, OW = (W + 1) / 2;
  return esgd::launch(subsample2_bwd_kernel, dim3(grid_for((int64_t)N * H * W * (C / 8))), 256, 0, stream,
                      (const __nv_bfloat16*)dy, (__nv_bfloat16*)dx, N, H, W, C, OH, OW);
}

// col: [N*Ho*Wo, Kpad] bf16; seg = roundup8(S*C) <= 32; Kpad a multiple of seg with Kpad >= R*seg.
// Element (r, j) of a row is x[.., h+r, (w0*C + j)] for j < S*C: weights must be laid out the same way.
int esgd_im2col_small_c(const void* x, void* col, int N, int H, int W, int C, int R, int S, int stride, int pad,
                        int seg, int Kpad, void* stream) {
  if (seg % 8 || seg < S * C || seg > 32 || Kpad % seg || Kpad < R * seg) return -1;
  const int Ho = (H + 2 * pad - R) / stride + 1, Wo = (W + 2 * pad - S) / stride + 1;
  const int rowbytes = W * C * 2;
  const int smem = R * (kImLeftGuard + rowbytes + kImRightGuard);
  // staged-row kernel: rows must be 16-byte multiples on a 16-byte base, the guards must cover the padding and
  // the over-read of the last window, and the rows must fit in the default shared-memory budget
  if (rowbytes % 16 == 0 && ((uintptr_t)x & 15) == 0 && pad * C * 2 <= kImLeftGuard &&
      ((Wo - 1) * stride - pad) * C * 2 + seg * 2 + 8 <= rowbytes + kImRightGuard && smem <= 48 * 1024) {
    return esgd::launch(im2col_rows_kernel, dim3(N * Ho), 256, smem, stream, (const __nv_bfloat16*)x, (__nv_bfloat16*)col, N,
                        H, W, C, R, S, stride, pad, Ho, Wo, seg, Kpad);
  }
  return esgd::launch(im2col_small_c_kernel<32>, dim3(grid_for((int64_t)N * Ho * Wo * (Kpad / seg))), 256, 0, stream,
                      (const __nv_bfloat16*)x, (__nv_bfloat16*)col, N, H, W, C, R, S, stride, pad, Ho, Wo, seg, Kpad);
}

// seg / Kpad as in esgd_im2col_small_c; w [Cout][R][S*C], sc = S*C.
int esgd_stem_pack(const void* w, void* out, int Cout, int R, int sc, int seg, int Kpad, void* stream) {
  return esgd::launch(stem_pack_kernel, dim3((Cout * Kpad + 255) / 256), 256, 0, stream, (const __nv_bfloat16*)w,
                      (__nv_bfloat16*)out, Cout, R, sc, seg, Kpad);
}
int esgd_stem_unpack(const float* col, void* dw, float* acc, int Cout, int R, int sc, int seg, int Kpad, void* stream) {
  return esgd::launch(stem_unpack_kernel, dim3((Cout * R * sc + 255) / 256), 256, 0, stream, col, (__nv_bfloat16*)dw, acc,
                      Cout, R, sc, seg, Kpad);
}

// out [M][np] bf16 (np a multiple of 8, zeros from column N on) = dy [M][N] fp32 with row stride ld; colsum (optional, zeroed
// by the caller) += column sums of dy.
int esgd_cast_colsum(const float* dy, int64_t ld, int M, int N, int np, void* out, float* colsum, void* stream) {
  if (np % 8 || np < N) return -1;
  const int vec = ld % 4 == 0 && ((uintptr_t)dy & 15) == 0;
  const int row_blocks = M / kCastRows + (M % kCastRows != 0);
  dim3 grid((np / 4 + 255) / 256, row_blocks < 65535 ? row_blocks : 65535);
  return esgd::launch(cast_colsum_kernel, grid, 256, 0, stream, dy, ld, M, N, np, (__nv_bfloat16*)out, colsum, vec);
}

int esgd_avgpool_fwd(const void* x, void* y, int N, int HW, int C, void* stream) {
  if (C % 8) return -1;
  if (N == 0) return 0;
  int cg = 1;
  while (cg < 16 && cg < C / 8) cg *= 2;
  return esgd::launch(avgpool_fwd_kernel, dim3(N, (C / 8 + cg - 1) / cg), 256, 0, stream, (const __nv_bfloat16*)x, (__nv_bfloat16*)y, N,
                      HW, C, cg);
}

int esgd_avgpool_bwd(const void* dy, void* dx, int N, int HW, int C, void* stream) {
  if (C % 8) return -1;
  return esgd::launch(avgpool_bwd_kernel, dim3(grid_for((int64_t)N * HW * (C / 8))), 256, 0, stream, (const __nv_bfloat16*)dy,
                      (__nv_bfloat16*)dx, N, HW, C);
}

}  // extern "C"
