// 3x3 convolutions of 16 and 32 channels over small images (the CIFAR ResNets): forward, data gradient, weight gradient; 64
// channels in small problems, forward and data gradient.
//
// A layer of 128 x 32 x 32 pixels and 16 channels is 0.6 GFLOP over 8 MB that sit in L2: it is bound by latency and by the
// instructions around the products, and the 128-row tcgen05 tiles fed 64 channels at a time spent 33 us on it, three quarters of
// each operand zero fill.  Here a block has a run of output rows (an even share of the rows of all images: 148 blocks, one an SM,
// so every address of the sums sees 148 atomics and not one per tile), copies the input rows it needs with their margin
// into shared memory (cp.async, a warp per row: an address per row instead of four divisions per 16 bytes), and every
// warp multiplies 16 pixels at a time with ldmatrix / mma.sync m16n8k16: the fragment rows are pixel addresses, so a tap, a
// stride or the filter's transposition is an address offset.  The tensor pipe is not what bounds these layers.  Pixel and
// filter rows are padded by 16 bytes, which makes every ldmatrix conflict-free.  Results leave by way of shared memory,
// eight channels of a pixel a lane, so that stores, shortcut and batch-norm operands are 16 bytes wide.
//
// Input rows are numbered as if every image had a row of zeros above and below it ("padded rows"); output row oh of image n
// reads padded rows n * (H + 2) + oh * stride and the two after it.
//
// Microseconds with sums, tiles of 256 pixels with their own index arithmetic -> now: 128 x 32 x 32, 16 channels, forward
// 15.4 -> 6.6, data gradient with batch norm 14.6 -> 7.0, weight gradient 12.3 -> 7.4; 128 x 16 x 16, 32 channels 8.6 -> 5.4, 11.1 -> 6.5,
// 12.9 -> 7.8.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include "bn_grad.h"
#include "launch.cuh"

namespace {

constexpr int kWarps = 16, kThreads = kWarps * 32;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void ldm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void unpack8(const uint4& w, float (&v)[8]) {
  const uint32_t x[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) { v[2 * q] = __uint_as_float(x[q] << 16); v[2 * q + 1] = __uint_as_float(x[q] & 0xffff0000u); }
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  uint4 raw;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
  for (int q = 0; q < 4; ++q) h[q] = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
  return raw;
}

// Division by a number known at launch, after Granlund and Montgomery (Division by Invariant Integers using Multiplication, 1994):
// multiply, add, shift; exact for dividends below 2^31.
struct FastDiv {
  uint32_t mul, shift, d;
  FastDiv() = default;
  explicit FastDiv(uint32_t d_) : d(d_) {
    for (shift = 0; shift < 31 && (1u << shift) < d; ++shift) {}
    mul = (uint32_t)((((uint64_t)1 << 32) * (((uint64_t)1 << shift) - d)) / d + 1);
  }
  __device__ __forceinline__ int div(int n) const { return (int)((__umulhi((uint32_t)n, mul) + (uint32_t)n) >> shift); }
};

struct Shape {
  int N, H, W, Ho, Wo, stride;   // H x W: the image the taps read, Ho x Wo: the pixels that are computed
  int pw;                        // pixel pitch of an input row (W + 2)
  int total;                     // output rows of all images
  int per_pass, slots;           // output rows that a block takes at a time, input rows that these need at most
  FastDiv by_wo, by_ho, by_hp;   // Wo, Ho, H + 2
};

// A pass: output rows v0 .. v1 - 1 of all images' rows.
struct Pass {
  int v0, v1, g0, rows;          // g0, rows: first padded row of the input that it reads, and how many
  __device__ __forceinline__ Pass(const Shape& s, int from, int to) : v0(from), v1(to) {
    g0 = padded(s, v0);
    rows = padded(s, v1 - 1) + 3 - g0;
  }
  static __device__ __forceinline__ int padded(const Shape& s, int v) {
    const int n = s.by_ho.div(v);
    return n * (s.H + 2) + (v - n * s.Ho) * s.stride;
  }
  // Where the window of output pixel p (counted from the pass's first) starts: a pixel of the input rows in shared memory.
  __device__ __forceinline__ int window(const Shape& s, int p) const {
    const int row = s.by_wo.div(p);
    return (padded(s, v0 + row) - g0) * s.pw + (p - row * s.Wo) * s.stride;
  }
};

struct Args {
  const __nv_bfloat16 *x, *w;
  __nv_bfloat16* y;
  const float *scale, *shift;
  const __nv_bfloat16* residual;
  int relu;
  float *sum, *sqsum;                                          // statistics of y; with bn_y dbeta and dgamma (bn_grad.h)
  const __nv_bfloat16* bn_y;
  const uint8_t* bn_mask;
  const float* bn_aux;
};

// The first output row of block b.
__device__ __forceinline__ int first_row(const Shape& s, int b) { return (int)((int64_t)s.total * b / (int)gridDim.x); }

// The left and right margin of every input row: zeros for as long as the block lives.
template <int C>
__device__ __forceinline__ void clear_margins(const Shape& s, uint8_t* sX) {
  constexpr int CH = C / 8, PX = C * 2 + 16;
  for (int i = threadIdx.x; i < s.slots * 2 * CH; i += blockDim.x) {
    const int r = i / (2 * CH), side = i / CH % 2, ch = i % CH;
    *reinterpret_cast<uint4*>(sX + (r * s.pw + side * (s.pw - 1)) * PX + ch * 16) = make_uint4(0, 0, 0, 0);
  }
}
// The input rows of a pass, a warp a row.
template <int C>
__device__ __forceinline__ void load_rows(const Shape& s, const Pass& ps, const __nv_bfloat16* x, uint8_t* sX) {
  constexpr int CH = C / 8, PX = C * 2 + 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  for (int r = warp; r < ps.rows; r += warps) {
    const int g = ps.g0 + r, n = s.by_hp.div(g), h = g - n * (s.H + 2) - 1;
    const bool ok = h >= 0 && h < s.H;
    const __nv_bfloat16* src = ok ? x + ((int64_t)n * s.H + h) * s.W * C : x;
    const uint32_t dst = smem_addr(sX + (r * s.pw + 1) * PX);
    for (int i = lane; i < s.W * CH; i += 32) cp_async16(dst + (i / CH) * PX + (i % CH) * 16, src + (ok ? i * 8 : 0), ok);
  }
}

// The batch norm in front of a convolution, applied to its rows on their way into shared memory: z = act(scale * y + shift), which
// is also stored, with its mask, for the backward pass.  As esgd_bn_fwd takes it, without a residual.
struct BnOutput {
  const __nv_bfloat16* y;                                      // the convolution's input is z
  __nv_bfloat16* z;
  uint8_t* mask;
  const float *sum, *sqsum, *gamma, *beta;
  float *running_mean, *running_var, *aux;
  float inv_count, unbias, momentum, eps;
  int relu;
};
// coef: [2][C] floats of shared memory
template <int C>
__device__ __forceinline__ void bn_coefficients(const BnOutput& b, float* coef) {
  if (threadIdx.x >= C) return;
  const int c = threadIdx.x;
  const float mean = b.sum[c] * b.inv_count, var = fmaxf(b.sqsum[c] * b.inv_count - mean * mean, 0.0f), invstd = rsqrtf(var + b.eps);
  const float sc = b.gamma[c] * invstd, sh = b.beta[c] - mean * sc;
  coef[c] = sc;
  coef[C + c] = sh;
  if (blockIdx.x == 0) {
    b.aux[c] = mean;
    b.aux[C + c] = invstd;
    b.aux[2 * C + c] = sc;
    b.aux[3 * C + c] = sh;
    if (b.running_mean != nullptr) {
      b.running_mean[c] = (1.0f - b.momentum) * b.running_mean[c] + b.momentum * mean;
      b.running_var[c] = (1.0f - b.momentum) * b.running_var[c] + b.momentum * var * b.unbias;
    }
  }
}
template <int C>
__device__ __forceinline__ void load_z_rows(const Shape& s, const Pass& ps, const BnOutput& b, const float* coef, uint8_t* sX) {
  constexpr int CH = C / 8, PX = C * 2 + 16, COLS = 4;         // loads in flight a lane
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5, n = s.W * CH;
  float sc[8], sh[8];                                          // every load of a lane is of the same channels
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    sc[q] = coef[lane % CH * 8 + q];
    sh[q] = coef[C + lane % CH * 8 + q];
  }
  for (int r = warp; r < ps.rows; r += warps) {
    const int g = ps.g0 + r, im = s.by_hp.div(g), h = g - im * (s.H + 2) - 1, row = im * s.H + h;
    const bool ok = h >= 0 && h < s.H, mine = ok && row >= ps.v0 && row < ps.v1;       // stride 1: output rows are input rows
    const int64_t at = ok ? (int64_t)row * s.W * C : 0;
    for (int i0 = lane; i0 < n; i0 += 32 * COLS) {
      uint4 ry[COLS];
#pragma unroll
      for (int k = 0; k < COLS; ++k)
        if (ok && i0 + k * 32 < n) ry[k] = *reinterpret_cast<const uint4*>(b.y + at + (i0 + k * 32) * 8);
#pragma unroll
      for (int k = 0; k < COLS; ++k) {
        const int i = i0 + k * 32;
        if (i >= n) continue;
        uint4 out = make_uint4(0, 0, 0, 0);                    // rows outside the image
        if (ok) {
          float v[8];
          unpack8(ry[k], v);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            v[q] = v[q] * sc[q] + sh[q];
            if (b.relu) v[q] = fmaxf(v[q], 0.0f);
          }
          out = pack8(v);
        }
        *reinterpret_cast<uint4*>(sX + (r * s.pw + 1 + i / CH) * PX + i % CH * 16) = out;
        if (mine) {
          *reinterpret_cast<uint4*>(b.z + at + i * 8) = out;
          if (b.mask != nullptr) {
            const uint32_t x[4] = {out.x, out.y, out.z, out.w};
            uint32_t m = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) m |= ((x[q] & 0x7fffu) ? 1u << (2 * q) : 0u) | ((x[q] & 0x7fff0000u) ? 2u << (2 * q) : 0u);
            b.mask[at / 8 + i] = (uint8_t)m;
          }
        }
      }
    }
  }
}

// A warp's share of the output: 16 pixels a time, NT tiles of 8 columns from column wn * NT * 8 on.
template <int CR, int CN, int WARPS = kWarps>
struct Tile {
  static constexpr int WN = CN == 64 ? 2 : 1, WM = WARPS / WN;       // warps along the output channels / along the pixels
  static constexpr int NT = CN / WN / 8;
  static constexpr int CHW = NT;                                     // 16-byte chunks of a pixel that a warp writes
  static constexpr int UNITS = 16 * CHW / 32;                        // ... and how many of the 16 pixels' a lane has
  static constexpr int PITCH = NT * 8 + 4;                           // floats of a pixel's row in the staging buffer
  static constexpr int STAGE = 16 * PITCH * 4;                       // its bytes per warp
  static constexpr bool kRegB = CR == 16 && CN == 16;                // the filters fit the registers
};

// Products of 16 pixels whose windows start at the lanes' address x0: acc = sum over taps and CR channels.
template <int CR, int CN, bool kT>
struct Products {
  using T = Tile<CR, CN>;
  static constexpr int PX = CR * 2 + 16;                       // bytes of a pixel in shared memory
  static constexpr int CIN = kT ? CN : CR, COUT = kT ? CR : CN;       // filter storage [COUT][9][CIN]
  static constexpr int WR = CIN * 2 + 16;                      // bytes of a filter row (tap, output channel)
  static constexpr int FILTER = 9 * COUT * WR;
  uint32_t w0;
  uint32_t breg[T::kRegB ? 9 : 1][4];
  // filters: [COUT][9][CIN] -> [9][COUT][CIN]
  static __device__ __forceinline__ void load_filters(const __nv_bfloat16* w, uint8_t* sW) {
    constexpr int CH = CIN / 8;
    for (int i = threadIdx.x; i < 9 * COUT * CH; i += blockDim.x) {
      const int ch = i % CH, rest = i / CH, tap = rest % 9, co = rest / 9;
      cp_async16(smem_addr(sW + (tap * COUT + co) * WR + ch * 16), w + i * 8, true);
    }
  }
  // fragments of two column tiles: rows are output columns (forward) or reduced channels (transposed)
  __device__ __forceinline__ void begin(const uint8_t* sW, int wn, int lane) {
    const uint32_t b_lane = kT ? (uint32_t)(((lane & 7) + ((lane >> 3) & 1) * 8) * WR + ((lane >> 4) & 1) * 16 + wn * T::NT * 16)
                               : (uint32_t)((wn * T::NT * 8 + (lane & 7) + ((lane >> 4) & 1) * 8) * WR + ((lane >> 3) & 1) * 16);
    w0 = smem_addr(sW) + b_lane;
    if constexpr (T::kRegB) {
#pragma unroll
      for (int tap = 0; tap < 9; ++tap) fragment(breg[tap], tap, 0, 0);
    }
  }
  __device__ __forceinline__ void fragment(uint32_t (&b)[4], int tap, int k, int t) const {
    const uint32_t wt = w0 + (uint32_t)((kT ? 8 - tap : tap) * COUT * WR);
    if (kT) ldm4t(b, wt + k * 16 * WR + t * 16);
    else ldm4(b, wt + t * 8 * WR + k * 32);
  }
  __device__ __forceinline__ void run(float (&acc)[T::NT][4], uint32_t x0, uint32_t row_bytes) const {
#pragma unroll
    for (int t = 0; t < T::NT; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.0f;
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
      const uint32_t xt = x0 + (uint32_t)(tap / 3) * row_bytes + (tap % 3) * PX;
#pragma unroll
      for (int k = 0; k < CR / 16; ++k) {
        uint32_t af[4];
        ldm4(af, xt + k * 32);
#pragma unroll
        for (int t = 0; t < T::NT; t += 2) {
          uint32_t bf[4];
          if constexpr (T::kRegB) {
#pragma unroll
            for (int q = 0; q < 4; ++q) bf[q] = breg[tap][q];
          } else {
            fragment(bf, tap, k, t);
          }
          mma16816(acc[t], af, bf[0], bf[1]);
          mma16816(acc[t + 1], af, bf[2], bf[3]);
        }
      }
    }
  }
};

// What happens to 16 pixels' products: affine map, residual, ReLU or mask, rounding, store, sums.  A lane has eight channels
// (its chunk) of UNITS pixels.
template <int CR, int CN, bool kBn, int WARPS = kWarps>
struct Output {
  using T = Tile<CR, CN, WARPS>;
  float s1[8], s2[8], neg_mean[kBn ? 8 : 1];
  float* stage;
  int lane, c0;                                                // c0: the lane's first channel
  __device__ __forceinline__ void begin(const Args& a, uint8_t* stages, int warp, int wn) {
    lane = threadIdx.x & 31;
    stage = reinterpret_cast<float*>(stages + warp * T::STAGE);
    c0 = wn * T::NT * 8 + lane % T::CHW * 8;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      s1[q] = s2[q] = 0.0f;
      if (kBn) neg_mean[kBn ? q : 0] = a.bn_y != nullptr ? -__ldg(a.bn_aux + c0 + q) : 0.0f;
    }
  }
  uint4 res[T::UNITS], by[kBn ? T::UNITS : 1];
  uint32_t keep[kBn ? T::UNITS : 1];
  __device__ __forceinline__ int pixel(int u) const { return lane / T::CHW + u * (32 / T::CHW); }
  // the epilogue's operands, on their way while the products run; pix: the first of the 16 pixels, n: how many there are
  __device__ __forceinline__ void prefetch(const Args& a, int64_t pix, int n) {
#pragma unroll
    for (int u = 0; u < T::UNITS; ++u) {
      if (pixel(u) >= n) continue;
      const int64_t at = (pix + pixel(u)) * CN + c0;
      if (a.residual != nullptr) res[u] = *reinterpret_cast<const uint4*>(a.residual + at);
      if (kBn && a.bn_y != nullptr) {
        by[kBn ? u : 0] = *reinterpret_cast<const uint4*>(a.bn_y + at);
        keep[kBn ? u : 0] = a.bn_mask != nullptr ? a.bn_mask[at / 8] : 0xffu;
      }
    }
  }
  __device__ __forceinline__ void finish(const Args& a, const float (&acc)[T::NT][4], int64_t pix, int n) {
    // fragment rows lane / 4 and + 8, columns 2 * (lane % 4), + 1 of every column tile
    __syncwarp();
#pragma unroll
    for (int t = 0; t < T::NT; ++t)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<float2*>(stage + ((lane >> 2) + h * 8) * T::PITCH + t * 8 + (lane & 3) * 2) = make_float2(acc[t][2 * h], acc[t][2 * h + 1]);
    __syncwarp();
#pragma unroll
    for (int u = 0; u < T::UNITS; ++u) {
      if (pixel(u) >= n) continue;
      const float* src = stage + pixel(u) * T::PITCH + lane % T::CHW * 8;
      const float4 lo = *reinterpret_cast<const float4*>(src), hi = *reinterpret_cast<const float4*>(src + 4);
      float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
      if (a.scale != nullptr) {
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = fmaf(v[q], __ldg(a.scale + c0 + q), __ldg(a.shift + c0 + q));
      }
      if (a.residual != nullptr) {
        float r[8];
        unpack8(res[u], r);
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] += r[q];
      }
      if (a.relu) {
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = fmaxf(v[q], 0.0f);
      }
      if (kBn && a.bn_y != nullptr) {
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = (keep[kBn ? u : 0] >> q) & 1u ? v[q] : 0.0f;
      }
      const uint4 o = pack8(v);
      *reinterpret_cast<uint4*>(a.y + (pix + pixel(u)) * CN + c0) = o;
      if (a.sum != nullptr) {
        float f[8], g[8];
        unpack8(o, f);
        if (kBn) {
          unpack8(by[kBn ? u : 0], g);
#pragma unroll
          for (int q = 0; q < 8; ++q) g[q] += neg_mean[kBn ? q : 0];
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          s1[q] += f[q];
          s2[q] = fmaf(f[q], kBn ? g[q] : f[q], s2[q]);
        }
      }
    }
  }
  // The warps' sums meet in shared memory (part: [WM][2][CN] floats), then one atomic per column and block.
  __device__ __forceinline__ void collect(const Args& a, float* part, int wm) {
    if (a.sum == nullptr) return;
#pragma unroll
    for (int q = 0; q < 8; ++q)
#pragma unroll
      for (int d = T::CHW; d < 32; d *= 2) {
        s1[q] += __shfl_xor_sync(0xffffffffu, s1[q], d);
        s2[q] += __shfl_xor_sync(0xffffffffu, s2[q], d);
      }
    if (lane < T::CHW) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        part[(wm * 2) * CN + c0 + q] = s1[q];
        part[(wm * 2 + 1) * CN + c0 + q] = s2[q];
      }
    }
  }
  static __device__ __forceinline__ void commit(const Args& a, const float* part) {
    if (a.sum == nullptr || threadIdx.x >= 2 * CN) return;
    float v = 0.0f;
#pragma unroll
    for (int m = 0; m < T::WM; ++m) v += part[m * 2 * CN + threadIdx.x];
    if (kBn && threadIdx.x >= CN) v *= __ldg(a.bn_aux + threadIdx.x);      // 1 / std
    atomicAdd((threadIdx.x < CN ? a.sum : a.sqsum) + threadIdx.x % CN, v);
  }
};

// y[pixel, CN] = sum over taps and CR channels; kT: the filters [CR][3][3][CN] are used transposed and rotated (data gradient).
// kBnIn: the input is a batch norm's output, made here (the 4 us of a launch of its own between two convolutions).
template <int CR, int CN, bool kT, bool kBnIn>
__global__ void __launch_bounds__(kThreads, 1) conv_narrow_kernel(const Shape s, const Args a, const BnOutput b) {
  using T = Tile<CR, CN>;
  using P = Products<CR, CN, kT>;
  extern __shared__ __align__(16) uint8_t smem[];
  uint8_t* sW = smem;
  uint8_t* sC = sW + P::FILTER;
  float* part = reinterpret_cast<float*>(sC + kWarps * T::STAGE);
  float* coef = part + T::WM * 2 * CN;
  uint8_t* sX = reinterpret_cast<uint8_t*>(coef + (kBnIn ? 2 * CR : 0));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wm = warp / T::WN, wn = warp % T::WN;
  clear_margins<CR>(s, sX);
  esgd::pdl_enter();
  P::load_filters(a.w, sW);
  if (kBnIn) {
    bn_coefficients<CR>(b, coef);
    __syncthreads();
  }
  P prod;
  Output<CR, CN, kT> out;
  out.begin(a, sC, warp, wn);
  const int end = first_row(s, blockIdx.x + 1);
  const int a_pix = (lane & 7) + ((lane >> 3) & 1) * 8, a_k = ((lane >> 4) & 1) * 16;
  bool first = true;
  for (int v0 = first_row(s, blockIdx.x); v0 < end; v0 += s.per_pass) {
    const Pass ps(s, v0, min(v0 + s.per_pass, end));
    if (!first) __syncthreads();                               // the previous pass has been read
    if constexpr (kBnIn) load_z_rows<CR>(s, ps, b, coef, sX);
    else load_rows<CR>(s, ps, a.x, sX);
    cp_async_wait();
    __syncthreads();
    if (first) prod.begin(sW, wn, lane);
    first = false;
    const int pixels = (ps.v1 - ps.v0) * s.Wo;
    const int64_t pix0 = (int64_t)ps.v0 * s.Wo;
    for (int m = wm * 16; m < pixels; m += T::WM * 16) {
      out.prefetch(a, pix0 + m, pixels - m);
      const uint32_t x0 = smem_addr(sX) + (uint32_t)(ps.window(s, min(m + a_pix, pixels - 1)) * P::PX + a_k);
      float acc[T::NT][4];
      prod.run(acc, x0, (uint32_t)(s.pw * P::PX));
      out.finish(a, acc, pix0 + m, pixels - m);
    }
  }
  out.collect(a, part, wm);
  __syncthreads();
  out.commit(a, part);
}

// dw[CO][3][3][CI] (fp32, added to) = sum over pixels of dy[pixel, CO] x[pixel + tap, CI].  Both operands are read transposed
// from their pixel rows.  A warp keeps the accumulators of TAPS taps; the warps of a tap group share the pixels.
template <int CI, int CO, int WARPS = kWarps>
struct WgradPlan {
  static constexpr int TILES = (CO / 16) * (CI / 8);                  // accumulator tiles per tap
  static constexpr int TAPS = TILES <= 2 ? 9 : (TILES <= 8 ? 3 : 1);  // at most 96 accumulator registers
  static constexpr int SETS = 9 / TAPS;
  static constexpr int SLICES = SETS == 3 && WARPS > 12 ? 4 : WARPS / SETS;      // (five banks of 32 channels would not fit shared memory)
  static constexpr int THREADS = SETS * SLICES * 32;
  static constexpr int BANK = CO * 9 * CI;                            // floats
  static constexpr int PITCH = 9 * CI + 8;                            // of an output channel in a slice's bank
  static constexpr int BYTES = (SLICES * CO * PITCH + BANK) * 4;
};

template <int CI, int CO, int WARPS = kWarps>
struct Wgrad {
  using P = WgradPlan<CI, CO, WARPS>;
  static constexpr int PX = CI * 2 + 16, PD = CO * 2 + 16, MT = CO / 16, NT = CI / 8;
  float acc[P::TAPS][MT][NT][4];
  int lane, set, slice;
  __device__ __forceinline__ void begin(int warp) {
    lane = threadIdx.x & 31;
    set = warp % P::SETS;
    slice = warp / P::SETS;
#pragma unroll
    for (int t = 0; t < P::TAPS; ++t)
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) acc[t][i][j][0] = acc[t][i][j][1] = acc[t][i][j][2] = acc[t][i][j][3] = 0.0f;
  }
  // 16 pixels: d0 the lanes' address of dy ([k][m] -> m x k fragments), x0 that of their windows ([k][n] -> k x n fragments)
  __device__ __forceinline__ void step(uint32_t d0, uint32_t x0, uint32_t row_bytes) {
    uint32_t af[MT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i) ldm4t(af[i], d0 + i * 32);
#pragma unroll
    for (int t = 0; t < P::TAPS; ++t) {
      const int tap = set * P::TAPS + t;
      const uint32_t xt = x0 + (uint32_t)(tap / 3) * row_bytes + (tap % 3) * PX;
#pragma unroll
      for (int j = 0; j < NT; j += 2) {
        uint32_t bf[4];
        ldm4t(bf, xt + j * 16);
#pragma unroll
        for (int i = 0; i < MT; ++i) {
          mma16816(acc[t][i][j], af[i], bf[0], bf[1]);
          mma16816(acc[t][i][j + 1], af[i], bf[2], bf[3]);
        }
      }
    }
  }
  __device__ __forceinline__ int d_pix() const { return (lane & 7) + ((lane >> 4) & 1) * 8; }
  __device__ __forceinline__ int d_col() const { return ((lane >> 3) & 1) * 16; }
  __device__ __forceinline__ int x_pix() const { return (lane & 7) + ((lane >> 3) & 1) * 8; }
  __device__ __forceinline__ int x_col() const { return ((lane >> 4) & 1) * 16; }
  // Every slice writes its sums to a bank of its own ([CO][9][CI], output channels a multiple of 32 words plus 8 apart: without
  // the 8 a store went to one bank eight times, 5 of the 11 us of 32 channels) ...
  __device__ __forceinline__ void collect(float* banks) {
    float* bank = banks + slice * (CO * P::PITCH);
#pragma unroll
    for (int t = 0; t < P::TAPS; ++t)
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            *reinterpret_cast<float2*>(bank + (i * 16 + (lane >> 2) + h * 8) * P::PITCH + (set * P::TAPS + t) * CI + j * 8 + (lane & 3) * 2) =
                make_float2(acc[t][i][j][2 * h], acc[t][i][j][2 * h + 1]);
  }
  // ... which all threads add up once they are there; the block adds the result to dw by bulk reductions, blocks in turn beginning
  // at another place.
  static __device__ __forceinline__ void commit(float* banks, float* dw) {
    float* sum = banks + P::SLICES * (CO * P::PITCH);
    for (int i = threadIdx.x * 4; i < P::BANK; i += blockDim.x * 4) {
      const float* at = banks + i + i / (9 * CI) * 8;
      float4 v = *reinterpret_cast<const float4*>(at);
#pragma unroll
      for (int sl = 1; sl < P::SLICES; ++sl) {
        const float4 o = *reinterpret_cast<const float4*>(at + sl * (CO * P::PITCH));
        v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
      }
      *reinterpret_cast<float4*>(sum + i) = v;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");    // the bulk copies below read what was written here
    __syncthreads();
    if (threadIdx.x == 0) {
      constexpr int PARTS = 4, PART = P::BANK / PARTS;
      for (int i = 0; i < PARTS; ++i) {
        const int at = (i + (int)blockIdx.x) % PARTS * PART;
        asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dw + at), "r"(smem_addr(sum + at)),
                     "r"((uint32_t)(PART * 4)) : "memory");
      }
      asm volatile("cp.async.bulk.commit_group;\n\tcp.async.bulk.wait_group 0;" ::: "memory");
    }
  }
};

template <int CI, int CO>
__global__ void __launch_bounds__(WgradPlan<CI, CO>::THREADS, 1) wgrad_narrow_kernel(const Shape s, const __nv_bfloat16* __restrict__ x,
                                                                                     const __nv_bfloat16* __restrict__ dy,
                                                                                     float* __restrict__ dw) {
  using P = WgradPlan<CI, CO>;
  using G = Wgrad<CI, CO>;
  extern __shared__ __align__(16) uint8_t smem[];
  uint8_t* sX = smem;
  uint8_t* sD = smem + s.slots * s.pw * G::PX;
  clear_margins<CI>(s, sX);
  esgd::pdl_enter();
  G g;
  g.begin(threadIdx.x >> 5);
  const int end = first_row(s, blockIdx.x + 1);
  bool first = true;
  for (int v0 = first_row(s, blockIdx.x); v0 < end; v0 += s.per_pass) {
    const Pass ps(s, v0, min(v0 + s.per_pass, end));
    if (!first) __syncthreads();
    first = false;
    load_rows<CI>(s, ps, x, sX);
    const int pixels = (ps.v1 - ps.v0) * s.Wo, padded = (pixels + 15) / 16 * 16;
    constexpr int CD = CO / 8;
    const __nv_bfloat16* d = dy + (int64_t)ps.v0 * s.Wo * CO;
    for (int i = threadIdx.x; i < padded * CD; i += P::THREADS) {      // the pass's pixels of dy, zeros past the end
      const bool ok = i < pixels * CD;
      cp_async16(smem_addr(sD + i / CD * G::PD + i % CD * 16), d + (ok ? i * 8 : 0), ok);
    }
    cp_async_wait();
    __syncthreads();
    for (int k = g.slice * 16; k < pixels; k += P::SLICES * 16) {
      const uint32_t d0 = smem_addr(sD + (k + g.d_pix()) * G::PD + g.d_col());
      const uint32_t x0 = smem_addr(sX) + (uint32_t)(ps.window(s, min(k + g.x_pix(), pixels - 1)) * G::PX + g.x_col());     // past the end dy is zero
      g.step(d0, x0, (uint32_t)(s.pw * G::PX));
    }
  }
  __syncthreads();                                                    // the banks lie where the rows were
  g.collect(reinterpret_cast<float*>(smem));
  __syncthreads();
  G::commit(reinterpret_cast<float*>(smem), dw);
}

// ---------------------------------------------------------------- a layer's whole backward pass
// Batch norm, data gradient and weight gradient of a stride-1 layer of C channels in one launch: the rows of the batch norm's
// gradient dy = a * dz + b * y + c are made on their way into shared memory (bf16, as a pass of its own would store them) and
// read there by eight warps that multiply them with the filters and by six or eight that multiply them with the input's rows.
// A block has one pass (with several the accumulators would have to outlive the loads, for which there are no registers):
// launch_bwd() refuses problems of more rows than that.  Microseconds, three launches (4.6 + 7.0 + 7.4) -> this one: 128 x 32 x 32, 16
// channels 19.0 -> 11.9; 128 x 16 x 16, 32 channels 17.6 -> 12.3.  The third ran on a stream of its own but did not overlap: each
// of them fills the SMs.
struct BnInput {
  const __nv_bfloat16 *dz, *y;
  const float *aux, *gamma, *dbeta, *dgamma;                   // as esgd_bn_bwd_apply takes them
  float *acc_dgamma, *acc_dbeta;
  float inv_count;
};

template <int C>
__device__ __forceinline__ void load_dy_rows(const Shape& s, const Pass& ps, const BnInput& b, const float* coef, uint8_t* sD) {
  constexpr int CH = C / 8, PX = C * 2 + 16, ROWS = 2, COLS = 2;      // eight loads in flight a lane
  float ca[8], cb[8], cc[8];                                   // every load of a lane is of the same channels
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int c = (int)(threadIdx.x & 31) % CH * 8 + q;
    ca[q] = coef[c];
    cb[q] = coef[C + c];
    cc[q] = coef[2 * C + c];
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5, n = s.W * CH;
  for (int r0 = warp; r0 < ps.rows; r0 += ROWS * warps) {
    const __nv_bfloat16 *dz[ROWS], *y[ROWS];
    bool ok[ROWS];
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      const int g = ps.g0 + r0 + j * warps, im = s.by_hp.div(g), h = g - im * (s.H + 2) - 1;
      ok[j] = r0 + j * warps < ps.rows && h >= 0 && h < s.H;
      const int64_t at = ok[j] ? ((int64_t)im * s.H + h) * s.W * C : 0;
      dz[j] = b.dz + at;
      y[j] = b.y + at;
    }
    for (int i0 = lane; i0 < n; i0 += 32 * COLS) {
      uint4 rd[ROWS][COLS], ry[ROWS][COLS];
#pragma unroll
      for (int j = 0; j < ROWS; ++j)
#pragma unroll
        for (int k = 0; k < COLS; ++k)
          if (ok[j] && i0 + k * 32 < n) {
            rd[j][k] = *reinterpret_cast<const uint4*>(dz[j] + (i0 + k * 32) * 8);
            ry[j][k] = *reinterpret_cast<const uint4*>(y[j] + (i0 + k * 32) * 8);
          }
#pragma unroll
      for (int j = 0; j < ROWS; ++j)
#pragma unroll
        for (int k = 0; k < COLS; ++k) {
          const int i = i0 + k * 32;
          if (r0 + j * warps >= ps.rows || i >= n) continue;
          uint4 out = make_uint4(0, 0, 0, 0);                  // rows outside the image
          if (ok[j]) {
            float d[8], yy[8];
            unpack8(rd[j][k], d);
            unpack8(ry[j][k], yy);
#pragma unroll
            for (int q = 0; q < 8; ++q) d[q] = ca[q] * d[q] + cb[q] * yy[q] + cc[q];
            out = pack8(d);
          }
          *reinterpret_cast<uint4*>(sD + ((r0 + j * warps) * s.pw + 1 + i / CH) * PX + i % CH * 16) = out;
        }
    }
  }
}

// Both groups of warps have read their rows.  They meet at a barrier with a name: __syncthreads() is for a place that the whole
// block reaches, and these are two.
__device__ __forceinline__ void rows_read(int threads) { asm volatile("barrier.sync 1, %0;" ::"r"(threads) : "memory"); }

template <int C>
struct BwdPlan {
  static constexpr int DGRAD = 8, WGRAD = C == 16 ? 8 : 6;     // warps
  static constexpr int THREADS = (DGRAD + WGRAD) * 32;
  using T = Tile<C, C, DGRAD>;
  using P = Products<C, C, true>;
  using G = Wgrad<C, C, WGRAD>;
  static constexpr int FIXED = P::FILTER + DGRAD * T::STAGE + T::WM * 2 * C * 4 + 3 * C * 4;
};

template <int C>
__global__ void __launch_bounds__(BwdPlan<C>::THREADS, 1) bwd_narrow_kernel(const Shape s, const Args a, const BnInput b, float* dw) {
  using B = BwdPlan<C>;
  using T = typename B::T;
  using P = typename B::P;
  using G = typename B::G;
  extern __shared__ __align__(16) uint8_t smem[];
  uint8_t* sW = smem;
  uint8_t* sC = sW + P::FILTER;
  float* part = reinterpret_cast<float*>(sC + B::DGRAD * T::STAGE);
  float* coef = part + T::WM * 2 * C;
  uint8_t* sX = reinterpret_cast<uint8_t*>(coef + 3 * C);
  uint8_t* sD = sX + s.slots * s.pw * P::PX;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  esgd::pdl_enter();
  P::load_filters(a.w, sW);
  if (threadIdx.x < C) {
    const int c = threadIdx.x;
    const float is = b.aux[C + c], gm = b.gamma[c], dgamma = b.dgamma[c], dbeta = b.dbeta[c], dg = dgamma * b.inv_count, db = dbeta * b.inv_count;
    coef[c] = gm * is;
    coef[C + c] = -gm * is * is * dg;
    coef[2 * C + c] = gm * is * (b.aux[c] * is * dg - db);
    if (blockIdx.x == 0) {                                     // the parameters' own gradient accumulators
      b.acc_dgamma[c] += dgamma;
      b.acc_dbeta[c] += dbeta;
    }
  }
  __syncthreads();
  const int end = first_row(s, blockIdx.x + 1);
  const uint32_t row_bytes = (uint32_t)(s.pw * P::PX);
  {
    const Pass ps(s, first_row(s, blockIdx.x), end);
    const int pixels = (ps.v1 - ps.v0) * s.Wo;
    clear_margins<C>(s, sX);
    clear_margins<C>(s, sD);
    load_rows<C>(s, ps, a.x, sX);
    load_dy_rows<C>(s, ps, b, coef, sD);
    cp_async_wait();
    __syncthreads();
    if (warp < B::DGRAD) {
      Output<C, C, true, B::DGRAD> out;
      out.begin(a, sC, warp, 0);
      P prod;
      prod.begin(sW, 0, lane);
      const int a_pix = (lane & 7) + ((lane >> 3) & 1) * 8, a_k = ((lane >> 4) & 1) * 16;
      const int64_t pix0 = (int64_t)ps.v0 * s.Wo;
      for (int m = warp * 16; m < pixels; m += T::WM * 16) {
        out.prefetch(a, pix0 + m, pixels - m);
        const uint32_t x0 = smem_addr(sD) + (uint32_t)(ps.window(s, min(m + a_pix, pixels - 1)) * P::PX + a_k);
        float acc[T::NT][4];
        prod.run(acc, x0, row_bytes);
        out.finish(a, acc, pix0 + m, pixels - m);
      }
      out.collect(a, part, warp);
      rows_read(B::THREADS);
    } else {
      G g;
      g.begin(warp - B::DGRAD);
      for (int k = g.slice * 16; k < pixels; k += G::P::SLICES * 16) {
        // past the end dy is the margin's zeros
        const int pd = k + g.d_pix(), px = min(k + g.x_pix(), pixels - 1);
        const uint32_t d0 = smem_addr(sD) + (uint32_t)((pd < pixels ? ps.window(s, pd) + s.pw + 1 : 0) * P::PX + g.d_col());
        const uint32_t x0 = smem_addr(sX) + (uint32_t)(ps.window(s, px) * P::PX + g.x_col());
        g.step(d0, x0, row_bytes);
      }
      rows_read(B::THREADS);                                   // the banks lie where the rows were
      g.collect(reinterpret_cast<float*>(sX));
    }
    __syncthreads();
    G::commit(reinterpret_cast<float*>(sX), dw);
    __syncthreads();
  }
  Output<C, C, true, B::DGRAD>::commit(a, part);
}

constexpr int kSmemMax = 220 * 1024;

// Every load of an operand is 16 bytes wide (cp.async).
bool aligned16(const void* a, const void* b) { return (((uintptr_t)a | (uintptr_t)b) & 15) == 0; }

// Input rows that `rows` consecutive output rows need at most: a window a row, and the rows between two images.
int slots_of(const Shape& s, int rows) {
  const int between = s.H + 2 - s.Ho * s.stride;
  return (rows - 1) * s.stride + 3 + (between > 0 ? (rows - 2 + s.Ho) / s.Ho * between : 0);
}

// The blocks' rows; `fixed` bytes of shared memory beside `row_bytes` of every input row and `out_bytes` of every output row.
// -1: there is nothing to compute; -100: one row at a time is too much.
int plan(Shape& s, int& grid, int& smem, int N, int H, int W, int stride, int fixed, int row_bytes, int out_bytes) {
  if (N < 1 || H < 1 || W < 1 || stride < 1) return -1;
  s.N = N; s.H = H; s.W = W; s.stride = stride;
  s.Ho = (H + 2 - 3) / stride + 1;
  s.Wo = (W + 2 - 3) / stride + 1;
  s.pw = W + 2;
  if ((int64_t)N * (H + 2) * s.pw >= (int64_t)1 << 30) return -100;
  s.total = N * s.Ho;
  s.by_wo = FastDiv((uint32_t)s.Wo);
  s.by_ho = FastDiv((uint32_t)s.Ho);
  s.by_hp = FastDiv((uint32_t)(H + 2));
  const int sms = esgd::sm_count();
  grid = s.total < sms ? s.total : sms;
  const auto bytes = [&](int rows) { return (int64_t)fixed + (int64_t)slots_of(s, rows) * row_bytes + (int64_t)rows * out_bytes; };
  int rows = (s.total + grid - 1) / grid;
  if (bytes(1) > kSmemMax) return -100;
  if (bytes(rows) > kSmemMax) {               // equal passes
    int passes = 2;
    while (bytes((rows + passes - 1) / passes) > kSmemMax) ++passes;
    rows = (rows + passes - 1) / passes;
  }
  s.per_pass = rows;
  s.slots = slots_of(s, rows);
  smem = (int)bytes(rows);
  return 0;
}

template <int CR, int CN, bool kT, bool kBnIn = false>
int launch_conv(const Args& a, int N, int H, int W, int stride, cudaStream_t stream, const BnOutput& b = BnOutput()) {
  using T = Tile<CR, CN>;
  using P = Products<CR, CN, kT>;
  Shape s;
  int grid, smem;
  const int rc = plan(s, grid, smem, N, H, W, stride, P::FILTER + kWarps * T::STAGE + T::WM * 2 * CN * 4 + (kBnIn ? 2 * CR * 4 : 0), (W + 2) * P::PX,
                      0);
  if (rc != 0) return rc;
  if (!aligned16(a.x, a.w) || !aligned16(a.y, a.residual) || !aligned16(a.bn_y, b.y) || !aligned16(b.z, nullptr)) return -100;
  static esgd::SmemAllowed allowed{0};
  if (const int e = esgd::allow_smem(conv_narrow_kernel<CR, CN, kT, kBnIn>, kSmemMax, allowed)) return e;
  return esgd::launch(conv_narrow_kernel<CR, CN, kT, kBnIn>, dim3(grid), kThreads, smem, stream, s, a, b);
}

template <int CI, int CO>
int launch_wgrad(const void* x, const void* dy, float* dw, int N, int H, int W, int stride, cudaStream_t stream) {
  using P = WgradPlan<CI, CO>;
  using G = Wgrad<CI, CO>;
  Shape s;
  int grid, smem;
  const int wo = stride < 1 ? 0 : (W + 2 - 3) / stride + 1;
  const int rc = plan(s, grid, smem, N, H, W, stride, 16 * G::PD, (W + 2) * G::PX, wo * G::PD);
  if (rc != 0) return rc;
  if (!aligned16(x, dy)) return -100;
  if (smem < P::BYTES) smem = P::BYTES;
  static esgd::SmemAllowed allowed{0};
  if (const int e = esgd::allow_smem(wgrad_narrow_kernel<CI, CO>, kSmemMax, allowed)) return e;
  return esgd::launch(wgrad_narrow_kernel<CI, CO>, dim3(grid), P::THREADS, smem, stream, s, (const __nv_bfloat16*)x,
                      (const __nv_bfloat16*)dy, dw);
}

template <int C>
int launch_bwd(const Args& a, const BnInput& b, float* dw, int N, int H, int W, cudaStream_t stream) {
  using B = BwdPlan<C>;
  Shape s;
  int grid, smem;
  const int rc = plan(s, grid, smem, N, H, W, 1, B::FIXED, 2 * (W + 2) * B::P::PX, 0);
  if (rc != 0) return rc;
  if (s.per_pass < (s.total + grid - 1) / grid) return -100;       // more rows a block than fit beside one another
  if (!aligned16(a.x, a.w) || !aligned16(a.y, a.residual) || !aligned16(a.bn_y, dw) || !aligned16(b.dz, b.y)) return -100;
  if (smem < B::FIXED + B::G::P::BYTES) smem = B::FIXED + B::G::P::BYTES;
  static esgd::SmemAllowed allowed{0};
  if (const int e = esgd::allow_smem(bwd_narrow_kernel<C>, kSmemMax, allowed)) return e;
  return esgd::launch(bwd_narrow_kernel<C>, dim3(grid), B::THREADS, smem, stream, s, a, b, dw);
}

}  // namespace

extern "C" {

// 64 input channels fill a k-block of the tile kernels, and only the smallest problems are better off here: blocks of one output row,
// of few pixels.  Microseconds back to back (100 launches in a graph), rows in shared memory / tiles, forward with sums, inference
// epilogue with a shortcut, data gradient with batch norm.  One row a block: 8 x 8 pixels, one image 4.1 / 5.1, 3.6 / 5.0, 4.3 / 5.8;
// 16 images 5.1 / 5.1, 4.6 / 5.1, 5.4 / 5.7; 14 x 14, ten 4.8 / 5.2, 4.3 / 5.2, 5.5 / 5.9; 28 x 28, five 5.1 / 5.3, 4.6 / 5.3, 5.6 /
// 6.0; 32 x 32, two 4.7 / 5.1, 4.2 / 5.1, 5.5 / 5.9.  Two: 8 x 8, 24 images 5.3 / 5.1, 4.9 / 5.1, 6.0 / 5.8; 14 x 14, twelve 5.7 / 5.2,
// 5.3 / 5.2, 6.2 / 5.9; 28 x 28, six 6.7 / 5.3, 6.4 / 5.2, 7.1 / 6.0.  Wider ones: 40 x 40, one image 5.2 / 5.1, 4.8 / 5.1, 5.6 /
// 5.8; 56 x 56, one 5.7 / 5.3, 5.5 / 5.2, 6.2 / 6.0.
//
// Inference, up to 4096 pixels in rows of at most 64: the two are within 0.6 us of one another on the device (64 images of 8 x 8 5.1 to
// 5.7 / 5.1, sixteen of 14 x 14 5.2 / 5.2, four of 28 x 28 5.2 / 5.2, one of 56 x 56 5.5 / 5.3; but one of 36 x 112 7.6 / 5.4), and a
// few images are bound by the host, which has three or four tensor maps less to make here: 3.0 us a call and 3.4.
bool rows_pay64(int N, int H, int W, bool inference) {
  if ((int64_t)N * H <= esgd::sm_count() && W <= 32) return true;
  return inference && (int64_t)N * H * W <= 4096 && W <= 64;
}

// With the batch norm in front of it, which is a launch of its own ahead of the tiles: 8 x 8, 128 images (8192 pixels) 7.6 / 9.1, 256
// images 10.1 / 11.3, 384 12.5 / 12.5; 14 x 14, 41 images (8036 pixels) 8.1 / 8.6, 48 9.1 / 8.8; 28 x 28, ten (7840 pixels) 8.0 / 8.8,
// twelve 9.8 / 8.7; 32 x 32, eight 8.2 / 9.2.  (Rows of more than 32 pixels: the caller's choice.)
constexpr int64_t kMaxNormPixels64 = 8192;

// Returns -100 for shapes this file does not take (the caller then uses the tile kernels).  3x3, padding 1, NHWC bf16.
// y = act(scale * conv + shift + residual), each part optional; sum / sqsum (caller-zeroed) receive y's statistics.
int esgd_conv_narrow_fwd(const void* x, const void* w, void* y, int N, int H, int W, int Cin, int Cout, int stride, const float* scale,
                         const float* shift, const void* residual, int relu, float* sum, float* sqsum, void* stream) {
  Args a{(const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (__nv_bfloat16*)y, scale, shift, (const __nv_bfloat16*)residual, relu, sum, sqsum,
         nullptr, nullptr, nullptr};
  cudaStream_t s = (cudaStream_t)stream;
  if (Cin == 16 && Cout == 16) return launch_conv<16, 16, false>(a, N, H, W, stride, s);
  if (Cin == 16 && Cout == 32) return launch_conv<16, 32, false>(a, N, H, W, stride, s);
  if (Cin == 32 && Cout == 32) return launch_conv<32, 32, false>(a, N, H, W, stride, s);
  if (Cin == 32 && Cout == 64) return launch_conv<32, 64, false>(a, N, H, W, stride, s);
  if (Cin == 64 && Cout == 64 && rows_pay64(N, H, W, sum == nullptr)) return launch_conv<64, 64, false>(a, N, H, W, stride, s);
  return -100;
}

// dx [N,H,W,Cin] from dy [N,H,W,Cout], stride 1; residual (optional) is added before the rounding; bn (optional): bn_grad.h.
int esgd_conv_narrow_dgrad(const void* dy, const void* w, void* dx, int N, int H, int W, int Cin, int Cout, const void* residual,
                           const esgd_bn_grad* bn, void* stream) {
  Args a{(const __nv_bfloat16*)dy, (const __nv_bfloat16*)w, (__nv_bfloat16*)dx, nullptr, nullptr, (const __nv_bfloat16*)residual, 0,
         nullptr, nullptr, nullptr, nullptr, nullptr};
  if (bn != nullptr) {
    a.sum = bn->sums; a.sqsum = bn->sums + Cin;
    a.bn_y = (const __nv_bfloat16*)bn->y; a.bn_mask = (const uint8_t*)bn->mask; a.bn_aux = bn->aux;
  }
  cudaStream_t s = (cudaStream_t)stream;
  if (Cin == 16 && Cout == 16) return launch_conv<16, 16, true>(a, N, H, W, 1, s);
  if (Cin == 32 && Cout == 32) return launch_conv<32, 32, true>(a, N, H, W, 1, s);
  if (Cin == 64 && Cout == 64 && rows_pay64(N, H, W, false)) return launch_conv<64, 64, true>(a, N, H, W, 1, s);
  return -100;
}

// The whole backward pass of z = act(batch_norm(conv(x, w))) for 3x3, stride 1, C channels in and out: dz [N,H,W,C] with the ReLU's
// mask applied, y the convolution's output; aux, gamma, dbeta, dgamma, acc_dgamma, acc_dbeta as in esgd_bn_bwd_apply; residual
// and bn as in esgd_conv_narrow_dgrad; dw as in esgd_conv_narrow_wgrad.
int esgd_conv_narrow_bwd(const void* x, const void* w, const void* dz, const void* y, const float* aux, const float* gamma, const float* dbeta,
                         const float* dgamma, float* acc_dgamma, float* acc_dbeta, void* dx, float* dw, int N, int H, int W, int C,
                         const void* residual, const esgd_bn_grad* bn, void* stream) {
  Args a{(const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (__nv_bfloat16*)dx, nullptr, nullptr, (const __nv_bfloat16*)residual, 0,
         nullptr, nullptr, nullptr, nullptr, nullptr};
  if (bn != nullptr) {
    a.sum = bn->sums; a.sqsum = bn->sums + C;
    a.bn_y = (const __nv_bfloat16*)bn->y; a.bn_mask = (const uint8_t*)bn->mask; a.bn_aux = bn->aux;
  }
  const BnInput b{(const __nv_bfloat16*)dz, (const __nv_bfloat16*)y, aux, gamma, dbeta, dgamma, acc_dgamma, acc_dbeta,
                  1.0f / ((float)N * (float)H * (float)W)};
  cudaStream_t s = (cudaStream_t)stream;
  if (C == 16) return launch_bwd<16>(a, b, dw, N, H, W, s);
  if (C == 32) return launch_bwd<32>(a, b, dw, N, H, W, s);
  return -100;
}

// y = conv(z, w) with y's statistics, for z = act(batch_norm(by)), C channels in and out, stride 1: z, mask, aux and the running
// statistics are written as esgd_bn_fwd writes them.
int esgd_conv_narrow_bn_fwd(const void* by, void* z, void* mask, const float* bsum, const float* bsqsum, const float* gamma, const float* beta,
                            float* running_mean, float* running_var, float* aux, int relu, float momentum, float eps, const void* w,
                            void* y, int N, int H, int W, int C, float* sum, float* sqsum, void* stream) {
  const int64_t m = (int64_t)N * H * W;
  Args a{(const __nv_bfloat16*)z, (const __nv_bfloat16*)w, (__nv_bfloat16*)y, nullptr, nullptr, nullptr, 0, sum, sqsum, nullptr, nullptr, nullptr};
  const BnOutput b{(const __nv_bfloat16*)by, (__nv_bfloat16*)z, (uint8_t*)mask, bsum, bsqsum, gamma, beta, running_mean, running_var, aux,
                   1.0f / (float)m, m > 1 ? (float)m / (float)(m - 1) : 1.0f, momentum, eps, relu};
  cudaStream_t s = (cudaStream_t)stream;
  if (C == 16) return launch_conv<16, 16, false, true>(a, N, H, W, 1, s, b);
  if (C == 32) return launch_conv<32, 32, false, true>(a, N, H, W, 1, s, b);
  if (C == 64 && m <= kMaxNormPixels64) return launch_conv<64, 64, false, true>(a, N, H, W, 1, s, b);
  return -100;
}

// dw [Cout][3][3][Cin] fp32, added to.
int esgd_conv_narrow_wgrad(const void* x, const void* dy, float* dw, int N, int H, int W, int Cin, int Cout, int stride, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if ((uintptr_t)dw & 15) return -100;
  if (Cin == 16 && Cout == 16) return launch_wgrad<16, 16>(x, dy, dw, N, H, W, stride, s);
  if (Cin == 16 && Cout == 32) return launch_wgrad<16, 32>(x, dy, dw, N, H, W, stride, s);
  if (Cin == 32 && Cout == 32) return launch_wgrad<32, 32>(x, dy, dw, N, H, W, stride, s);
  if (Cin == 32 && Cout == 64) return launch_wgrad<32, 64>(x, dy, dw, N, H, W, stride, s);
  return -100;
}

}  // extern "C"
