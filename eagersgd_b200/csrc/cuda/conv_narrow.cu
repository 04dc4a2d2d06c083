// 3x3 convolutions of 16 and 32 channels over small images (the CIFAR ResNets): forward, data gradient, weight gradient; 64
// channels in small forward problems.
//
// A layer of 128 x 32 x 32 pixels and 16 channels is 0.6 GFLOP over 8 MB that sit in L2: it is bound by latency, and the
// 128-row tcgen05 tiles fed 64 channels at a time spent 33 us on it, three quarters of each operand zero fill.  Here a block
// of eight warps copies a few image rows with their margin into shared memory (cp.async, only the channels there are) and
// every warp multiplies 16 pixels at a time with ldmatrix / mma.sync m16n8k16: the fragment rows are pixel addresses, so a
// tap, a stride or the filter's transposition is an address offset.  The tensor pipe is not what bounds these layers.
// Pixel and filter rows are padded by 16 bytes, which makes every ldmatrix conflict-free.
//
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <atomic>
#include "bn_grad.h"
#include "launch.cuh"

namespace {

constexpr int kThreads = 256;

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

struct Shape {
  int N, H, W, Ho, Wo, stride;   // H x W: the image the taps read, Ho x Wo: the pixels that are computed
  int tr, ti;                    // output rows of an image and images per tile (ti > 1 only with tr == Ho)
  int rows, pw;                  // input rows per image in a tile, pixel pitch (W + 2)
  int row_tiles, tiles;
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

// The input rows of a tile with a margin of one pixel (zeros outside the image): [ti][rows][pw] pixels of C channels.
template <int C>
__device__ __forceinline__ void load_tile(const __nv_bfloat16* x, const Shape& s, int n0, int oh0, uint8_t* dst) {
  constexpr int CH = C / 8, PX = C * 2 + 16;
  const int per_img = s.rows * s.pw * CH;
  for (int i = threadIdx.x; i < s.ti * per_img; i += kThreads) {
    const int im = i / per_img, j = i - im * per_img;
    const int px = j / CH, ch = j - px * CH, row = px / s.pw, col = px - row * s.pw;
    const int n = n0 + im, h = oh0 * s.stride - 1 + row, w = col - 1;
    const bool ok = n < s.N && h >= 0 && h < s.H && w >= 0 && w < s.W;
    const __nv_bfloat16* src = ok ? x + (((int64_t)n * s.H + h) * s.W + w) * C + ch * 8 : x;
    cp_async16(smem_addr(dst + (im * s.rows * s.pw + px) * PX + ch * 16), src, ok);
  }
}

// y[pixel, CN] = sum over taps and CR channels; kT: the filters [CR][3][3][CN] are used transposed and rotated (data gradient).
template <int CR, int CN, bool kT>
__global__ void __launch_bounds__(kThreads) conv_narrow_kernel(const Shape s, const Args a) {
  constexpr int PX = CR * 2 + 16;                              // bytes of a pixel in shared memory
  constexpr int CIN = kT ? CN : CR, COUT = kT ? CR : CN;       // filter storage [COUT][9][CIN]
  constexpr int WR = CIN * 2 + 16;                             // bytes of a filter row (tap, output channel)
  constexpr int WN = CN == 64 ? 2 : 1, WM = 8 / WN;            // warps along the output channels / along the pixels
  constexpr int NT = CN / WN / 8;                              // 8-column tiles of a warp
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ float s_stat[2 * CN];
  uint8_t* sW = smem;                                          // [9][COUT] rows
  uint8_t* sX = smem + 9 * COUT * WR;
  esgd::pdl_enter();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wm = warp / WN, wn = warp % WN;
  for (int i = threadIdx.x; i < 9 * COUT * (CIN / 8); i += kThreads) {      // filters: [COUT][9][CIN] -> [9][COUT][CIN]
    const int ch = i % (CIN / 8), rest = i / (CIN / 8), tap = rest % 9, co = rest / 9;
    cp_async16(smem_addr(sW + (tap * COUT + co) * WR + ch * 16), a.w + (int64_t)i * 8, true);
  }
  if (threadIdx.x < 2 * CN) s_stat[threadIdx.x] = 0.0f;
  float st[NT][4];                                             // sum, sum, squares, squares of this thread's two columns
#pragma unroll
  for (int t = 0; t < NT; ++t) st[t][0] = st[t][1] = st[t][2] = st[t][3] = 0.0f;
  const int a_pix = (lane & 7) + ((lane >> 3) & 1) * 8, a_k = ((lane >> 4) & 1) * 16;
  // filter fragments of two column tiles: rows are output columns (forward) or reduced channels (transposed)
  const uint32_t b_lane = kT ? (uint32_t)(((lane & 7) + ((lane >> 3) & 1) * 8) * WR + ((lane >> 4) & 1) * 16 + wn * NT * 16)
                             : (uint32_t)((wn * NT * 8 + (lane & 7) + ((lane >> 4) & 1) * 8) * WR + ((lane >> 3) & 1) * 16);
  const uint32_t w0 = smem_addr(sW) + b_lane;
  const int pixels = s.ti * s.tr * s.Wo;
  for (int tile = blockIdx.x; tile < s.tiles; tile += gridDim.x) {
    const int n0 = tile / s.row_tiles * s.ti, oh0 = tile % s.row_tiles * s.tr;
    __syncthreads();                                           // the previous tile has been read
    load_tile<CR>(a.x, s, n0, oh0, sX);
    cp_async_wait();
    __syncthreads();
    for (int m = wm; m * 16 < pixels; m += WM) {
      const int p = min(m * 16 + a_pix, pixels - 1);
      const int im = p / (s.tr * s.Wo), q = p - im * s.tr * s.Wo, oh = q / s.Wo, ow = q - oh * s.Wo;
      const uint32_t x0 = smem_addr(sX) + (uint32_t)(((im * s.rows + oh * s.stride) * s.pw + ow * s.stride) * PX + a_k);
      float acc[NT][4];
#pragma unroll
      for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.0f;
      // batch-norm input and mask of this thread's outputs: on their way while the products run
      __nv_bfloat162 by[kT ? NT : 1][2];
      uint32_t keep[2] = {0xffffffffu, 0xffffffffu};           // bits 8t + (c % 8) of the thread's columns
      if (kT && a.bn_y != nullptr) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int pp = m * 16 + (lane >> 2) + h * 8, im2 = pp / (s.tr * s.Wo);
          if (pp >= pixels || n0 + im2 >= s.N) continue;
          const int64_t pix = ((int64_t)(n0 + im2) * s.Ho + oh0) * s.Wo + (pp - im2 * s.tr * s.Wo);
#pragma unroll
          for (int t = 0; t < NT; ++t)
            by[t][h] = *reinterpret_cast<const __nv_bfloat162*>(a.bn_y + pix * CN + wn * NT * 8 + t * 8 + (lane & 3) * 2);
          if (a.bn_mask != nullptr) {
            const uint8_t* mp = a.bn_mask + pix * (CN / 8) + wn * NT;
            keep[h] = NT == 2 ? *reinterpret_cast<const uint16_t*>(mp) : *reinterpret_cast<const uint32_t*>(mp);
          }
        }
      }
#pragma unroll
      for (int tap = 0; tap < 9; ++tap) {
        const uint32_t xt = x0 + (uint32_t)((tap / 3 * s.pw + tap % 3) * PX);
        const uint32_t wt = w0 + (uint32_t)((kT ? 8 - tap : tap) * COUT * WR);
#pragma unroll
        for (int k = 0; k < CR / 16; ++k) {
          uint32_t af[4];
          ldm4(af, xt + k * 32);
#pragma unroll
          for (int t = 0; t < NT; t += 2) {
            uint32_t bf[4];
            if (kT) ldm4t(bf, wt + k * 16 * WR + t * 16);
            else ldm4(bf, wt + t * 8 * WR + k * 32);
            mma16816(acc[t], af, bf[0], bf[1]);
            mma16816(acc[t + 1], af, bf[2], bf[3]);
          }
        }
      }
      // fragment rows lane / 4 and + 8, columns 2 * (lane % 4), + 1 of every column tile
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int pp = m * 16 + (lane >> 2) + h * 8;
        const int im2 = pp / (s.tr * s.Wo);
        if (pp >= pixels || n0 + im2 >= s.N) continue;
        const int64_t pix = ((int64_t)(n0 + im2) * s.Ho + oh0) * s.Wo + (pp - im2 * s.tr * s.Wo);
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const int c = wn * NT * 8 + t * 8 + (lane & 3) * 2;
          float v0 = acc[t][2 * h], v1 = acc[t][2 * h + 1];
          if (a.scale != nullptr) {
            v0 = fmaf(v0, __ldg(a.scale + c), __ldg(a.shift + c));
            v1 = fmaf(v1, __ldg(a.scale + c + 1), __ldg(a.shift + c + 1));
          }
          if (a.residual != nullptr) {
            const float2 r = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(a.residual + pix * CN + c));
            v0 += r.x;
            v1 += r.y;
          }
          if (a.relu) { v0 = fmaxf(v0, 0.0f); v1 = fmaxf(v1, 0.0f); }
          if (kT) {
            const uint32_t bits = keep[h] >> (t * 8 + (lane & 3) * 2);
            v0 = bits & 1u ? v0 : 0.0f;
            v1 = bits & 2u ? v1 : 0.0f;
          }
          const __nv_bfloat162 o = __floats2bfloat162_rn(v0, v1);
          *reinterpret_cast<__nv_bfloat162*>(a.y + pix * CN + c) = o;
          if (a.sum != nullptr) {
            const float2 f = __bfloat1622float2(o);
            float2 g = f;
            if (kT) {
              g = __bfloat1622float2(by[kT ? t : 0][h]);
              g.x -= __ldg(a.bn_aux + c);
              g.y -= __ldg(a.bn_aux + c + 1);
            }
            st[t][0] += f.x; st[t][1] += f.y;
            st[t][2] = fmaf(f.x, g.x, st[t][2]); st[t][3] = fmaf(f.y, g.y, st[t][3]);
          }
        }
      }
    }
  }
  if (a.sum != nullptr) {      // lanes with equal lane % 4, then the block's warps, then one atomic per column and block
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float v = st[t][q];
        v += __shfl_xor_sync(0xffffffffu, v, 4);
        v += __shfl_xor_sync(0xffffffffu, v, 8);
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        if (lane < 4) atomicAdd(&s_stat[(q >> 1) * CN + wn * NT * 8 + t * 8 + lane * 2 + (q & 1)], v);
      }
    __syncthreads();
    if (threadIdx.x < 2 * CN) {
      const float scale = kT && threadIdx.x >= CN ? __ldg(a.bn_aux + threadIdx.x) : 1.0f;      // 1 / std
      atomicAdd((threadIdx.x < CN ? a.sum : a.sqsum) + threadIdx.x % CN, s_stat[threadIdx.x] * scale);
    }
  }
}

// dw[CO][3][3][CI] (fp32, added to) = sum over pixels of dy[pixel, CO] x[pixel + tap, CI].  Both operands are read transposed
// from their pixel rows.  A warp keeps the accumulators of TAPS taps; the warps of a tap group share the pixels.
template <int CI, int CO>
struct WgradPlan {
  static constexpr int TILES = (CO / 16) * (CI / 8);                  // accumulator tiles per tap
  static constexpr int TAPS = TILES <= 2 ? 9 : (TILES <= 8 ? 3 : 1);  // at most 96 accumulator registers
  static constexpr int SETS = 9 / TAPS;
  static constexpr int SLICES = TAPS == 9 ? 8 : (TAPS == 3 ? 3 : 1);
  static constexpr int THREADS = SETS * SLICES * 32;
};

template <int CI, int CO>
__global__ void __launch_bounds__(WgradPlan<CI, CO>::THREADS) wgrad_narrow_kernel(const Shape s, const __nv_bfloat16* __restrict__ x,
                                                                                 const __nv_bfloat16* __restrict__ dy,
                                                                                 float* __restrict__ dw) {
  using P = WgradPlan<CI, CO>;
  constexpr int PX = CI * 2 + 16, PD = CO * 2 + 16, MT = CO / 16, NT = CI / 8;
  extern __shared__ __align__(16) uint8_t smem[];
  uint8_t* sX = smem;
  uint8_t* sD = smem + s.ti * s.rows * s.pw * PX;
  esgd::pdl_enter();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, set = warp % P::SETS, slice = warp / P::SETS;
  float acc[P::TAPS][MT][NT][4];
#pragma unroll
  for (int t = 0; t < P::TAPS; ++t)
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j) acc[t][i][j][0] = acc[t][i][j][1] = acc[t][i][j][2] = acc[t][i][j][3] = 0.0f;
  const int d_pix = (lane & 7) + ((lane >> 4) & 1) * 8, d_col = ((lane >> 3) & 1) * 16;      // dy: [k][m] -> m x k fragments
  const int x_pix = (lane & 7) + ((lane >> 3) & 1) * 8, x_col = ((lane >> 4) & 1) * 16;      // x:  [k][n] -> k x n fragments
  const int pixels = s.ti * s.tr * s.Wo, padded = (pixels + 15) / 16 * 16;
  for (int tile = blockIdx.x; tile < s.tiles; tile += gridDim.x) {
    const int n0 = tile / s.row_tiles * s.ti, oh0 = tile % s.row_tiles * s.tr;
    __syncthreads();
    {      // input rows with margin, and the tile's pixels of dy (zeros past the end)
      constexpr int CH = CI / 8;
      const int per_img = s.rows * s.pw * CH;
      for (int i = threadIdx.x; i < s.ti * per_img; i += P::THREADS) {
        const int im = i / per_img, j = i - im * per_img;
        const int px = j / CH, ch = j - px * CH, row = px / s.pw, col = px - row * s.pw;
        const int n = n0 + im, h = oh0 * s.stride - 1 + row, w = col - 1;
        const bool ok = n < s.N && h >= 0 && h < s.H && w >= 0 && w < s.W;
        cp_async16(smem_addr(sX + (im * s.rows * s.pw + px) * PX + ch * 16), ok ? x + (((int64_t)n * s.H + h) * s.W + w) * CI + ch * 8 : x, ok);
      }
      constexpr int CD = CO / 8;
      for (int i = threadIdx.x; i < padded * CD; i += P::THREADS) {
        const int px = i / CD, ch = i - px * CD, im = px / (s.tr * s.Wo);
        const bool ok = px < pixels && n0 + im < s.N;
        const int64_t pix = ((int64_t)(n0 + im) * s.Ho + oh0) * s.Wo + (px - im * s.tr * s.Wo);
        cp_async16(smem_addr(sD + px * PD + ch * 16), ok ? dy + pix * CO + ch * 8 : dy, ok);
      }
    }
    cp_async_wait();
    __syncthreads();
    for (int k = slice; k * 16 < pixels; k += P::SLICES) {
      uint32_t af[MT][4];
      const uint32_t d0 = smem_addr(sD + (k * 16 + d_pix) * PD + d_col);
#pragma unroll
      for (int i = 0; i < MT; ++i) ldm4t(af[i], d0 + i * 32);
      const int p = min(k * 16 + x_pix, pixels - 1);               // past the end dy is zero
      const int im = p / (s.tr * s.Wo), q = p - im * s.tr * s.Wo, oh = q / s.Wo, ow = q - oh * s.Wo;
      const uint32_t x0 = smem_addr(sX) + (uint32_t)(((im * s.rows + oh * s.stride) * s.pw + ow * s.stride) * PX + x_col);
#pragma unroll
      for (int t = 0; t < P::TAPS; ++t) {
        const int tap = set * P::TAPS + t;
        const uint32_t xt = x0 + (uint32_t)((tap / 3 * s.pw + tap % 3) * PX);
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
  }
  // The pixel slices meet in shared memory, and the block adds its filter bank to dw with one bulk reduction.
  float* bank = reinterpret_cast<float*>(smem);                      // [CO][9][CI]
  __syncthreads();
  for (int sl = 0; sl < P::SLICES; ++sl) {
    if (slice == sl) {
#pragma unroll
      for (int t = 0; t < P::TAPS; ++t)
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              float2* d = reinterpret_cast<float2*>(bank + ((i * 16 + (lane >> 2) + h * 8) * 9 + set * P::TAPS + t) * CI + j * 8 + (lane & 3) * 2);
              float2 v = make_float2(acc[t][i][j][2 * h], acc[t][i][j][2 * h + 1]);
              if (sl > 0) { const float2 o = *d; v.x += o.x; v.y += o.y; }
              *d = v;
            }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");    // the bulk copy below reads what was written here
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dw), "r"(smem_addr(bank)),
                 "r"((uint32_t)(CO * 9 * CI * 4)) : "memory");
    asm volatile("cp.async.bulk.commit_group;\n\tcp.async.bulk.wait_group 0;" ::: "memory");
  }
}

// Tiles of about `target` pixels: whole rows of an image, or whole images when they are small.  False: there is nothing to tile.
bool plan(Shape& s, int N, int H, int W, int stride, int target, int min_tiles) {
  if (N < 1 || H < 1 || W < 1 || stride < 1) return false;
  s.N = N; s.H = H; s.W = W; s.stride = stride;
  s.Ho = (H + 2 - 3) / stride + 1;
  s.Wo = (W + 2 - 3) / stride + 1;
  s.pw = W + 2;
  const auto rows_of = [&](int px) {
    int best = 1;
    for (int d = 1; d <= s.Ho && d * s.Wo <= px; ++d) if (s.Ho % d == 0) best = d;
    return best;
  };
  // smaller tiles rather than idle SMs
  while (target > 64 && (int64_t)N * s.Ho * s.Wo / target < min_tiles) target /= 2;
  s.tr = rows_of(target);
  s.ti = 1;
  if (s.tr == s.Ho) {
    s.ti = target / (s.Ho * s.Wo);
    if (s.ti < 1) s.ti = 1;
    if (s.ti > N) s.ti = N;
  }
  s.rows = (s.tr - 1) * stride + 3;
  s.row_tiles = s.Ho / s.tr;
  s.tiles = s.row_tiles * ((N + s.ti - 1) / s.ti);
  return true;
}

constexpr int kSmemMax = 200 * 1024;

// Every load of an operand is 16 bytes wide (cp.async).
bool aligned16(const void* a, const void* b) { return (((uintptr_t)a | (uintptr_t)b) & 15) == 0; }

// Resident blocks per SM (kept per kernel for the newest shared-memory size; a layer's is always the same).
struct Occupancy { std::atomic<uint64_t> last{0}; };
template <class K>
int blocks_per_sm(K kernel, int threads, int smem, Occupancy& o) {
  const uint64_t seen = o.last.load(std::memory_order_relaxed);
  if ((int)(seen >> 32) == smem) return (int)(seen & 0xffffffffu);
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem) != cudaSuccess || n < 1) n = 1;
  o.last.store(((uint64_t)smem << 32) | (uint64_t)n, std::memory_order_relaxed);
  return n;
}

template <int CR, int CN, bool kT>
int launch_conv(const Args& a, int N, int H, int W, int stride, cudaStream_t stream) {
  static Occupancy occ;
  Shape s;
  if (!plan(s, N, H, W, stride, 256, esgd::sm_count())) return -1;
  if (!aligned16(a.x, a.w)) return -100;
  const int cin = kT ? CN : CR, cout = kT ? CR : CN;
  const int smem = 9 * cout * (cin * 2 + 16) + s.ti * s.rows * s.pw * (CR * 2 + 16);
  if (smem > kSmemMax) return -100;
  const int resident = blocks_per_sm(conv_narrow_kernel<CR, CN, kT>, kThreads, smem, occ) * esgd::sm_count();
  return esgd::launch(conv_narrow_kernel<CR, CN, kT>, dim3(s.tiles < resident ? s.tiles : resident), kThreads, smem, stream, s, a);
}

template <int CI, int CO>
int launch_wgrad(const void* x, const void* dy, float* dw, int N, int H, int W, int stride, cudaStream_t stream) {
  static Occupancy occ;
  Shape s;
  if (!plan(s, N, H, W, stride, 256, esgd::sm_count())) return -1;
  if (!aligned16(x, dy)) return -100;
  const int px = (s.ti * s.tr * s.Wo + 15) / 16 * 16;
  int smem = s.ti * s.rows * s.pw * (CI * 2 + 16) + px * (CO * 2 + 16);
  if (smem < CO * 9 * CI * 4) smem = CO * 9 * CI * 4;
  if (smem > kSmemMax) return -100;
  blocks_per_sm(wgrad_narrow_kernel<CI, CO>, WgradPlan<CI, CO>::THREADS, smem, occ);
  // one block per SM at most: every block ends with a reduction of the whole filter bank
  const int grid = s.tiles < esgd::sm_count() ? s.tiles : esgd::sm_count();
  return esgd::launch(wgrad_narrow_kernel<CI, CO>, dim3(grid), WgradPlan<CI, CO>::THREADS, smem, stream, s, (const __nv_bfloat16*)x,
                      (const __nv_bfloat16*)dy, dw);
}

}  // namespace

extern "C" {

// 64 input channels fill a k-block of the tile kernels, and only small forward problems are better off here.  Microseconds back
// to back, rows in shared memory / tiles: 8 x 8 pixels, 64 images, inference epilogue 7.7 / 9.0, statistics 8.2 / 8.2; 96
// images 9.0 / 9.5 and 9.6 / 8.2; 14 x 14, 16 images (3136 pixels) 7.8 / 9.0 and 7.5 / 8.4, 32 images 10.6 / 9.1 and
// 11.6 / 8.5; 8 x 8, 512 images 18.6 / 12.4.  The data gradient with its batch norm lost from the first image on (8.8 / 7.7 at
// 8 x 8, 20.2 / 13.8 at 512 images) and is the tile kernels'.
constexpr int64_t kMaxPixels64 = 4096;

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
  if (Cin == 64 && Cout == 64 && (int64_t)N * H * W <= kMaxPixels64) return launch_conv<64, 64, false>(a, N, H, W, stride, s);
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
