// The 7x7 / 2 convolution of RGB images (padding 3, 64 output channels): forward and weight gradient without the matrix of windows.
//
// Pixels of 6 bytes are nothing that TMA or a tensor-core operand could step through, so the windows have to be cut out by
// threads.  As a matrix in memory (im2col: 1.2 GB at 256 x 224 x 224, written once and read by both products) they cost more than
// the products.  Here bands of eight output rows (21 input rows) come into shared memory as they are, bulk copies between
// margins of zeros, and threads cut the windows of 128 output pixels at a time out of them: twelve words and eleven funnel
// shifts a filter row and pixel (a window starts in the middle of a word).
//   forward          a thread's window is its row of the A operand, which goes to tensor memory (K = 7 rows x 24, 22 of them zeros
//                    of the packed filters' layout): no shared-memory traffic but the reads.  16 x 11 MMAs of 128 x 64 x 16 a band
//   weight gradient  the reduction runs over pixels: windows are rows of 16 bytes in swizzled shared memory, read MN-major as two
//                    tiles of 128 window elements; dy comes by TMA.  Sums stay in tensor memory until the end, then one bulk
//                    reduction per output channel and CTA
// 256 x 224 x 224 before and after: forward with statistics 294 (windows) + 250 us -> 134 (141 with the copy of the images that it
// leaves for the backward pass), weight gradient 250 -> 155; inference of 125 images 152 + 125 -> 63.  Bounds: y is 411 MB, 75 us
// with the images.  A bare product takes 105; the affine map and the statistics are the rest (epilogue warps; two groups of them took
// 134 and 159 where three take 125 and 134, a third set of warps that build gave nothing).  The weight gradient is at the bandwidth
// of shared memory: windows written once (21 KB a tile) and read with dy by two products (96 KB).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include "launch.cuh"
#include "sm100_primitives.cuh"
#include "tensormap.cuh"

using namespace sm100;

namespace {

constexpr int kR = 7;                         // filter rows
constexpr int kSeg = 24;                      // elements of a window's row as the packed filters have them (21 and three zeros)
constexpr int kK = kR * kSeg;                 // 168
constexpr int kSteps = (kK + 15) / 16;        // K steps of a product: 11, the last one half zeros
constexpr int kOut = 64;
constexpr int kLead = 32;                     // bytes in front of a row's first pixel
constexpr int kSmemLimit = 227 * 1024;

struct StemShape {
  int N, H, W, Ho, Wo;
  int band, rows;                             // output rows of a band, its input rows
  int per_image, bands;                       // bands of an image, of all
  int tiles, pixels;                          // tiles of 128 pixels of a band, its pixels
  int pitch;                                  // bytes of a row
};

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src),
               "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void umma_bf16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st_x4(uint32_t taddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void tmem_st_x8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// The input rows of the CTA's bands, two bands in flight.
struct Bands {
  uint8_t* buf;                               // [2][rows][pitch], then a row of zeros
  uint64_t *full, *empty;
  __device__ __forceinline__ uint8_t* at(const StemShape& s, int k) const { return buf + (k & 1) * s.rows * s.pitch; }
  __device__ __forceinline__ void clear(const StemShape& s) const {
    uint4* p = reinterpret_cast<uint4*>(buf);
    for (int i = threadIdx.x; i < bytes(s) / 16; i += blockDim.x) p[i] = make_uint4(0, 0, 0, 0);
  }
  __host__ __device__ static int bytes(const StemShape& s) { return (2 * s.rows + 1) * s.pitch; }
  // The rows that are band `band`'s alone, to where they are kept (the thread that loads, once they are there).
  __device__ __forceinline__ void store(const StemShape& s, __nv_bfloat16* keep, int band, int k) const {
    const int64_t h = (int64_t)2 * s.band * band;                      // an image has whole bands
    for (int i = 0; i < 2 * s.band; ++i)
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(keep + (h + i) * s.W * 3),
                   "r"(smem_u32(at(s, k) + (i + 3) * s.pitch + kLead)), "r"((uint32_t)(s.W * 6)) : "memory");
    tma_store_commit();
  }
  // Band `band`, the CTA's k-th (one thread).
  __device__ __forceinline__ bool load(const StemShape& s, const __nv_bfloat16* x, int band, int k, volatile int* abort_flag) const {
    if (!mbar_wait(&empty[k & 1], ((uint32_t)(k >> 1) & 1u) ^ 1u, abort_flag)) return false;
    const int n = band / s.per_image, h0 = 2 * s.band * (band - n * s.per_image) - 3;
    const int lo = max(h0, 0), hi = min(h0 + s.rows, s.H);
    mbar_expect_tx(&full[k & 1], (uint32_t)((hi - lo) * s.W * 6));
    for (int h = lo; h < hi; ++h)
      bulk_load(at(s, k) + (h - h0) * s.pitch + kLead, x + ((int64_t)n * s.H + h) * s.W * 3, (uint32_t)(s.W * 6), &full[k & 1]);
    return true;
  }
};

// The window of a pixel of a band, row by row: out[12] words of the row's 24 elements.
struct Window {
  const uint8_t* rows;                        // the band's first input row
  const uint8_t* zero;
  int h0, H, pitch, top, at;                  // image row of the band's first; the window's first row, word of its first column
  __device__ __forceinline__ Window(const StemShape& s, const Bands& b, int band, int k, int pixel) {
    const int n = band / s.per_image, p = min(pixel, s.pixels - 1), row = p / s.Wo;
    rows = b.at(s, k);
    zero = b.buf + 2 * s.rows * s.pitch;
    h0 = 2 * s.band * (band - n * s.per_image) - 3;
    H = s.H;
    pitch = s.pitch;
    top = 2 * row;
    at = (kLead - 20) / 4 + 3 * (p - row * s.Wo);          // three pixels of margin are 18 bytes: it starts two bytes further on
  }
  __device__ __forceinline__ void row(int r, uint32_t (&out)[12]) const {
    const int h = h0 + top + r;
    const uint32_t* w = reinterpret_cast<const uint32_t*>(h >= 0 && h < H ? rows + (top + r) * pitch : zero) + at;
    uint32_t v[12];
#pragma unroll
    for (int i = 0; i < 12; ++i) v[i] = w[i];
#pragma unroll
    for (int i = 0; i < 11; ++i) out[i] = __funnelshift_r(v[i], v[i + 1], 16);
    out[10] &= 0xffffu;                       // the 21st element; what follows belongs to the next window
    out[11] = 0;
  }
};

// ---------------------------------------------------------------- forward
constexpr int kAStride = 96;                  // tensor-memory columns of an A stage (88 are used)
constexpr int kSets = 2, kGroups = 3;         // sets of four warps that build, groups of four of the epilogue
constexpr int kAccs = 4;
constexpr int kACol = kAccs * kOut;           // accumulators, then the A stages
constexpr int kFwdThreads = (4 + 4 * kSets + 4 * kGroups) * 32;
constexpr int kPanel = 128 * 128;

struct StemFwd {
  CUtensorMap tmW, tmY;                       // packed filters [64][Kpad]; y as [bands][pixels of a band][64]
  const __nv_bfloat16* x;
  __nv_bfloat16* keep;                        // x for the backward pass, or nullptr
  StemShape s;
  const float *scale, *shift;
  int relu;
  float *sum, *sqsum;
  int* error_flag;
};

__global__ void __launch_bounds__(kFwdThreads, 1) stem_fwd_kernel(const __grid_constant__ StemFwd p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const StemShape& s = p.s;
  uint8_t* sB = smem;                                         // three blocks of 64 filters x 64 elements
  uint8_t* sC = sB + 3 * 8192;                                // the epilogue groups' panels
  float* sAff = reinterpret_cast<float*>(sC + kGroups * kPanel);    // factors, summands
  float* sSum = sAff + 128;                                   // [2][64]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sSum + 128);
  uint64_t *afull = bars + 4, *aempty = bars + 6, *dfull = bars + 8, *dempty = bars + 12, *wfull = bars + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const Bands bands{reinterpret_cast<uint8_t*>(bars + 18), bars, bars + 2};
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bands.full[i], 1);
      mbar_init(&bands.empty[i], 4 * kSets);
    }
    for (int i = 0; i < kSets; ++i) { mbar_init(&afull[i], 4); mbar_init(&aempty[i], 1); }
    for (int i = 0; i < kAccs; ++i) { mbar_init(&dfull[i], 1); mbar_init(&dempty[i], 4); }
    mbar_init(wfull, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&p.tmW);
    tma_prefetch_desc(&p.tmY);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  bands.clear(s);
  if (threadIdx.x < 128) sSum[threadIdx.x] = 0.0f;
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  esgd::pdl_enter();

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(wfull, 3 * 8192);
      for (int b = 0; b < 3; ++b) tma_load_2d(sB + b * 8192, &p.tmW, wfull, b * 64, 0);
      bool ok = true;
      int k = 0;
      for (int band = blockIdx.x; ok && band < s.bands; band += gridDim.x, ++k) {
        ok = bands.load(s, p.x, band, k, abort_flag);
        if (p.keep == nullptr) continue;
        if (k == 0 && band + (int)gridDim.x < s.bands) continue;                  // one band behind the loads
        const bool last = band + (int)gridDim.x >= s.bands;
        for (int b = k > 0 ? k - 1 : 0; ok && b <= (last ? k : k - 1); ++b) {
          ok = mbar_wait(&bands.full[b & 1], (uint32_t)(b >> 1) & 1u, abort_flag);
          if (ok) bands.store(s, p.keep, blockIdx.x + b * gridDim.x, b);
        }
        tma_store_wait_read<0>();
      }
      tma_store_wait_all();
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(128, kOut, 0, 0);
      const uint64_t b_desc = umma_smem_desc(smem_u32(sB), 16, 1024);
      bool ok = mbar_wait(wfull, 0u, abort_flag);
      const int total = ((s.bands - 1 - (int)blockIdx.x) / (int)gridDim.x + 1) * s.tiles;
      for (int it = 0; ok && it < total; ++it) {
        const int st = it % kSets, acc = it % kAccs;
        ok = mbar_wait(&dempty[acc], ((uint32_t)(it / kAccs) & 1u) ^ 1u, abort_flag) && mbar_wait(&afull[st], (uint32_t)(it / kSets) & 1u, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint32_t a = tmem + (uint32_t)(kACol + st * kAStride), d = tmem + (uint32_t)(acc * kOut);
#pragma unroll
        for (int j = 0; j < kSteps; ++j) umma_bf16_ta(d, a + j * 8, b_desc + (uint64_t)((j >> 2) * 512 + (j & 3) * 2), idesc, j > 0 ? 1u : 0u);
        umma_commit(&aempty[st]);
        umma_commit(&dfull[acc]);
      }
    }
  } else if (warp >= 4 && warp < 4 + 4 * kSets) {
    // ------------------------------------------------------------ windows
    const int set = (warp - 4) >> 2, q = warp & 3;
    const uint32_t a = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(kACol + set * kAStride);
    tmem_st_x4(a + kK / 2, 0u, 0u, 0u, 0u);                   // the second half of the last K step
    bool ok = true;
    int it = 0, k = 0;
    for (int band = blockIdx.x; ok && band < s.bands; band += gridDim.x, ++k) {
      ok = __all_sync(0xffffffffu, mbar_wait(&bands.full[k & 1], (uint32_t)(k >> 1) & 1u, abort_flag));
      for (int j = 0; ok && j < s.tiles; ++j, ++it) {
        if (it % kSets != set) continue;
        const Window w(s, bands, band, k, j * 128 + q * 32 + lane);
        ok = __all_sync(0xffffffffu, mbar_wait(&aempty[set], ((uint32_t)(it / kSets) & 1u) ^ 1u, abort_flag));
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int r = 0; r < kR; ++r) {
          uint32_t v[12];
          w.row(r, v);
          tmem_st_x8(a + r * 12, v);
          tmem_st_x4(a + r * 12 + 8, v[8], v[9], v[10], v[11]);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&afull[set]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&bands.empty[k & 1]);
    }
  } else if (warp >= 4 + 4 * kSets) {
    // ------------------------------------------------------------ epilogue
    const int grp = ((warp - 4) >> 2) - kSets, q = warp & 3, gt = (int)threadIdx.x - (4 + 4 * kSets) * 32 - grp * 128, row = q * 32 + lane;
    uint8_t* panel = sC + grp * kPanel;
    const bool leader = gt == 0;
    if (p.shift != nullptr && grp == 0) sAff[gt] = gt >= 64 ? __ldg(p.shift + gt - 64) : p.scale != nullptr ? __ldg(p.scale + gt) : 1.0f;
    named_barrier_sync(1 + kGroups, kGroups * 128);
    const int cp = gt & 31, rg = gt >> 5;                     // sums: columns 2cp, 2cp + 1 of rows 32rg .. + 31
    float s0 = 0.0f, s1 = 0.0f, q0 = 0.0f, q1 = 0.0f;
    bool ok = true;
    int it = 0;
    for (int band = blockIdx.x; band < s.bands; band += gridDim.x) {               // to the end, whatever `ok` is: the group's barriers
      for (int j = 0; j < s.tiles; ++j, ++it) {
        if (it % kGroups != grp) continue;
        const int acc = it % kAccs;
        ok = __all_sync(0xffffffffu, ok && mbar_wait(&dfull[acc], (uint32_t)(it / kAccs) & 1u, abort_flag));
        tc_fence_after();
        const uint32_t t_row = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * kOut);
        uint32_t r[32];
        tmem_ld_32x32b_x32(t_row, r);
        if (leader) tma_store_wait_read<0>();                 // the previous panel has left the buffer
        named_barrier_sync(1 + grp, 128);
        tmem_ld_wait();
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          if (half == 1) {
            tmem_ld_32x32b_x32(t_row + 32, r);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&dempty[acc]);
          }
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[g * 8 + i]);
            if (p.shift != nullptr) {
              const float* aff = sAff + half * 32 + g * 8;
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] = fmaf(v[i], aff[i], aff[64 + i]);
            }
            if (p.relu) {
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] = fmaxf(v[i], 0.0f);
            }
            uint4 pk;
            __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
            for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            *reinterpret_cast<uint4*>(panel + row * 128 + (((half * 4 + g) ^ (row & 7)) << 4)) = pk;
          }
        }
        fence_proxy_async();
        named_barrier_sync(1 + grp, 128);
        if (leader) {
          tma_store_4d(&p.tmY, panel, 0, j * 128, band, 0);   // clipped at the end of the band
          tma_store_commit();
        }
        if (p.sum != nullptr) {
          const int rows = min(32, s.pixels - j * 128 - rg * 32);
          const uint8_t* colp = panel + rg * 32 * 128 + (cp & 3) * 4;
#pragma unroll 8
          for (int rr = 0; rr < 32; ++rr) {
            uint32_t w = *reinterpret_cast<const uint32_t*>(colp + rr * 128 + (((cp >> 2) ^ (rr & 7)) << 4));
            if (rr >= rows) w = 0u;
            const float a0 = __uint_as_float(w << 16), a1 = __uint_as_float(w & 0xffff0000u);
            s0 += a0; s1 += a1;
            q0 = fmaf(a0, a0, q0); q1 = fmaf(a1, a1, q1);
          }
        }
      }
    }
    if (p.sum != nullptr) {
      atomicAdd(sSum + 2 * cp, s0);
      atomicAdd(sSum + 2 * cp + 1, s1);
      atomicAdd(sSum + 64 + 2 * cp, q0);
      atomicAdd(sSum + 65 + 2 * cp, q1);
      named_barrier_sync(1 + kGroups, kGroups * 128);
      if (grp == 0) atomicAdd((gt < 64 ? p.sum : p.sqsum - 64) + gt, sSum[gt]);
    }
    if (leader) tma_store_wait_all();
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    __nanosleep(1000000);                                     // copies in flight land
    if (threadIdx.x == 0 && p.error_flag != nullptr) atomicExch(p.error_flag, 1);
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ---------------------------------------------------------------- weight gradient
constexpr int kBlock = 128 * 128;             // 128 pixels x 64 window elements
constexpr int kWgThreads = 12 * 32;

struct StemWgrad {
  CUtensorMap tmDY;                           // dy as [bands][pixels of a band][64]
  const __nv_bfloat16* x;
  StemShape s;
  float* col;                                 // [64][Kpad], added to
  int kpad;
  int* error_flag;
};

__global__ void __launch_bounds__(kWgThreads, 1) stem_wgrad_kernel(const __grid_constant__ StemWgrad p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const StemShape& s = p.s;
  // Window elements 0..63, 64..127 and 128..167 (and zeros) of a stage are blocks of their own; the second tile of 128 pairs the
  // third block with one of zeros, a fixed distance behind it.
  uint8_t* third = smem;                                      // [2]
  uint8_t* zeros = third + 2 * kBlock;
  uint8_t* pairs = zeros + kBlock;                            // [2][2]
  uint8_t* sD = pairs + 4 * kBlock;                           // dy [2]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sD + 2 * kBlock);
  uint64_t *cfull = bars + 4, *empty = bars + 6, *yfull = bars + 8, *done = bars + 10;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 11);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const Bands bands{reinterpret_cast<uint8_t*>(bars + 12), bars, bars + 2};
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bands.full[i], 1);
      mbar_init(&bands.empty[i], 8);
      mbar_init(&cfull[i], 4);
      mbar_init(&empty[i], 1);
      mbar_init(&yfull[i], 1);
    }
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&p.tmDY);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 128);
    tmem_relinquish();
  }
  bands.clear(s);
  for (int i = threadIdx.x; i < 7 * kBlock / 16; i += kWgThreads) reinterpret_cast<uint4*>(smem)[i] = make_uint4(0, 0, 0, 0);
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  esgd::pdl_enter();
  const int total = ((s.bands - 1 - (int)blockIdx.x) / (int)gridDim.x + 1) * s.tiles;

  if (warp == 0) {
    if (elect_one()) {
      bool ok = bands.load(s, p.x, blockIdx.x, 0, abort_flag);
      int it = 0, k = 0;
      for (int band = blockIdx.x; ok && band < s.bands; band += gridDim.x, ++k) {
        if (band + (int)gridDim.x < s.bands) ok = bands.load(s, p.x, band + gridDim.x, k + 1, abort_flag);      // one ahead
        for (int j = 0; ok && j < s.tiles; ++j, ++it) {
          ok = mbar_wait(&empty[it & 1], ((uint32_t)(it >> 1) & 1u) ^ 1u, abort_flag);
          if (!ok) break;
          mbar_expect_tx(&yfull[it & 1], kBlock);
          tma_load_4d(sD + (it & 1) * kBlock, &p.tmDY, &yfull[it & 1], 0, j * 128, band, 0);                    // zeros past the band
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(128, kOut, 1, 1);
      bool ok = true;
      for (int it = 0; ok && it < total; ++it) {
        const int st = it & 1;
        ok = mbar_wait(&yfull[st], (uint32_t)(it >> 1) & 1u, abort_flag) && mbar_wait(&cfull[st], (uint32_t)(it >> 1) & 1u, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint64_t b = umma_smem_desc(smem_u32(sD + st * kBlock), kBlock, 1024);
        const uint64_t a0 = umma_smem_desc(smem_u32(pairs + st * 2 * kBlock), kBlock, 1024);
        const uint64_t a1 = umma_smem_desc(smem_u32(third + st * kBlock), (uint32_t)((2 - st) * kBlock), 1024);
#pragma unroll
        for (int j = 0; j < 8; ++j) {                         // 16 pixels: 16 rows of 128 bytes
          umma_bf16(tmem, a0 + j * 128, b + j * 128, idesc, it > 0 || j > 0 ? 1u : 0u);
          umma_bf16(tmem + kOut, a1 + j * 128, b + j * 128, idesc, it > 0 || j > 0 ? 1u : 0u);
        }
        umma_commit(&empty[st]);
      }
      if (ok) umma_commit(done);
    }
  } else if (warp >= 4) {
    const int set = (warp - 4) >> 2, q = warp & 3, px = q * 32 + lane;
    uint8_t* b01 = pairs + set * 2 * kBlock + px * 128;
    uint8_t* b2 = third + set * kBlock + px * 128;
    bool ok = true;
    int it = 0, k = 0;
    for (int band = blockIdx.x; ok && band < s.bands; band += gridDim.x, ++k) {
      ok = __all_sync(0xffffffffu, mbar_wait(&bands.full[k & 1], (uint32_t)(k >> 1) & 1u, abort_flag));
      for (int j = 0; ok && j < s.tiles; ++j, ++it) {
        if ((it & 1) != set) continue;
        const Window w(s, bands, band, k, j * 128 + px);
        ok = __all_sync(0xffffffffu, mbar_wait(&empty[set], ((uint32_t)(it >> 1) & 1u) ^ 1u, abort_flag));
        if (!ok) break;
#pragma unroll
        for (int r = 0; r < kR; ++r) {
          uint32_t v[12];
          w.row(r, v);
#pragma unroll
          for (int c = 0; c < 3; ++c) {                       // chunk of eight elements
            const int chunk = 3 * r + c, block = chunk >> 3;
            uint8_t* to = block < 2 ? b01 + block * kBlock : b2;
            *reinterpret_cast<uint4*>(to + (((chunk & 7) ^ (px & 7)) << 4)) = make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
          }
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&cfull[set]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&bands.empty[k & 1]);
    }
    // the sums: window element (lane of tensor memory) x output channel -> [channel][168] of shared memory, then to col
    ok = __all_sync(0xffffffffu, ok && mbar_wait(done, 0u, abort_flag));
    float* bank = reinterpret_cast<float*>(pairs);
    if (ok) {
      tc_fence_after();
      const int tile = set, elem = tile * 128 + px;           // the first four warps have elements 0..127, the others 128..167
      if (tile == 0 || q * 32 < kK - 128) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(tile * kOut + half * 32), r);
          tmem_ld_wait();
          if (elem < kK) {
#pragma unroll
            for (int i = 0; i < 32; ++i) bank[(half * 32 + i) * kK + elem] = __uint_as_float(r[i]);
          }
        }
        tc_fence_before();
      }
      fence_proxy_async();
    }
    named_barrier_sync(1, 256);
    const int co = (int)threadIdx.x - 4 * 32;
    if (ok && co < kOut) {
      asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(p.col + (int64_t)co * p.kpad),
                   "r"(smem_u32(bank + co * kK)), "r"((uint32_t)(kK * 4)) : "memory");
      asm volatile("cp.async.bulk.commit_group;\n\tcp.async.bulk.wait_group 0;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    __nanosleep(1000000);
    if (threadIdx.x == 0 && p.error_flag != nullptr) atomicExch(p.error_flag, 1);
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 128);
  }
}

int fwd_smem(const StemShape& s) { return 3 * 8192 + kGroups * kPanel + 1024 + 18 * 8 + Bands::bytes(s); }
int wgrad_smem(const StemShape& s) { return 9 * kBlock + 12 * 8 + Bands::bytes(s); }

// Which images: rows of whole 16 bytes (copied as they are), whole bands, and at most 320 pixels in a row (shared memory of the
// weight gradient, the larger of the two).  -100: not these.
int shape(StemShape& s, const void* x, int N, int H, int W, int C, int Cout, int R, int S, int stride, int pad, int kpad) {
  if (N < 1 || C != 3 || Cout != kOut || R != kR || S != 7 || stride != 2 || pad != 3 || H < 16 || W < 8 || H % 16 || W % 8 ||
      kpad < 192 || kpad % 8 || ((uintptr_t)x & 15)) return -100;
  s.N = N; s.H = H; s.W = W;
  s.Ho = H / 2;
  s.Wo = W / 2;
  if ((int64_t)N * s.Ho >= (int64_t)1 << 30) return -100;
  s.pitch = 6 * W + 48;                       // both margins
  s.band = 8;
  s.rows = 2 * 8 + 5;
  if (wgrad_smem(s) > kSmemLimit) return -100;
  // Bands of two rows give every SM some from few images on; bands of eight bring fewer rows twice (21 for 16, 9 for 4).  Forward with
  // statistics, two rows and eight: 5.0 and 8.5 us for one image of 224 x 224, 11 and 13.5 for eleven, 33 and 29 for 48, 43 and 39 for
  // 64, 162 and 134 for 256.  The line is where eight rows have stopped losing to rounds that are not full.
  if (N * s.Ho / 8 < 6 * esgd::sm_count()) {
    s.band = 2;
    s.rows = 2 * 2 + 5;
  }
  s.per_image = s.Ho / s.band;
  s.bands = N * s.per_image;
  s.pixels = s.band * s.Wo;
  s.tiles = (s.pixels + 127) / 128;
  return 0;
}

int map_of(CUtensorMap* tm, const void* t, const StemShape& s) {
  uint64_t dims[4] = {kOut, (uint64_t)s.pixels, (uint64_t)s.bands, 1};
  uint64_t strides[3] = {kOut * 2, (uint64_t)s.pixels * kOut * 2, (uint64_t)s.bands * s.pixels * kOut * 2};
  uint32_t box[4] = {kOut, 128, 1, 1};
  return esgd::make_tensormap_bf16(tm, t, 4, dims, strides, box, nullptr);
}

}  // namespace

extern "C" {

// y [N,H/2,W/2,64] = act(scale * conv(x, w) + shift), x [N,H,W,3] bf16, w2d the filters as esgd_stem_pack leaves them (rows of Kpad >=
// 192 elements); sum / sqsum (optional, zeroed) receive y's statistics, keep
// (optional) a copy of x.  -100: a shape that this file does not take.
int esgd_stem_fwd(const void* x, const void* w2d, void* y, void* keep, int N, int H, int W, int C, int Cout, int R, int S, int stride, int pad, int kpad,
                  const float* scale, const float* shift, int relu, float* sum, float* sqsum, int* error_flag, void* stream) {
  StemFwd p;
  int rc = shape(p.s, x, N, H, W, C, Cout, R, S, stride, pad, kpad);
  if (rc != 0) return rc;
  uint64_t dims[2] = {(uint64_t)kpad, kOut}, strides[1] = {(uint64_t)kpad * 2};
  uint32_t box[2] = {64, kOut};
  if ((rc = esgd::make_tensormap_bf16(&p.tmW, w2d, 2, dims, strides, box, nullptr)) != 0) return 1000 + rc;
  if ((rc = map_of(&p.tmY, y, p.s)) != 0) return 2000 + rc;
  p.x = (const __nv_bfloat16*)x;
  p.keep = (__nv_bfloat16*)keep;
  p.scale = scale; p.shift = shift; p.relu = relu; p.sum = sum; p.sqsum = sqsum; p.error_flag = error_flag;
  static esgd::SmemAllowed allowed{0};
  if ((rc = esgd::allow_smem(stem_fwd_kernel, kSmemLimit, allowed)) != 0) return rc;
  const int sms = esgd::sm_count();
  return esgd::launch(stem_fwd_kernel, dim3(p.s.bands < sms ? p.s.bands : sms), kFwdThreads, fwd_smem(p.s), stream, p);
}

// col [64][kpad] fp32 (in the packed filters' layout) += the filter gradient.
int esgd_stem_wgrad(const void* x, const void* dy, float* col, int N, int H, int W, int C, int Cout, int R, int S, int stride, int pad, int kpad,
                    int* error_flag, void* stream) {
  StemWgrad p;
  int rc = shape(p.s, x, N, H, W, C, Cout, R, S, stride, pad, kpad);
  if (rc != 0) return rc;
  if ((rc = map_of(&p.tmDY, dy, p.s)) != 0) return 1000 + rc;
  p.x = (const __nv_bfloat16*)x;
  p.col = col; p.kpad = kpad; p.error_flag = error_flag;
  static esgd::SmemAllowed allowed{0};
  if ((rc = esgd::allow_smem(stem_wgrad_kernel, kSmemLimit, allowed)) != 0) return rc;
  const int sms = esgd::sm_count();
  return esgd::launch(stem_wgrad_kernel, dim3(p.s.bands < sms ? p.s.bands : sms), kWgThreads, wgrad_smem(p.s), stream, p);
}

}  // extern "C"
