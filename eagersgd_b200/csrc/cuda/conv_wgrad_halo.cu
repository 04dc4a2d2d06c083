// Weight gradient of stride-1 convolutions with shared input boxes (sm_100a, tcgen05 / TMEM / TMA).
//
//   dw[k, r, s, c] = sum over output pixels p of dy[p, k] * x[p + (r, s) - pad, c]
//
// The per-tap kernel (conv_tcgen05.cu) loads a dy box and an x box for every (tap, 64-pixel block): the
// activations cross L2 -> SM once per tap.  Here a CTA owns a SET of taps (accumulators of their own in tensor memory; how many is
// wg_plan's choice) and, for every block of full output rows, loads ONE dy box and ONE x box (the rows plus
// the filter margin); the taps are shifted views of the x box, exactly as in the forward halo mode: both boxes
// are indexed by the x box's pixel pitch PW = Wo + S - 1, dy's margin columns are zero-filled by TMA, and tap
// (r, s) reads x (r * PW + s) rows further on.  Both operands are MN-major (the pixel is the K index), the
// accumulators stay in tensor memory over the CTA's whole pixel range and are added to dw in fp32 at the end.
// Layers of 64 channels have a kernel that takes all nine taps at once (conv_wgrad_packed_kernel).
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>
#include "launch.cuh"
#include "sm100_primitives.cuh"
#include "tensormap.cuh"

using namespace sm100;

namespace {

constexpr int WG_THREADS = 192;       // warp 0: TMA, warp 1: MMA issue, warps 2-5: epilogue
constexpr int WG_SMEM = 226 * 1024;

struct WgHaloParams {
  CUtensorMap tmDY, tmX;
  int N, Ho, Wo, Cout, Cin, R, S, pad;
  int BH, PW, h_tiles;                 // output rows per box, pixel pitch, boxes per image
  int ksteps;                          // ceil(BH * PW / 16)
  int abox, xbox;                      // bytes of one 64-channel atom of the dy / x box (multiples of 1024)
  int nstages;
  int sets, taps_per_set, m_tiles, n_tiles, splits, boxes_total, boxes_per_split;
  float* dw;                           // [Cout][R*S][Cin] fp32
  int* error_flag;
};

// Sums of a tap on their way out: 128 rows of an odd number of 16 bytes (no bank conflicts).
__host__ __device__ constexpr int wg_bank_bytes(int BN) { return 128 * (BN * 4 + 16); }

template <int BN>
__global__ void __launch_bounds__(WG_THREADS, 1) conv_wgrad_halo_kernel(const __grid_constant__ WgHaloParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int NA = 2, NB = BN / 64;                  // 64-channel atoms of the dy (128 rows) and x operands
  const int stage_bytes = NA * p.abox + NB * p.xbox;
  constexpr int kBank = wg_bank_bytes(BN), kPitch = kBank / 128;     // sums on their way out
  uint8_t* bar_area = smem + max(p.nstages * stage_bytes, kBank);
  uint64_t* full = reinterpret_cast<uint64_t*>(bar_area);
  uint64_t* empty = full + 4;
  uint64_t* done = empty + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

  // work item of this CTA
  int id = blockIdx.x;
  const int set = id % p.sets; id /= p.sets;
  const int n_idx = id % p.n_tiles; id /= p.n_tiles;
  const int m_idx = id % p.m_tiles; id /= p.m_tiles;
  const int split = id;
  const int tap0 = set * p.taps_per_set;
  const int ntaps = min(p.taps_per_set, p.R * p.S - tap0);
  const int box0 = split * p.boxes_per_split;
  const int box1 = min(box0 + p.boxes_per_split, p.boxes_total);
  const int m0 = m_idx * 128, n0 = n_idx * BN;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.nstages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&p.tmDY);
    tma_prefetch_desc(&p.tmX);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  {
    // Rows the boxes do not cover are read as K padding (dy) or by the most shifted views (x): they must hold
    // zeros (dy) or at least finite values (x) for ever, so the stages start out cleared.
    uint4* p4 = reinterpret_cast<uint4*>(smem);
    const int n16 = p.nstages * stage_bytes / 16;
    for (int i = threadIdx.x; i < n16; i += WG_THREADS) p4[i] = make_uint4(0, 0, 0, 0);
    fence_proxy_async();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  esgd::pdl_enter();

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      const int na = min(NA, (p.Cout - m0 + 63) / 64);     // atoms of dy that hold channels; the other stays zero
      const uint32_t tx = (uint32_t)(na * p.BH * p.PW * 128 + NB * (p.BH + p.R - 1) * p.PW * 128);
      for (int b = box0; b < box1; ++b) {
        if (!mbar_wait(&empty[stage], phase ^ 1u, abort_flag)) break;
        const int h0 = (b % p.h_tiles) * p.BH, n = b / p.h_tiles;
        uint8_t* sa = smem + stage * stage_bytes;
        uint8_t* sb = sa + NA * p.abox;
        mbar_expect_tx(&full[stage], tx);
#pragma unroll
        for (int i = 0; i < NA; ++i)
          if (i < na) tma_load_4d(sa + i * p.abox, &p.tmDY, &full[stage], m0 + 64 * i, 0, h0, n);
#pragma unroll
        for (int i = 0; i < NB; ++i)
          tma_load_4d(sb + i * p.xbox, &p.tmX, &full[stage], n0 + 64 * i, -p.pad, h0 - p.pad, n);
        if (++stage == p.nstages) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(128, min(BN, (p.Cin - n0 + 15) / 16 * 16), 1, 1);
      int stage = 0;
      uint32_t phase = 0;
      uint32_t accumulate = 0;
      bool ok = true;
      constexpr uint64_t kstep = 2048 >> 4;                      // 16 pixel rows
      // The issuing lane has nothing to hide its own instruction latency behind, so the loop below is fully
      // unrolled over (tap, K step) with compile-time offsets; the taps' view offsets are computed once.
      constexpr int MAXT = 512 / BN;                             // accumulators that fit in tensor memory
      uint64_t view_off[MAXT];
#pragma unroll
      for (int tl = 0; tl < MAXT; ++tl) {
        const int tap = tap0 + (tl < ntaps ? tl : 0);
        const int r = tap / p.S, s = tap - r * p.S;
        view_off[tl] = (uint64_t)((r * p.PW + s) * 8);           // (r * PW + s) rows of 128 bytes, in 16-byte units
      }
      const int ksteps = p.ksteps;                               // <= 8: a box has at most 128 pixel rows
      for (int b = box0; ok && b < box1; ++b) {
        if (!mbar_wait(&full[stage], phase, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t sa = smem_u32(smem + stage * stage_bytes);
        const uint64_t a_desc = umma_smem_desc(sa, (uint32_t)p.abox, 1024);
        const uint64_t b_desc0 = umma_smem_desc(sa + NA * p.abox, (uint32_t)p.xbox, 1024);
#pragma unroll
        for (int tl = 0; tl < MAXT; ++tl) {
          if (tl < ntaps) {
            const uint64_t b_desc = b_desc0 + view_off[tl];
            const uint32_t d = tmem_base + (uint32_t)(tl * BN);
            umma_bf16(d, a_desc, b_desc, idesc, accumulate);
#pragma unroll
            for (int ks = 1; ks < 8; ++ks)
              if (ks < ksteps) umma_bf16(d, a_desc + ks * kstep, b_desc + ks * kstep, idesc, 1u);
          }
        }
        accumulate = 1;
        umma_commit(&empty[stage]);
        if (++stage == p.nstages) { stage = 0; phase ^= 1u; }
      }
      umma_commit(done);
    }
  } else {
    // ---- epilogue: once, after the CTA's whole pixel range.  A tap's sums go to shared memory, then a bulk reduction for each output
    // channel; rows of 64 channels are short for that, and a reduction of 16 bytes for each thread and four columns is quicker
    // (16 bytes at a time and in bulk: 64 x 28 x 28 x 128 20.5 and 18.3 us, 64 x 7 x 7 x 512 20.9 and 19.0, 128 x 8 x 8 x 64 5.3 and 6.0).
    const int q = warp & 3, row = q * 32 + lane, banks = 2 * kBank <= p.nstages * stage_bytes ? 2 : 1;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(done, 0u, abort_flag)) && box1 > box0;
    const int out = ((int)threadIdx.x - 64 + split * 37) & 127;      // the CTAs of a range meet on different lines
    if (ok) tc_fence_after();
    if (BN == 64 && ok) {
      const int k = m0 + row;
      for (int tl = 0; tl < ntaps; ++tl) {
        float* to = k < p.Cout ? p.dw + ((size_t)k * (p.R * p.S) + tap0 + tl) * p.Cin : nullptr;
#pragma unroll 1
        for (int c = 0; c < BN / 32; ++c) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(tl * BN + c * 32), v);
          tmem_ld_wait();
          const int col0 = n0 + c * 32;
          if (to != nullptr) {
#pragma unroll
            for (int j = 0; j < 32; j += 4)
              if (col0 + j < p.Cin)
                atomicAdd(reinterpret_cast<float4*>(to + col0 + j),
                          make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3])));
          }
        }
      }
    }
    for (int tl = 0; BN > 64 && tl < ntaps; ++tl) {
      uint8_t* bank = smem + (tl & (banks - 1)) * kBank;
      if (tl >= banks) {
        if (banks == 2) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        else asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        named_barrier_sync(1, 128);
      }
      if (ok) {
#pragma unroll 1
        for (int c = 0; c < BN / 32; ++c) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(tl * BN + c * 32), v);
          tmem_ld_wait();
          float4* to = reinterpret_cast<float4*>(bank + row * kPitch + c * 128);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            to[j] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
        }
        fence_proxy_async();
      }
      named_barrier_sync(1, 128);
      if (ok && m0 + out < p.Cout)
        asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(
                         p.dw + ((size_t)(m0 + out) * (p.R * p.S) + tap0 + tl) * p.Cin + n0),
                     "r"(smem_u32(bank + out * kPitch)), "r"((uint32_t)(min(BN, p.Cin - n0) * 4)) : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    tc_fence_before();
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    __nanosleep(1000000);
    if (threadIdx.x == 0 && p.error_flag != nullptr) atomicExch(p.error_flag, 1);
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// 3x3 layers of 64 input and at most 64 output channels, all nine taps in one CTA and two products a K step.  A product of 128 x 64 is
// bound by the bytes it reads from shared memory (49 cycles where 32 would do), and of its 128 rows such a layer fills 64.  So
// the rows are output channels of two taps, dy and dy one pixel earlier (blocks of 64 rows 128 bytes apart):
//   sum over p of dy[p] x[p + r PW + 1]  =  sum over q of dy[q - 1] x[q + r PW],
// and the columns are three blocks of 64, x one box row of pixels apart: taps (0..2, 0..1) in one product of 128 x 192, taps (0..2, 2)
// in another (its lower rows are not used).  193 cycles a K step where taps one by one took 441, and dy and x are read once.
// The sums leave by way of shared memory, a bulk reduction for each output channel.
constexpr int kPackedLead = 1024;             // zeros in front of dy: the pixel before the first
constexpr int kPackedPitch = 9 * 64 + 4;      // floats of an output channel's sums (an odd number of 16 bytes: no bank conflicts)
constexpr int kPackedBank = 64 * kPackedPitch * 4;

__global__ void __launch_bounds__(WG_THREADS, 1) conv_wgrad_packed_kernel(const __grid_constant__ WgHaloParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int stage_bytes = p.abox + p.xbox;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + max(p.nstages * stage_bytes, kPackedBank));
  uint64_t* empty = full + 4;
  uint64_t* done = empty + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int box0 = blockIdx.x * p.boxes_per_split, box1 = min(box0 + p.boxes_per_split, p.boxes_total);

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.nstages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&p.tmDY);
    tma_prefetch_desc(&p.tmX);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  {
    // what the boxes do not cover reads as zeros (dy: the pixel in front, K padding) or as finite values (x) for ever
    uint4* p4 = reinterpret_cast<uint4*>(smem);
    for (int i = threadIdx.x; i < p.nstages * stage_bytes / 16; i += WG_THREADS) p4[i] = make_uint4(0, 0, 0, 0);
    fence_proxy_async();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  esgd::pdl_enter();

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      int n = box0 / p.h_tiles, h = box0 - n * p.h_tiles;
      for (int b = box0; b < box1; ++b) {
        if (!mbar_wait(&empty[stage], phase ^ 1u, abort_flag)) break;
        uint8_t* sa = smem + stage * stage_bytes;
        mbar_expect_tx(&full[stage], (uint32_t)((2 * p.BH + 2) * p.PW * 128));
        tma_load_4d(sa + kPackedLead, &p.tmDY, &full[stage], 0, 0, h * p.BH, n);
        tma_load_4d(sa + p.abox, &p.tmX, &full[stage], 0, -p.pad, h * p.BH - p.pad, n);
        if (++h == p.h_tiles) { h = 0; ++n; }
        if (++stage == p.nstages) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(128, 192, 1, 1);
      int stage = 0;
      uint32_t phase = 0, accumulate = 0;
      bool ok = true;
      constexpr uint64_t kstep = 2048 >> 4;                      // 16 pixel rows
      const int ksteps = p.ksteps;                               // <= 8
      for (int b = box0; ok && b < box1; ++b) {
        if (!mbar_wait(&full[stage], phase, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t sa = smem_u32(smem + stage * stage_bytes);
        const uint64_t a0 = umma_smem_desc(sa + kPackedLead - 128, 128, 1024), a1 = a0 + 8;      // one pixel further on
        const uint64_t x0 = umma_smem_desc(sa + p.abox, (uint32_t)(p.PW * 128), 1024), x1 = x0 + 16;   // two pixels further on
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          if (ks < ksteps) {
            umma_bf16(tmem_base, a0 + ks * kstep, x0 + ks * kstep, idesc, ks > 0 ? 1u : accumulate);
            umma_bf16(tmem_base + 192, a1 + ks * kstep, x1 + ks * kstep, idesc, ks > 0 ? 1u : accumulate);
          }
        accumulate = 1;
        umma_commit(&empty[stage]);
        if (++stage == p.nstages) { stage = 0; phase ^= 1u; }
      }
      if (ok) umma_commit(done);
    }
  } else {
    // ---- epilogue: once, after the CTA's whole pixel range
    const int q = warp & 3;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(done, 0u, abort_flag)) && box1 > box0;
    float* bank = reinterpret_cast<float*>(smem);
    if (ok) {
      tc_fence_after();
      float* row = bank + ((q & 1) * 32 + lane) * kPackedPitch;
      for (int part = 0; part < (q < 2 ? 2 : 1); ++part) {       // the second product has its rows in the first half alone
        const int s = part == 1 ? 2 : q < 2 ? 1 : 0;
#pragma unroll 1
        for (int c = 0; c < 6; ++c) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(part * 192 + c * 32), v);
          tmem_ld_wait();
          float4* to = reinterpret_cast<float4*>(row + ((c >> 1) * 3 + s) * 64 + (c & 1) * 32);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            to[j] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
        }
      }
      tc_fence_before();
      fence_proxy_async();
    }
    named_barrier_sync(1, 128);
    const int k0 = (int)threadIdx.x - 64;
    if (ok && k0 < p.Cout) {
      // CTAs start with different channels: they would meet on the same lines
      const int k = (int)((k0 + blockIdx.x * 7) % p.Cout);
      asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(p.dw + (size_t)k * 576),
                   "r"(smem_u32(bank + k * kPackedPitch)), "r"(576u * 4u) : "memory");
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
    tmem_dealloc(tmem_base, 512);
  }
}

// Geometry of a launch (host arithmetic only, shared by the launcher and by the plan query that the CPU tests
// sweep): box sizes, stages, tap sets, pixel splits.  Returns -7 when two stages do not fit.
int wg_plan(WgHaloParams& p, int BN, int N, int H, int W, int Cin, int Cout, int R, int S, int pad, int bh, int sms, double* cost_out = nullptr) {
  p.N = N; p.Cout = Cout; p.Cin = Cin; p.R = R; p.S = S; p.pad = pad;
  p.Ho = H + 2 * pad - R + 1;
  p.Wo = W + 2 * pad - S + 1;
  p.BH = bh;
  p.PW = p.Wo + S - 1;
  p.h_tiles = p.Ho / bh;
  p.ksteps = (bh * p.PW + 15) / 16;
  const int off_max = (R - 1) * p.PW + (S - 1);
  p.abox = (p.ksteps * 16 * 128 + 1023) / 1024 * 1024;
  p.xbox = ((p.ksteps * 16 + off_max) * 128 + 1023) / 1024 * 1024;
  const int stage_bytes = 2 * p.abox + (BN / 64) * p.xbox;
  p.nstages = (WG_SMEM - 1024 - 256) / stage_bytes;
  if (p.nstages > 4) p.nstages = 4;
  if (p.nstages < 2) return -7;
  p.m_tiles = (Cout + 127) / 128;
  p.n_tiles = (Cin + BN - 1) / BN;
  p.boxes_total = p.h_tiles * N;
  // One wave of CTAs; taps of a CTA by what they cost.  Many taps share the boxes they read; few leave fewer pixel ranges, whose sums
  // meet in L2.  A box takes its loads (50 bytes a cycle and SM) or its products (49, 65, 129 cycles for 64, 128, 256 columns),
  // sums 900 bytes a cycle of the chip (in bulk 1800).  Measured with 1, 2, 3 and 5 taps, 5 the most that fit (it was that, in two waves of CTAs:
  // 15.1, 42, 124 us): 128 x 8 x 8 x 64 5.4, 6.3, 7.8, 9.8 us; 64 x 56 x 56 x 64 40, 33, 32, 36; 256 images of these 199, 121, 109,
  // 116.  With 1 and 2 taps (2 in two waves: 45 and 85 us): 64 x 7 x 7 x 512 19.8 and 26.5, 256 images 53 and 69.
  const int most = 512 / BN < R * S ? 512 / BN : R * S, per_mma = BN == 64 ? 49 : BN + 1;
  const int box_bytes = ((Cout < 128 ? (Cout + 63) / 64 : 2) * bh + BN / 64 * (bh + R - 1)) * p.PW * 128;
  double best = 0.0;
  for (int n = 1; n <= most; ++n) {
    const int sets = (R * S + n - 1) / n, taps = (R * S + sets - 1) / sets;      // balanced (9 taps: 5 + 4, or 3 + 3 + 3)
    const int base = sets * p.m_tiles * p.n_tiles;
    int splits = sms / base;
    if (splits > p.boxes_total) splits = p.boxes_total;
    if (splits < 1) splits = 1;
    const int boxes = (p.boxes_total + splits - 1) / splits, products = taps * p.ksteps * per_mma;
    splits = (p.boxes_total + boxes - 1) / boxes;
    const double cost = (double)((base * splits + sms - 1) / sms) * boxes * (products > box_bytes / 50 ? products : box_bytes / 50) +
                        (double)base * splits * taps * BN * (Cout < 128 ? Cout : 128) * 4 / (BN == 64 ? 900 : 1800);
    if (n > 1 && cost >= best) continue;
    best = cost;
    p.sets = sets;
    p.taps_per_set = taps;
    p.boxes_per_split = boxes;
    p.splits = splits;
  }
  if (cost_out != nullptr) *cost_out = best;
  return 0;
}

// The packed kernel's geometry and what it costs, in the terms of wg_plan (bulk reductions: 1400 bytes a cycle); false: not its shape.
// 64 channels, taps one by one and packed: 4 x 56 x 56 6.3 and 9.3 us, 8 images 8.3 and 10.5, 16 13.3 and 12.5, 64 32 and 21, 256 108 and
// 62; 128 x 8 x 8 5.3 and 8.7, 2048 x 8 x 8 33 and 17, 1024 x 16 x 16 59 and 24.  The model draws the line between 8 and 16, 512 and 2048.
bool wg_packed_plan(WgHaloParams& p, int Cin, int Cout, int R, int S, int sms, double* cost) {
  if (R != 3 || S != 3 || Cin != 64 || Cout > 64) return false;
  p.abox = kPackedLead + (p.ksteps * 16 + 1) * 128;
  p.abox = (p.abox + 1023) / 1024 * 1024;
  p.nstages = (WG_SMEM - 1024 - 256) / (p.abox + p.xbox);
  if (p.nstages > 4) p.nstages = 4;
  if (p.nstages < 2) return false;
  p.splits = sms < p.boxes_total ? sms : p.boxes_total;
  p.boxes_per_split = (p.boxes_total + p.splits - 1) / p.splits;
  p.splits = (p.boxes_total + p.boxes_per_split - 1) / p.boxes_per_split;
  const int box_bytes = (2 * p.BH + 2) * p.PW * 128, products = p.ksteps * 2 * 97;
  *cost = (double)p.boxes_per_split * (products > box_bytes / 50 ? products : box_bytes / 50) + (double)p.splits * kPackedBank / 1400;
  return true;
}

// What a launch will be; -7 as wg_plan.  aligned16: dw is a multiple of 16 bytes (the packed kernel's bulk reductions need it).
int wg_choose(WgHaloParams& p, bool& packed, int BN, int N, int H, int W, int Cin, int Cout, int R, int S, int pad, int bh, int sms, bool aligned16) {
  double cost = 0.0, packed_cost = 0.0;
  const int rc = wg_plan(p, BN, N, H, W, Cin, Cout, R, S, pad, bh, sms, &cost);
  packed = false;
  if (rc != 0 || BN != 64 || !aligned16) return rc;
  WgHaloParams q = p;
  if (wg_packed_plan(q, Cin, Cout, R, S, sms, &packed_cost) && packed_cost < cost) {
    p = q;
    packed = true;
  }
  return 0;
}

// Input channels of a tile.  128 leave room for the sums of four taps, 256 for two.  128 and 256: 8 x 14 x 14 x 256 6.7 and 8.7 us, 64
// images 18.0 and 19.3, 256 images 45.5 and 53.6; but 64 x 7 x 7 x 512, whose boxes are small, 24.5 and 20.0, 256 images 68 and 53.
int columns(int Cin) { return Cin <= 64 ? 64 : (Cin <= 256 ? 128 : 256); }

// Largest number of full output rows whose pitched pixels fit one 128-row K range; 0: outside this kernel's range.
int wg_pick_bh(int H, int W, int Cin, int Cout, int R, int S, int pad) {
  if (Cin % 8 || Cout % 8 || R * S < 2) return 0;
  const int Ho = H + 2 * pad - R + 1, Wo = W + 2 * pad - S + 1;
  const int PW = Wo + S - 1;
  if (Ho < 1 || Wo < 1 || PW > 128) return 0;
  int bh = 0;
  for (int d = 1; d * PW <= 128 && d <= Ho; ++d) if (Ho % d == 0) bh = d;
  if (bh == 0 || bh * Wo < 48) return 0;
  if (bh + R - 1 > 256) return 0;
  return bh;
}

template <int BN>
int launch_wgrad_halo(const void* x, const void* dy, float* dw, int N, int H, int W, int Cin, int Cout, int R, int S,
                      int pad, int bh, int* error_flag, cudaStream_t stream) {
  static esgd::SmemAllowed allowed{0};
  if (const int e = esgd::allow_smem(conv_wgrad_halo_kernel<BN>, WG_SMEM, allowed)) return e;
  WgHaloParams p;
  bool packed = false;
  const int pr = wg_choose(p, packed, BN, N, H, W, Cin, Cout, R, S, pad, bh, esgd::sm_count(), ((uintptr_t)dw & 15) == 0);
  if (pr != 0) return pr;
  p.dw = dw;
  p.error_flag = error_flag;
  {
    uint64_t dims[4] = {(uint64_t)Cout, (uint64_t)p.Wo, (uint64_t)p.Ho, (uint64_t)N};
    uint64_t strides[3] = {(uint64_t)Cout * 2, (uint64_t)p.Wo * Cout * 2, (uint64_t)p.Ho * p.Wo * Cout * 2};
    uint32_t box[4] = {64, (uint32_t)p.PW, (uint32_t)bh, 1};
    int r = esgd::make_tensormap_bf16(&p.tmDY, dy, 4, dims, strides, box, nullptr);
    if (r != 0) return 1000 + r;
  }
  {
    uint64_t dims[4] = {(uint64_t)Cin, (uint64_t)W, (uint64_t)H, (uint64_t)N};
    uint64_t strides[3] = {(uint64_t)Cin * 2, (uint64_t)W * Cin * 2, (uint64_t)H * W * Cin * 2};
    uint32_t box[4] = {64, (uint32_t)p.PW, (uint32_t)(bh + R - 1), 1};
    int r = esgd::make_tensormap_bf16(&p.tmX, x, 4, dims, strides, box, nullptr);
    if (r != 0) return 2000 + r;
  }
  if (packed) {
    static esgd::SmemAllowed packed_allowed{0};
    if (const int e = esgd::allow_smem(conv_wgrad_packed_kernel, WG_SMEM, packed_allowed)) return e;
    return esgd::launch(conv_wgrad_packed_kernel, dim3(p.splits), WG_THREADS, WG_SMEM, stream, p);
  }
  const int grid = p.sets * p.m_tiles * p.n_tiles * p.splits;
  return esgd::launch(conv_wgrad_halo_kernel<BN>, dim3(grid), WG_THREADS, WG_SMEM, stream, p);
}

}  // namespace

extern "C" {

// Returns -100 when the shape is outside this kernel's range (the caller then uses the per-tap kernel).
// dw: fp32 [Cout][R][S][Cin], zeroed by the caller.  Stride 1 only; Cin % 8 == 0, Cout % 8 == 0.
int esgd_conv2d_wgrad_halo(const void* x, const void* dy, float* dw, int N, int H, int W, int Cin, int Cout, int R,
                           int S, int pad, int* error_flag, void* stream) {
  {
    const char* e = getenv("ESGD_CONV_HALO");          // the same switch as the forward halo mode
    if (e != nullptr && e[0] == '0') return -100;
  }
  const int bh = wg_pick_bh(H, W, Cin, Cout, R, S, pad);
  if (bh == 0) return -100;
  cudaStream_t s = (cudaStream_t)stream;
  int rc;
  if (columns(Cin) == 64) rc = launch_wgrad_halo<64>(x, dy, dw, N, H, W, Cin, Cout, R, S, pad, bh, error_flag, s);
  else if (columns(Cin) == 128) rc = launch_wgrad_halo<128>(x, dy, dw, N, H, W, Cin, Cout, R, S, pad, bh, error_flag, s);
  else rc = launch_wgrad_halo<256>(x, dy, dw, N, H, W, Cin, Cout, R, S, pad, bh, error_flag, s);
  return rc == -7 ? -100 : rc;          // boxes too large for two stages: the per-tap kernel takes the shape
}

// Host arithmetic of a launch without launching anything (no device needed).  out[0..11]: applicable (0/1), BH, PW,
// ksteps, abox, xbox, nstages, sets, taps_per_set, splits, boxes_per_split, grid; out[12] = BN, out[13] = shared
// memory requested, out[14] = m_tiles, out[15] = n_tiles; out[16]: 1 for the packed kernel (all nine taps, sets, m_tiles and n_tiles
// of 1), out[17]: bytes that the sums of a CTA take on their way out, where the stages were.
void esgd_conv2d_wgrad_halo_plan(int N, int H, int W, int Cin, int Cout, int R, int S, int pad, int sms, int* out) {
  for (int i = 0; i < 18; ++i) out[i] = 0;
  const int bh = wg_pick_bh(H, W, Cin, Cout, R, S, pad);
  if (bh == 0) return;
  const int BN = columns(Cin);
  WgHaloParams p;
  bool packed = false;
  if (wg_choose(p, packed, BN, N, H, W, Cin, Cout, R, S, pad, bh, sms, true) != 0) return;
  if (packed) {
    p.sets = p.m_tiles = p.n_tiles = 1;
    p.taps_per_set = 9;
  }
  out[0] = 1; out[1] = p.BH; out[2] = p.PW; out[3] = p.ksteps; out[4] = p.abox; out[5] = p.xbox; out[6] = p.nstages;
  out[7] = p.sets; out[8] = p.taps_per_set; out[9] = p.splits; out[10] = p.boxes_per_split;
  out[11] = p.sets * p.m_tiles * p.n_tiles * p.splits; out[12] = BN; out[13] = WG_SMEM; out[14] = p.m_tiles;
  out[15] = p.n_tiles; out[16] = packed; out[17] = packed ? kPackedBank : wg_bank_bytes(BN);
}

}  // extern "C"
