// Persistent warp-specialised tcgen05 pipeline shared by the GEMM and the
// implicit-GEMM convolution kernels.
//
//   warp 0     : TMA producer — the Problem policy issues the loads of one k-block
//   warp 1     : tcgen05.mma issuer (one elected thread); two TMEM accumulators of 256 columns or four narrower
//                ones, so that the epilogues of earlier tiles overlap the main loop of the next
//   warps 2..17: epilogue, four groups of four warps.  A unit of work is one 64-column panel of a tile: tcgen05.ld, affine
//                map / residual / ReLU, the panel staged in shared memory in the 128-byte-swizzled layout and written
//                with a TMA store (coalesced, clipped at the tensor edge); per-channel sum and sum of squares of the
//                stored panel are taken from shared memory and flushed with one atomic per column per CTA (batch-norm
//                statistics).  The groups work on different panels with barriers of their own: one group of eight warps
//                in lock step left the SM idle in every barrier and load it waited for (64-deep products with
//                statistics ran at half the speed of those without).  fp32 outputs leave the same way, 32 columns at a
//                time; split-K sums are TMA reductions (whole rows into L2 instead of one atomic per 16 bytes).
//
// B-resident mode: when a CTA keeps one column range for all of its tiles and the whole K
// extent of B for that range fits beside four A stages, B is loaded ONCE and stays in shared
// memory; the ring then carries A only (up to eight stages).  Short-K, long-M problems (1x1
// convolutions over early feature maps, 3x3 over 64 channels) otherwise re-read B from L2 for
// every tile, which is a quarter of their L2 traffic.
//
// A tile is 128 rows x BN columns; a k-block is 64 bf16 (one 128-byte swizzle row).
// Every mbarrier wait is bounded; on expiry the CTA raises an error flag, lets the
// copies in flight land, frees its tensor memory and returns.  A role that has given up still meets its group at the
// barriers, so nobody waits for it.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <stdlib.h>
#include "bn_grad.h"
#include "launch.cuh"
#include "sm100_primitives.cuh"

namespace umma {

using namespace sm100;

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int A_STAGE_BYTES = BM * BK * 2;   // 16 KB
constexpr int PANEL_BYTES = BM * 64 * 2;     // one 128 x 64 bf16 output panel
constexpr int NUM_GROUPS = 4;                // epilogue groups, each with a staging buffer of one panel
constexpr int GROUP_THREADS = 128;
constexpr int NUM_THREADS = 64 + NUM_GROUPS * GROUP_THREADS;

enum BiasKind { BIAS_F32 = 0, BIAS_BF16 = 1, BIAS_F32_UNALIGNED = 2 };
enum OutMode { OUT_BF16 = 0, OUT_F32 = 1, OUT_F32_ADD = 2 };

struct Epilogue {
  int out_mode;
  int relu;
  int n_total;             // number of valid output columns (channels)
  const float* scale;      // per column factor applied before the bias, may be null (needs a bias)
  const float* bias;       // per column, may be null
  int bias_kind;           // BIAS_F32 (16-byte aligned, like scale), BIAS_BF16 or BIAS_F32_UNALIGNED
  float* col_sum;          // optional per-column statistics of the stored bf16 values
  float* col_sqsum;
  int* error_flag;
  uint32_t tx_bytes;       // bytes the loads of one k-block deliver (0: full A and B stage tiles)
  uint32_t tx_bytes_a;     // bytes of the A loads alone (B-resident mode; 0: a full A stage tile)
  const void* residual;    // optional bf16 tensor added to the product before rounding (same shape as the output)
  int ldr;                 // its row stride in elements (GEMM)
  uint32_t res_bytes;      // bytes one panel of it delivers
  // Data gradients: the product is the gradient of z = act(batch_norm(bn_y)).  Elements whose bit in bn_mask is clear are
  // stored as zeros, and col_sum / col_sqsum receive dbeta and dgamma: sum g and sum g * (bn_y - mean) / std.
  const __nv_bfloat16* bn_y = nullptr;       // [rows][n_total], n_total a multiple of 64
  const uint8_t* bn_mask = nullptr;          // [rows][n_total / 8], null: no ReLU
  const float* bn_aux = nullptr;             // mean [n_total], 1 / std [n_total]
};

// False: the kernels do not take this many channels.
inline bool set_bn_grad(Epilogue& ep, const esgd_bn_grad* bn) {
  if (bn == nullptr) return true;
  if (ep.n_total % 64 || ((uintptr_t)bn->mask & 7) || ((uintptr_t)bn->aux & 7)) return false;
  ep.bn_y = (const __nv_bfloat16*)bn->y;
  ep.bn_mask = (const uint8_t*)bn->mask;
  ep.bn_aux = bn->aux;
  ep.col_sum = bn->sums;
  ep.col_sqsum = bn->sums + ep.n_total;
  return true;
}

template <int BN>
struct Cfg {
  static constexpr int B_STAGE_BYTES = BN * BK * 2;
  static constexpr int STAGES = BN == 256 ? 3 : (BN == 128 ? 5 : 6);             // with one panel per group
  static constexpr int ACCS = BN == 256 ? 2 : 4;       // accumulators in tensor memory: tiles in flight
  static constexpr int TMEM_COLS = ACCS * BN;
  static constexpr int PAIR_STAGES = 5;                // a pair's stage: 128 rows of A and half of B's columns in each CTA
  static constexpr int MAX_STAGES = 8;                 // A-only ring of the B-resident mode
  static constexpr int STAGE_AREA = 160 * 1024;        // operand stages (ring, or A ring + resident B)
  static constexpr int STAGE_AREA2 = STAGE_AREA - NUM_GROUPS * PANEL_BYTES;      // ... beside two panels per group
  static constexpr int AFFINE_BYTES = NUM_GROUPS * 2 * 64 * 4;                    // the groups' columns of the affine map
  static constexpr int SMEM_BYTES = STAGE_AREA + NUM_GROUPS * PANEL_BYTES + AFFINE_BYTES + 512;      // (starts on 1024 bytes)
  static_assert(STAGES * (A_STAGE_BYTES + B_STAGE_BYTES) <= STAGE_AREA, "ring does not fit");
  static_assert(SMEM_BYTES <= 227 * 1024, "over the shared-memory limit of a CTA");
  // k-blocks of B that may stay resident: four A stages must still fit
  static constexpr int MAX_RES_KB = (STAGE_AREA - 4 * A_STAGE_BYTES) / B_STAGE_BYTES;
  static constexpr int MAX_RES_KB2 = (STAGE_AREA2 - 4 * A_STAGE_BYTES) / B_STAGE_BYTES;
};

// Halo mode (policies with kHalo): a convolution tile loads, per 64-channel block, ONE box of input pixels
// that covers all filter taps (the output rows of the tile plus the filter's margin, full width), and the
// taps are shifted VIEWS of that box: the A descriptor of tap (r, s) starts (r * PW + s) rows of 128 bytes
// into it (the swizzle is a function of the absolute shared-memory address, so a view that starts in the
// middle of a 1024-byte pattern reads what TMA wrote there; the descriptor's base-offset field stays 0 --
// putting the row phase there gives wrong results, as a test run showed).  GEMM rows then run over the box's pixel pitch PW (the margin columns compute values that are
// never stored), and the input crosses L2 -> SM once instead of once per tap.  The box ring has its own
// barriers; the operand ring carries the filter tiles only (or nothing, when they are resident).
constexpr int HALO_BYTES = 32 * 1024;        // one input box (incl. the rows a shifted view may touch past it)
constexpr int MAX_HALOS = 3;

// Columns of a tile for `n` output columns and `m_tiles` row tiles.  Wide tiles re-read the rows least, but a problem with
// few of them leaves SMs idle while each CTA walks the whole reduction: as long as twice the tiles still fit one wave,
// half the width is faster (one image, 7x7 pixels, 3x3 over 512 channels: 2 CTAs of 72 blocks become 8).
inline int tile_columns(int n, int m_tiles, int sms) {
  int bn = n <= 64 ? 64 : (n <= 128 ? 128 : 256);
  while (bn > 64 && 2 * m_tiles * ((n + bn - 1) / bn) <= sms) bn /= 2;
  return bn;
}

// ESGD_GEMM_B_RESIDENT=0 in the environment turns the B-resident mode off (for A/B timing).
inline bool resident_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("ESGD_GEMM_B_RESIDENT");
    v = (e != nullptr && e[0] == '0') ? 0 : 1;
  }
  return v == 1;
}

__device__ __forceinline__ float bias_at(const Epilogue& ep, int col) {
  if (col >= ep.n_total) return 0.0f;
  return ep.bias_kind == BIAS_BF16 ? __bfloat162float(__ldg(reinterpret_cast<const __nv_bfloat16*>(ep.bias) + col)) : __ldg(ep.bias + col);
}

// Eight columns of the affine map, from its copy in shared memory: aff[0..63] factors, aff[64..127] summands of a panel's columns.
// (Read from memory where they are used, loads one after the other behind the products, they were 3.0 of the 5.9 us of a single
// image's 3136 x 64 x 64 layer.)
__device__ __forceinline__ void affine8(const float* aff, int col, float* v) {
#pragma unroll
  for (int q = 0; q < 8; q += 4) {
    const float4 a = *reinterpret_cast<const float4*>(aff + col + q), b = *reinterpret_cast<const float4*>(aff + 64 + col + q);
    v[q] = fmaf(v[q], a.x, b.x); v[q + 1] = fmaf(v[q + 1], a.y, b.y); v[q + 2] = fmaf(v[q + 2], a.z, b.z); v[q + 3] = fmaf(v[q + 3], a.w, b.w);
  }
}

// 32 accumulator columns of one row -> bf16 -> four 16-byte chunks of the swizzled staging panel.
// The plain kind leaves out the affine / residual / ReLU code altogether: as run-time options they would be predicated
// instructions that still take issue slots in the common case that uses none.
enum PackKind { PACK_PLAIN, PACK_AFFINE, PACK_MASKED };      // affine map, residual, ReLU; residual, bit mask
template <int kKind>
__device__ __forceinline__ void pack_row_to_panel(const uint32_t* r, uint8_t* panel, const uint8_t* rpanel, int row, int half,
                                                  const float* aff, const Epilogue& ep, bool has_residual, uint32_t keep = 0xffffffffu) {
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[g * 8 + j]);
    const int chunk = half * 4 + g;          // 16-byte chunk within the 128-byte row
    const int slot = row * 128 + ((chunk ^ (row & 7)) << 4);
    if (kKind != PACK_PLAIN) {
      if (kKind == PACK_AFFINE && ep.bias != nullptr) affine8(aff, half * 32 + g * 8, v);
      if (has_residual) {     // its panel was brought by TMA, possibly into this very buffer
        const uint4 rv = *reinterpret_cast<const uint4*>(rpanel + slot);
        const uint32_t* rw = reinterpret_cast<const uint32_t*>(&rv);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          v[2 * j] += __uint_as_float(rw[j] << 16);
          v[2 * j + 1] += __uint_as_float(rw[j] & 0xffff0000u);
        }
      }
      if (kKind == PACK_AFFINE && ep.relu) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = fmaxf(v[j], 0.0f);
      }
      if (kKind == PACK_MASKED) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = (keep >> (g * 8 + j)) & 1u ? v[j] : 0.0f;
      }
    }
    uint4 pk;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
    *reinterpret_cast<uint4*>(panel + slot) = pk;
  }
}

// 32 fp32 accumulator columns of one row -> eight 16-byte chunks of a staging panel of 32 columns.
__device__ __forceinline__ void stage_row_f32(const uint32_t* r, uint8_t* panel, int row, const float* aff, int col, const Epilogue& ep) {
#pragma unroll
  for (int c = 0; c < 8; c += 2) {
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[c * 4 + j]);
    if (ep.bias != nullptr) affine8(aff, col + c * 4, v);
    if (ep.relu) {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = fmaxf(v[j], 0.0f);
    }
    *reinterpret_cast<float4*>(panel + row * 128 + ((c ^ (row & 7)) << 4)) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(panel + row * 128 + (((c + 1) ^ (row & 7)) << 4)) = make_float4(v[4], v[5], v[6], v[7]);
  }
}

// Two fp32 additions / multiply-adds in one instruction.
__device__ __forceinline__ uint64_t pack_f32x2(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ void add_f32x2(uint64_t& a, uint64_t b) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(a) : "l"(b)); }
__device__ __forceinline__ void fma_f32x2(uint64_t& acc, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }
__device__ __forceinline__ uint64_t bf16x2_to_f32x2(uint32_t w) { return pack_f32x2(w << 16, w & 0xffff0000u); }
__device__ __forceinline__ float2 unpack_f32x2(uint64_t v) {
  uint32_t lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
  return make_float2(__uint_as_float(lo), __uint_as_float(hi));
}

// Problem policy requirements (all __device__ const):
//   static constexpr int BN; static constexpr bool A_MN, B_MN, kZeroStages;
//   struct Tile { int kb0, kb1, n0; ... };
//   int ksteps, n_mma                              16-wide K steps of a k-block that hold anything; MMA columns
//   bool tile(int it, Tile&)                       enumerate this CTA's tiles
//   struct Step; Step begin(const Tile&); void advance(Step&)    where a k-block lies, from the tile's first one on.  Counted, not
//                                                  divided out of the block's number: divisions by run-time numbers made the one
//                                                  thread that loads the bound of 3x3 layers (125 x 28 x 28 x 128: 37.4 -> 27.4 us)
//   void load(const Tile&, const Step&, uint8_t* a, uint8_t* b, uint64_t* bar)
//   void load_a(...a, bar) / load_b(...b, bar)     the two halves of load(); int res_kb (0: B not resident)
//   void store_panel(const Tile&, int panel, const void* smem)   TMA store of a 128x64 bf16 panel
//   static constexpr bool kPair                    the CTA is one of a pair (below): tile() gives it its own 128 rows, load()
//                                                  takes its half of B's columns and the address of the leader's barrier
//   static constexpr int kTwoPanels                residual panels in buffers of their own: 0 no, 1 in kBn kernels, 2 in all
//   void load_res_panel(const Tile&, int panel, void* smem, uint64_t* bar)   TMA load of the residual's panel
//   static constexpr bool kHalo; int out_row(int row)   row of the stored tile for a GEMM row (identity unless kHalo)
//   kHalo only: int cblks, R, S, PW; void load_halo(const Tile&, int cb, void* smem, uint64_t* bar)
//   int valid_prefix(const Tile&)                  rows [0, n) of the stored tile are real outputs
//   int64_t first_row(const Tile&)                 row 0 of the tile in the dense output matrix; the others follow
//   void store_f32(const Tile&, int col, const void* smem, bool add)   TMA store / reduction of 128 x 32 fp32 columns
// kBn: the batch-norm part of the epilogue (bn_y and so on); a kernel of its own, because its registers cost the others
// a tenth of their speed.
template <class P, bool kBn = false>
__device__ __forceinline__ void run(const P& prob, const Epilogue& ep) {
  constexpr int BN = P::BN;
  using C = Cfg<BN>;
  constexpr int STAGES = C::STAGES;
  // The swizzle counts from multiples of 1024 bytes.  Nothing else is in front of it in these kernels; rounding up would cost the
  // kilobyte that the affine map needs.
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023u) {
    if (threadIdx.x == 0 && ep.error_flag != nullptr) atomicExch(ep.error_flag, 1);
    return;
  }
  const int res_kb = prob.res_kb;            // > 0: B-resident mode
  constexpr bool kHalo = P::kHalo;
  // The residual's panels land in buffers of their own (four stages' worth of shared memory), so that the next one travels
  // while this one is stored and its sums are taken: 340 -> 260 us for 802816 x 256 x 64.
  const bool two_panels = (P::kTwoPanels == 2 || (kBn && P::kTwoPanels)) && ep.residual != nullptr;
  const int area = two_panels ? C::STAGE_AREA2 : C::STAGE_AREA;
  const int nhalo = kHalo ? (res_kb > 0 ? 2 : MAX_HALOS) : 0;
  constexpr bool kPair = P::kPair;
  const bool leads = !kPair || (blockIdx.x & 1) == 0;
  constexpr int kBStage = kPair ? C::B_STAGE_BYTES / 2 : C::B_STAGE_BYTES;
  const int nstages = kHalo ? (res_kb > 0 ? 1 : min(C::MAX_STAGES, (C::STAGE_AREA - nhalo * HALO_BYTES) / kBStage))
                      : kPair ? C::PAIR_STAGES
                            : (res_kb > 0 ? min(C::MAX_STAGES, (area - res_kb * C::B_STAGE_BYTES) / A_STAGE_BYTES)
                                          : min(STAGES, area / (A_STAGE_BYTES + C::B_STAGE_BYTES)));
  uint8_t* sA = smem;                        // halo mode: the input boxes
  uint8_t* sB = kHalo ? sA + nhalo * HALO_BYTES : sA + nstages * A_STAGE_BYTES;
  uint8_t* sC = smem + area;                 // the groups' output panels, then their residual panels
  float* sAff = reinterpret_cast<float*>(smem + C::STAGE_AREA + NUM_GROUPS * PANEL_BYTES);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::STAGE_AREA + NUM_GROUPS * PANEL_BYTES + C::AFFINE_BYTES);
  uint64_t* empty = full + C::MAX_STAGES;
  uint64_t* tfull = empty + C::MAX_STAGES;
  uint64_t* tempty = tfull + C::ACCS;
  uint64_t* bres = tempty + C::ACCS;         // the resident B tiles have landed
  uint64_t* rfull = bres + 1;                // residual panel has landed in the staging buffer of a group
  uint64_t* hfull = rfull + NUM_GROUPS;      // halo mode: input box has landed / has been consumed [MAX_HALOS]
  uint64_t* hempty = hfull + MAX_HALOS;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(hempty + MAX_HALOS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::MAX_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < C::ACCS; ++a) { mbar_init(&tfull[a], 1); mbar_init(&tempty[a], (kPair ? 2 : 1) * BN / 64 * GROUP_THREADS / 32); }
    mbar_init(bres, 1);
    for (int b = 0; b < NUM_GROUPS; ++b) mbar_init(&rfull[b], 1);
    for (int b = 0; b < MAX_HALOS; ++b) { mbar_init(&hfull[b], 1); mbar_init(&hempty[b], 1); }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    if (kPair) {
      tmem_alloc_pair(tmem_slot, C::TMEM_COLS);
    } else {
      tmem_alloc(tmem_slot, C::TMEM_COLS);
      tmem_relinquish();
    }
  }
  if (P::kZeroStages) {
    // partial boxes leave the tail rows of a stage untouched: they must read as zeros for ever
    uint4* p4 = reinterpret_cast<uint4*>(sA);
    const int n16 = STAGES * (A_STAGE_BYTES + C::B_STAGE_BYTES) / 16;
    for (int i = threadIdx.x; i < n16; i += NUM_THREADS) p4[i] = make_uint4(0, 0, 0, 0);
    fence_proxy_async();
  }
  tc_fence_before();
  __syncthreads();
  if (kPair) cluster_sync_all();             // the peer's barriers are there, too
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  esgd::pdl_enter();       // the setup above overlaps the end of the kernel before; from here on its results are there

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      typename P::Tile t;
      if (res_kb > 0 && prob.tile(0, t)) {
        mbar_expect_tx(bres, (uint32_t)(res_kb * C::B_STAGE_BYTES));
        typename P::Step at = prob.begin(t);
        for (int kb = 0; kb < res_kb; ++kb, prob.advance(at)) prob.load_b(t, at, sB + kb * C::B_STAGE_BYTES, bres);
      }
      const uint32_t tx_a = ep.tx_bytes_a ? ep.tx_bytes_a : (uint32_t)A_STAGE_BYTES;
      const uint32_t tx_ab = ep.tx_bytes ? ep.tx_bytes : (uint32_t)(A_STAGE_BYTES + C::B_STAGE_BYTES);
      if constexpr (kHalo) {
        // One input box per (tile, channel block), issued one step ahead of the filter tiles it goes with.
        const int cblks = prob.cblks;
        typename P::Tile tn;                     // box iterator, one (tile, block) ahead
        int it_n = 0, cb_n = 0, hs_n = 0;
        uint32_t hph_n = 0;
        bool more = prob.tile(0, tn);
        auto issue_box = [&]() -> bool {
          if (!more) return true;
          if (!mbar_wait(&hempty[hs_n], hph_n ^ 1u, abort_flag)) return false;
          if (leads) mbar_expect_tx(&hfull[hs_n], (kPair ? 2 : 1) * ep.tx_bytes_a);
          prob.load_halo(tn, cb_n, sA + hs_n * HALO_BYTES, &hfull[hs_n]);
          if (++hs_n == nhalo) { hs_n = 0; hph_n ^= 1u; }
          if (++cb_n == cblks) { cb_n = 0; more = prob.tile(++it_n, tn); }
          return true;
        };
        ok = issue_box();
        for (int it = 0; ok && prob.tile(it, t); ++it) {
          for (int cb = 0; ok && cb < cblks; ++cb) {
            ok = issue_box();                    // the next box travels while this block's filter tiles are fed
            if (res_kb > 0) continue;
            for (int r = 0; ok && r < prob.R; ++r)
            for (int s = 0; s < prob.S; ++s) {
              if (!mbar_wait(&empty[stage], phase ^ 1u, abort_flag)) { ok = false; break; }
              if (leads) mbar_expect_tx(&full[stage], (uint32_t)C::B_STAGE_BYTES);          // a pair's halves together
              prob.load_b(t, typename P::Step{r, s, cb}, sB + stage * kBStage, &full[stage]);
              if (++stage == nstages) { stage = 0; phase ^= 1u; }
            }
          }
        }
      } else
      for (int it = 0; ok && prob.tile(it, t); ++it) {
        typename P::Step at = prob.begin(t);
        for (int kb = t.kb0; kb < t.kb1; ++kb, prob.advance(at)) {
          if (!mbar_wait(&empty[stage], phase ^ 1u, abort_flag)) { ok = false; break; }
          if constexpr (kPair) {
            // both CTAs' loads arrive at the leader's barrier; it may see the peer's bytes before it expects them
            if (leads) mbar_expect_tx(&full[stage], 2 * (tx_a + (uint32_t)kBStage));
            prob.load(t, at, sA + stage * A_STAGE_BYTES, sB + stage * kBStage, leader_addr(&full[stage]));
          } else if (res_kb > 0) {
            mbar_expect_tx(&full[stage], tx_a);
            prob.load_a(t, at, sA + stage * A_STAGE_BYTES, &full[stage]);
          } else {
            mbar_expect_tx(&full[stage], tx_ab);
            prob.load(t, at, sA + stage * A_STAGE_BYTES, sB + stage * C::B_STAGE_BYTES, &full[stage]);
          }
          if (++stage == nstages) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (leads && elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(kPair ? 2 * BM : BM, prob.n_mma, P::A_MN ? 1 : 0, P::B_MN ? 1 : 0);
      // Products of one k-block.  Below 64 reduced channels (narrow convolutions) the last steps would multiply zero fill;
      // the full block is a path of its own because a predicate per instruction slows the issue loop of narrow tiles.
      const int ksteps = prob.ksteps;
      auto commit = [](uint64_t* bar) {
        if constexpr (kPair) umma_commit_pair(bar);
        else umma_commit(bar);
      };
      auto issue_full = [&](uint32_t d, uint64_t a, uint64_t b, uint32_t& accumulate) {
        constexpr uint64_t sa = P::A_MN ? (2048 >> 4) : (32 >> 4), sb = P::B_MN ? (2048 >> 4) : (32 >> 4);   // 16 K elements
#pragma unroll
        for (int j = 0; j < BK / 16; ++j) {
          umma_bf16(d, a + j * sa, b + j * sb, idesc, j > 0 ? 1u : accumulate);
        }
        accumulate = 1;
      };
      auto issue_block = [&](uint32_t d, uint64_t a, uint64_t b, uint32_t& accumulate) {
        constexpr uint64_t sa = P::A_MN ? (2048 >> 4) : (32 >> 4), sb = P::B_MN ? (2048 >> 4) : (32 >> 4);   // 16 K elements
        if constexpr (kPair) {
          umma_bf16_pair(d, a, b, idesc, accumulate);
#pragma unroll
          for (int j = 1; j < BK / 16; ++j) umma_bf16_pair(d, a + j * sa, b + j * sb, idesc, 1u);
        } else if (ksteps == BK / 16) {
          umma_bf16(d, a, b, idesc, accumulate);
#pragma unroll
          for (int j = 1; j < BK / 16; ++j) umma_bf16(d, a + j * sa, b + j * sb, idesc, 1u);
        } else {
          umma_bf16(d, a, b, idesc, accumulate);
          for (int j = 1; j < ksteps; ++j) umma_bf16(d, a + j * sa, b + j * sb, idesc, 1u);
        }
        accumulate = 1;
      };
      // The issuing thread is one lane with nothing to hide its instruction latency behind: every instruction
      // between two tcgen05.mma widens the gap between them.  (It has to be elected: under lane == 0, which the compiler
      // does not know to be one lane, every MMA sat in a loop over the active lanes, and 128 x 64 x 16 ones went out ~115
      // cycles apart, 32 of them tensor-pipe work; 3x3 on 256 x 64 x 56 x 56: 148 -> 98 us.)  Descriptors are built once and
      // advanced by adding to their address field (bits 0-13, in 16-byte units; shared memory is < 256 KB, so no carry).
      const uint64_t a_desc0 = P::A_MN ? umma_smem_desc(smem_u32(sA), 8192, 1024) : umma_smem_desc(smem_u32(sA), 16, 1024);
      const uint64_t b_desc0 = P::B_MN ? umma_smem_desc(smem_u32(sB), 8192, 1024) : umma_smem_desc(smem_u32(sB), 16, 1024);
      int stage = 0, acc = 0, hs = 0;
      uint32_t phase = 0, acc_phase = 0, hphase = 0;
      bool ok = true;
      typename P::Tile t;
      if (res_kb > 0 && prob.tile(0, t)) ok = mbar_wait(bres, 0u, abort_flag);
      for (int it = 0; ok && prob.tile(it, t); ++it) {
        if (!mbar_wait(&tempty[acc], acc_phase ^ 1u, abort_flag)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(acc * BN);
        uint32_t accumulate = 0;                  // the tile's first MMA overwrites the accumulator
        if constexpr (kHalo) {
          const int cblks = prob.cblks, R = prob.R, S = prob.S;
          const uint64_t row_step = (uint64_t)(prob.PW * 8);           // one box row of pixels, in 16-byte units
          for (int cb = 0; ok && cb < cblks; ++cb) {
            if (!mbar_wait(&hfull[hs], hphase, abort_flag)) { ok = false; break; }
            tc_fence_after();
            // the window of tap (r, s): the same box, (r * PW + s) pixel rows (128 bytes each) further on
            uint64_t a_row = a_desc0 + (uint64_t)(hs * (HALO_BYTES >> 4));
            uint64_t b_tap = b_desc0 + (uint64_t)(cb * (C::B_STAGE_BYTES >> 4));       // resident: k-block tap*cblks+cb
            const uint64_t b_tap_step = (uint64_t)(cblks * (C::B_STAGE_BYTES >> 4));
            if (!kPair && res_kb > 0 && R == 3 && S == 3 && ksteps == BK / 16) {
              // the common filter, all of it there: the 36 products in one straight line
#pragma unroll
              for (int tap = 0; tap < 9; ++tap)
                issue_full(d_tmem, a_row + (uint64_t)(tap / 3) * row_step + (tap % 3) * 8, b_tap + tap * b_tap_step, accumulate);
            } else
            for (int r = 0; ok && r < R; ++r, a_row += row_step) {
              uint64_t a_tap = a_row;
              for (int sx = 0; sx < S; ++sx, a_tap += 8, b_tap += b_tap_step) {
                uint64_t b_cur = b_tap;
                if (res_kb == 0) {
                  if (!mbar_wait(&full[stage], phase, abort_flag)) { ok = false; break; }
                  tc_fence_after();
                  b_cur = b_desc0 + (uint64_t)(stage * (kBStage >> 4));
                }
                issue_block(d_tmem, a_tap, b_cur, accumulate);
                if (res_kb == 0) {
                  commit(&empty[stage]);
                  if (++stage == nstages) { stage = 0; phase ^= 1u; }
                }
              }
            }
            if (!ok) break;
            commit(&hempty[hs]);
            if (++hs == nhalo) { hs = 0; hphase ^= 1u; }
          }
        } else
        for (int kb = t.kb0; kb < t.kb1; ++kb) {
          if (!mbar_wait(&full[stage], phase, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint64_t a_cur = a_desc0 + (uint64_t)(stage * (A_STAGE_BYTES >> 4));
          const uint64_t b_cur = b_desc0 + (uint64_t)((res_kb > 0 ? kb : stage) * (kBStage >> 4));
          issue_block(d_tmem, a_cur, b_cur, accumulate);
          commit(&empty[stage]);
          if (++stage == nstages) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        commit(&tfull[acc]);
        if (++acc == C::ACCS) { acc = 0; acc_phase ^= 1u; }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    // A warp may only touch TMEM lanes [32*(warp%4), +32); four consecutive warps cover all rows.  Group g works on
    // panel g % PANELS of the tiles it is dealt, so its columns within a tile never change.
    constexpr int PANELS = BN / 64, TURNS = NUM_GROUPS / PANELS;     // groups per panel: they take turns over the tiles
    const int q = warp & 3, grp = (warp - 2) >> 2;
    const int gt = (int)threadIdx.x - 64 - grp * GROUP_THREADS;      // 0..127 among the group's threads
    const int pnl = grp % PANELS, turn = grp / PANELS;
    const int row = q * 32 + lane;          // tile row owned by this thread
    const int drow = prob.out_row(row);     // its row in the stored tile (halo mode: margin rows have none)
    uint8_t* panel = sC + grp * PANEL_BYTES;
    uint8_t* rpanel = two_panels ? panel + NUM_GROUPS * PANEL_BYTES : panel;
    const bool leader = gt == 0;            // issues the group's copies
    const bool has_res = ep.residual != nullptr;
    const bool plain = ep.bias == nullptr && !ep.relu && !has_res;
    // statistics: thread (cp, rg) covers columns 2cp, 2cp+1 of the panel, rows 32rg .. 32rg+31
    const int cp = gt & 31, rg = gt >> 5;
    uint64_t st_sum = 0, st_sq = 0;
    uint32_t res_phase = 0;
    bool ok = true;
    typename P::Tile t, next;               // this tile and the group's next one: where a tile lies takes divisions, once is enough
    bool more = prob.tile(turn, t);
    auto release_acc = [&](int a) {
      if (kPair) mbar_arrive_at(leader_addr(&tempty[a]));
      else mbar_arrive(&tempty[a]);
    };
    // The residual panel of a unit travels while the group finishes the one before it.
    auto fetch_residual = [&](const typename P::Tile& n) {
      if (!leader || !more || n.n0 + pnl * 64 >= ep.n_total) return;
      mbar_expect_tx(&rfull[grp], ep.res_bytes);
      prob.load_res_panel(n, pnl, rpanel, &rfull[grp]);
    };
    // ... and the lines that a unit will read go to L2 meanwhile, a row per thread: bn_y, or a residual panel that can only be
    // asked for when the panel before it has left their common buffer (392000 x 256 x 64 with a residual: 93 -> 84 us, 98000 x 512 x
    // 128: 54 -> 49; in pairs of CTAs, whose products are the longer part, 6125 x 2048 x 512, it took 22.7 for 22.1).
    auto prefetch = [&](const void* p, int ld, const typename P::Tile& n) {
      if (!more || n.n0 + pnl * 64 >= ep.n_total || gt >= prob.valid_prefix(n)) return;
      asm volatile("prefetch.global.L2 [%0];" ::"l"((const __nv_bfloat16*)p + (prob.first_row(n) + gt) * ld + n.n0 + pnl * 64));
    };
    uint64_t neg_mean = 0;
    if (kBn && more && t.n0 + pnl * 64 < ep.n_total) {      // a CTA's tiles share their columns
      const float2 m = __ldg(reinterpret_cast<const float2*>(ep.bn_aux + t.n0 + pnl * 64) + cp);
      neg_mean = pack_f32x2(__float_as_uint(-m.x), __float_as_uint(-m.y));
      prefetch(ep.bn_y, ep.n_total, t);
    }
    if (has_res) fetch_residual(t);
    // The affine map of the group's columns: a thread has one factor or summand, asked for a tile ahead and put down when the
    // columns change.
    float* aff = sAff + grp * 128;
    int aff_n0 = -1;
    float aff_next = 0.0f;
    auto ask_affine = [&](const typename P::Tile& n) {
      if (ep.bias == nullptr || !more) return;
      const int col = n.n0 + pnl * 64 + (gt & 63);
      aff_next = gt >= 64 ? bias_at(ep, col) : ep.scale != nullptr && col < ep.n_total ? __ldg(ep.scale + col) : 1.0f;
    };
    if (!kBn) ask_affine(t);
    for (int it = turn; more; it += TURNS, t = next) {
      more = prob.tile(it + TURNS, next);
      const int acc = it % C::ACCS;
      if (!kBn && ep.bias != nullptr) {
        if (t.n0 != aff_n0) {                                  // the same for all of the group
          named_barrier_sync(1 + grp, GROUP_THREADS);
          aff[gt] = aff_next;
          aff_n0 = t.n0;
          named_barrier_sync(1 + grp, GROUP_THREADS);
        }
        ask_affine(next);
      }
      // bn: the mask of this thread's row, and of bn_y this thread's column pair of rows 32rg .. +15 (later +16 .. +31), asked
      // for before the waits
      uint32_t ya[kBn ? 16 : 1];
      uint2 keep = make_uint2(0xffffffffu, 0xffffffffu);
      const uint32_t* ysrc = nullptr;
      auto load_y = [&](uint32_t (&v)[kBn ? 16 : 1], int r0) {
        const int rows = prob.valid_prefix(t) - rg * 32 - r0;
#pragma unroll
        for (int rr = 0; rr < (kBn ? 16 : 1); ++rr) v[rr] = rr < rows ? __ldg(ysrc + (size_t)(r0 + rr) * (ep.n_total >> 1)) : 0u;
      };
      if (kBn && t.n0 + pnl * 64 < ep.n_total) {
        const int64_t row0 = prob.first_row(t);
        const int c0 = t.n0 + pnl * 64;
        if (ep.bn_mask != nullptr && drow >= 0 && drow < prob.valid_prefix(t))
          keep = __ldg(reinterpret_cast<const uint2*>(ep.bn_mask + ((row0 + drow) * ep.n_total + c0) / 8));
        ysrc = reinterpret_cast<const uint32_t*>(ep.bn_y + (row0 + rg * 32) * ep.n_total + c0) + cp;
        load_y(ya, 0);
      }
      ok = __all_sync(0xffffffffu, ok && mbar_wait(&tfull[acc], (uint32_t)(it / C::ACCS) & 1u, abort_flag));
      tc_fence_after();
      const int col0 = t.n0 + pnl * 64;
      if (kBn) prefetch(ep.bn_y, ep.n_total, next);
      else if (!kPair && !kHalo && has_res) prefetch(ep.residual, ep.ldr, next);
      if (col0 < ep.n_total) {              // uniform across the group
        const int prefix = prob.valid_prefix(t);              // rows [0, prefix) are real outputs
        const int yrows = min(32, max(0, prefix - rg * 32));
        const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * BN + pnl * 64);
        uint32_t r[32];                       // 32 columns at a time: two halves would not fit 96 registers beside the rest
        tmem_ld_32x32b_x32(t_row, r);
        if (has_res) {
          ok = __all_sync(0xffffffffu, ok && mbar_wait(&rfull[grp], res_phase, abort_flag));
          res_phase ^= 1u;
        }
        if (!has_res || two_panels) {
          if (leader) tma_store_wait_read<0>();               // the group's previous panel has left the buffer
          named_barrier_sync(1 + grp, GROUP_THREADS);
        }
        tmem_ld_wait();
        auto next_half = [&]() {                              // the accumulator is free once every panel has been read
          tmem_ld_32x32b_x32(t_row + 32, r);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) release_acc(acc);
        };
        if (kBn || ep.out_mode == OUT_BF16) {
          if (!kBn && plain) {
            if (drow >= 0) pack_row_to_panel<PACK_PLAIN>(r, panel, rpanel, drow, 0, aff, ep, false);
            next_half();
            if (drow >= 0) pack_row_to_panel<PACK_PLAIN>(r, panel, rpanel, drow, 1, aff, ep, false);
          } else if (!kBn) {
            if (drow >= 0) pack_row_to_panel<PACK_AFFINE>(r, panel, rpanel, drow, 0, aff, ep, has_res);
            next_half();
            if (drow >= 0) pack_row_to_panel<PACK_AFFINE>(r, panel, rpanel, drow, 1, aff, ep, has_res);
          } else {
            if (drow >= 0) pack_row_to_panel<PACK_MASKED>(r, panel, rpanel, drow, 0, aff, ep, has_res, keep.x);
            next_half();
            if (drow >= 0) pack_row_to_panel<PACK_MASKED>(r, panel, rpanel, drow, 1, aff, ep, has_res, keep.y);
          }
          fence_proxy_async();
          named_barrier_sync(1 + grp, GROUP_THREADS);         // the panel is complete and visible to the TMA engine
          if (leader) {
            prob.store_panel(t, pnl, panel);
            tma_store_commit();
            if (two_panels) fetch_residual(next);        // everybody has read this one
          }
          if (kBn || ep.col_sum != nullptr) {
            const uint8_t* colp = panel + rg * 32 * 128 + (cp & 3) * 4;
            const int chunk = cp >> 2;
            uint64_t s = 0, sq = 0;
            if (kBn) {
              // dbeta and dgamma: y comes from L2 (the previous unit asked for it), coalesced over the panel's columns
              uint32_t yb[kBn ? 16 : 1];
              load_y(yb, 16);
#pragma unroll
              for (int rr = 0; rr < 32; ++rr) {
                uint32_t w = *reinterpret_cast<const uint32_t*>(colp + rr * 128 + ((chunk ^ (rr & 7)) << 4));
                if (rr >= yrows) w = 0u;
                const uint64_t f = bf16x2_to_f32x2(w);
                uint64_t d = bf16x2_to_f32x2(rr < 16 ? ya[kBn ? rr & 15 : 0] : yb[kBn ? rr & 15 : 0]);
                add_f32x2(d, neg_mean);
                add_f32x2(s, f);
                fma_f32x2(sq, f, d);
              }
            } else if (yrows == 32) {
#pragma unroll 16
              for (int rr = 0; rr < 32; ++rr) {
                const uint32_t w = *reinterpret_cast<const uint32_t*>(colp + rr * 128 + ((chunk ^ (rr & 7)) << 4));
                const uint64_t f = bf16x2_to_f32x2(w);
                add_f32x2(s, f);
                fma_f32x2(sq, f, f);
              }
            } else {
#pragma unroll 8
              for (int rr = 0; rr < 32; ++rr) {
                uint32_t w = *reinterpret_cast<const uint32_t*>(colp + rr * 128 + ((chunk ^ (rr & 7)) << 4));
                if (rr >= yrows) w = 0u;                      // rows outside the tensor count as zeros
                const uint64_t f = bf16x2_to_f32x2(w);
                add_f32x2(s, f);
                fma_f32x2(sq, f, f);
              }
            }
            add_f32x2(st_sum, s);
            add_f32x2(st_sq, sq);
          }
        } else {
          // fp32 outputs (logits, split-K weight gradients): 32 columns at a time through the same buffer
          const bool add = ep.out_mode == OUT_F32_ADD;
          stage_row_f32(r, panel, row, aff, 0, ep);
          next_half();
          fence_proxy_async();
          named_barrier_sync(1 + grp, GROUP_THREADS);
          if (leader) {
            prob.store_f32(t, col0, panel, add);
            tma_store_commit();
            tma_store_wait_read<0>();
          }
          named_barrier_sync(1 + grp, GROUP_THREADS);
          if (col0 + 32 < ep.n_total) {
            stage_row_f32(r, panel, row, aff, 32, ep);
            fence_proxy_async();
            named_barrier_sync(1 + grp, GROUP_THREADS);
            if (leader) {
              prob.store_f32(t, col0 + 32, panel, add);
              tma_store_commit();
            }
          }
        }
        if (has_res && !two_panels) {
          named_barrier_sync(1 + grp, GROUP_THREADS);         // the statistics are done with the panel, too
          if (leader) {
            tma_store_wait_read<0>();
            fetch_residual(next);
          }
        }
      } else {
        if (lane == 0) release_acc(acc);
        if (has_res && leader) {
          tma_store_wait_read<0>();
          fetch_residual(next);
        }
      }
    }
    if (ep.col_sum != nullptr && prob.tile(0, t)) {
      // One atomic per column and CTA (its tiles share the column range): the threads' sums meet in shared memory first.
      // Flushed thread by thread, a 64-channel layer sent 2400 atomics to every address and waited 17 us for them.
      float* sums = reinterpret_cast<float*>(sC);             // [2][BN]
      const int tid = (int)threadIdx.x - 64;
      if (leader) tma_store_wait_read<0>();
      named_barrier_sync(1 + NUM_GROUPS, NUM_GROUPS * GROUP_THREADS);
      if (tid < 2 * BN) sums[tid] = 0.0f;
      named_barrier_sync(1 + NUM_GROUPS, NUM_GROUPS * GROUP_THREADS);
      const float2 s = unpack_f32x2(st_sum), sq = unpack_f32x2(st_sq);
      float* mine = sums + pnl * 64 + cp * 2;
      atomicAdd(mine, s.x);
      atomicAdd(mine + 1, s.y);
      atomicAdd(mine + BN, sq.x);
      atomicAdd(mine + BN + 1, sq.y);
      named_barrier_sync(1 + NUM_GROUPS, NUM_GROUPS * GROUP_THREADS);
      const int c = tid % BN, col = t.n0 + c;
      if (tid < 2 * BN && col < ep.n_total)
        atomicAdd((tid < BN ? ep.col_sum : ep.col_sqsum) + col, kBn && tid >= BN ? sums[tid] * __ldg(ep.bn_aux + ep.n_total + col) : sums[tid]);
    }
    if (leader) tma_store_wait_all();                // shared memory must outlive the bulk stores
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    __nanosleep(1000000);
    if (threadIdx.x == 0 && ep.error_flag != nullptr) atomicExch(ep.error_flag, 1);
  }
  if (kPair) cluster_sync_all();             // nobody leaves while the peer's barriers or products may still use this CTA
  if (warp == 1) {
    tc_fence_after();
    if (kPair) tmem_dealloc_pair(tmem_base, C::TMEM_COLS);
    else tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

}  // namespace umma
