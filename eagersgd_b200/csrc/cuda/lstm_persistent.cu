// The recurrence of an LSTM layer as ONE persistent kernel per direction (sm_100a: tcgen05 / TMEM / TMA / clusters).
//
// A time step is a product with the recurrent weights (32 MB of bf16 at 2048 units) and a few hundred bytes of state per
// SM; as two launches per step (split-K GEMM + cell kernel) it cost 13.8 us forward and 15.3 us backward at batch 16, bound
// by the two kernel boundaries and by re-reading the weights from L2.  Here every CTA keeps its share of the weights on
// chip for the whole sequence and a step is: fetch the previous step's state as it appears (32 KB), 64 MMAs, exchange
// partial sums inside the cluster, apply the cell to 16 units, publish.
//
//   weights   the A operand of tcgen05.mma, 64 columns of K at a time: up to 14 such blocks (224 KB) in tensor memory, the
//             rest in shared memory, as the room left by the state and the partial sums allows
//   forward   128 rows = 4 gates x 32 units, K = half of the hidden state: clusters of 2, H/16 CTAs
//   backward  128 rows = 128 units of dh (weights transposed), K = 4H split over clusters of up to 8 CTAs: the largest
//             cluster size whose whole grid is resident (of 16 clusters, a B200's GPCs hold 15 of size 8 or 7 but all of size 6)
//   cluster   each finalising CTA owns 16 (forward) or 32 (backward) units x batch: partial sums go to its shared memory
//             (st.async: the bytes carry their own arrival), double buffered by step parity; a CTA can be at most one step ahead of a cluster mate (it needs a
//             state that transitively needs the mate's previous one), so two buffers are enough
//   grid      the state is published by writing it to y (forward) or dG (backward), which are filled with a bit pattern that
//             no result has (0xffff per bf16; conversions round every NaN to 0x7fff) before the launch: eight warps read the
//             words they need until none of them is the pattern, and put them where the tensor core reads them.  The data is
//             its own flag, so no fence, counter or second trip to L2 stands between a store and its use.  With counters, a
//             release and a TMA load the way from a stored state to the first MMA took 3 of the step's 5.2 us.
//             Launched cooperatively (all CTAs resident); every wait is bounded and ends in the error flag.
//
// Cell state (forward) and cell gradient (backward) of an element stay in the register of the thread that owns it.
// Gate order i, f, g, o as in torch.nn.LSTM.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include "launch_count.cuh"
#include "sm100_primitives.cuh"
#include "tensormap.cuh"

using namespace sm100;

namespace {

constexpr int kRows = 128;          // weight rows of a CTA (MMA M)
constexpr int kEpiThreads = 256;
constexpr int kFetchWarps = 8;
constexpr int kIssuers = 4;         // warps that issue MMAs, one on each scheduler of the SM
constexpr int kIssue0 = kEpiThreads / 32, kFetch0 = kIssue0 + kIssuers;
constexpr int kThreads = (kFetch0 + kFetchWarps) * 32;
constexpr int kATile = kRows * 128; // one 64-column block of A
constexpr int kPiece = kIssuers;    // K blocks of a piece of the state, one per issuer: the MMAs of one run while the next is fetched
constexpr int kMaxPieces = 8;
constexpr int kSmemLimit = 227 * 1024;
constexpr uint32_t kUnset = 0xffffffffu;      // two bf16 that have not been written yet
constexpr uint64_t kWaitNs = 4000000000ull;   // bound on every wait

struct SeqParams {
  CUtensorMap tmW;                  // recurrent weights
  const __nv_bfloat16* w;           // [4H][H]
  int T, B, H, S;                   // S: cluster size, the split of K
  const __nv_bfloat16* xproj;       // forward: [T][B][4H]
  const float* bias;                // forward: [4H]
  float* c;                         // [T][B][H]
  __nv_bfloat16* y;                 // forward: [T][B][H]
  __nv_bfloat16* gates;             // [T][B][4H]
  const __nv_bfloat16* dy;          // backward: [T][B][H]
  __nv_bfloat16* dG;                // backward: [T][B][4H]
  float* db;                        // backward: [4H] bias gradient, added to (may be null)
  int* error_flag;
};

__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + __expf(-x)); }
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
// 16 bytes into a mate's shared memory, counted by its barrier.
__device__ __forceinline__ void st_async_x4(uint32_t addr, const uint32_t* v, uint32_t bar_addr) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(bar_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ bool try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded waits without a sleep between the polls (a step is a chain of them); they raise the CTA's abort flag on expiry
// and give up at once when it is up.
struct Patience {
  uint64_t t0 = 0;
  __device__ __forceinline__ bool over(uint32_t it, volatile int* abort_flag) {
    if ((it & 63u) != 63u) return false;
    uint64_t now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    if (t0 == 0) t0 = now;
    if (now - t0 > kWaitNs) *abort_flag = 1;
    return *abort_flag != 0;
  }
};
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  Patience p;
  for (uint32_t it = 0; !try_wait_cluster(bar, parity); ++it)
    if (p.over(it, abort_flag)) return false;
  return true;
}
__device__ __forceinline__ uint4 ld_state(const void* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool unset(const uint4& v) { return v.x == kUnset || v.y == kUnset || v.z == kUnset || v.w == kUnset; }
__device__ __forceinline__ uint32_t bf16_bits(float v) { return (uint32_t)__bfloat16_as_ushort(__float2bfloat16(v)); }
// Four lanes' values, in lane order, in each of the four.
__device__ __forceinline__ uint2 gather_quad(uint32_t v, int lane) {
  const uint32_t other = __shfl_xor_sync(0xffffffffu, v, 1);
  const uint32_t pair = lane & 1 ? other | (v << 16) : v | (other << 16);
  const uint32_t far = __shfl_xor_sync(0xffffffffu, pair, 2);
  return lane & 2 ? make_uint2(far, pair) : make_uint2(pair, far);
}
template <int N>
__device__ __forceinline__ void ld_shared_vec(float (&v)[N], const float* p) {
  if constexpr (N == 1) v[0] = *p;
  else if constexpr (N == 2) { const float2 x = *reinterpret_cast<const float2*>(p); v[0] = x.x; v[1] = x.y; }
  else { const float4 x = *reinterpret_cast<const float4*>(p); v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; }
}
__device__ __forceinline__ void publish(void* p, uint2 v) {
  asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(v.x), "r"(v.y) : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]: A holds two consecutive K elements of a row per 32-bit cell, K-major.
__device__ __forceinline__ void umma_bf16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st_x8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_ld_x8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}

template <bool kBwd, int N>
struct Layout {
  static constexpr int kUnits = kBwd ? 32 : 16;                       // units a finalising CTA owns
  static constexpr int kFinal = kBwd ? 4 : 2;                         // finalising CTAs of a cluster
  static constexpr int kPer = kUnits * N / kEpiThreads;               // elements of a finalising thread
  static constexpr int kTBlocks = 16 - kIssuers * N / 32;             // K blocks of the weights in tensor memory, 32 columns each
  static constexpr int kDCol = kTBlocks * 32;                         // the issuers' accumulators, N columns each
  static constexpr int kPitch = N + 4;                                // floats of a unit's batch in the partial sums
  int kblocks, per, tblocks, sblocks, part;                           // per: K blocks of a CTA (the last may have fewer);
                                                                      // part: floats for one step's partial sums
  __host__ __device__ Layout(int H, int S) {
    kblocks = (kBwd ? 4 * H : H) / 64;
    per = (kblocks + S - 1) / S;
    tblocks = per < kTBlocks ? per : kTBlocks;
    sblocks = per - tblocks;
    part = S * (kBwd ? 1 : 4) * kUnits * kPitch;
  }
  int smem() const { return 1024 + sblocks * kATile + per * (N * 128) + 2 * part * 4 + 256; }
};

template <bool kBwd, int N>
__global__ void __launch_bounds__(kThreads, 1) lstm_sequence_kernel(const __grid_constant__ SeqParams p) {
  using L = Layout<kBwd, N>;
  constexpr int PER = L::kPer, UNITS = L::kUnits;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int H = p.H, B = p.B, T = p.T, S = p.S;
  const L lay(H, S);
  const int rank = (int)cluster_rank(), group = blockIdx.x / S;
  const int kblocks = min(lay.per, lay.kblocks - rank * lay.per);     // K blocks of this CTA: the first tblocks of them
  const int tblocks = min(kblocks, lay.tblocks);                      // in tensor memory, the others in shared memory
  const int kbase = rank * lay.per * 64;                              // its K range: h units, or rows of the weights (gates)
  uint8_t* sA = smem;
  uint8_t* sB = sA + lay.sblocks * kATile;
  float* sP = reinterpret_cast<float*>(sB + lay.per * (N * 128));
  uint64_t* full = reinterpret_cast<uint64_t*>(sP + 2 * lay.part);    // [kMaxPieces] pieces of the state are in place
  uint64_t* wfull = full + kMaxPieces;                                 // the weights have landed
  uint64_t* dfull = wfull + 1;                                        // the step's product is in tensor memory
  uint64_t* dfree = dfull + 1;                                        // ... and has been read out of it
  uint64_t* pfull = dfree + 1;                                        // [2] partial sums of all cluster mates are here
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pfull + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const bool final_cta = rank < L::kFinal;
  const int u0 = (kBwd ? group * 128 : group * 32) + rank * UNITS;    // first unit this CTA finalises
  const int npieces = (kblocks + kPiece - 1) / kPiece;
  const int p0 = group % npieces;        // CTAs start at different pieces: 128 SMs asking for one line queue up at its L2 slice

  if (threadIdx.x == 0) {
    for (int i = 0; i < kMaxPieces; ++i) mbar_init(&full[i], kFetchWarps);
    mbar_init(wfull, 1);
    mbar_init(dfull, kIssuers);
    mbar_init(dfree, kEpiThreads / 32);
    mbar_init(&pfull[0], 1);
    mbar_init(&pfull[1], 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&p.tmW);
  }
  if (warp == kIssue0) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  for (int i = threadIdx.x; i < lay.per * N * 8; i += kThreads)       // batch rows that do not exist stay zero
    reinterpret_cast<uint4*>(sB)[i] = make_uint4(0, 0, 0, 0);
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // ---- the weights: shared-memory part by TMA, tensor-memory part through registers
  if (warp == kIssue0) {
    if (elect_one()) {
      mbar_expect_tx(wfull, (uint32_t)((kblocks - tblocks) * kATile));
      for (int kb = tblocks; kb < kblocks; ++kb) {
        uint8_t* a = sA + (kb - tblocks) * kATile;
        if (kBwd) {     // A[unit][gate row] = w[gate row][unit]: MN-major, two 64-unit atoms
          for (int i = 0; i < 2; ++i) tma_load_2d(a + i * 8192, &p.tmW, wfull, group * 128 + 64 * i, kbase + kb * 64);
        } else {        // rows: gate q, units of the group
          for (int q = 0; q < 4; ++q) tma_load_2d(a + q * 4096, &p.tmW, wfull, kbase + kb * 64, q * H + group * 32);
        }
      }
    }
  } else if (warp < kIssue0) {
    const int q = warp & 3, row = q * 32 + lane;
    for (int k0 = (warp >> 2) * 16; k0 < tblocks * 64; k0 += 32) {            // 16 K elements = 8 columns at a time
      uint32_t r[8];
      if (kBwd) {
        const __nv_bfloat16* src = p.w + (size_t)(kbase + k0) * H + group * 128 + row;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint32_t lo = __bfloat16_as_ushort(src[(size_t)(2 * i) * H]), hi = __bfloat16_as_ushort(src[(size_t)(2 * i + 1) * H]);
          r[i] = lo | (hi << 16);
        }
      } else {
        const uint4* src = reinterpret_cast<const uint4*>(p.w + ((size_t)q * H + group * 32 + lane) * H + kbase + k0);
        const uint4 a = __ldg(src), b = __ldg(src + 1);
        r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w; r[4] = b.x; r[5] = b.y; r[6] = b.z; r[7] = b.w;
      }
      tmem_st_x8(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(k0 / 2), r);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  cluster_sync();          // barriers of all mates are initialised, every thread's part of the weights is in place
  tc_fence_after();

  if (warp >= kIssue0 && warp < kFetch0) {
    // ------------------------------------------------------------ issue the products
    const uint32_t idesc_s = umma_idesc_bf16(kRows, N, kBwd ? 1 : 0, 0), idesc_t = umma_idesc_bf16(kRows, N, 0, 0);
    const uint64_t a_desc0 = kBwd ? umma_smem_desc(smem_u32(sA), 8192, 1024) : umma_smem_desc(smem_u32(sA), 16, 1024);
    const uint64_t b_desc0 = umma_smem_desc(smem_u32(sB), 16, 1024);
    constexpr uint64_t kStepA = kBwd ? (2048 >> 4) : (32 >> 4), kStepB = 32 >> 4;
    // The thread's own instructions between two MMAs bound it (one issuer: 40 to 57 cycles apart, 128 x 16 x 16 is a
    // fraction of that), so four of them share the K blocks of a piece, each with an accumulator of its own.
    const int issuer = warp - kIssue0;
    const uint32_t d_tmem = tmem + (uint32_t)(L::kDCol + issuer * N);
    if (elect_one()) {
      bool ok = wait_bar(wfull, 0u, abort_flag);
      for (int s = 1; ok && s < T; ++s) {                    // step 0 has no recurrent product
        const uint32_t ph = (uint32_t)(s - 1) & 1u;
        if (s > 1) ok = wait_bar(dfree, ph ^ 1u, abort_flag);               // the previous product has been read
        uint32_t acc = 0;
        for (int j = 0; ok && j < npieces; ++j) {
          const int piece = p0 + j < npieces ? p0 + j : p0 + j - npieces;
          ok = wait_bar(&full[piece], ph, abort_flag);
          tc_fence_after();
          const int kb = piece * kPiece + issuer;
          if (!ok || kb >= kblocks) continue;
          const uint64_t b_desc = b_desc0 + (uint64_t)(kb * (N * 128 >> 4));
          if (kb >= tblocks) {
            const uint64_t a_desc = a_desc0 + (uint64_t)((kb - tblocks) * (kATile >> 4));
#pragma unroll
            for (int i = 0; i < 4; ++i) { umma_bf16(d_tmem, a_desc + i * kStepA, b_desc + i * kStepB, idesc_s, acc); acc = 1; }
          } else {
            const uint32_t a_t = tmem + (uint32_t)(kb * 32);
#pragma unroll
            for (int i = 0; i < 4; ++i) { umma_bf16_ta(d_tmem, a_t + i * 8, b_desc + i * kStepB, idesc_t, acc); acc = 1; }
          }
        }
        if (ok) umma_commit(dfull);
      }
    }
    __syncwarp();
  } else if (warp >= kFetch0) {
    // ------------------------------------------------------------ fetch the state
    // A load of a warp is four batch rows of one K block (64 values), up to eight are in flight.  All of them poll (asking for
    // the first piece alone until it is there costs a second trip to L2: 2.4 instead of 2.2 us a step at 256 units).
    constexpr int kLoads = N / 8;                            // loads of a warp per piece, at most
    constexpr int kWindow = 8 / kLoads;                      // pieces in flight
    const int fw = warp - kFetch0, width = kBwd ? 4 * H : H, quads = B / 4;
    const __nv_bfloat16* state = (kBwd ? p.dG : p.y) + kbase + (size_t)(lane >> 3) * width + (lane & 7) * 8;
    bool ok = true;
    for (int s = 1; ok && s < T; ++s) {
      const uint32_t ph = (uint32_t)(s - 1) & 1u;
      const __nv_bfloat16* from = state + (size_t)(kBwd ? T - s : s - 1) * B * width;
      for (int j0 = 0; ok && j0 < npieces; j0 += kWindow) {
        uint4 v[kWindow][kLoads];
        auto chunk = [&](int w, int l, int& kb, int& b) {    // the l-th load of this warp in piece j0 + w; false: none
          const int j = j0 + w, piece = p0 + j < npieces ? p0 + j : p0 + j - npieces, c = fw + l * kFetchWarps;
          kb = piece * kPiece + c / quads;
          b = c % quads * 4;
          return j < npieces && c < kPiece * quads && kb < kblocks;
        };
        auto load_unset = [&](int w, bool all) {
#pragma unroll
          for (int l = 0; l < kLoads; ++l) {
            int kb, b;
            if (chunk(w, l, kb, b) && (all || unset(v[w][l]))) v[w][l] = ld_state(from + (size_t)b * width + kb * 64);
          }
        };
        auto complete = [&](int w) {
          bool missing = false;
#pragma unroll
          for (int l = 0; l < kLoads; ++l) {
            int kb, b;
            missing |= chunk(w, l, kb, b) && unset(v[w][l]);
          }
          return !__any_sync(0xffffffffu, missing);
        };
        Patience patience;
#pragma unroll
        for (int w = 0; w < kWindow; ++w) load_unset(w, true);
        if (s > 1 && j0 == 0 && ok) ok = __all_sync(0xffffffffu, wait_bar(dfull, ph ^ 1u, abort_flag));   // the last product has been taken
#pragma unroll
        for (int w = 0; w < kWindow; ++w) {
          const int j = j0 + w;
          if (!ok || j >= npieces) break;
          for (uint32_t it = 0; ok && !complete(w); ++it) {
#pragma unroll
            for (int x = w; x < kWindow; ++x) load_unset(x, false);
            ok = !__any_sync(0xffffffffu, patience.over(it, abort_flag));
          }
#pragma unroll
          for (int l = 0; l < kLoads; ++l) {
            int kb, b;
            if (!chunk(w, l, kb, b)) continue;
            b += lane >> 3;
            *reinterpret_cast<uint4*>(sB + kb * (N * 128) + b * 128 + (((lane & 7) ^ (b & 7)) << 4)) = v[w][l];
          }
          fence_proxy_async();                               // the tensor core reads what was written here
          __syncwarp();
          if (ok && lane == 0) mbar_arrive(&full[p0 + j < npieces ? p0 + j : p0 + j - npieces]);
        }
      }
    }
  } else {
    // ------------------------------------------------------------ cells
    const int q = warp & 3, half = warp >> 2;                // TMEM lane quarter, half of the batch columns
    const int dest = kBwd ? q : lane >> 4;                   // the mate that finalises this lane's unit
    const uint32_t p_remote = map_to_rank(smem_u32(sP), (uint32_t)dest);
    const uint32_t bar_remote = map_to_rank(smem_u32(&pfull[0]), (uint32_t)dest);
    const uint32_t part_bytes = (uint32_t)(S * (kBwd ? 1 : 4) * UNITS * N * 4);
    const int u = u0 + threadIdx.x % UNITS, b0 = threadIdx.x / UNITS * PER;        // this thread's unit and its PER batch rows
    float state[PER];                                        // c (forward) / dc (backward) of this thread's elements
#pragma unroll
    for (int e = 0; e < PER; ++e) state[e] = 0.0f;
    float db[4] = {0.0f, 0.0f, 0.0f, 0.0f};                  // backward: bias gradient of this thread's unit
    bool ok = true;        // same in all lanes of a warp; a warp that has given up still meets the others at the barriers
    for (int s = 0; s < T; ++s) {
      const int t = kBwd ? T - 1 - s : s;
      // what does not depend on the recurrence is on its way before the wait
      if (s > 0 && final_cta && threadIdx.x == 0) mbar_expect_tx(&pfull[(s - 1) & 1], part_bytes);
      float in[PER][4], cc[PER], dyv[PER], fgate[PER];
#pragma unroll
      for (int e = 0; e < PER; ++e) {
        const int b = b0 + e;
        if (b < B && final_cta) {
          const size_t row = (size_t)t * B + b;
          const __nv_bfloat16* g4 = (kBwd ? p.gates : p.xproj) + row * 4 * H + u;
#pragma unroll
          for (int k = 0; k < 4; ++k) in[e][k] = __bfloat162float(g4[(size_t)k * H]);
          if (kBwd) {
            // d(gate) = dc * in[gate] (output gate: dh * in), dc = state + dh * cc
            const float ig = in[e][0], fg = in[e][1], gg = in[e][2], og = in[e][3];
            const float tc = tanhf(p.c[row * H + u]), before = t > 0 ? p.c[(row - B) * H + u] : 0.0f;
            dyv[e] = __bfloat162float(p.dy[row * H + u]);
            cc[e] = og * (1.0f - tc * tc);
            in[e][0] = gg * ig * (1.0f - ig);
            in[e][1] = before * fg * (1.0f - fg);
            in[e][2] = ig * (1.0f - gg * gg);
            in[e][3] = tc * og * (1.0f - og);
            fgate[e] = fg;
          } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) in[e][k] += __ldg(p.bias + k * H + u);
          }
        }
      }
      const uint32_t ph = (uint32_t)(s - 1) & 1u;
      if (s > 0 && ok) ok = __all_sync(0xffffffffu, wait_bar(dfull, ph, abort_flag));
      if (s > 0 && ok) {
        tc_fence_after();
        uint32_t r[N / 2];
        const uint32_t t_row = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(L::kDCol + half * (N / 2));
#pragma unroll
        for (int i = 0; i < N / 16; ++i) tmem_ld_x8(t_row + i * 8, r + i * 8);
        constexpr int kAtOnce = N == 16 ? 3 : 1;
#pragma unroll
        for (int a0 = 1; a0 < kIssuers; a0 += kAtOnce) {
          uint32_t x[kAtOnce][N / 2];
#pragma unroll
          for (int a = 0; a < kAtOnce; ++a)
            if (a0 + a < kblocks) {
#pragma unroll
              for (int i = 0; i < N / 16; ++i) tmem_ld_x8(t_row + (a0 + a) * N + i * 8, x[a] + i * 8);
            }
          tmem_ld_wait();
#pragma unroll
          for (int a = 0; a < kAtOnce; ++a)
            if (a0 + a < kblocks) {
#pragma unroll
              for (int j = 0; j < N / 2; ++j) {
                asm volatile("" : "+r"(r[j]), "+r"(x[a][j]));        // no addition moves above the wait
                r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(x[a][j]));
              }
            }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(dfree);
        // partial sums to the finaliser: [parity][source rank][gate][unit][batch]
        const uint32_t dst = p_remote + 4u * (uint32_t)((int)ph * lay.part + ((kBwd ? rank : rank * 4 + q) * UNITS + lane % UNITS) * L::kPitch +
                                                        half * (N / 2));
#pragma unroll
        for (int j = 0; j < N / 2; j += 4) st_async_x4(dst + 4u * j, r + j, bar_remote + 8u * ph);
        if (final_cta) ok = __all_sync(0xffffffffu, wait_bar(&pfull[ph], (uint32_t)((s - 1) >> 1) & 1u, abort_flag));
      }
      if (final_cta && b0 < B) {          // a batch that is not there is a whole warp's, or none of its lanes'
        constexpr int SRC = 8, PITCH = UNITS * L::kPitch;  // blocks of [unit][batch]: up to 8 ranks; 2 ranks x 4 gates
        const float* part = sP + ((s - 1) & 1) * lay.part + threadIdx.x % UNITS * L::kPitch + b0;
        float sum[kBwd ? 1 : 4][PER];
#pragma unroll
        for (int e = 0; e < PER; ++e) {
          if (kBwd) sum[0][e] = dyv[e];
          else {
#pragma unroll
            for (int k = 0; k < 4; ++k) sum[kBwd ? 0 : k][e] = in[e][k];
          }
        }
        if (s > 0) {
          float v[SRC][PER];
#pragma unroll
          for (int k = 0; k < SRC; ++k)
            if (!kBwd || k < S) ld_shared_vec<PER>(v[k], part + k * PITCH);
#pragma unroll
          for (int k = 0; k < SRC; ++k)
            if (!kBwd || k < S) {
#pragma unroll
              for (int e = 0; e < PER; ++e) sum[kBwd ? 0 : k & 3][e] += v[k][e];
            }
        }
        if (!kBwd) {
          uint2 h4[PER];
#pragma unroll
          for (int e = 0; e < PER; ++e) {
            const float ig = sigmoidf_(sum[0][e]), fg = sigmoidf_(sum[kBwd ? 0 : 1][e]), gg = tanhf(sum[kBwd ? 0 : 2][e]),
                        og = sigmoidf_(sum[kBwd ? 0 : 3][e]);
            const float c = fg * state[e] + ig * gg;
            state[e] = c;
            h4[e] = gather_quad(bf16_bits(og * tanhf(c)), lane);
            in[e][0] = ig; in[e][1] = fg; in[e][2] = gg; in[e][3] = og;
          }
#pragma unroll
          for (int e = 0; e < PER; ++e)
            if ((lane & 3) == 0) publish(p.y + ((size_t)t * B + b0 + e) * H + u, h4[e]);
        } else {
          uint2 d4[PER];                                     // lane k of four publishes gate k
#pragma unroll
          for (int e = 0; e < PER; ++e) {
            const float dh = sum[0][e], dct = state[e] + dh * cc[e];
            state[e] = dct * fgate[e];
            const float d[4] = {dct * in[e][0], dct * in[e][1], dct * in[e][2], dh * in[e][3]};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint2 g = gather_quad(bf16_bits(d[k]), lane);
              if (k == 0 || (lane & 3) == k) d4[e] = g;
              db[k] += d[k];
            }
          }
#pragma unroll
          for (int e = 0; e < PER; ++e)
            publish(p.dG + (((size_t)t * B + b0 + e) * 4 + (lane & 3)) * H + (u & ~3), d4[e]);
        }
      }
      if (!kBwd) {                        // what only the backward pass reads leaves after the hand-over
#pragma unroll
        for (int e = 0; e < PER; ++e) {
          const int b = b0 + e;
          if (b < B) {
            const size_t row = (size_t)t * B + b;
            p.c[row * H + u] = state[e];
            __nv_bfloat16* gp = p.gates + row * 4 * H + u;
#pragma unroll
            for (int k = 0; k < 4; ++k) gp[(size_t)k * H] = __float2bfloat16(in[e][k]);
          }
        }
      }
    }
    if (kBwd && p.db != nullptr && final_cta) {              // a lane's elements all belong to unit u0 + lane
#pragma unroll
      for (int k = 0; k < 4; ++k) atomicAdd(p.db + (size_t)k * H + u0 + lane, db[k]);
    }
  }
  // ---------------------------------------------------------------- teardown: nobody leaves while a mate may still write here
  tc_fence_before();
  cluster_sync();
  __syncthreads();
  if (*abort_flag) {
    __nanosleep(1000000);
    if (threadIdx.x == 0 && p.error_flag != nullptr) atomicExch(p.error_flag, 1);
  }
  if (warp == kIssue0) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

int grid_of(bool bwd, int H, int S) { return (bwd ? H / 128 : H / 32) * S; }

// The cluster size for a layer of H units on the current device: the largest whose CTAs' share of the weights fits on the
// chip and whose whole grid can be resident at once; 0: none (asked once per kernel, H and device).
template <bool kBwd, int N>
int cluster_size(int H) {
  static int cache[64][17] = {};                  // 0 unknown, else 1 + size
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 0;
  int& v = cache[dev][H / 128];
  if (v == 0) {
    int found = 0;
    cudaError_t e = cudaFuncSetAttribute(lstm_sequence_kernel<kBwd, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
    for (int S = kBwd ? 8 : 2; e == cudaSuccess && found == 0 && S >= Layout<kBwd, N>::kFinal; --S) {
      const Layout<kBwd, N> lay(H, S);
      if (lay.smem() > kSmemLimit || lay.per * (S - 1) >= lay.kblocks ||      // too much per CTA; an empty CTA
          lay.per > kPiece * kMaxPieces) continue;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(grid_of(kBwd, H, S));
      cfg.blockDim = dim3(kThreads);
      cfg.dynamicSmemBytes = lay.smem();
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = S;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, lstm_sequence_kernel<kBwd, N>, &cfg) != cudaSuccess) cudaGetLastError();
      else if (n * S >= grid_of(kBwd, H, S)) found = S;
    }
    if (e != cudaSuccess) cudaGetLastError();
    v = 1 + found;
  }
  return v - 1;
}

template <bool kBwd, int N>
int launch(SeqParams& p, cudaStream_t stream) {
  const int H = p.H;
  p.S = cluster_size<kBwd, N>(H);
  if (p.S == 0) return -1;
  const Layout<kBwd, N> lay(H, p.S);
  {
    uint64_t dims[2] = {(uint64_t)H, (uint64_t)4 * H}, strides[1] = {(uint64_t)H * 2};
    uint32_t box[2] = {64, kBwd ? 64u : 32u};
    int r = esgd::make_tensormap_bf16(&p.tmW, p.w, 2, dims, strides, box, nullptr);
    if (r != 0) return 1000 + r;
  }
  cudaError_t e = cudaMemsetAsync(kBwd ? (void*)p.dG : (void*)p.y, 0xff, (size_t)p.T * p.B * H * (kBwd ? 8 : 2), stream);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid_of(kBwd, H, p.S));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = lay.smem();
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = p.S;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeCooperative;      // the CTAs wait for one another: all of them or none
  at[1].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  esgd::count_launch();
  return (int)cudaLaunchKernelEx(&cfg, lstm_sequence_kernel<kBwd, N>, (const SeqParams)p);
}

}  // namespace

extern "C" {

// Whether the persistent kernels take this shape on the current device: units a multiple of 128 up to 2048 (the weights
// must fit on the chip), a batch of up to 32 that is a multiple of 8, and every CTA resident.  1 yes, 0 no.  On a B200 that is
// every such shape but one: backward at 2048 units with a batch of 24 or 32 needs clusters of 8 for its shared memory, and only
// 15 of the 16 would be resident.
int esgd_lstm_persistent_ok(int B, int H, int backward) {
  if (B <= 0 || B > 32 || B % 8 || H < 128 || H > 2048 || H % 128) return 0;
  if (backward) return (B <= 16 ? cluster_size<true, 16>(H) : cluster_size<true, 32>(H)) > 0;
  return (B <= 16 ? cluster_size<false, 16>(H) : cluster_size<false, 32>(H)) > 0;
}

// xproj [T*B, 4H] bf16, w_hh [4H, H] bf16, bias [4H] fp32; out: c [T, B, H] fp32, y [T, B, H] bf16, gates [T, B, 4H] bf16.
int esgd_lstm_persistent_fwd(const void* xproj, const void* w_hh, const float* bias, float* c, void* y, void* gates,
                             int T, int B, int H, int* error_flag, void* stream) {
  if (T <= 0 || !esgd_lstm_persistent_ok(B, H, 0)) return -1;
  SeqParams p = {};
  p.w = (const __nv_bfloat16*)w_hh; p.T = T; p.B = B; p.H = H;
  p.xproj = (const __nv_bfloat16*)xproj; p.bias = bias; p.c = c; p.y = (__nv_bfloat16*)y; p.gates = (__nv_bfloat16*)gates;
  p.error_flag = error_flag;
  return B <= 16 ? launch<false, 16>(p, (cudaStream_t)stream) : launch<false, 32>(p, (cudaStream_t)stream);
}

// dG [T, B, 4H] bf16 (pre-activation gradients of every step) from dy [T, B, H] bf16 and the saved gates and cell states;
// db [4H] fp32 (or null) += their sum over steps and batch.
int esgd_lstm_persistent_bwd(const void* gates, const float* c, const void* dy, const void* w_hh, void* dG, float* db,
                             int T, int B, int H, int* error_flag, void* stream) {
  if (T <= 0 || !esgd_lstm_persistent_ok(B, H, 1)) return -1;
  SeqParams p = {};
  p.w = (const __nv_bfloat16*)w_hh; p.T = T; p.B = B; p.H = H;
  p.gates = (__nv_bfloat16*)gates; p.c = const_cast<float*>(c); p.dy = (const __nv_bfloat16*)dy; p.dG = (__nv_bfloat16*)dG; p.db = db;
  p.error_flag = error_flag;
  return B <= 16 ? launch<true, 16>(p, (cudaStream_t)stream) : launch<true, 32>(p, (cudaStream_t)stream);
}

}  // extern "C"
