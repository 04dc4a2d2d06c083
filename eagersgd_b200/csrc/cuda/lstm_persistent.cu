// The recurrence of an LSTM layer as ONE persistent kernel per direction (sm_100a: tcgen05 / TMEM / TMA / clusters).
//
// A time step is a product with the recurrent weights (32 MB of bf16 at 2048 units) and a few hundred bytes of state per
// SM; as two launches per step (split-K GEMM + cell kernel) it cost 13.8 us forward and 15.3 us backward at batch 16, bound
// by the two kernel boundaries and by re-reading the weights from L2.  Here every CTA keeps its share of the weights on
// chip for the whole sequence and a step is: fetch the previous step's state as it appears (32 KB), 64 MMAs, exchange
// partial sums inside the cluster, apply the cell to 16 units, publish.
//
//   weights   the A operand of tcgen05.mma, 64 columns of K at a time: the last 14 such blocks (224 KB; 12 forward with a
//             batch of 32, whose four accumulators are wider) in tensor memory, the others in shared memory, as the room left
//             by the state and the partial sums allows.  128 x 16 x 16 takes 12 cycles with A in tensor memory and 41 with A in
//             shared memory, so the latter go first, while the state arrives
//   forward   128 rows = 4 gates x 32 units, K = half of the hidden state: clusters of 2, H/16 CTAs
//   backward  128 rows = 128 units of dh (weights transposed), K = 4H split over clusters of up to 8 CTAs: the largest
//             cluster size whose whole grid is resident (of 16 clusters, a B200's GPCs hold 15 of size 8 or 7 but all of size 6)
//   cluster   each finalising CTA owns 16 (forward) or 32 (backward) units x batch: partial sums go to its shared memory, a
//             row of memory per store of a warp (st.async: the bytes carry their own arrival; 8 KB in pieces of 16 bytes took
//             1100 cycles, half of it here and rows of 256 bytes take 560), double buffered by step parity; a CTA can be at
//             most one step ahead of a cluster mate (it needs a state that transitively needs the mate's previous one), so
//             two buffers are enough
//   grid      the state is published by writing it to y (forward) or dG (backward), which are filled with a bit pattern that
//             no result has (0xffff per bf16; conversions round every NaN to 0x7fff) before the launch: eight warps fetch the
//             words they need until none of them is the pattern.  The data is its own flag, so no fence, counter or second
//             trip to L2 stands between a store and its use.  See hold_cycles() for when they begin.
//             Launched cooperatively (all CTAs resident); every wait is bounded and ends in the error flag.
//
// A step is bound by a chain of latencies.  Cycles at 2048 units and 16 sequences, forward / backward: from publishing to the
// state's being in shared memory 2400 / 2600 (a store is seen from the other die after 900, and an SM keeps 16 KB of loads in
// flight), the products behind the last of it 800 / 2100, reading them 500 / 450, the exchange 320 / 500, the cells 470 / 540.
// Microseconds a step, polling all the time, handing on pieces of four blocks and exchanging 16 bytes at a time as before / now,
// forward and backward: 256 units 2.4 / 1.8 and 2.7 / 1.9, 1024 units 3.3 / 2.1 and 3.7 / 2.3, 2048 units (in a training step)
// 4.1 / 2.4 and 5.5 / 3.2; 32 sequences, 1024 units 4.7 / 2.7 and 6.1 / 3.2.
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
constexpr int kIssue0 = kEpiThreads / 32;
constexpr int kATile = kRows * 128; // one 64-column block of A
constexpr int kMaxBlocks = 32;      // K blocks of a CTA
constexpr int kSmemLimit = 227 * 1024;
constexpr int kAhead = 4;           // steps
constexpr uint32_t kUnset = 0xffffffffu;      // two bf16 that have not been written yet
constexpr uint64_t kWaitNs = 4000000000ull;   // bound on every wait

struct SeqParams {
  CUtensorMap tmW;                  // recurrent weights
  const __nv_bfloat16* w;           // [4H][H]
  int T, B, H, S;                   // S: cluster size, the split of K
  uint32_t hold;                    // cycles between publishing and the first look at the others' part
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
// 16 bytes into a mate's shared memory, counted by its barrier.  The barrier takes in a row of memory at a time, so a warp's
// addresses have to be consecutive.
__device__ __forceinline__ void st_async_x4(uint32_t addr, const uint32_t* v, uint32_t bar_addr) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(bar_addr) : "memory");
}
// Orders nothing: with release semantics it waits for this thread's stores to memory first, which took 2000 cycles here.
__device__ __forceinline__ void mbar_arrive_relaxed_at(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
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
// kCluster: what the barrier announces came from another CTA.
template <bool kCluster = false>
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  Patience p;
  for (uint32_t it = 0; !(kCluster ? try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity)); ++it)
    if (p.over(it, abort_flag)) return false;
  return true;
}
__device__ __forceinline__ uint32_t clock32() {
  uint32_t t;
  asm volatile("mov.u32 %0, %%clock;" : "=r"(t));
  return t;
}
__device__ __forceinline__ uint4 ld_state(const void* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t newest(uint4 v) { return max(max(v.x, v.y), max(v.z, v.w)); }    // kUnset: one is not there
__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float2 f32_pair(uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void publish(void* p, uint32_t v) { asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
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
  // Warps that issue MMAs, one on each scheduler of the SM, each with an accumulator of its own.  With a batch of 32 the backward
  // pass would spill over reading four of them (1024 units: 3.9 us a step, with two 3.2).
  static constexpr int kIssuers = kBwd && N == 32 ? 2 : 4;
  static constexpr int kFetch0 = kIssue0 + kIssuers;
  static constexpr int kThreads = (kFetch0 + kFetchWarps) * 32;
  static constexpr int kUnits = kBwd ? 32 : 16;                       // units a finalising CTA owns
  static constexpr int kFinal = kBwd ? 4 : 2;                         // finalising CTAs of a cluster
  static constexpr int kActive = kUnits / 2 * N < kEpiThreads ? kUnits / 2 * N : kEpiThreads;       // finalising threads, and how
  static constexpr int kPer = kUnits / 2 * N / kActive;               // many elements of a pair of units each of them has
  static constexpr int kTBlocks = 16 - kIssuers * N / 32;             // K blocks of the weights in tensor memory, 32 columns each
  static constexpr int kDCol = kTBlocks * 32;                         // the issuers' accumulators, N columns each
  static constexpr int kLocal = kBwd ? 2 : kEpiThreads / 32;          // warps of a finalising CTA that sum for it themselves
  int kblocks, per, tblocks, sblocks, part;                           // per: K blocks of a CTA (the last may have fewer);
                                                                      // part: floats for one step's partial sums
  __host__ __device__ Layout(int H, int S) {
    kblocks = (kBwd ? 4 * H : H) / 64;
    per = (kblocks + S - 1) / S;
    tblocks = per < kTBlocks ? per : kTBlocks;
    sblocks = per - tblocks;
    part = S * (kBwd ? 1 : 4) * kUnits * N;
  }
  int smem() const { return 1024 + sblocks * kATile + per * (N * 128) + 2 * part * 4 + 512; }
};

template <bool kBwd, int N>
__global__ void __launch_bounds__(Layout<kBwd, N>::kThreads, 1) lstm_sequence_kernel(const __grid_constant__ SeqParams p) {
  using L = Layout<kBwd, N>;
  constexpr int kIssuers = L::kIssuers, kFetch0 = L::kFetch0, kThreads = L::kThreads;
  constexpr int PER = L::kPer, UNITS = L::kUnits;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int H = p.H, B = p.B, T = p.T, S = p.S;
  const L lay(H, S);
  const int rank = (int)cluster_rank(), group = blockIdx.x / S;
  const int kblocks = min(lay.per, lay.kblocks - rank * lay.per);     // K blocks of this CTA: the last tblocks of them in tensor
  const int tblocks = min(kblocks, lay.tblocks), sblocks = kblocks - tblocks;      // memory, the others in shared memory
  const int kbase = rank * lay.per * 64;                              // its K range: h units, or rows of the weights (gates)
  uint8_t* sA = smem;
  uint8_t* sB = sA + lay.sblocks * kATile;
  float* sP = reinterpret_cast<float*>(sB + lay.per * (N * 128));
  uint64_t* full = reinterpret_cast<uint64_t*>(sP + 2 * lay.part);    // [kMaxBlocks] a block of the state is in place
  uint64_t* wfull = full + kMaxBlocks;                                 // the weights have landed
  uint64_t* dfull = wfull + 1;                                        // the step's product is in tensor memory
  uint64_t* dfree = dfull + 1;                                        // ... and has been read out of it
  uint64_t* pfull = dfree + 1;                                        // [2] partial sums of all cluster mates are here
  uint64_t* pub = pfull + 2;                                          // the cells here, or a mate's, have published the step
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pub + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const bool final_cta = rank < L::kFinal;
  const int u0 = (kBwd ? group * 128 : group * 32) + rank * UNITS;    // first unit this CTA finalises

  if (threadIdx.x == 0) {
    for (int i = 0; i < kMaxBlocks; ++i) mbar_init(&full[i], 1);
    mbar_init(wfull, 1);
    mbar_init(dfull, kIssuers);
    mbar_init(dfree, kEpiThreads / 32);
    mbar_init(&pfull[0], 1 + L::kLocal);
    mbar_init(&pfull[1], 1 + L::kLocal);
    mbar_init(pub, L::kActive / 32);
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
      mbar_expect_tx(wfull, (uint32_t)(sblocks * kATile));
      for (int kb = 0; kb < sblocks; ++kb) {
        uint8_t* a = sA + kb * kATile;
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
        const __nv_bfloat16* src = p.w + (size_t)(kbase + sblocks * 64 + k0) * H + group * 128 + row;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint32_t lo = __bfloat16_as_ushort(src[(size_t)(2 * i) * H]), hi = __bfloat16_as_ushort(src[(size_t)(2 * i + 1) * H]);
          r[i] = lo | (hi << 16);
        }
      } else {
        const uint4* src = reinterpret_cast<const uint4*>(p.w + ((size_t)q * H + group * 32 + lane) * H + kbase + sblocks * 64 + k0);
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
    constexpr uint64_t kStepA = kBwd ? (2048 >> 4) : (32 >> 4), kStepB = 32 >> 4;
    // The thread's own instructions between two MMAs bound it (one issuer: 40 to 57 cycles apart, 128 x 16 x 16 is a
    // fraction of that), so four of them share the K blocks of a piece, each with an accumulator of its own.
    const int issuer = warp - kIssue0;
    const uint32_t d_tmem = tmem + (uint32_t)(L::kDCol + issuer * N);
    const uint64_t b_desc0 = umma_smem_desc(smem_u32(sB) + issuer * (N * 128), 16, 1024);
    const uint64_t a_desc0 = kBwd ? umma_smem_desc(smem_u32(sA), 8192, 1024) : umma_smem_desc(smem_u32(sA), 16, 1024);
    if (elect_one()) {
      bool ok = wait_bar(wfull, 0u, abort_flag);
      for (int s = 1; ok && s < T; ++s) {                    // step 0 has no recurrent product
        const uint32_t ph = (uint32_t)(s - 1) & 1u;
        if (s > 1) ok = wait_bar(dfree, ph ^ 1u, abort_flag);               // the previous product has been read
        uint32_t acc = 0;
        uint64_t b_desc = b_desc0;
        for (int kb = issuer; kb < kblocks; kb += kIssuers, b_desc += kIssuers * (N * 128 >> 4)) {
          ok = wait_bar(&full[kb], ph, abort_flag);
          if (!ok) break;
          tc_fence_after();
          if (kb >= sblocks) {
            const uint32_t a_t = tmem + (uint32_t)((kb - sblocks) * 32);
#pragma unroll
            for (int i = 0; i < 4; ++i) { umma_bf16_ta(d_tmem, a_t + i * 8, b_desc + i * kStepB, idesc_t, acc); acc = 1; }
          } else {
            const uint64_t a_desc = a_desc0 + (uint64_t)(kb * (kATile >> 4));
#pragma unroll
            for (int i = 0; i < 4; ++i) { umma_bf16(d_tmem, a_desc + i * kStepA, b_desc + i * kStepB, idesc_s, acc); acc = 1; }
          }
        }
        if (ok) umma_commit(dfull);
      }
    }
    __syncwarp();
  } else if (warp >= kFetch0) {
    // ------------------------------------------------------------ fetch the state
    // A warp has every eighth K block, loads of 64 values of four batch rows each.  All loads poll (asking for some of them alone
    // until they are there costs a second trip to L2).  A block is handed on as soon as it is complete, with as few instructions
    // as that takes: the warps have latency and no parallelism to hide it (divisions for the place of a load cost 250 cycles a block).
    constexpr int kQuads = N / 4;                            // loads of a block
    constexpr int kWindow = N == 16 ? 2 : 1;                 // blocks of a warp in flight
    const int fw = warp - kFetch0, quads = B / 4, width = kBwd ? 4 * H : H;
    bool ok = true;
    const uint32_t row_step = (uint32_t)width * 8, at = (uint32_t)(lane >> 3) * width * 2 + fw * 128 + (lane & 7) * 16;       // bytes
    const char* const state = reinterpret_cast<const char*>((kBwd ? p.dG : p.y) + kbase) + at;
    uint8_t* const landing = sB + fw * (N * 128) + (lane >> 3) * 128;
    const int swz[2] = {((lane & 7) ^ (lane >> 3)) << 4, ((lane & 7) ^ (4 + (lane >> 3))) << 4};
    // A CTA with fewer blocks than warps: a warp without one stays out.  Nothing makes a step wait for it, so it could fall two
    // steps behind `pub`, whose parity would then hide them from it.  (A warp with a block is waited for: its block is part of the
    // product without which nobody publishes the next step.)
    for (int s = 1; ok && fw < kblocks && s < T; ++s) {
      const char* const from = state + (size_t)(kBwd ? T - s : s - 1) * B * width * 2;
      uint4 v[kWindow][kQuads];
      auto load = [&](uint4 (&x)[kQuads], int kb, bool all) {
#pragma unroll
        for (int q = 0; q < kQuads; ++q)
          if (q < quads && (all || newest(x[q]) == kUnset)) x[q] = ld_state(from + q * row_step + (kb - fw) * 128);
      };
      // not before this cluster's cells have published, too: the last product has been taken, and the others' are no earlier
      ok = __all_sync(0xffffffffu, wait_bar(pub, (uint32_t)(s - 1) & 1u, abort_flag));
      for (const uint32_t t0 = clock32(); clock32() - t0 < p.hold;) {}
#pragma unroll
      for (int w = 0; w < kWindow; ++w)
        if (fw + w * kFetchWarps < kblocks) load(v[w], fw + w * kFetchWarps, true);
      for (int k0 = fw; ok && k0 < kblocks; k0 += kWindow * kFetchWarps) {
#pragma unroll
        for (int w = 0; w < kWindow; ++w) {
          const int kb = k0 + w * kFetchWarps;
          if (!ok || kb >= kblocks) break;
          Patience patience;
          for (uint32_t it = 0;; ++it) {
            uint32_t worst = 0;
#pragma unroll
            for (int q = 0; q < kQuads; ++q)
              if (q < quads) worst = max(worst, newest(v[w][q]));
            if (!__any_sync(0xffffffffu, worst == kUnset)) break;
            load(v[w], kb, false);
            ok = !__any_sync(0xffffffffu, patience.over(it, abort_flag));
            if (!ok) break;
          }
          uint8_t* dst = landing + (kb - fw) * (N * 128);
#pragma unroll
          for (int q = 0; q < kQuads; ++q)
            if (q < quads) *reinterpret_cast<uint4*>(dst + q * 512 + swz[q & 1]) = v[w][q];
          if (kb + kWindow * kFetchWarps < kblocks) load(v[w], kb + kWindow * kFetchWarps, true);
          fence_proxy_async();                               // the tensor core reads what was written here
          __syncwarp();
          if (ok && lane == 0) mbar_arrive(&full[kb]);
        }
      }
    }
  } else {
    // ------------------------------------------------------------ cells
    const int q = warp & 3, half = warp >> 2;                // TMEM lane quarter, half of the batch columns
    const int dest = kBwd ? q : lane >> 4;                   // the mate that finalises this lane's unit
    const uint32_t p_remote = map_to_rank(smem_u32(sP), (uint32_t)dest);
    const uint32_t bar_remote = map_to_rank(smem_u32(&pfull[0]), (uint32_t)dest);
    const uint32_t part_bytes = (uint32_t)((S - 1) * (kBwd ? 1 : 4) * UNITS * N * 4);      // from the mates
    // the partial sums of a step: [source rank][gate][four batch rows][unit][4], so that a store of a warp is one row of memory
    const int p_at = ((kBwd ? rank : rank * 4 + q) * (N / 4) + half * (N / 8)) * UNITS * 4 + (lane % UNITS / 2 + (lane & 1) * (UNITS / 2)) * 4;
    const uint32_t pub_remote = map_to_rank(smem_u32(pub), (uint32_t)(rank + L::kFinal < S ? rank + L::kFinal : 0));
    // this thread's units, u and u + 1, and its batch rows, b0 and b0 + N / PER: a warp has eight pairs of four rows
    const int pair = UNITS == 16 ? threadIdx.x % 8 : threadIdx.x % 8 + (threadIdx.x / 32 & 1) * 8;
    const int u = u0 + 2 * pair, b0 = UNITS == 16 ? threadIdx.x / 8 : threadIdx.x / 8 % 4 + threadIdx.x / 64 * 4;
    const bool finalises = final_cta && threadIdx.x < L::kActive;
    float state[PER][2];                                     // c (forward) / dc (backward) of this thread's elements
#pragma unroll
    for (int e = 0; e < PER; ++e) state[e][0] = state[e][1] = 0.0f;
    float db[4][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}};       // backward: bias gradient of this thread's units
    bool ok = true;        // same in all lanes of a warp; a warp that has given up still meets the others at the barriers
    for (int s = 0; s < T; ++s) {
      const int t = kBwd ? T - 1 - s : s;
      // what does not depend on the recurrence is on its way before the wait
      if (s > 0 && final_cta && threadIdx.x == 0) mbar_expect_tx(&pfull[(s - 1) & 1], part_bytes);
      float in[PER][4][2], cc[PER][2], dyv[PER][2], fgate[PER][2];
#pragma unroll
      for (int e = 0; e < PER; ++e) {
        const int b = b0 + e * (N / PER);
        if (b < B && finalises) {
          const size_t row = (size_t)t * B + b;
          const __nv_bfloat16* g4 = (kBwd ? p.gates : p.xproj) + row * 4 * H + u;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 f = f32_pair(*reinterpret_cast<const uint32_t*>(g4 + (size_t)k * H));
            in[e][k][0] = f.x;
            in[e][k][1] = f.y;
          }
          if (kBwd) {
            const float2 c = *reinterpret_cast<const float2*>(p.c + row * H + u);
            const float2 before = t > 0 ? *reinterpret_cast<const float2*>(p.c + (row - B) * H + u) : make_float2(0.0f, 0.0f);
            const float2 d = f32_pair(*reinterpret_cast<const uint32_t*>(p.dy + row * H + u));
            dyv[e][0] = d.x;
            dyv[e][1] = d.y;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              // d(gate) = dc * in[gate] (output gate: dh * in), dc = state + dh * cc
              const float ig = in[e][0][i], fg = in[e][1][i], gg = in[e][2][i], og = in[e][3][i], tc = tanhf(i ? c.y : c.x);
              cc[e][i] = og * (1.0f - tc * tc);
              in[e][0][i] = gg * ig * (1.0f - ig);
              in[e][1][i] = (i ? before.y : before.x) * fg * (1.0f - fg);
              in[e][2][i] = ig * (1.0f - gg * gg);
              in[e][3][i] = tc * og * (1.0f - og);
              fgate[e][i] = fg;
            }
          } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              in[e][k][0] += __ldg(p.bias + k * H + u);
              in[e][k][1] += __ldg(p.bias + k * H + u + 1);
            }
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
        constexpr int kAtOnce = kIssuers - 1;
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
        const int at = (int)ph * lay.part + p_at;
        if (dest == rank) {
#pragma unroll
          for (int j = 0; j < N / 2; j += 4) *reinterpret_cast<uint4*>(sP + at + j * UNITS) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
        } else {
#pragma unroll
          for (int j = 0; j < N / 2; j += 4) st_async_x4(p_remote + 4u * (uint32_t)(at + j * UNITS), r + j, bar_remote + 8u * ph);
        }
        if (!kBwd || q == rank) {
          __syncwarp();
          if (lane == 0) mbar_arrive(&pfull[ph]);
        }
        if (final_cta) ok = __all_sync(0xffffffffu, wait_bar<true>(&pfull[ph], (uint32_t)((s - 1) >> 1) & 1u, abort_flag));
      }
      if (finalises) {
        constexpr int SRC = kBwd ? 8 : 4;                  // blocks of one source: up to 8 ranks; 2 ranks x 4 gates
        const float* part = sP + ((s - 1) & 1) * lay.part + (b0 / 4 * UNITS + pair) * 4 + b0 % 4;
        float sum[PER][kBwd ? 1 : 4][2];
#pragma unroll
        for (int e = 0; e < PER; ++e)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (kBwd) sum[e][0][i] = dyv[e][i];
            else {
#pragma unroll
              for (int k = 0; k < 4; ++k) sum[e][kBwd ? 0 : k][i] = in[e][k][i];
            }
          }
        if (s > 0) {
#pragma unroll
          for (int k = 0; k < SRC; ++k)
#pragma unroll
            for (int e = 0; e < PER; ++e)
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                const float* at = part + k * UNITS * N + e * (N / PER) * UNITS + i * UNITS * 2;
                if (!kBwd) sum[e][kBwd ? 0 : k][i] += at[0] + at[4 * UNITS * N];
                else if (k < S) sum[e][0][i] += at[0];
              }
        }
        if (!kBwd) {
#pragma unroll
          for (int e = 0; e < PER; ++e) {
            float h[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const float ig = sigmoidf_(sum[e][0][i]), fg = sigmoidf_(sum[e][kBwd ? 0 : 1][i]), gg = tanhf(sum[e][kBwd ? 0 : 2][i]),
                          og = sigmoidf_(sum[e][kBwd ? 0 : 3][i]);
              const float c = fg * state[e][i] + ig * gg;
              state[e][i] = c;
              h[i] = og * tanhf(c);
              in[e][0][i] = ig; in[e][1][i] = fg; in[e][2][i] = gg; in[e][3][i] = og;
            }
            const int b = b0 + e * (N / PER);
            if (b < B) publish(p.y + ((size_t)t * B + b) * H + u, bf16_pair(h[0], h[1]));
          }
        } else {
#pragma unroll
          for (int e = 0; e < PER; ++e) {
            const int b = b0 + e * (N / PER);
            if (b >= B) continue;
            float d[4][2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const float dh = sum[e][0][i], dct = state[e][i] + dh * cc[e][i];
              state[e][i] = dct * fgate[e][i];
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                d[k][i] = (k < 3 ? dct : dh) * in[e][k][i];
                db[k][i] += d[k][i];
              }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) publish(p.dG + (((size_t)t * B + b) * 4 + k) * H + u, bf16_pair(d[k][0], d[k][1]));
          }
        }
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(pub);
          if (rank + L::kFinal < S) mbar_arrive_relaxed_at(pub_remote);
        }
        // The lines that this thread's units are published to some steps on, filled before the launch, may have left L2 since; a
        // reader would then wait for memory.
        if ((lane & 7) == 0 && s + kAhead < T) {
          const int64_t row = (int64_t)(kBwd ? t - kAhead : t + kAhead) * B;
#pragma unroll
          for (int e = 0; e < PER; ++e) {
            const int b = b0 + e * (N / PER);
#pragma unroll
            for (int k = 0; k < (kBwd ? 4 : 1); ++k)
              if (b < B) prefetch_l2(kBwd ? p.dG + ((row + b) * 4 + k) * H + u : p.y + (row + b) * H + u);
          }
        }
        if (!kBwd) {                      // what only the backward pass reads leaves after the hand-over
#pragma unroll
          for (int e = 0; e < PER; ++e) {
            const int b = b0 + e * (N / PER);
            if (b < B) {
              const size_t row = (size_t)t * B + b;
              *reinterpret_cast<float2*>(p.c + row * H + u) = make_float2(state[e][0], state[e][1]);
#pragma unroll
              for (int k = 0; k < 4; ++k)
                *reinterpret_cast<uint32_t*>(p.gates + (row * 4 + k) * H + u) = bf16_pair(in[e][k][0], in[e][k][1]);
            }
          }
        }
      }
    }
    if (kBwd && p.db != nullptr && finalises) {              // lanes 8 apart have the same units
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float v = db[k][i];
          v += __shfl_xor_sync(0xffffffffu, v, 8);
          v += __shfl_xor_sync(0xffffffffu, v, 16);
          if (lane < 8) atomicAdd(p.db + (size_t)k * H + u + i, v);
        }
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

// How long after the cluster has published its own part a CTA asks for the others'.  Who asks too early asks twice, and one
// CTA that is late makes all of them late; the other die sees a store after 900 cycles, and a grid of few CTAs sits on one.
// Forward, microseconds a step without / with it (16 CTAs are 256 units), 8, 16 and 32 sequences: 16 CTAs 1.59 / 1.66, 1.70 / 1.76,
// 2.26 / 2.23; 48 1.93 / 1.93, 2.02 / 1.99, 2.77 / 2.67; 56 1.97 / 1.97, 2.07 / 2.05, 2.86 / 2.73; 64 1.97 / 1.97, 2.07 / 2.06, 2.87 /
// 2.75; 72 2.16 / 2.07, 2.26 / 2.18, 3.03 / 3.05; 80 2.31 / 2.08, 2.44 / 2.17, 3.20 / 3.08; 128 2.60 / 2.38, 2.75 / 2.49, 3.55 / 3.42.
// With 64 it has stopped costing and from 72 on it gives.  Backward, whose CTAs read more and are later anyway, in a training step
// of 16 sequences: 64 CTAs (1024 units) 2.26 / 2.29, 96 (2048) 3.20 / 3.37.
uint32_t hold_cycles(bool bwd, int ctas) { return !bwd && ctas >= 64 ? 350u : 0u; }

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
          lay.per > kMaxBlocks) continue;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(grid_of(kBwd, H, S));
      cfg.blockDim = dim3(Layout<kBwd, N>::kThreads);
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
  p.hold = hold_cycles(kBwd, grid_of(kBwd, H, p.S));
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
  cfg.blockDim = dim3(Layout<kBwd, N>::kThreads);
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
