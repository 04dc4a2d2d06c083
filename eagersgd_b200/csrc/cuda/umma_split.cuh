// Products with few output tiles and a long reduction (the last layers for one image: 49 x 512 over 4608): the reduction of a tile
// is split over a cluster of CTAs.
//
// The persistent pipeline (umma_pipeline.cuh) gives a tile to one CTA, which then reads all of the tile's filters by itself, 24 KB a
// k-block at the 50 to 60 bytes a cycle that one SM gets out of L2, while the others have nothing to do.  Here each CTA of a cluster
// multiplies a share of the k-blocks, leaves its 128 x 64 partial sums (fp32) in its own shared memory, and finishes 1 / S of the
// rows: it adds the partial sums of all by way of the cluster's shared memory, in the order of the reduction, then the affine map,
// residual and ReLU.
// One image, pipeline and split: 7 x 7 x 512, 3x3 15.8 us and 6.5; 14 x 14 x 256 10.0 and 6.5; 28 x 28 x 128 8.2 and 6.3; 49 x 512 x 2048
// 7.9 and 5.1.  Sixteen images of the first: 16.4 and 12.3; of the second the pipeline, 10.6.
#pragma once
#include "umma_pipeline.cuh"

namespace umma {

struct SplitOut {
  __nv_bfloat16* out;        // [rows][ld], dense in the tiles' order
  int ld, n_tiles, kb_total, kb_per_cta;
};

constexpr int SPLIT_THREADS = 192;                    // loads, products, four epilogue warps
constexpr int SPLIT_STAGES = 8;
constexpr int SPLIT_PITCH = 64 * 4 + 16;              // bytes of a row of partial sums: an odd number of 16
constexpr int SPLIT_STAGE_BYTES = A_STAGE_BYTES + 64 * BK * 2;
constexpr int SPLIT_SMEM = SPLIT_STAGES * SPLIT_STAGE_BYTES + 256;

// CTAs of a cluster for `tiles` tiles of `blocks` k-blocks; 1: the pipeline takes them.  All clusters have to be resident at once, and
// a cluster lies within one of the GPU's groups of SMs: 16 clusters of eight do not fit a B200 (2 x 14 x 14 x 256, 3x3: 12.2 us, the
// pipeline 10.1, clusters of four 6.6).  With eight blocks sharing them costs more than it gives (7 x 7, 512 to 2048 channels: 5.2 us,
// the pipeline 4.8), with 16 it begins to pay (1x1, 1024 to 2048 channels: 5.7 and 6.5; 1024 to 256: clusters of eight
// 6.0, of four 5.4, the pipeline 5.9).
constexpr int kOutside8 = 28, kOutside4 = 16;         // of a B200's 148 SMs, the ones that no cluster of eight, of four takes
inline int split_ctas(int64_t tiles, int blocks, int sms) {
  if (blocks < 16) return 1;
  if (tiles * 8 <= sms - kOutside8 && blocks > 16) return 8;
  if (tiles * 4 <= sms - kOutside4) return 4;
  return tiles * 2 <= sms ? 2 : 1;
}

__device__ __forceinline__ float4 ld_cluster(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}

template <class P, int S>
__device__ __forceinline__ void run_split(const P& prob, const Epilogue& ep, const SplitOut& so) {
  static_assert(P::BN == 64 && !P::kPair && !P::kHalo && !P::kZeroStages, "plain tiles of 64 columns");
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + SPLIT_STAGES * SPLIT_STAGE_BYTES);
  uint64_t* empty = full + SPLIT_STAGES;
  uint64_t* done = empty + SPLIT_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int rank = blockIdx.x % S, id = blockIdx.x / S;
  if (smem_u32(smem) & 1023u) {                       // the same for all
    if (threadIdx.x == 0 && ep.error_flag != nullptr) atomicExch(ep.error_flag, 1);
    return;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < SPLIT_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 64);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  typename P::Tile t;
  prob.place(id / so.n_tiles, id % so.n_tiles, t);
  t.kb0 = min(rank * so.kb_per_cta, so.kb_total);
  t.kb1 = min(t.kb0 + so.kb_per_cta, so.kb_total);    // the last ones may have none
  esgd::pdl_enter();

  // what the rows that this CTA finishes need, asked for before the products: thread e has columns 8 (e % 8) .. + 7 of every 16th row
  constexpr int kRows = 128 / S, kTurns = kRows * 8 / 128 > 0 ? kRows * 8 / 128 : 1;
  const int e = (int)threadIdx.x - 64, col = t.n0 + (e & 7) * 8, prefix = prob.valid_prefix(t);
  const int64_t row0 = prob.first_row(t);
  float scale[8], shift[8];
  uint4 res[kTurns];
  bool mine[kTurns];
  if (warp == 0) {
    if (elect_one()) {
      typename P::Step at = prob.begin(t);
      const uint32_t tx = ep.tx_bytes ? ep.tx_bytes : (uint32_t)SPLIT_STAGE_BYTES;
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = t.kb0; kb < t.kb1; ++kb, prob.advance(at)) {
        if (!mbar_wait(&empty[stage], phase ^ 1u, abort_flag)) break;
        mbar_expect_tx(&full[stage], tx);
        uint8_t* a = smem + stage * SPLIT_STAGE_BYTES;
        prob.load(t, at, a, a + A_STAGE_BYTES, &full[stage]);
        if (++stage == SPLIT_STAGES) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(BM, prob.n_mma, P::A_MN ? 1 : 0, P::B_MN ? 1 : 0);
      constexpr uint64_t sa = P::A_MN ? (2048 >> 4) : (32 >> 4), sb = P::B_MN ? (2048 >> 4) : (32 >> 4);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = t.kb0; kb < t.kb1; ++kb) {
        ok = mbar_wait(&full[stage], phase, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint32_t base = smem_u32(smem + stage * SPLIT_STAGE_BYTES);
        const uint64_t a = P::A_MN ? umma_smem_desc(base, 8192, 1024) : umma_smem_desc(base, 16, 1024);
        const uint64_t b = P::B_MN ? umma_smem_desc(base + A_STAGE_BYTES, 8192, 1024) : umma_smem_desc(base + A_STAGE_BYTES, 16, 1024);
        for (int j = 0; j < prob.ksteps; ++j) umma_bf16(tmem, a + j * sa, b + j * sb, idesc, kb > t.kb0 || j > 0 ? 1u : 0u);
        umma_commit(&empty[stage]);
        if (++stage == SPLIT_STAGES) { stage = 0; phase ^= 1u; }
      }
      if (ok) umma_commit(done);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const bool in = col + i < ep.n_total;
      scale[i] = ep.scale != nullptr && in ? __ldg(ep.scale + col + i) : 1.0f;
      shift[i] = ep.bias != nullptr && in ? __ldg(ep.bias + col + i) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < kTurns; ++u) {
      const int r = rank * kRows + (e >> 3) + u * 16;
      mine[u] = (e >> 3) + u * 16 < kRows && r < prefix && col < ep.n_total;
      res[u] = make_uint4(0, 0, 0, 0);
      if (mine[u] && ep.residual != nullptr)
        res[u] = __ldg(reinterpret_cast<const uint4*>((const __nv_bfloat16*)ep.residual + (row0 + r) * ep.ldr + col));
    }
    const int q = warp & 3;
    if (__all_sync(0xffffffffu, t.kb1 > t.kb0 && mbar_wait(done, 0u, abort_flag))) {
      tc_fence_after();
      // every load and product of this CTA is done: the stages are free
      float4* to = reinterpret_cast<float4*>(smem + (q * 32 + lane) * SPLIT_PITCH);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t v[32];
        tmem_ld_32x32b_x32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * 32), v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j)
          to[half * 8 + j] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
      }
      tc_fence_before();
    }
  }
  __syncwarp();
  cluster_sync_all();
  if (warp >= 2) {
    const int parts = (so.kb_total + so.kb_per_cta - 1) / so.kb_per_cta;
#pragma unroll
    for (int u = 0; u < kTurns; ++u) {
      if (!mine[u]) continue;
      const int r = rank * kRows + (e >> 3) + u * 16;
      const uint32_t here = smem_u32(smem + r * SPLIT_PITCH + (e & 7) * 32);
      float4 lo[S], hi[S];
#pragma unroll
      for (int p = 0; p < S; ++p) {
        uint32_t there;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(here), "r"(p));
        lo[p] = hi[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (p < parts) {
          lo[p] = ld_cluster(there);
          hi[p] = ld_cluster(there + 16);
        }
      }
      float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int p = 0; p < S; ++p) {
        v[0] += lo[p].x; v[1] += lo[p].y; v[2] += lo[p].z; v[3] += lo[p].w;
        v[4] += hi[p].x; v[5] += hi[p].y; v[6] += hi[p].z; v[7] += hi[p].w;
      }
      const uint32_t* rw = reinterpret_cast<const uint32_t*>(&res[u]);
      uint4 pk;
      __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float a = v[2 * i], b = v[2 * i + 1];
        if (ep.bias != nullptr) {
          a = fmaf(a, scale[2 * i], shift[2 * i]);
          b = fmaf(b, scale[2 * i + 1], shift[2 * i + 1]);
        }
        if (ep.residual != nullptr) {
          a += __uint_as_float(rw[i] << 16);
          b += __uint_as_float(rw[i] & 0xffff0000u);
        }
        if (ep.relu) {
          a = fmaxf(a, 0.0f);
          b = fmaxf(b, 0.0f);
        }
        h[i] = __floats2bfloat162_rn(a, b);
      }
      *reinterpret_cast<uint4*>(so.out + (row0 + r) * so.ld + col) = pk;
    }
  }
  __syncwarp();
  cluster_sync_all();                                 // nobody leaves while its sums are being read
  if (*abort_flag) {
    __nanosleep(1000000);
    if (threadIdx.x == 0 && ep.error_flag != nullptr) atomicExch(ep.error_flag, 1);
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 64);
  }
}

template <int S, class K, class P>
int launch_split(K kernel, int tiles, cudaStream_t stream, const P& p, const Epilogue& ep, const SplitOut& so) {
  static esgd::SmemAllowed allowed{0};       // one for each kernel: its type is the instance's
  if (const int e = esgd::allow_smem(kernel, SPLIT_SMEM, allowed)) return e;
  return esgd::launch<S>(kernel, dim3(tiles * S), SPLIT_THREADS, SPLIT_SMEM, stream, p, ep, so);
}

}  // namespace umma
