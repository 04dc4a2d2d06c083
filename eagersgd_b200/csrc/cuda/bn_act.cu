// Fused batch-norm kernels for NHWC bf16 activations viewed as [M = N*H*W, C].
//
//   bn_stats        : per-channel sum / sum of squares (fp32) of a conv output
//   bn_fwd          : mean / inv-std, scale / shift, running-statistics update and
//                     z = act(scale*y + shift [+ residual])           (one read, one write)
//   bn_coefficients : inference scale / shift of every layer of a network
//   bn_bwd_reduce   : g = dz * [z > 0];  dbeta = sum g, dgamma = sum g*xhat
//   bn_bwd_apply    : dy = gamma*invstd*(g - dbeta/M - xhat*dgamma/M), optional dres = g
//
// Training-mode semantics, momentum and eps follow the reference model
// (official/resnet/resnet_model.py:51-60: decay 0.997, eps 1e-5, fused=True) and its
// CPU restatement (deep500 .../cpp/operators/batchnormalization_op_training.cpp:48-329).
// A thread owns a group of 8 channels (one 16-byte vector) of every k-th row.  A block covers up to 16 groups (256-byte row
// segments) and 16 or more rows at a time; the grid splits rows and, for wide layers, channels: with whole rows per block a
// 2048-channel reduction sent 1.2 million atomics and reloaded all coefficients every five rows.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include "launch.cuh"

namespace {

using esgd::pdl_enter;

__device__ __forceinline__ uint4 st8(__nv_bfloat16* p, const float v[8]) {
  uint4 raw;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
  for (int q = 0; q < 4; ++q) h[q] = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
  *reinterpret_cast<uint4*>(p) = raw;
  return raw;
}
// Bit q: element q of eight stored bf16 values (none negative) is above zero.
__device__ __forceinline__ uint8_t sign_bits(const uint4& w) {
  const uint32_t x[4] = {w.x, w.y, w.z, w.w};
  uint32_t m = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) m |= ((x[q] & 0x7fffu) ? 1u << (2 * q) : 0u) | ((x[q] & 0x7fff0000u) ? 2u << (2 * q) : 0u);
  return (uint8_t)m;
}

// Blocks of a kernel that are resident on an SM, and the size of its grid.  With more of them every block beyond these starts
// over with its coefficients and the last wave is partly empty; with more registers a thread instead (the backward apply pass
// of two resident blocks) too few loads are in flight.  12544 x 2048 and 802816 x 256, 8 blocks an SM -> now: forward 31 -> 28
// and 161 -> 145 us, with a residual 41 -> 37 and 213 -> 199, apply 49 -> 35 and 249 -> 208.
constexpr int kStatsBlocks = 4;
constexpr int fwd_blocks(bool res) { return res ? 2 : 3; }
constexpr int reduce_blocks(int mode) { return mode == 2 ? 2 : 3; }
constexpr int apply_blocks(int mode, bool res) { return mode == 0 && !res ? 3 : 2; }

struct Map {
  int groups;      // C / 8
  int cg;          // channel groups of a block (a power of two)
  int rows_par;    // rows a block processes in parallel
};

// Sums of a thread's 8 channels meet over the block's rows in shared memory, then one atomic per channel and block.
__device__ __forceinline__ void flush_sums(const float (&a)[8], const float (&b)[8], const Map& mp, float* out_a, float* out_b) {
  __shared__ float s_a[256 * 9], s_b[256 * 9];                 // 9: the row lanes of a channel fall into different banks
#pragma unroll
  for (int q = 0; q < 8; ++q) { s_a[threadIdx.x * 9 + q] = a[q]; s_b[threadIdx.x * 9 + q] = b[q]; }
  __syncthreads();
  // cg * 8 <= 128 channels, 256 / (cg * 8) helpers each
  const int ch = mp.cg * 8, helpers = 256 / ch, c = threadIdx.x % ch, h = threadIdx.x / ch;
  float ta = 0.0f, tb = 0.0f;
  for (int r = h; r < mp.rows_par; r += helpers) {
    ta += s_a[(r * mp.cg + c / 8) * 9 + c % 8];
    tb += s_b[(r * mp.cg + c / 8) * 9 + c % 8];
  }
  __syncthreads();
  s_a[threadIdx.x] = ta;                                       // reuses the front of the arrays
  s_b[threadIdx.x] = tb;
  __syncthreads();
  const int gg = blockIdx.y * mp.cg + c / 8;
  if (h == 0 && gg < mp.groups) {
    for (int k = 1; k < helpers; ++k) { ta += s_a[k * ch + c]; tb += s_b[k * ch + c]; }
    atomicAdd(out_a + gg * 8 + c % 8, ta);
    atomicAdd(out_b + gg * 8 + c % 8, tb);
  }
}

__global__ void __launch_bounds__(256, kStatsBlocks) bn_stats_kernel(const __nv_bfloat16* __restrict__ y, int64_t M, int C, Map mp,
                                                       float* __restrict__ sum, float* __restrict__ sqsum) {
  pdl_enter();
  const int gl = threadIdx.x % mp.cg, rl = threadIdx.x / mp.cg, g = blockIdx.y * mp.cg + gl;
  float a[8] = {0, 0, 0, 0, 0, 0, 0, 0}, b[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (g < mp.groups) {
    const int64_t step = (int64_t)gridDim.x * mp.rows_par;
    for (int64_t r = (int64_t)blockIdx.x * mp.rows_par + rl; r < M; r += 4 * step) {
      uint4 raw[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (r + u * step < M) raw[u] = *reinterpret_cast<const uint4*>(y + (r + u * step) * C + g * 8);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (r + u * step < M) {
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[u]);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float2 f = __bfloat1622float2(h[q]);
            a[2 * q] += f.x; a[2 * q + 1] += f.y; b[2 * q] += f.x * f.x; b[2 * q + 1] += f.y * f.y;
          }
        }
      }
    }
  }
  flush_sums(a, b, mp, sum, sqsum);
}

// z = act(scale * y + shift [+ residual]) with scale / shift from the batch sums.  Every thread derives the coefficients
// of its own 8 channels (32 loads and 8 reciprocal roots against thousands of elements: a launch of its own for
// them cost 4 us a layer); the first block also leaves them, and the running statistics, for later.  Threads keep a
// fixed group of 8 channels and walk over rows, last row first: the producer of y wrote its end last, so that part
// is still in L2, and what is left there afterwards is z's beginning, where the next layer starts.
// With a residual the sign of z cannot be told from y alone, and a convolution's data gradient has no y to tell it from: the
// backward passes then read one bit per element (mask) instead of z, a sixteenth of the bytes.
template <bool kRes>
__global__ void __launch_bounds__(256, fwd_blocks(kRes))
bn_fwd_kernel(const __nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ res, __nv_bfloat16* __restrict__ z,
              uint8_t* __restrict__ mask, const float* __restrict__ sum, const float* __restrict__ sqsum,
              const float* __restrict__ gamma, const float* __restrict__ beta, float* running_mean, float* running_var,
              float* __restrict__ aux, int64_t M, int C, Map mp, int relu, float inv_count, float unbias, float momentum, float eps) {
  pdl_enter();
  const int gl = threadIdx.x % mp.cg, rl = threadIdx.x / mp.cg, g = blockIdx.y * mp.cg + gl;
  if (g >= mp.groups) return;
  float sc[8], sh[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int c = g * 8 + q;
    const float mean = sum[c] * inv_count;
    const float var = fmaxf(sqsum[c] * inv_count - mean * mean, 0.0f);
    const float invstd = rsqrtf(var + eps);
    sc[q] = gamma[c] * invstd;
    sh[q] = beta[c] - mean * sc[q];
    if (blockIdx.x == 0 && rl == 0) {
      aux[c] = mean;
      aux[C + c] = invstd;
      aux[2 * C + c] = sc[q];
      aux[3 * C + c] = sh[q];
      if (running_mean != nullptr) {
        running_mean[c] = (1.0f - momentum) * running_mean[c] + momentum * mean;
        running_var[c] = (1.0f - momentum) * running_var[c] + momentum * var * unbias;
      }
    }
  }
  const int64_t step = (int64_t)gridDim.x * mp.rows_par;
  for (int64_t r = M - 1 - ((int64_t)blockIdx.x * mp.rows_par + rl); r >= 0; r -= 4 * step) {
    uint4 ry[4], rr_[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t rr = r - u * step;
      if (rr >= 0) {
        ry[u] = *reinterpret_cast<const uint4*>(y + rr * C + g * 8);
        if (kRes) rr_[u] = *reinterpret_cast<const uint4*>(res + rr * C + g * 8);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t rr = r - u * step;
      if (rr >= 0) {
        const __nv_bfloat162* hy = reinterpret_cast<const __nv_bfloat162*>(&ry[u]);
        const __nv_bfloat162* hr = reinterpret_cast<const __nv_bfloat162*>(&rr_[u]);
        float v[8];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float2 f = __bfloat1622float2(hy[q]);
          v[2 * q] = f.x * sc[2 * q] + sh[2 * q];
          v[2 * q + 1] = f.y * sc[2 * q + 1] + sh[2 * q + 1];
          if (kRes) {
            float2 rf = __bfloat1622float2(hr[q]);
            v[2 * q] += rf.x; v[2 * q + 1] += rf.y;
          }
          if (relu) { v[2 * q] = fmaxf(v[2 * q], 0.0f); v[2 * q + 1] = fmaxf(v[2 * q + 1], 0.0f); }
        }
        const uint4 out = st8(z + rr * C + g * 8, v);
        if (mask != nullptr) mask[rr * mp.groups + g] = sign_bits(out);
      }
    }
  }
}

// The gradient behind the ReLU: kMode 0 no ReLU, 1 from the mask the forward pass left, 2 recomputed from y.
template <int kMode>
__device__ __forceinline__ void masked(const uint4& rd, const uint4& ry, uint32_t bits, const float (&fsc)[8], const float (&fsh)[8],
                                       float (&d)[8], float (&yy)[8]) {
  const __nv_bfloat162* hd = reinterpret_cast<const __nv_bfloat162*>(&rd);
  const __nv_bfloat162* hy = reinterpret_cast<const __nv_bfloat162*>(&ry);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float2 dd = __bfloat1622float2(hd[q]), f = __bfloat1622float2(hy[q]);
    d[2 * q] = dd.x; d[2 * q + 1] = dd.y;
    yy[2 * q] = f.x; yy[2 * q + 1] = f.y;
  }
  if (kMode == 1) {
#pragma unroll
    for (int q = 0; q < 8; ++q) d[q] = (bits >> q) & 1u ? d[q] : 0.0f;
  } else if (kMode == 2) {
#pragma unroll
    for (int q = 0; q < 8; ++q) d[q] = yy[q] * fsc[q] + fsh[q] > 0.0f ? d[q] : 0.0f;
  }
}

template <int kMode>
__global__ void __launch_bounds__(256, reduce_blocks(kMode))
bn_bwd_reduce_kernel(const __nv_bfloat16* __restrict__ dz, const uint8_t* __restrict__ mask, const __nv_bfloat16* __restrict__ y,
                     const float* __restrict__ aux, int64_t M, int C, Map mp, float* __restrict__ dbeta, float* __restrict__ dgamma) {
  pdl_enter();
  const int gl = threadIdx.x % mp.cg, rl = threadIdx.x / mp.cg, g = blockIdx.y * mp.cg + gl;
  float a[8] = {0, 0, 0, 0, 0, 0, 0, 0}, b[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (g < mp.groups) {
    float mu[8], fsc[8], fsh[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      mu[q] = aux[g * 8 + q];
      fsc[q] = kMode == 2 ? aux[2 * C + g * 8 + q] : 0.0f;
      fsh[q] = kMode == 2 ? aux[3 * C + g * 8 + q] : 0.0f;
    }
    const int64_t step = (int64_t)gridDim.x * mp.rows_par;
    // sum g and g*(y - mean); the 1/std factor is applied once at the end.  Four rows in flight, last rows first
    // (dz was produced front to back); the apply pass then goes front to back over what this one read last.
    for (int64_t r = M - 1 - ((int64_t)blockIdx.x * mp.rows_par + rl); r >= 0; r -= 4 * step) {
      uint4 rd[4], ry[4];
      uint32_t bits[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t rr = r - u * step;
        if (rr >= 0) {
          const int64_t off = rr * C + g * 8;
          rd[u] = *reinterpret_cast<const uint4*>(dz + off);
          ry[u] = *reinterpret_cast<const uint4*>(y + off);
          if (kMode == 1) bits[u] = mask[rr * mp.groups + g];
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (r - u * step >= 0) {
          float d[8], yy[8];
          masked<kMode>(rd[u], ry[u], bits[u], fsc, fsh, d, yy);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            a[q] += d[q];
            b[q] += d[q] * (yy[q] - mu[q]);
          }
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) b[q] *= aux[C + g * 8 + q];
  }
  flush_sums(a, b, mp, dbeta, dgamma);
}

// dy = a*g + b*y + c per channel, with a = gamma*invstd, b = -gamma*invstd^2*dgamma/M,
// c = gamma*invstd*(mean*invstd*dgamma - dbeta)/M held in registers.
template <int kMode, bool kRes>
__global__ void __launch_bounds__(256, apply_blocks(kMode, kRes))
bn_bwd_apply_kernel(const __nv_bfloat16* __restrict__ dz, const uint8_t* __restrict__ mask, const __nv_bfloat16* __restrict__ y,
                    const float* __restrict__ aux, const float* __restrict__ gamma, const float* __restrict__ dbeta,
                    const float* __restrict__ dgamma, __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ dres, int64_t M,
                    int C, Map mp, float inv_count, float* acc_dgamma, float* acc_dbeta, int last_first) {
  pdl_enter();
  const int gl = threadIdx.x % mp.cg, rl = threadIdx.x / mp.cg, g = blockIdx.y * mp.cg + gl;
  if (g >= mp.groups) return;
  float ca[8], cb[8], cc[8], fsc[8], fsh[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int c = g * 8 + q;
    fsc[q] = kMode == 2 ? aux[2 * C + c] : 0.0f;
    fsh[q] = kMode == 2 ? aux[3 * C + c] : 0.0f;
    const float is = aux[C + c], gm = gamma[c], dg = dgamma[c] * inv_count, db = dbeta[c] * inv_count;
    ca[q] = gm * is;
    cb[q] = -gm * is * is * dg;
    cc[q] = gm * is * (aux[c] * is * dg - db);
    if (blockIdx.x == 0 && rl == 0) {       // the parameters' own gradient accumulators, when the caller gives them
      if (acc_dgamma != nullptr) acc_dgamma[c] += dgamma[c];
      if (acc_dbeta != nullptr) acc_dbeta[c] += dbeta[c];
    }
  }
  const int64_t step = (int64_t)gridDim.x * mp.rows_par;
  // last_first: straight after a data gradient, which wrote dz (and read y) front to back
  const int64_t flip = last_first ? M - 1 : 0, sign = last_first ? -1 : 1;
  for (int64_t r = (int64_t)blockIdx.x * mp.rows_par + rl; r < M; r += 4 * step) {
    uint4 rd[4], ry[4];
    uint32_t bits[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (r + u * step < M) {
        const int64_t rr = flip + sign * (r + u * step), off = rr * C + g * 8;
        rd[u] = *reinterpret_cast<const uint4*>(dz + off);
        ry[u] = *reinterpret_cast<const uint4*>(y + off);
        if (kMode == 1) bits[u] = mask[rr * mp.groups + g];
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (r + u * step < M) {
        const int64_t rr = flip + sign * (r + u * step);
        const int64_t off = rr * C + g * 8;
        float d[8], yy[8], o[8];
        masked<kMode>(rd[u], ry[u], bits[u], fsc, fsh, d, yy);
#pragma unroll
        for (int q = 0; q < 8; ++q) o[q] = ca[q] * d[q] + cb[q] * yy[q] + cc[q];
        if (kRes) st8(dres + off, d);
        st8(dy + off, o);
      }
    }
  }
}

// Inference: the affine maps of all batch norms of a network in one launch, one block per layer.
struct CoefLayer {
  const float *gamma, *beta, *mean, *var;
  float* out;            // [2][C]: scale, shift
  int64_t C;
};
__global__ void __launch_bounds__(256) bn_coefficients_kernel(const CoefLayer* __restrict__ layers, float eps) {
  pdl_enter();
  const CoefLayer l = layers[blockIdx.x];
  for (int c = threadIdx.x; c < l.C; c += 256) {
    const float sc = l.gamma[c] * rsqrtf(l.var[c] + eps);
    l.out[c] = sc;
    l.out[l.C + c] = l.beta[c] - l.mean[c] * sc;
  }
}

Map make_map(int C) {
  Map m;
  m.groups = C / 8;
  if (m.groups % 16 == 0) m.cg = 16;
  else if (m.groups % 8 == 0) m.cg = 8;
  else if (m.groups % 4 == 0) m.cg = 4;
  else for (m.cg = 1; m.cg < m.groups && m.cg < 16; m.cg *= 2) {}
  m.rows_par = 256 / m.cg;
  return m;
}
// Four rows per thread as long as that does not fill the machine, then as many blocks as are resident.
dim3 grid_for(const Map& m, int64_t M, int blocks_per_sm) {
  const int64_t chunks = (m.groups + m.cg - 1) / m.cg;
  int64_t rows = (M + m.rows_par * 4 - 1) / (m.rows_par * 4), most = esgd::sm_count() * blocks_per_sm / chunks;
  if (most < 1) most = 1;
  if (rows > most) rows = most;
  return dim3((unsigned)(rows < 1 ? 1 : rows), (unsigned)chunks);
}

}  // namespace

extern "C" {

// sum / sqsum must be zeroed by the caller (they accumulate).
int esgd_bn_stats(const void* y, int64_t M, int C, float* sum, float* sqsum, void* stream) {
  if (C < 8 || C % 8) return -1;
  const Map mp = make_map(C);
  return esgd::launch(bn_stats_kernel, grid_for(mp, M, kStatsBlocks), 256, 0, stream, (const __nv_bfloat16*)y, M, C, mp, sum, sqsum);
}

// sum / sqsum: the batch sums of y.  aux [4][C] receives mean, inverse standard deviation, scale and shift; mask (optional,
// [M][C / 8] bytes) which elements of z are above zero.
int esgd_bn_fwd(const void* y, const void* residual, void* z, void* mask, const float* sum, const float* sqsum, const float* gamma,
                const float* beta, float* running_mean, float* running_var, float* aux, int64_t M, int C, int relu,
                float momentum, float eps, void* stream) {
  if (C < 8 || C % 8) return -1;
  const float unbias = M > 1 ? (float)M / (float)(M - 1) : 1.0f;
  const Map mp = make_map(C);
  auto kernel = residual != nullptr ? bn_fwd_kernel<true> : bn_fwd_kernel<false>;
  return esgd::launch(kernel, grid_for(mp, M, fwd_blocks(residual != nullptr)), 256, 0, stream, (const __nv_bfloat16*)y, (const __nv_bfloat16*)residual,
                      (__nv_bfloat16*)z, (uint8_t*)mask, sum, sqsum, gamma, beta, running_mean, running_var, aux, M, C, mp, relu,
                      1.0f / (float)M, unbias, momentum, eps);
}

int esgd_bn_coefficients(const void* layers, int n, float eps, void* stream) {
  return esgd::launch(bn_coefficients_kernel, dim3(n), 256, 0, stream, (const CoefLayer*)layers, eps);
}

// dbeta / dgamma must be zeroed by the caller.
// mode: 0 no ReLU, 1 its mask as esgd_bn_fwd left it (needed with a residual), 2 mask recomputed from y with the forward
// scale / shift.
int esgd_bn_bwd_reduce(const void* dz, const void* mask, const void* y, const float* aux, int64_t M, int C, int mode, float* dbeta,
                       float* dgamma, void* stream) {
  if (C < 8 || C % 8 || mode < 0 || mode > 2 || (mode == 1 && mask == nullptr)) return -1;
  const Map mp = make_map(C);
  auto kernel = mode == 0 ? bn_bwd_reduce_kernel<0> : (mode == 1 ? bn_bwd_reduce_kernel<1> : bn_bwd_reduce_kernel<2>);
  return esgd::launch(kernel, grid_for(mp, M, reduce_blocks(mode)), 256, 0, stream, (const __nv_bfloat16*)dz, (const uint8_t*)mask,
                      (const __nv_bfloat16*)y, aux, M, C, mp, dbeta, dgamma);
}

// dres (optional): the gradient behind the ReLU, for the shortcut.  last_first: rows in descending order.
// acc_dgamma / acc_dbeta (optional): fp32 accumulators the two parameter gradients are added to.
int esgd_bn_bwd_apply(const void* dz, const void* mask, const void* y, const float* aux, const float* gamma, const float* dbeta,
                      const float* dgamma, void* dy, void* dres, int64_t M, int C, int mode, int last_first, float* acc_dgamma,
                      float* acc_dbeta, void* stream) {
  if (C < 8 || C % 8 || mode < 0 || mode > 2 || (mode == 1 && mask == nullptr)) return -1;
  const Map mp = make_map(C);
  auto kernel = dres != nullptr ? (mode == 0 ? bn_bwd_apply_kernel<0, true> : mode == 1 ? bn_bwd_apply_kernel<1, true> : bn_bwd_apply_kernel<2, true>)
                                : (mode == 0 ? bn_bwd_apply_kernel<0, false> : mode == 1 ? bn_bwd_apply_kernel<1, false> : bn_bwd_apply_kernel<2, false>);
  return esgd::launch(kernel, grid_for(mp, M, apply_blocks(mode, dres != nullptr)), 256, 0, stream, (const __nv_bfloat16*)dz, (const uint8_t*)mask,
                      (const __nv_bfloat16*)y, aux, gamma, dbeta, dgamma, (__nv_bfloat16*)dy, (__nv_bfloat16*)dres, M, C, mp,
                      1.0f / (float)M, acc_dgamma, acc_dbeta, last_first);
}

}  // extern "C"
