// Training-mode batch normalisation for channels-last bf16 activations, fused with the ReLU
// and the residual add that follow it in a ResNet block.
//
// Why this is here: in the ResNet-50 data-parallel benchmark (64 images per GPU) the framework
// library's channels-last batch-norm kernels took 54 % of the device time of a training step,
// 5-15x off what one pass over the activations costs at HBM speed.  A batch-norm layer is pure
// streaming work:
//
//   forward   stats:  one read of x                      -> per-channel mean / inverse std
//             apply:  y = relu(x*a + b [+ residual])      one read (two with residual), one write
//   backward  reduce: sums of dy' and dy'*(x - mean), dy' = dy * (y > 0)
//             elemt:  dx = dy'*a + x*k2 + k3 [, dres = dy']
//
// What the backward pass wants of y is a bit per element.  The apply kernel can leave those (a byte for a thread's
// eight channels), and both backward kernels then read a sixteenth of what y is: with activations of 103 MB they take
// 43 and 70 us, and 57 and 86 with y.
//
// Every kernel uses the same geometry: a CTA owns a tile of up to 256 channels and a contiguous
// range of rows (row = one pixel of one image, C contiguous bf16 values).  A thread owns 8
// adjacent channels (one 16-byte load per row) for the whole kernel, so per-channel constants
// sit in registers, and four rows are in flight per thread.  The two reductions store one
// partial result per CTA and channel; a small finalize kernel (32 channels per CTA, 32 warps
// striding over the partials, merged in a fixed order, so results are deterministic) combines
// them -- the variance with Chan's parallel update, so no precision is lost to
// E[x^2] - E[x]^2 over the whole batch -- and writes the coefficients the elementwise kernel
// needs.  The three kernels of a direction overlap at their ends (launch.cuh).  (When the last CTA to finish
// combines all partials instead, one thread per channel walking ~1,200 of them in sequence takes 6x longer
// than reading the activations.)
//
// The reference has no model code; this belongs to the model zoo built around its codecs.
#include <cuda_bf16.h>

#include "kernels.h"
#include "launch.cuh"
#include "nhwc.cuh"

namespace hipress {
namespace cuda {

namespace {

// ---------------------------------------------------------------- forward: statistics
__global__ void __launch_bounds__(kBnThreads)
bn_stats_kernel(const __nv_bfloat16* __restrict__ x, int64_t M, int C, int tx_count, int64_t rows_per_block,
                float2* __restrict__ partial) {
  __shared__ float sh[2 * kBnThreads * kBnVec];
  const Lane l = lane_of(tx_count, M, rows_per_block);
  float s[kBnVec], q[kBnVec];
#pragma unroll
  for (int k = 0; k < kBnVec; ++k) s[k] = q[k] = 0.f;
  const __nv_bfloat16* base = x + l.c0;
  int64_t r = l.r_begin + l.ty;
  for (; r + 3 * l.TY < l.r_end; r += 4 * l.TY) {
    float v[4][kBnVec];
#pragma unroll
    for (int u = 0; u < 4; ++u) load8(base + (r + u * l.TY) * C, v[u]);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int k = 0; k < kBnVec; ++k) {
        s[k] += v[u][k];
        q[k] += v[u][k] * v[u][k];
      }
  }
  for (; r < l.r_end; r += l.TY) {
    float v[kBnVec];
    load8(base + r * C, v);
#pragma unroll
    for (int k = 0; k < kBnVec; ++k) {
      s[k] += v[k];
      q[k] += v[k] * v[k];
    }
  }
  let_next_start();
  float S, Q;
  reduce_rows(s, q, tx_count, sh, S, Q);
  const int ct = tx_count * kBnVec;
  const int c = blockIdx.x * ct + threadIdx.x;
  if (int(threadIdx.x) < ct) {
    const float cnt = float(l.r_end - l.r_begin);
    const float mean_b = cnt > 0.f ? S / cnt : 0.f;
    partial[int64_t(blockIdx.y) * C + c] = make_float2(mean_b, fmaxf(Q - S * mean_b, 0.f));
  }
}

constexpr int kFinChannels = 32;  // channels per finalize CTA (one per lane)
constexpr int kFinThreads = 1024;
constexpr int kFinWarps = kFinThreads / 32;
constexpr int kFinHeld = 20;      // partials per thread, all requested at once: their load latencies overlap
static_assert(kFinHeld * kFinWarps >= 148 * 4, "covers the row blocks of nhwc.cuh's geometry");

// Chan et al.: merges the (count, mean, M2) of disjoint sets, one after another, into (cnt, mean, m2).  The
// weights follow from the counts alone: they are all computed first, so that the chain of dependent
// operations is a subtraction and a multiply-add per set, and not a divide.  nb[j] <= 0: no such set.
template <int N>
__device__ __forceinline__ void chan_merge(float& cnt, float& mean, float& m2, const float (&nb)[N], const float (&mb)[N],
                                           const float (&m2b)[N]) {
  float frac[N], before[N];
#pragma unroll
  for (int j = 0; j < N; ++j) {
    before[j] = cnt;
    const float tot = cnt + nb[j];
    frac[j] = __fdividef(nb[j], tot);  // weights of a mean: 2 ulp is plenty, an IEEE divide per step is not free
    if (nb[j] > 0.f) cnt = tot;
  }
#pragma unroll
  for (int j = 0; j < N; ++j) {
    if (nb[j] <= 0.f) continue;
    const float delta = mb[j] - mean;
    mean += delta * frac[j];
    m2 += m2b[j] + delta * delta * (before[j] * frac[j]);
  }
}

// grid = C / 32.  Lane = channel, warp w merges row blocks w, w+32, ... and the warp results are merged in
// warp order (always the same order: results are deterministic).  A few CTAs with little to do: what counts
// is the length of the dependent chain, so all partials of a thread are requested at once, the weights are
// taken out of the chain, and the kernel starts while the one before it ends.  A ResNet-50 step of 64 images:
// 8.46 ms, and 8.85 with the weights in the chain, plain launches and the codecs' former decode.
__global__ void __launch_bounds__(kFinThreads)
bn_stats_finalize_kernel(const float2* __restrict__ partial, int row_blocks, int64_t M, int C,
                         int64_t rows_per_block, const float* __restrict__ gamma,
                         const float* __restrict__ beta, float* running_mean, float* running_var,
                         long long* num_batches, float momentum, float eps, float* __restrict__ mean_out,
                         float* __restrict__ invstd_out, float2* __restrict__ ab_out) {
  __shared__ float sh[3][kFinWarps][kFinChannels];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * kFinChannels + lane;
  let_next_start();
  // per-channel scalars of the epilogue, requested now so that they arrive during the sums
  float w_c = 1.f, b_c = 0.f, rm_c = 0.f, rv_c = 0.f;
  if (warp == 0 && c < C) {
    if (gamma) w_c = gamma[c];
    if (beta) b_c = beta[c];
  }
  wait_for_previous();
  if (warp == 0 && c < C && running_mean) {
    rm_c = running_mean[c];
    rv_c = running_var[c];
  }
  float cnt = 0.f, mean = 0.f, m2 = 0.f;
  {
    float2 p[kFinHeld];
#pragma unroll
    for (int j = 0; j < kFinHeld; ++j) {
      const int y = warp + j * kFinWarps;
      p[j] = c < C && y < row_blocks ? load_written(&partial[int64_t(y) * C + c]) : make_float2(0.f, 0.f);
    }
    const int full_blocks = int(M / rows_per_block), blocks = c < C ? row_blocks : 0;
    const float full_rows = float(rows_per_block), last_rows = float(M % rows_per_block);
#pragma unroll
    for (int j0 = 0; j0 < kFinHeld; j0 += 5) {
      float nb[5], mb[5], m2b[5];
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        const int y = warp + (j0 + j) * kFinWarps;
        nb[j] = y < blocks ? (y < full_blocks ? full_rows : last_rows) : 0.f;
        mb[j] = p[j0 + j].x;
        m2b[j] = p[j0 + j].y;
      }
      chan_merge<5>(cnt, mean, m2, nb, mb, m2b);
    }
  }
  sh[0][warp][lane] = cnt;
  sh[1][warp][lane] = mean;
  sh[2][warp][lane] = m2;
  __syncthreads();
  if (warp != 0 || c >= C) return;
#pragma unroll
  for (int w0 = 1; w0 < kFinWarps; w0 += 8) {
    float nb[8], mb[8], m2b[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int w = w0 + j;
      nb[j] = w < kFinWarps ? sh[0][w][lane] : 0.f;
      mb[j] = w < kFinWarps ? sh[1][w][lane] : 0.f;
      m2b[j] = w < kFinWarps ? sh[2][w][lane] : 0.f;
    }
    chan_merge<8>(cnt, mean, m2, nb, mb, m2b);
  }
  const float var = m2 / cnt;
  const float invstd = rsqrtf(var + eps);
  mean_out[c] = mean;
  invstd_out[c] = invstd;
  const float a = w_c * invstd;
  ab_out[c] = make_float2(a, b_c - mean * a);
  if (running_mean) {
    running_mean[c] = (1.f - momentum) * rm_c + momentum * mean;
    running_var[c] = (1.f - momentum) * rv_c + momentum * (cnt > 1.f ? m2 / (cnt - 1.f) : var);
  }
  if (num_batches && c == 0) *num_batches += 1;
}

// ---------------------------------------------------------------- forward: apply
// Bit k: the value that store8 writes for v[k], rounded, is positive.
__device__ __forceinline__ uint8_t positive8(const float (&v)[kBnVec]) {
  uint32_t bits = 0;
#pragma unroll
  for (int k = 0; k < kBnVec; ++k) bits |= __bfloat162float(__float2bfloat16_rn(v[k])) > 0.f ? 1u << k : 0u;
  return uint8_t(bits);
}
template <bool RELU, bool ADD>
__global__ void __launch_bounds__(kBnThreads)
bn_apply_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                __nv_bfloat16* __restrict__ y, uint8_t* __restrict__ mask, int64_t M, int C, int tx_count,
                int64_t rows_per_block, const float2* ab) {
  wait_for_previous();
  const Lane l = lane_of(tx_count, M, rows_per_block);
  float a[kBnVec], b[kBnVec];
#pragma unroll
  for (int k = 0; k < kBnVec; ++k) {
    const float2 t = ab[l.c0 + k];
    a[k] = t.x;
    b[k] = t.y;
  }
  int64_t r = l.r_begin + l.ty;
  for (; r + 3 * l.TY < l.r_end; r += 4 * l.TY) {
    float v[4][kBnVec], w[4][kBnVec];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      load8(x + (r + u * l.TY) * C + l.c0, v[u]);
      if (ADD) load8(res + (r + u * l.TY) * C + l.c0, w[u]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
#pragma unroll
      for (int k = 0; k < kBnVec; ++k) {
        float o = fmaf(v[u][k], a[k], b[k]);
        if (ADD) o += w[u][k];
        v[u][k] = RELU ? fmaxf(o, 0.f) : o;
      }
      store8(y + (r + u * l.TY) * C + l.c0, v[u]);
      if (RELU && mask != nullptr) mask[((r + u * l.TY) * C + l.c0) / kBnVec] = positive8(v[u]);
    }
  }
  for (; r < l.r_end; r += l.TY) {
    float v[kBnVec], w[kBnVec];
    load8(x + r * C + l.c0, v);
    if (ADD) load8(res + r * C + l.c0, w);
#pragma unroll
    for (int k = 0; k < kBnVec; ++k) {
      float o = fmaf(v[k], a[k], b[k]);
      if (ADD) o += w[k];
      v[k] = RELU ? fmaxf(o, 0.f) : o;
    }
    store8(y + r * C + l.c0, v);
    if (RELU && mask != nullptr) mask[(r * C + l.c0) / kBnVec] = positive8(v);
  }
}

// Where the gradient passes the ReLU: everywhere, where y is positive, or where the apply kernel left a bit.
enum Gate { kOpen = 0, kOutput = 1, kMask = 2 };
template <int GATE>
__device__ __forceinline__ void load_gate(const __nv_bfloat16* y, const uint8_t* mask, int64_t at, float (&o)[kBnVec], uint32_t& bits) {
  if (GATE == kOutput) load8(y + at, o);
  if (GATE == kMask) bits = mask[at / kBnVec];
}
template <int GATE>
__device__ __forceinline__ bool passes(const float (&o)[kBnVec], uint32_t bits, int k) {
  return GATE == kOpen || (GATE == kOutput ? o[k] > 0.f : ((bits >> k) & 1u) != 0);
}

// ---------------------------------------------------------------- backward: reductions
template <int GATE>
__global__ void __launch_bounds__(kBnThreads)
bn_bwd_reduce_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                     const __nv_bfloat16* __restrict__ y, const uint8_t* __restrict__ mask, int64_t M, int C, int tx_count,
                     int64_t rows_per_block, const float* __restrict__ mean, float2* __restrict__ partial) {
  __shared__ float sh[2 * kBnThreads * kBnVec];
  const Lane l = lane_of(tx_count, M, rows_per_block);
  float mu[kBnVec], s1[kBnVec], s2[kBnVec];
#pragma unroll
  for (int k = 0; k < kBnVec; ++k) {
    mu[k] = mean[l.c0 + k];
    s1[k] = s2[k] = 0.f;
  }
  int64_t r = l.r_begin + l.ty;
  for (; r + 1 * l.TY < l.r_end; r += 2 * l.TY) {
    float g[2][kBnVec], v[2][kBnVec], o[2][kBnVec];
    uint32_t bits[2] = {};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      load8(dy + (r + u * l.TY) * C + l.c0, g[u]);
      load8(x + (r + u * l.TY) * C + l.c0, v[u]);
      load_gate<GATE>(y, mask, (r + u * l.TY) * C + l.c0, o[u], bits[u]);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int k = 0; k < kBnVec; ++k) {
        const float d = passes<GATE>(o[u], bits[u], k) ? g[u][k] : 0.f;
        s1[k] += d;
        s2[k] += d * (v[u][k] - mu[k]);
      }
  }
  for (; r < l.r_end; r += l.TY) {
    float g[kBnVec], v[kBnVec], o[kBnVec];
    uint32_t bits = 0;
    load8(dy + r * C + l.c0, g);
    load8(x + r * C + l.c0, v);
    load_gate<GATE>(y, mask, r * C + l.c0, o, bits);
#pragma unroll
    for (int k = 0; k < kBnVec; ++k) {
      const float d = passes<GATE>(o, bits, k) ? g[k] : 0.f;
      s1[k] += d;
      s2[k] += d * (v[k] - mu[k]);
    }
  }
  let_next_start();
  float S1, S2;
  reduce_rows(s1, s2, tx_count, sh, S1, S2);
  const int ct = tx_count * kBnVec;
  const int c = blockIdx.x * ct + threadIdx.x;
  if (int(threadIdx.x) < ct) partial[int64_t(blockIdx.y) * C + c] = make_float2(S1, S2);
}

// grid = C / 32; same layout as bn_stats_finalize_kernel, plain sums.
__global__ void __launch_bounds__(kFinThreads)
bn_bwd_finalize_kernel(const float2* __restrict__ partial, int row_blocks, int64_t M, int C,
                       const float* __restrict__ mean, const float* __restrict__ invstd,
                       const float* __restrict__ gamma, float* __restrict__ dgamma,
                       float* __restrict__ dbeta, float4* __restrict__ coef) {
  __shared__ float sh[2][kFinWarps][kFinChannels];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * kFinChannels + lane;
  let_next_start();
  float is = 0.f, m = 0.f, wgt = 1.f;  // requested now, used after the sums; older than the kernel before
  if (warp == 0 && c < C) {
    is = invstd[c];
    m = mean[c];
    if (gamma) wgt = gamma[c];
  }
  wait_for_previous();
  float2 p[kFinHeld];
#pragma unroll
  for (int j = 0; j < kFinHeld; ++j) {
    const int y = warp + j * kFinWarps;
    p[j] = c < C && y < row_blocks ? load_written(&partial[int64_t(y) * C + c]) : make_float2(0.f, 0.f);
  }
  float t1 = 0.f, t2 = 0.f;
#pragma unroll
  for (int j = 0; j < kFinHeld; ++j) {
    t1 += p[j].x;
    t2 += p[j].y;
  }
  sh[0][warp][lane] = t1;
  sh[1][warp][lane] = t2;
  __syncthreads();
  if (warp != 0 || c >= C) return;
#pragma unroll 8
  for (int w = 1; w < kFinWarps; ++w) {
    t1 += sh[0][w][lane];
    t2 += sh[1][w][lane];
  }
  if (dbeta) dbeta[c] = t1;
  if (dgamma) dgamma[c] = t2 * is;
  // dx = a*(dy' - mean(dy') - xhat*mean(dy'*xhat)),  xhat = (x - m)*is,  a = w*is
  const float a = wgt * is;
  const float inv_count = 1.f / float(M);
  const float k2 = -a * is * is * t2 * inv_count;
  const float k3 = -a * t1 * inv_count - m * k2;
  coef[c] = make_float4(a, k2, k3, 0.f);
}

// ---------------------------------------------------------------- backward: elementwise
template <int GATE, bool ADD>
__global__ void __launch_bounds__(kBnThreads)
bn_bwd_elemt_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                    const __nv_bfloat16* __restrict__ y, const uint8_t* __restrict__ mask, __nv_bfloat16* __restrict__ dx,
                    __nv_bfloat16* __restrict__ dres, int64_t M, int C, int tx_count,
                    int64_t rows_per_block, const float4* coef) {
  wait_for_previous();
  const Lane l = lane_of(tx_count, M, rows_per_block);
  float a[kBnVec], k2[kBnVec], k3[kBnVec];
#pragma unroll
  for (int k = 0; k < kBnVec; ++k) {
    const float4 t = coef[l.c0 + k];
    a[k] = t.x;
    k2[k] = t.y;
    k3[k] = t.z;
  }
  int64_t r = l.r_begin + l.ty;
  for (; r + 1 * l.TY < l.r_end; r += 2 * l.TY) {
    float g[2][kBnVec], v[2][kBnVec], o[2][kBnVec];
    uint32_t bits[2] = {};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      load8(dy + (r + u * l.TY) * C + l.c0, g[u]);
      load8(x + (r + u * l.TY) * C + l.c0, v[u]);
      load_gate<GATE>(y, mask, (r + u * l.TY) * C + l.c0, o[u], bits[u]);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
#pragma unroll
      for (int k = 0; k < kBnVec; ++k) {
        const float d = passes<GATE>(o[u], bits[u], k) ? g[u][k] : 0.f;
        g[u][k] = d;
        v[u][k] = fmaf(d, a[k], fmaf(v[u][k], k2[k], k3[k]));
      }
      store8(dx + (r + u * l.TY) * C + l.c0, v[u]);
      if (ADD) store8(dres + (r + u * l.TY) * C + l.c0, g[u]);
    }
  }
  for (; r < l.r_end; r += l.TY) {
    float g[kBnVec], v[kBnVec], o[kBnVec];
    uint32_t bits = 0;
    load8(dy + r * C + l.c0, g);
    load8(x + r * C + l.c0, v);
    load_gate<GATE>(y, mask, r * C + l.c0, o, bits);
#pragma unroll
    for (int k = 0; k < kBnVec; ++k) {
      const float d = passes<GATE>(o, bits, k) ? g[k] : 0.f;
      g[k] = d;
      v[k] = fmaf(d, a[k], fmaf(v[k], k2[k], k3[k]));
    }
    store8(dx + r * C + l.c0, v);
    if (ADD) store8(dres + r * C + l.c0, g);
  }
}

}  // namespace

bool bn_supported(int64_t rows, int channels) {
  Geom g;
  return geometry(rows, channels, &g);
}

int64_t bn_partial_elems(int64_t rows, int channels) {
  Geom g;
  if (!geometry(rows, channels, &g)) return 0;
  return int64_t(g.row_blocks) * channels;
}

cudaError_t bn_forward(const void* x, const void* residual, void* y, int64_t rows, int channels,
                       const float* gamma, const float* beta, float* running_mean, float* running_var,
                       long long* num_batches, float momentum, float eps, int relu, float* mean,
                       float* invstd, float* ab, float* partial, cudaStream_t stream, uint8_t* mask) {
  Geom g;
  if (!geometry(rows, channels, &g) || !x || !y || !mean || !invstd || !ab || !partial)
    return cudaErrorInvalidValue;
  const dim3 grid(static_cast<unsigned>(g.tiles), static_cast<unsigned>(g.row_blocks), 1);
  const int fin_grid = (channels + kFinChannels - 1) / kFinChannels;
  const auto* xb = static_cast<const __nv_bfloat16*>(x);
  const auto* rb = static_cast<const __nv_bfloat16*>(residual);
  auto* yb = static_cast<__nv_bfloat16*>(y);
  auto* part = reinterpret_cast<float2*>(partial);
  bn_stats_kernel<<<grid, kBnThreads, 0, stream>>>(xb, rows, channels, g.tx, g.rows_per_block, part);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  e = launch_after(bn_stats_finalize_kernel, dim3(fin_grid), dim3(kFinThreads), 0, stream, part, g.row_blocks, rows, channels,
                   g.rows_per_block, gamma, beta, running_mean, running_var, num_batches, momentum, eps, mean, invstd,
                   reinterpret_cast<float2*>(ab));
  if (e != cudaSuccess) return e;
  const float2* abp = reinterpret_cast<const float2*>(ab);
#define HP_BN_APPLY(R, A)                                                                                          \
  e = launch_after(bn_apply_kernel<R, A>, grid, dim3(kBnThreads), 0, stream, xb, rb, yb, mask, rows, channels, g.tx, \
                   g.rows_per_block, abp)
  if (relu && rb) HP_BN_APPLY(true, true);
  else if (relu) HP_BN_APPLY(true, false);
  else if (rb) HP_BN_APPLY(false, true);
  else HP_BN_APPLY(false, false);
#undef HP_BN_APPLY
  return e;
}

cudaError_t bn_backward(const void* dy, const void* x, const void* y, void* dx, void* dres, int64_t rows,
                        int channels, const float* gamma, const float* mean, const float* invstd,
                        int relu, float* dgamma, float* dbeta, float* coef, float* partial,
                        cudaStream_t stream, const uint8_t* mask) {
  Geom g;
  if (!geometry(rows, channels, &g) || !dy || !x || !dx || !mean || !invstd || !coef || !partial ||
      (relu && !y && !mask))
    return cudaErrorInvalidValue;
  const dim3 grid(static_cast<unsigned>(g.tiles), static_cast<unsigned>(g.row_blocks), 1);
  const int fin_grid = (channels + kFinChannels - 1) / kFinChannels;
  const auto* gb = static_cast<const __nv_bfloat16*>(dy);
  const auto* xb = static_cast<const __nv_bfloat16*>(x);
  const auto* yb = static_cast<const __nv_bfloat16*>(y);
  auto* dxb = static_cast<__nv_bfloat16*>(dx);
  auto* drb = static_cast<__nv_bfloat16*>(dres);
  auto* part = reinterpret_cast<float2*>(partial);
  auto* cf = reinterpret_cast<float4*>(coef);
  const int gate = !relu ? kOpen : (mask != nullptr ? kMask : kOutput);
  (gate == kMask ? bn_bwd_reduce_kernel<kMask> : (gate == kOutput ? bn_bwd_reduce_kernel<kOutput> : bn_bwd_reduce_kernel<kOpen>))
      <<<grid, kBnThreads, 0, stream>>>(gb, xb, yb, mask, rows, channels, g.tx, g.rows_per_block, mean, part);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  e = launch_after(bn_bwd_finalize_kernel, dim3(fin_grid), dim3(kFinThreads), 0, stream, part, g.row_blocks, rows, channels,
                   mean, invstd, gamma, dgamma, dbeta, cf);
  if (e != cudaSuccess) return e;
#define HP_BN_ELEMT(G)                                                                                             \
  e = launch_after(drb ? bn_bwd_elemt_kernel<G, true> : bn_bwd_elemt_kernel<G, false>, grid, dim3(kBnThreads), 0,  \
                   stream, gb, xb, yb, mask, dxb, drb, rows, channels, g.tx, g.rows_per_block, cf)
  if (gate == kMask) HP_BN_ELEMT(kMask);
  else if (gate == kOutput) HP_BN_ELEMT(kOutput);
  else HP_BN_ELEMT(kOpen);
#undef HP_BN_ELEMT
  return e;
}

}  // namespace cuda
}  // namespace hipress
