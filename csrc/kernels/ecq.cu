// ECQ: error-compensated stochastic quantisation with a history tensor H, for
// sm_100a.  Payload layout follows the reference (ecq_body.h:266-276):
//   {i32 total = 10 + M, f32 max, u8 bitwidth, u8 unused_slots} + M data bytes.
// Semantics are the corrected ones implemented by the CPU codec
// (csrc/codec_cpu/codec_cpu.cpp): v = G + alpha*H keeps its sign, every data
// byte is produced, and the header is written on the device once the maximum
// is known (the reference reads the maximum on the host before the copy that
// delivers it has completed, ecq_body.h:203-214).
//
// Two kernels, no host synchronisation: abs-max grid reduction (+ header), then
// quantise / update H / pack / store to every destination / publish flag.  Both read
// with 16-byte loads when the arrays are aligned, take the step's epoch (flag value, slot
// parity, rounding seed) from the device when asked to, and return at once when an earlier
// kernel of the step recorded a failure.  Callers that have the GPU to themselves get both in one launch where
// the tensor fits the chip (ecq_hold_kernel).
#include "../common/codec_math.h"
#include "hold.cuh"
#include "kernels.h"
#include "launch.cuh"
#include "p2p.cuh"
#include "reduce.cuh"
#include "unpack_lut.cuh"

#include <type_traits>

namespace hipress {
namespace cuda {

namespace {

constexpr int kThreads = 256;
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
inline int grid_for(int64_t items, int threads, int max_blocks) {
  int64_t blocks = (items + threads - 1) / threads;
  if (blocks < 1) blocks = 1;
  if (blocks > max_blocks) blocks = max_blocks;
  return int(blocks);
}

struct EcqScale {
  float mx, gap, inv;
  bool zero;   // nothing to send: every level is 0
};
__device__ __forceinline__ EcqScale ecq_scale(float absmax, int bw) {
  EcqScale s;
  s.zero = absmax < kEcqZeroCutoff;
  s.mx = s.zero ? 0.0f : absmax;
  s.gap = s.zero ? 0.0f : ecq_gap(absmax, bw);
  s.inv = s.zero ? 0.0f : ecq_gap_inverse(s.gap);
  return s;
}
__device__ __forceinline__ void ecq_put_header(const PushTargets& dst, int64_t n, int bw, float mx) {
  const int dpb = 8 / bw;
  const int64_t M = (n + dpb - 1) / dpb;
  const uint32_t total = uint32_t(kEcqHeaderBytes + M);
  const uint32_t mb = __float_as_uint(mx);
  uint8_t header[kEcqHeaderBytes];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    header[k] = uint8_t(total >> (8 * k));
    header[4 + k] = uint8_t(mb >> (8 * k));
  }
  header[8] = uint8_t(bw);
  header[9] = uint8_t(M * dpb - n);
  push_bytes(dst, 0, header, kEcqHeaderBytes);
}

// `count` elements of one payload byte: v = g + alpha * h in, h takes the new history; returns the byte.
template <int BW>
__device__ __forceinline__ uint32_t ecq_quant_byte(const float* v, float* h, int count, float beta, const EcqScale& s, uint64_t seed,
                                                   int64_t byte_index) {
  uint8_t q = 0;
  Lcg32 rng(tern_byte_seed(seed, byte_index));
#pragma unroll
  for (int j = 0; j < 8 / BW; ++j) {
    if (j < count) {
      uint8_t t = 0;
      if (!s.zero) t = ecq_quant(v[j], s.mx, s.inv, rng.next_unit());
      q = uint8_t(q | (int(t) << (BW * j)));
      const uint32_t kept = uint32_t(t) & ((1u << BW) - 1u);
      h[j] = ecq_history(h[j], beta, v[j], ecq_dequant(kept, s.gap, s.mx));
    }
  }
  return q;
}

template <bool VEC>
__global__ void __launch_bounds__(kThreads)
ecq_absmax_header_kernel(const float* grad, const float* hist, int64_t n, float alpha, int bw, PushTargets dst,
                         MinMaxScratch* scratch) {
  wait_for_previous();
  if (push_guarded(dst)) return;
  resolve_epoch(dst);
  float mx = 0.0f, unused = 0.0f;
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  const int64_t tid = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t nv = VEC ? (n >> 2) : 0;  // 16-byte loads when both arrays are aligned
  auto fold = [&](float4 g, float4 h) {
    mx = fmaxf(mx, fmaxf(fmaxf(fabsf(ecq_compensated(g.x, h.x, alpha)), fabsf(ecq_compensated(g.y, h.y, alpha))),
                         fmaxf(fabsf(ecq_compensated(g.z, h.z, alpha)), fabsf(ecq_compensated(g.w, h.w, alpha)))));
  };
  int64_t q = tid;
  for (; q + 3 * stride < nv; q += 4 * stride) {   // four loads of each array in flight
    float4 g[4], h[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      g[u] = reinterpret_cast<const float4*>(grad)[q + u * stride];
      h[u] = reinterpret_cast<const float4*>(hist)[q + u * stride];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) fold(g[u], h[u]);
  }
  for (; q < nv; q += stride)
    fold(reinterpret_cast<const float4*>(grad)[q], reinterpret_cast<const float4*>(hist)[q]);
  for (int64_t i = (nv << 2) + tid; i < n; i += stride)
    mx = fmaxf(mx, fabsf(ecq_compensated(grad[i], hist[i], alpha)));
  let_next_start();
  float gmn, gmx;
  if (!grid_minmax_last_block<kThreads>(scratch, unused, mx, gmn, gmx)) return;
  if (threadIdx.x == 0) {
    const EcqScale scale = ecq_scale(gmx, bw);
    scratch->mx = scale.mx;
    scratch->mn = scale.zero ? 1.0f : 0.0f;  // for kernel 2
    scratch->gap = scale.gap;
    scratch->inv = scale.inv;
    ecq_put_header(dst, n, bw, scale.mx);
  }
}

constexpr int kStageBytes = 512;  // payload bytes a warp gathers before it stores them

// One thread quantises four consecutive elements (one 16-byte load of the gradient and of the
// history, one 16-byte store of the history) into BW/2 payload bytes; lanes then combine their
// bytes into 32-bit words, so that every destination gets word stores.  The random generator is
// seeded per payload byte, as in the CPU codec.  shift >= 0: large tensors whose destinations start
// equally far past a 16-byte boundary; a warp then gathers 512 payload bytes in shared memory, with the
// loads of four sub-steps in flight, and stores them 16 bytes per lane (put_chunk512).
template <int BW, bool VEC>
__global__ void __launch_bounds__(kThreads)
ecq_quant_kernel(const float* __restrict__ grad, float* __restrict__ hist, int64_t n, float alpha,
                 float beta, uint64_t seed, PushTargets dst, const MinMaxScratch* scratch, int shift) {
  wait_for_previous();
  if (push_guarded(dst)) return;
  resolve_epoch(dst);
  if (dst.epoch_dev != nullptr) seed += uint64_t(dst.epoch) * kEpochSeedStride;
  constexpr int DPB = 8 / BW;
  constexpr int BPT = 4 / DPB;  // bytes per thread: 1, 2, 4
  const EcqScale scale{scratch->mx, scratch->gap, scratch->inv, scratch->mn != 0.0f};
  auto quant_byte = [&](const float* g, float* h, int count, int64_t byte_index) -> uint32_t {
    float v[DPB];
#pragma unroll
    for (int j = 0; j < DPB; ++j) v[j] = j < count ? ecq_compensated(g[j], h[j], alpha) : 0.0f;
    return ecq_quant_byte<BW>(v, h, count, beta, scale, seed, byte_index);
  };
  int64_t unit0 = 0;   // first unit of the rest
  if (VEC && shift >= 0) {
    constexpr int64_t CU = int64_t(kStageBytes) / BPT;   // units per chunk
    __shared__ __align__(16) uint8_t stages[kThreads / 32][kStageBytes + 16];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint8_t* const stage = stages[warp] + shift;
    const PushCursor all{nullptr};
    const int64_t chunks = (n >> 2) / CU;
    const int64_t warps = int64_t(gridDim.x) * (blockDim.x >> 5);
    for (int64_t c = int64_t(blockIdx.x) * (blockDim.x >> 5) + warp; c < chunks; c += warps) {
#pragma unroll 1
      for (int j = 0; j < int(CU) / 32; j += 4) {
        float4 gv[4], hv[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int64_t u = c * CU + (j + k) * 32 + lane;
          gv[k] = __ldg(reinterpret_cast<const float4*>(grad) + u);
          hv[k] = reinterpret_cast<const float4*>(hist)[u];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int at = (j + k) * 32 + lane;
          const int64_t u = c * CU + at;
          const float g[4] = {gv[k].x, gv[k].y, gv[k].z, gv[k].w};
          float h[4] = {hv[k].x, hv[k].y, hv[k].z, hv[k].w};
          uint32_t bytes = 0;
#pragma unroll
          for (int b = 0; b < BPT; ++b)
            bytes |= quant_byte(g + b * DPB, h + b * DPB, DPB, u * BPT + b) << (8 * b);
          reinterpret_cast<float4*>(hist)[u] = make_float4(h[0], h[1], h[2], h[3]);
          if (BPT == 1) {
            stage[at] = uint8_t(bytes);
          } else if (BPT == 2) {
            reinterpret_cast<uint16_t*>(stage)[at] = uint16_t(bytes);
          } else if ((shift & 3) == 0) {
            reinterpret_cast<uint32_t*>(stage)[at] = bytes;
          } else {
            reinterpret_cast<uint16_t*>(stage)[2 * at] = uint16_t(bytes);
            reinterpret_cast<uint16_t*>(stage)[2 * at + 1] = uint16_t(bytes >> 16);
          }
        }
      }
      __syncwarp();
      put_chunk512(dst, all, kEcqHeaderBytes + c * kStageBytes, stages[warp], shift, lane);
      __syncwarp();
    }
    unit0 = chunks * CU;
  }
  const int64_t units = n >> 2;
  const int64_t units_padded = (units + 31) & ~int64_t(31);   // unit0 is a multiple of 32
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  for (int64_t u = unit0 + int64_t(blockIdx.x) * blockDim.x + threadIdx.x; u < units_padded; u += stride) {
    uint32_t bytes = 0;
    if (u < units) {
      float g[4], h[4];
      if (VEC) {
        const float4 gv = __ldg(reinterpret_cast<const float4*>(grad) + u);
        const float4 hv = reinterpret_cast<const float4*>(hist)[u];
        g[0] = gv.x; g[1] = gv.y; g[2] = gv.z; g[3] = gv.w;
        h[0] = hv.x; h[1] = hv.y; h[2] = hv.z; h[3] = hv.w;
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          g[k] = grad[4 * u + k];
          h[k] = hist[4 * u + k];
        }
      }
#pragma unroll
      for (int b = 0; b < BPT; ++b)
        bytes |= quant_byte(g + b * DPB, h + b * DPB, DPB, u * BPT + b) << (8 * b);
      if (VEC) {
        reinterpret_cast<float4*>(hist)[u] = make_float4(h[0], h[1], h[2], h[3]);
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) hist[4 * u + k] = h[k];
      }
    }
    if (BPT == 1) {
      const uint32_t word = gather4_bytes(bytes);
      if ((threadIdx.x & 3) == 0 && u < units) {
        if (u + 3 < units) {
          push_u32(dst, kEcqHeaderBytes + u, word);
        } else {
          for (int64_t b = u; b < units; ++b) push_u8(dst, kEcqHeaderBytes + b, uint8_t(word >> (8 * (b - u))));
        }
      }
    } else if (BPT == 2) {
      const uint32_t word = gather2_halves(bytes);
      if ((threadIdx.x & 1) == 0 && u < units) {
        if (u + 1 < units) {
          push_u32(dst, kEcqHeaderBytes + 2 * u, word);
        } else {
          push_u8(dst, kEcqHeaderBytes + 2 * u, uint8_t(word));
          push_u8(dst, kEcqHeaderBytes + 2 * u + 1, uint8_t(word >> 8));
        }
      }
    } else {
      if (u < units) push_u32(dst, kEcqHeaderBytes + 4 * u, bytes);
    }
  }
  // fewer than four leftover elements
  const int64_t done = units << 2;
  if (done < n && blockIdx.x == 0 && threadIdx.x == 0) {
    int64_t byte_index = done / DPB;
    for (int64_t e = done; e < n; e += DPB, ++byte_index) {
      const int count = (n - e) >= DPB ? DPB : int(n - e);
      float g[DPB], h[DPB];
      for (int j = 0; j < count; ++j) {
        g[j] = grad[e + j];
        h[j] = hist[e + j];
      }
      push_u8(dst, kEcqHeaderBytes + byte_index, uint8_t(quant_byte(g, h, count, byte_index)));
      for (int j = 0; j < count; ++j) hist[e + j] = h[j];
    }
  }
  publish_when_grid_done(dst);
}

// Medium tensors, callers that have the GPU to themselves: both passes in one launch that reads the gradient
// once.  What a CTA keeps in shared memory is v = g + alpha * h; the history itself is read again, from L2,
// where it and the gradient (two tensors of 30 MB at most) still are.  All CTAs have to be resident at once, each
// with an SM to itself: the exchange engine, whose compressor runs beside the backward pass, keeps the two launches.
// 25 MB, 4 bits, in a chain of calls: 24.8 us; 28.4 in two launches.  256 KB: 6.4 and 8.1 (with a slower exchange of
// the extremes).  A thread of 25 MB has eleven words: with the last three loaded one after another, in both walks,
// compress and decode take 37.9 us, and 37.2 so.
constexpr int kHoldAhead = 4;   // history words of a thread in flight
template <int BW>
__global__ void __launch_bounds__(kHoldThreads, 1)
ecq_hold_kernel(const float* __restrict__ grad, float* hist, int64_t n, int64_t part, float alpha, float beta, uint64_t seed,
                PushTargets dst, MinMaxScratch* scratch, int shift, uint64_t wait_ns, int* status) {
  constexpr int DPB = 8 / BW, BPT = 4 / DPB;
  extern __shared__ __align__(16) float hold[];           // [part], then the payload bytes
  __shared__ EcqScale shared_scale;
  uint8_t* const bytes_at = reinterpret_cast<uint8_t*>(hold + part);
  const int tid = threadIdx.x;
  GridPlace place;
  grid_arrive(scratch, place);
  const int64_t begin = int64_t(blockIdx.x) * part;       // a multiple of 512
  const int64_t left = n - begin;
  const int len = int(left < 0 ? 0 : (left < part ? left : part));
  const float4* g4 = reinterpret_cast<const float4*>(grad + begin);
  float4* h4 = reinterpret_cast<float4*>(hist + begin);
  float mn = 0.0f, mx = 0.0f;
  const int quads = len >> 2;
  auto take = [&](int i, float4 g, float4 h) {
    const float4 v = make_float4(ecq_compensated(g.x, h.x, alpha), ecq_compensated(g.y, h.y, alpha),
                                 ecq_compensated(g.z, h.z, alpha), ecq_compensated(g.w, h.w, alpha));
    mx = fmaxf(mx, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
    reinterpret_cast<float4*>(hold)[i] = v;
  };
  for (int q = tid; q < quads; q += kHoldAhead * kHoldThreads) {   // the last, partial round keeps its loads together too
    float4 g[kHoldAhead], h[kHoldAhead];
#pragma unroll
    for (int u = 0; u < kHoldAhead; ++u) {
      if (q + u * kHoldThreads < quads) {
        g[u] = __ldg(g4 + q + u * kHoldThreads);
        h[u] = h4[q + u * kHoldThreads];
      }
    }
#pragma unroll
    for (int u = 0; u < kHoldAhead; ++u)
      if (q + u * kHoldThreads < quads) take(q + u * kHoldThreads, g[u], h[u]);
  }
  for (int e = 4 * quads + tid; e < len; e += kHoldThreads)   // fewer than four
    mx = fmaxf(mx, fabsf(ecq_compensated(grad[begin + e], hist[begin + e], alpha)));
  if (!grid_minmax_all<kHoldThreads>(scratch, mn, mx, wait_ns, status, place)) {
    grid_leave(scratch, place);
    return;
  }
  if (tid == 0) {
    shared_scale = ecq_scale(mx, BW);
    if (blockIdx.x == 0) ecq_put_header(dst, n, BW, shared_scale.mx);
  }
  __syncthreads();
  const EcqScale scale = shared_scale;
  const int64_t byte0 = begin / DPB;                       // first payload byte of the part
  auto quantise = [&](int u, float4 old) {
    const float4 held = reinterpret_cast<const float4*>(hold)[u];
    const float v[4] = {held.x, held.y, held.z, held.w};
    float h[4] = {old.x, old.y, old.z, old.w};
    uint32_t bytes = 0;
#pragma unroll
    for (int b = 0; b < BPT; ++b)
      bytes |= ecq_quant_byte<BW>(v + b * DPB, h + b * DPB, DPB, beta, scale, seed, byte0 + int64_t(u) * BPT + b) << (8 * b);
    h4[u] = make_float4(h[0], h[1], h[2], h[3]);
    hold_unit_bytes<BPT>(bytes_at + shift + u * BPT, bytes);   // shift is even
  };
  for (int u = tid; u < quads; u += kHoldAhead * kHoldThreads) {
    float4 h[kHoldAhead];
#pragma unroll
    for (int k = 0; k < kHoldAhead; ++k)
      if (u + k * kHoldThreads < quads) h[k] = h4[u + k * kHoldThreads];
#pragma unroll
    for (int k = 0; k < kHoldAhead; ++k)
      if (u + k * kHoldThreads < quads) quantise(u + k * kHoldThreads, h[k]);
  }
  __syncthreads();
  hold_put(dst, kEcqHeaderBytes, byte0, bytes_at, shift, quads * BPT);
  if (tid == 32) {   // fewer than four leftover elements
    for (int e = 4 * quads; e < len; e += DPB) {
      const int count = len - e < DPB ? len - e : DPB;
      float v[DPB], h[DPB];
      for (int j = 0; j < count; ++j) {
        h[j] = hist[begin + e + j];
        v[j] = ecq_compensated(grad[begin + e + j], h[j], alpha);
      }
      push_u8(dst, kEcqHeaderBytes + byte0 + e / DPB, uint8_t(ecq_quant_byte<BW>(v, h, count, beta, scale, seed, byte0 + e / DPB)));
      for (int j = 0; j < count; ++j) hist[begin + e + j] = h[j];
    }
  }
  grid_leave(scratch, place);
}

// Headers of all payloads -> mx, gap, bw (shared memory); false, with the status word set, when one of
// them does not fit or their bitwidths differ.  Whole CTA.
__device__ __forceinline__ bool ecq_read_headers(const UnpackSources& src, int64_t n, float* s_mx, float* s_gap, int* s_bw,
                                                 int* status) {
  __shared__ int all_ok;
  if (threadIdx.x == 0) all_ok = 1;
  __syncthreads();
  const int r = int(threadIdx.x);   // thread r reads header r, all at the same time
  if (r < src.world) {
    const uint8_t* p = select_payload(src, r) + src.parity_off;
    uint32_t total = 0, mb = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      total |= uint32_t(p[k]) << (8 * k);
      mb |= uint32_t(p[4 + k]) << (8 * k);
    }
    const int bw = p[8], unused = p[9], first_bw = src.payload[0][src.parity_off + 8];
    bool ok = ecq_bitwidth_ok(bw) && int64_t(total) <= select_payload_bytes(src, r);
    if (ok) ok = (int64_t(total) - kEcqHeaderBytes) * (8 / bw) - unused == n;
    const float mx = __uint_as_float(mb);
    s_mx[r] = mx;
    s_bw[r] = bw;
    s_gap[r] = (ok && mx > 0.0f) ? ecq_gap(mx, bw) : 0.0f;
    if (!ok || bw != first_bw) all_ok = 0;
  }
  __syncthreads();
  if (!all_ok) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && status) atomicExch(status, int(kBadHeader));
    return false;
  }
  return true;
}

// One thread decodes one payload byte of every rank: DPB consecutive elements.
__global__ void __launch_bounds__(kThreads)
ecq_unpack_kernel(UnpackSources src, float* __restrict__ out, int64_t n, int add, float post_scale,
                  int* status) {
  if (status_guarded(src.guard)) return;
  resolve_epoch(src);
  __shared__ float s_mx[kMaxWorld], s_gap[kMaxWorld];
  __shared__ int s_bw[kMaxWorld];
  if (!ecq_read_headers(src, n, s_mx, s_gap, s_bw, status)) return;
  const int bw = s_bw[0], dpb = 8 / bw;
  const uint32_t mask = (1u << bw) - 1u;
  const int64_t M = (n + dpb - 1) / dpb;
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  for (int64_t b = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; b < M; b += stride) {
    uint32_t byte[kMaxWorld];
#pragma unroll
    for (int r = 0; r < kMaxWorld; ++r)
      byte[r] = r < src.world ? uint32_t(src.payload[r][src.parity_off + kEcqHeaderBytes + b]) : 0u;
    for (int j = 0; j < dpb; ++j) {
      const int64_t i = b * dpb + j;
      if (i >= n) break;
      float acc = add ? out[i] : 0.0f;
#pragma unroll
      for (int r = 0; r < kMaxWorld; ++r) {
        if (r < src.world) {
          const float v = ecq_dequant((byte[r] >> (j * bw)) & mask, s_gap[r], s_mx[r]);
          acc = (r == 0 && !add) ? v : hp_add(acc, v);
        }
      }
      if (post_scale != 1.0f) acc = hp_mul(acc, post_scale);
      out[i] = acc;
    }
  }
}

// The same into a dense array that is overwritten, 16-byte aligned, by index tables (see unpack_lut.cuh)
// whose sums run rank by rank: this codec's order.  The bitwidth is in the headers, which only the
// device reads: all three decode loops are compiled, and the shared memory is sized for the largest.
// The byte loop above costs one scalar load per rank and one scalar store per element:
// 4 bits, four payloads, 25 MB: 11.3 us in a chain of calls; (ncu, cold) 34.9 by bytes.
template <int WORLD>
__global__ void __launch_bounds__(index_threads(WORLD), index_ctas(WORLD))
ecq_unpack_index_kernel(UnpackSources src, float* __restrict__ out, int64_t n, float post_scale, int* status, int align) {
  wait_for_previous();
  if (status_guarded(src.guard)) return;
  resolve_epoch(src);
  extern __shared__ __align__(16) float smem[];
  __shared__ float s_mx[kMaxWorld], s_gap[kMaxWorld];
  __shared__ int s_bw[kMaxWorld];
  if (!ecq_read_headers(src, n, s_mx, s_gap, s_bw, status)) return;
  const int64_t data_offset = kEcqHeaderBytes + src.parity_off;
  const SgdApply none;
  if (s_bw[0] == 8) {
    float mx[WORLD], gap[WORLD];
#pragma unroll
    for (int r = 0; r < WORLD; ++r) {
      mx[r] = s_mx[r];
      gap[r] = s_gap[r];
    }
    unpack_bytes_body<false, WORLD, true>(src, data_offset, align, out, n, 0, post_scale, none,
                                          [&](int r, uint32_t q) { return ecq_dequant(q, gap[r], mx[r]); });
    return;
  }
  auto value = [&](int r, uint32_t q) { return ecq_dequant(q, s_gap[r], s_mx[r]); };
  auto decode = [&](auto bits) {
    constexpr int BW = decltype(bits)::value;
    PayloadWords<WORLD> w;
    index_prefetch<BW, WORLD>(src, kEcqHeaderBytes, n, align, w);
    build_index_tables<BW, WORLD, false, true>(smem, value);
    __syncthreads();
    unpack_index_body<BW, false, WORLD, false, true>(smem, w, 0u, src, data_offset, align, out, n, 0, post_scale, none);
  };
  if (s_bw[0] == 2) decode(std::integral_constant<int, 2>{});
  else decode(std::integral_constant<int, 4>{});
}

template <int WORLD>
cudaError_t launch_ecq_index(const UnpackSources& src, float* out, int64_t n, float post_scale, int* status,
                             cudaStream_t stream, bool overlap) {
  constexpr size_t b2 = IndexLayout<2, WORLD, false, true>::kBytes, b4 = IndexLayout<4, WORLD, false, true>::kBytes;
  constexpr size_t smem = b2 > b4 ? b2 : b4;
  if (smem > 40 * 1024) {   // with the static part, past the default limit
    const cudaError_t e = cudaFuncSetAttribute(ecq_unpack_index_kernel<WORLD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               int(smem));
    if (e != cudaSuccess) return e;
  }
  // sized by the smallest chunk (4 bits); at 8 bits the loop strides over what there is
  const int grid = index_grid(n, IndexForm<4>::kChunk, WORLD, smem);
  return launch_with(overlap, 1, ecq_unpack_index_kernel<WORLD>, dim3(grid), dim3(index_threads(WORLD)), smem, stream, src, out, n,
                     post_scale, status, payload_alignment(src, kEcqHeaderBytes));
}

}  // namespace

cudaError_t ecq_compress(const float* grad, float* history, int64_t n, float alpha, float beta,
                         int bitwidth, uint64_t seed, const PushTargets& dst, void* scratch,
                         cudaStream_t stream, bool whole_gpu, int* status, uint64_t grid_wait_ns, bool overlap) {
  if (n <= 0 || !ecq_bitwidth_ok(bitwidth) || scratch == nullptr) return cudaErrorInvalidValue;
  auto* s = static_cast<MinMaxScratch*>(scratch);
  PushTargets hdr_dst = dst;
  hdr_dst.done = nullptr;
  const bool vec = aligned16(grad) && aligned16(history);
  const int shift = chunk_shift(dst, kEcqHeaderBytes);
  if (hold_alone(whole_gpu, dst) && status != nullptr && vec && shift >= 0) {
    HoldPlan hold;
    cudaError_t e = hold_plan(n, bitwidth, hold);
    if (e != cudaSuccess) return e;
    if (hold.part > 0) {
      auto kernel = bitwidth == 2 ? ecq_hold_kernel<2> : (bitwidth == 4 ? ecq_hold_kernel<4> : ecq_hold_kernel<8>);
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(hold.smem));
      if (e != cudaSuccess) return e;
      e = launch_resident(kernel, dim3(hold.ctas), dim3(kHoldThreads), hold.smem, stream, grad, history, n, hold.part, alpha, beta,
                          seed, dst, s, shift, grid_wait_ns, status);
      if (e != cudaErrorCooperativeLaunchTooLarge) return e;
      cudaGetLastError();   // fewer SMs than the device has: the two launches below
    }
  }
  const int hgrid = grid_for((n + 3) >> 2, kThreads, 148 * 4);
  const cudaError_t e = launch_with(overlap, 1, vec ? ecq_absmax_header_kernel<true> : ecq_absmax_header_kernel<false>, dim3(hgrid),
                                    dim3(kThreads), 0, stream, grad, history, n, alpha, bitwidth, hdr_dst, s);
  if (e != cudaSuccess) return e;
  // chunked path once there is a chunk per warp of a half-filled GPU
  const int64_t chunks = n / (int64_t(kStageBytes) * (8 / bitwidth));
  const bool wide = vec && shift >= 0 && chunks >= 148 * 2;
  const int threads = wide ? 128 : kThreads;
  const int grid = wide ? grid_for(chunks * 32, threads, 148 * 16) : grid_for((n + 3) >> 2, kThreads, 148 * 8);
#define HP_ECQ(BW)                                                                                                   \
  return vec ? launch_after(ecq_quant_kernel<BW, true>, dim3(grid), dim3(threads), 0, stream, grad, history, n,      \
                            alpha, beta, seed, dst, s, wide ? shift : -1)                                            \
             : launch_after(ecq_quant_kernel<BW, false>, dim3(grid), dim3(threads), 0, stream, grad, history, n,     \
                            alpha, beta, seed, dst, s, -1)
  switch (bitwidth) {
    case 2: HP_ECQ(2);
    case 4: HP_ECQ(4);
    default: HP_ECQ(8);
  }
#undef HP_ECQ
}

cudaError_t ecq_unpack_accum(const UnpackSources& src, float* out, int64_t n, int add,
                             float post_scale, int* status, cudaStream_t stream, bool overlap) {
  if (n <= 0 || src.world < 1 || src.world > kMaxWorld) return cudaErrorInvalidValue;
  if (!add && aligned16(out)) {
#define HP_INDEX(W) case W: return launch_ecq_index<W>(src, out, n, post_scale, status, stream, overlap)
    switch (src.world) {
      HP_INDEX(1); HP_INDEX(2); HP_INDEX(3); HP_INDEX(4); HP_INDEX(5); HP_INDEX(6); HP_INDEX(7); HP_INDEX(8);
    }
#undef HP_INDEX
  }
  // one thread per payload byte (at least two elements)
  ecq_unpack_kernel<<<grid_for((n + 1) >> 1, kThreads, 148 * 8), kThreads, 0, stream>>>(src, out, n, add,
                                                                                        post_scale, status);
  return cudaGetLastError();
}

}  // namespace cuda
}  // namespace hipress
