// Min-max k-bit quantiser ("TernGrad" codec of the reference) for sm_100a.
//
// Compress is two kernels and no host synchronisation:
//   1. minmax_header_kernel  grid reduction of min/max over grad (+ residual);
//      the last CTA derives gap and 1/(gap+1e-8) (in double, as the reference's
//      host code does: terngrad_body.h:205-206), stores them for kernel 2 and
//      writes the 10-byte header into every destination.
//   2. tern_quant_kernel     quantises with per-byte LCG stochastic rounding
//      (or round-half-even), packs, stores the bytes into every destination,
//      optionally writes the error-feedback residual, handles the always
//      deterministic partial last byte in-kernel, then publishes the flag.
// The reference needs minmax_element + D2H + sync, a header H2D, a transform,
// and a second D2H/sync/H2D for the tail (terngrad_body.h:186-298).
//
// Unpack-accumulate decodes the payloads of all ranks in one pass, each with
// its own header, in ascending rank order.
#include "../common/codec_math.h"
#include "hold.cuh"
#include "kernels.h"
#include "launch.cuh"
#include "p2p.cuh"
#include "reduce.cuh"
#include "unpack_lut.cuh"

#include <algorithm>

#include <cooperative_groups.h>

namespace hipress {
namespace cuda {

namespace {

namespace cg = cooperative_groups;

constexpr int kThreads = 256;

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
inline int grid_for(int64_t items, int threads, int max_blocks) {
  int64_t blocks = (items + threads - 1) / threads;
  if (blocks < 1) blocks = 1;
  if (blocks > max_blocks) blocks = max_blocks;
  return int(blocks);
}

__device__ __forceinline__ void put_header(const PushTargets& dst, const PushCursor& cur, int64_t n, int bw, float mn,
                                           float mx) {
  uint8_t header[kTernHeaderBytes];
  header[0] = uint8_t(bw);
  header[1] = uint8_t(tern_tail(n, bw));
  const uint32_t a = __float_as_uint(mn), b = __float_as_uint(mx);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    header[2 + k] = uint8_t(a >> (8 * k));
    header[6 + k] = uint8_t(b >> (8 * k));
  }
  put_bytes(dst, cur, 0, header, kTernHeaderBytes);
}

template <bool VEC, bool EF>
__global__ void __launch_bounds__(kThreads)
minmax_header_kernel(const float* grad, const float* residual, int64_t n, int bw, PushTargets dst, MinMaxScratch* scratch) {
  wait_for_previous();
  if (push_guarded(dst)) return;
  resolve_epoch(dst);
  // scatter mode: blockIdx.y is the shard; each shard has its own reduction state and header
  PushCursor cur{nullptr};
  if (dst.shard_elems > 0) {
    const int j = blockIdx.y;
    const int64_t cnt = shard_len(n, dst.shard_elems, j);
    if (cnt == 0) return;
    grad += int64_t(j) * dst.shard_elems;
    if (EF) residual += int64_t(j) * dst.shard_elems;
    n = cnt;
    scratch += j;
    cur.one = select_dest(dst, j);
  }
  float mn = INFINITY, mx = -INFINITY;
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  const int64_t tid = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (VEC) {
    const int64_t nv = n >> 2;
    auto fold = [&](float4 g, float4 r) {
      if (EF) {
        g.x = hp_add(g.x, r.x); g.y = hp_add(g.y, r.y);
        g.z = hp_add(g.z, r.z); g.w = hp_add(g.w, r.w);
      }
      mn = fminf(mn, fminf(fminf(g.x, g.y), fminf(g.z, g.w)));
      mx = fmaxf(mx, fmaxf(fmaxf(g.x, g.y), fmaxf(g.z, g.w)));
    };
    int64_t i = tid;
    for (; i + 3 * stride < nv; i += 4 * stride) {   // four loads of each array in flight
      float4 g[4], r[4] = {};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        g[u] = reinterpret_cast<const float4*>(grad)[i + u * stride];
        if (EF) r[u] = reinterpret_cast<const float4*>(residual)[i + u * stride];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) fold(g[u], r[u]);
    }
    for (; i < nv; i += stride)
      fold(reinterpret_cast<const float4*>(grad)[i],
           EF ? reinterpret_cast<const float4*>(residual)[i] : make_float4(0.f, 0.f, 0.f, 0.f));
    for (int64_t i = (nv << 2) + tid; i < n; i += stride) {
      const float v = EF ? hp_add(grad[i], residual[i]) : grad[i];
      mn = fminf(mn, v);
      mx = fmaxf(mx, v);
    }
  } else {
    for (int64_t i = tid; i < n; i += stride) {
      const float v = EF ? hp_add(grad[i], residual[i]) : grad[i];
      mn = fminf(mn, v);
      mx = fmaxf(mx, v);
    }
  }
  let_next_start();
  float gmn, gmx;
  if (!grid_minmax_last_block<kThreads>(scratch, mn, mx, gmn, gmx)) return;
  if (threadIdx.x == 0) {
    const float gap = tern_gap(gmn, gmx, bw);
    scratch->mn = gmn;
    scratch->mx = gmx;
    scratch->gap = gap;
    scratch->inv = tern_gap_inverse(gap);
    put_header(dst, cur, n, bw, gmn, gmx);
  }
}

// Elements handled by one thread and bytes it produces.
template <int BW> struct Unit {
  static constexpr int DPB = 8 / BW;
  static constexpr int EPT = DPB > 4 ? DPB : 4;  // elements per thread
  static constexpr int BPT = EPT / DPB;          // bytes per thread: 1,1,2,4
};

constexpr int kStageBytes = 512;  // payload bytes a warp gathers before it stores them

// Quantise the EPT elements of one unit; returns its BPT payload bytes (little-endian).
template <int BW, bool EF>
__device__ __forceinline__ uint32_t tern_quant_unit(float (&x)[Unit<BW>::EPT], int64_t first_byte, float mn,
                                                    float inv, float gap, int random, uint64_t seed,
                                                    float (&ef)[Unit<BW>::EPT]) {
  constexpr int DPB = Unit<BW>::DPB, BPT = Unit<BW>::BPT;
  uint32_t bytes = 0;
#pragma unroll
  for (int b = 0; b < BPT; ++b) {
    const uint8_t q = tern_pack_byte<BW>(x + b * DPB, DPB, mn, inv, random != 0,
                                         tern_byte_seed(seed, first_byte + b), gap,
                                         EF ? ef + b * DPB : nullptr);
    bytes |= uint32_t(q) << (8 * b);
  }
  return bytes;
}

// The payload bytes of unit u, one unit per lane: the lanes combine theirs into 32-bit words.  Whole
// warp; u < units tells the lanes that hold one.
template <int BPT>
__device__ __forceinline__ void put_unit_bytes(const PushTargets& dst, const PushCursor& cur, int64_t u, int64_t units,
                                               uint32_t bytes) {
  if (BPT == 1) {
    const uint32_t word = gather4_bytes(bytes);
    if ((threadIdx.x & 3) == 0 && u < units) {
      if (u + 3 < units) {
        put_u32(dst, cur, kTernHeaderBytes + u, word);
      } else {
        for (int64_t b = u; b < units; ++b)
          put_u8(dst, cur, kTernHeaderBytes + b, uint8_t(word >> (8 * (b - u))));
      }
    }
  } else if (BPT == 2) {
    const uint32_t word = gather2_halves(bytes);
    if ((threadIdx.x & 1) == 0 && u < units) {
      if (u + 1 < units) {
        put_u32(dst, cur, kTernHeaderBytes + 2 * u, word);
      } else {
        put_u8(dst, cur, kTernHeaderBytes + 2 * u, uint8_t(word));
        put_u8(dst, cur, kTernHeaderBytes + 2 * u + 1, uint8_t(word >> 8));
      }
    }
  } else {
    if (u < units) put_u32(dst, cur, kTernHeaderBytes + 4 * u, bytes);
  }
}

// Elements from `done` to the end of a tensor (or shard), fewer than a unit: whole bytes keep the
// requested rounding mode, the partial last byte is always deterministic.  One thread.
template <int BW, bool EF>
__device__ __forceinline__ void tern_leftover(const float* grad, float* residual, int64_t done, int64_t n, float mn,
                                              float inv, float gap, int random, uint64_t seed, const PushTargets& dst,
                                              const PushCursor& cur) {
  constexpr int DPB = 8 / BW;
  int64_t byte_index = done / DPB;
  for (int64_t e = done; e < n; e += DPB, ++byte_index) {
    const int count = (n - e) >= DPB ? DPB : int(n - e);
    float x[DPB], ef[DPB];
    for (int j = 0; j < count; ++j) x[j] = EF ? hp_add(grad[e + j], residual[e + j]) : grad[e + j];
    const bool rnd = random != 0 && count == DPB;
    const uint8_t q = tern_pack_byte<BW>(x, count, mn, inv, rnd, tern_byte_seed(seed, byte_index), gap,
                                         EF ? ef : nullptr);
    put_u8(dst, cur, kTernHeaderBytes + byte_index, q);
    if (EF)
      for (int j = 0; j < count; ++j) residual[e + j] = ef[j];
  }
}

// shift >= 0: large tensors whose destinations start equally far past a 16-byte boundary.  A warp
// then works on chunks of 512 payload bytes: in each of J = 16/BPT sub-steps lane L quantises unit
// j*32+L of the chunk (coalesced 16-byte loads), the bytes are gathered in shared memory, and every
// lane stores 16 of them to each destination (put_chunk512) -- 512 contiguous bytes per warp and
// destination, against the 32 bytes per warp of the word path, which is what NVLink peer stores need
// to run near link speed, and half the instructions.  The rest of the tensor (less than one chunk)
// takes the word path.  A payload at the start of a tensor has its packed data 10 bytes past a
// boundary: against 2-byte stores, and together with the cheaper draws of Lcg32::unit_from_raw, chunks save 2 us of
// compressing 9.4 MB at 4 bits in two launches and 4 us of 25 MB with ECQ.
template <int BW, bool VEC, bool EF>
__global__ void __launch_bounds__(kThreads)
tern_quant_kernel(const float* __restrict__ grad, float* __restrict__ residual, int64_t n,
                  int random, uint64_t seed, PushTargets dst, const MinMaxScratch* scratch, int shift) {
  wait_for_previous();
  if (push_guarded(dst)) return;
  resolve_epoch(dst);
  if (dst.epoch_dev != nullptr) seed += uint64_t(dst.epoch) * kEpochSeedStride;
  constexpr int DPB = Unit<BW>::DPB, EPT = Unit<BW>::EPT, BPT = Unit<BW>::BPT;
  const int64_t S = dst.shard_elems;
  // state of the shard in hand (the whole tensor unless in scatter mode)
  int cur_j = -1;
  PushCursor cur{nullptr};
  float mn = 0.f, inv = 0.f, gap = 0.f;
  uint64_t cur_seed = seed;
  auto enter = [&](int j) {   // (re)load what depends on the shard
    if (j == cur_j) return;
    cur_j = j;
    const MinMaxScratch* s = scratch + (S > 0 ? j : 0);
    mn = s->mn; inv = s->inv; gap = s->gap;
    if (S > 0) {
      cur.one = select_dest(dst, j);
      cur_seed = seed + uint64_t(j) * kShardSeedStride;
    }
  };
  if (S == 0) enter(0);

  // ---- chunks of 512 payload bytes
  constexpr int64_t CH = int64_t(kStageBytes) * DPB;
  int64_t chunks = 0;
  if (VEC && shift >= 0) {
    __shared__ __align__(16) uint8_t stages[kThreads / 32][kStageBytes + 16];
    constexpr int J = 16 / BPT;           // sub-steps per chunk
    constexpr int U = EPT == 8 ? 2 : 4;   // sub-steps whose loads are issued together
    chunks = n / CH;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint8_t* const stage = stages[warp] + shift;
    const int64_t warps = int64_t(gridDim.x) * (blockDim.x >> 5);
    for (int64_t c = int64_t(blockIdx.x) * (blockDim.x >> 5) + warp; c < chunks; c += warps) {
      int64_t ebase = c * CH;        // first element of the chunk in the tensor
      int64_t lbase = ebase;         // ... and relative to its shard
      if (S > 0) {
        const int j = int(ebase / S);
        enter(j);
        lbase = ebase - int64_t(j) * S;
      }
      const int64_t bbase = lbase / DPB;  // first payload byte of the chunk
#pragma unroll 1
      for (int j0 = 0; j0 < J; j0 += U) {
        float x[U][EPT], ef[U][EPT];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int64_t e0 = ebase + int64_t((j0 + u) * 32 + lane) * EPT;
#pragma unroll
          for (int v = 0; v < EPT / 4; ++v) {
            float4 g = __ldg(reinterpret_cast<const float4*>(grad + e0) + v);
            if (EF) {
              const float4 r = reinterpret_cast<const float4*>(residual + e0)[v];
              g.x = hp_add(g.x, r.x); g.y = hp_add(g.y, r.y);
              g.z = hp_add(g.z, r.z); g.w = hp_add(g.w, r.w);
            }
            x[u][4 * v] = g.x; x[u][4 * v + 1] = g.y; x[u][4 * v + 2] = g.z; x[u][4 * v + 3] = g.w;
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int unit = (j0 + u) * 32 + lane;
          const uint32_t bytes = tern_quant_unit<BW, EF>(x[u], bbase + int64_t(unit) * BPT, mn, inv, gap, random,
                                                         cur_seed, ef[u]);
          if (EF) {
            const int64_t e0 = ebase + int64_t(unit) * EPT;
#pragma unroll
            for (int v = 0; v < EPT / 4; ++v)
              reinterpret_cast<float4*>(residual + e0)[v] =
                  make_float4(ef[u][4 * v], ef[u][4 * v + 1], ef[u][4 * v + 2], ef[u][4 * v + 3]);
          }
          if (BPT == 1) {
            stage[unit] = uint8_t(bytes);
          } else if (BPT == 2) {
            reinterpret_cast<uint16_t*>(stage)[unit] = uint16_t(bytes);
          } else if ((shift & 3) == 0) {
            reinterpret_cast<uint32_t*>(stage)[unit] = bytes;
          } else {
            reinterpret_cast<uint16_t*>(stage)[2 * unit] = uint16_t(bytes);
            reinterpret_cast<uint16_t*>(stage)[2 * unit + 1] = uint16_t(bytes >> 16);
          }
        }
      }
      __syncwarp();
      put_chunk512(dst, cur, kTernHeaderBytes + bbase, stages[warp], shift, lane);
      __syncwarp();
    }
  }

  // ---- the rest, one unit per thread: lanes combine their bytes into 32-bit words
  const int64_t rest_begin = chunks * CH;         // element
  int64_t rest_local = rest_begin;                // relative to its shard
  int64_t rest_n = n;                             // end of the rest, relative to its shard
  if (S > 0 && rest_begin < n) {
    const int j = int(rest_begin / S);
    enter(j);
    rest_local = rest_begin - int64_t(j) * S;
    rest_n = rest_local + (n - rest_begin);
  }
  const float* g_rest = grad + (rest_begin - rest_local);      // shard base
  float* r_rest = EF ? residual + (rest_begin - rest_local) : nullptr;
  const int64_t unit0 = rest_local / EPT;
  const int64_t units = rest_n / EPT;             // complete units of the shard
  const int64_t span = units - unit0;
  const int64_t span_padded = (span + 31) & ~int64_t(31);
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  for (int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; k < span_padded; k += stride) {
    const int64_t u = unit0 + k;
    uint32_t bytes = 0;
    if (u < units) {
      float x[EPT], ef[EPT];
      const int64_t e0 = u * EPT;
      if (VEC) {
#pragma unroll
        for (int v = 0; v < EPT / 4; ++v) {
          float4 g = __ldg(reinterpret_cast<const float4*>(g_rest + e0) + v);
          if (EF) {
            const float4 r = reinterpret_cast<const float4*>(r_rest + e0)[v];
            g.x = hp_add(g.x, r.x); g.y = hp_add(g.y, r.y);
            g.z = hp_add(g.z, r.z); g.w = hp_add(g.w, r.w);
          }
          x[4 * v] = g.x; x[4 * v + 1] = g.y; x[4 * v + 2] = g.z; x[4 * v + 3] = g.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < EPT; ++i)
          x[i] = EF ? hp_add(g_rest[e0 + i], r_rest[e0 + i]) : g_rest[e0 + i];
      }
      bytes = tern_quant_unit<BW, EF>(x, u * BPT, mn, inv, gap, random, cur_seed, ef);
      if (EF) {
        if (VEC) {
#pragma unroll
          for (int v = 0; v < EPT / 4; ++v)
            reinterpret_cast<float4*>(r_rest + e0)[v] =
                make_float4(ef[4 * v], ef[4 * v + 1], ef[4 * v + 2], ef[4 * v + 3]);
        } else {
#pragma unroll
          for (int i = 0; i < EPT; ++i) r_rest[e0 + i] = ef[i];
        }
      }
    }
    // (k and u differ by a multiple of 32 units only when unit0 is one; the lane pattern of
    // put_unit_bytes depends on the lane, not on u)
    put_unit_bytes<BPT>(dst, cur, u, units, bytes);
  }
  if (units * EPT < rest_n && blockIdx.x == 0 && threadIdx.x == 0)
    tern_leftover<BW, EF>(g_rest, r_rest, units * EPT, rest_n, mn, inv, gap, random, cur_seed, dst, cur);
  publish_when_grid_done(dst);
}

// Small tensors: both passes in one launch.  A cluster of eight CTAs holds the tensor in registers (16
// elements per thread), the CTAs exchange their extremes through distributed shared memory, and the
// quantising pass starts from the registers.  At these sizes a launch costs more than the work: eight
// SMs take the tensor in and quantise it in less time than the second launch and its ramp-up need.
// 256 KB, compress and decode of two payloads: 16.4 us in three launches, 14.3 in two.
// A cluster starts when eight neighbouring SMs have room for 1,024 threads each, so this form is for callers
// that say the GPU is theirs (whole_gpu): beside 16384^3 matrix products a 256 KB task takes 560 us in it
// and 153 in two launches; beside a chain of 4096^3 ones the op takes 96 and 55 us.
constexpr int kSmallCtas = 8, kSmallThreads = 1024, kSmallPerThread = 16;
constexpr int64_t kSmallElems = int64_t(kSmallCtas) * kSmallThreads * kSmallPerThread;
template <int BW, bool VEC, bool EF>
__global__ void __cluster_dims__(kSmallCtas, 1, 1) __launch_bounds__(kSmallThreads)
tern_small_kernel(const float* grad, float* residual, int64_t n, int random, uint64_t seed, PushTargets dst) {
  wait_for_previous();
  constexpr int EPT = Unit<BW>::EPT, BPT = Unit<BW>::BPT, UPT = kSmallPerThread / EPT;
  __shared__ float ext_mn[kSmallCtas], ext_mx[kSmallCtas], scale[4];
  const cg::cluster_group cluster = cg::this_cluster();
  const int64_t units = n / EPT;
  const int64_t tid = int64_t(blockIdx.x) * kSmallThreads + threadIdx.x;
  constexpr int64_t kStride = int64_t(kSmallCtas) * kSmallThreads;
  float x[UPT][EPT];
  float mn = INFINITY, mx = -INFINITY;
#pragma unroll
  for (int q = 0; q < UPT; ++q) {
    const int64_t u = tid + q * kStride;
    if (u < units) {
      if (VEC) {
#pragma unroll
        for (int v = 0; v < EPT / 4; ++v) {
          float4 g = reinterpret_cast<const float4*>(grad + u * EPT)[v];
          if (EF) {
            const float4 r = reinterpret_cast<const float4*>(residual + u * EPT)[v];
            g.x = hp_add(g.x, r.x); g.y = hp_add(g.y, r.y);
            g.z = hp_add(g.z, r.z); g.w = hp_add(g.w, r.w);
          }
          x[q][4 * v] = g.x; x[q][4 * v + 1] = g.y; x[q][4 * v + 2] = g.z; x[q][4 * v + 3] = g.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < EPT; ++i)
          x[q][i] = EF ? hp_add(grad[u * EPT + i], residual[u * EPT + i]) : grad[u * EPT + i];
      }
#pragma unroll
      for (int i = 0; i < EPT; ++i) {
        mn = fminf(mn, x[q][i]);
        mx = fmaxf(mx, x[q][i]);
      }
    }
  }
  if (tid == 0) {
    for (int64_t e = units * EPT; e < n; ++e) {
      const float v = EF ? hp_add(grad[e], residual[e]) : grad[e];
      mn = fminf(mn, v);
      mx = fmaxf(mx, v);
    }
  }
  block_minmax<kSmallThreads>(mn, mx);
  cluster.sync();   // the other CTAs' shared memory exists from here on
  if (threadIdx.x == 0) {
    for (int c = 0; c < kSmallCtas; ++c) {
      cluster.map_shared_rank(ext_mn, c)[blockIdx.x] = mn;
      cluster.map_shared_rank(ext_mx, c)[blockIdx.x] = mx;
    }
  }
  cluster.sync();
  PushCursor cur{nullptr};
  if (threadIdx.x == 0) {
    mn = ext_mn[0];
    mx = ext_mx[0];
    for (int c = 1; c < kSmallCtas; ++c) {
      mn = fminf(mn, ext_mn[c]);
      mx = fmaxf(mx, ext_mx[c]);
    }
    const float gap = tern_gap(mn, mx, BW);
    scale[0] = mn;
    scale[1] = gap;
    scale[2] = tern_gap_inverse(gap);
    if (blockIdx.x == 0) put_header(dst, cur, n, BW, mn, mx);
  }
  __syncthreads();
  mn = scale[0];
  const float gap = scale[1], inv = scale[2];
#pragma unroll
  for (int q = 0; q < UPT; ++q) {
    const int64_t u = tid + q * kStride;
    if (q * kStride + (tid & ~int64_t(31)) >= units) break;   // whole warps leave together
    uint32_t bytes = 0;
    if (u < units) {
      float ef[EPT];
      bytes = tern_quant_unit<BW, EF>(x[q], u * BPT, mn, inv, gap, random, seed, ef);
      if (EF) {
        if (VEC) {
#pragma unroll
          for (int v = 0; v < EPT / 4; ++v)
            reinterpret_cast<float4*>(residual + u * EPT)[v] =
                make_float4(ef[4 * v], ef[4 * v + 1], ef[4 * v + 2], ef[4 * v + 3]);
        } else {
#pragma unroll
          for (int i = 0; i < EPT; ++i) residual[u * EPT + i] = ef[i];
        }
      }
    }
    put_unit_bytes<BPT>(dst, cur, u, units, bytes);
  }
  if (tid == 0 && units * EPT < n)
    tern_leftover<BW, EF>(grad, residual, units * EPT, n, mn, inv, gap, random, seed, dst, cur);
}

// Medium tensors: both passes in one launch that reads the inputs once.  One CTA per SM keeps its part of
// grad + residual in shared memory (up to 208 KB of it: 30 MB over the chip), the CTAs exchange their
// extremes through the scratch, and quantise from shared memory.  The two-launch form reads both arrays
// twice, the second time from L2, and drains and refills the chip in between.  All CTAs have to be resident
// at once and each needs an SM to itself, so this form too is for callers that say the GPU is theirs: the
// exchange engine and the task API, whose compressors run beside the backward pass, keep the two launches.
// Beside a chain of 16384^3 matrix products a 4 MB task takes 850 us in this form (it waits for SMs to fall
// free) and 260 in two launches; on an idle GPU 64 and 71 us.
// 25 MB with error feedback, 2 bits (ncu, cold): 21.3 us with a slower exchange of the extremes; 14.3 + 18.0 in two
// launches.  9.4 MB at 4 bits, compress and decode: 12.3; two launches were 4 us slower.  A thread of 25 MB has eleven
// words: with the last three loaded one after another, compress and the decode of eight payloads take 35.3 us, and
// 34.9 so.  Inside the kernel: 11.5 us for 52 MB of inputs, 1.9 the exchange, 6 the quantiser and its stores.
template <int BW, bool EF>
__global__ void __launch_bounds__(kHoldThreads, 1)
tern_hold_kernel(const float* __restrict__ grad, float* __restrict__ residual, int64_t n, int64_t part, int random,
                 uint64_t seed, PushTargets dst, MinMaxScratch* scratch, int shift, uint64_t wait_ns, int* status) {
  constexpr int DPB = 8 / BW, EPT = Unit<BW>::EPT, BPT = Unit<BW>::BPT;
  extern __shared__ __align__(16) float hold[];           // [part], then the payload bytes
  __shared__ float scale[3];
  uint8_t* const bytes_at = reinterpret_cast<uint8_t*>(hold + part);
  const int tid = threadIdx.x;
  GridPlace place;
  grid_arrive(scratch, place);
  const int64_t begin = int64_t(blockIdx.x) * part;       // a multiple of 512
  const int64_t left = n - begin;
  const int len = int(left < 0 ? 0 : (left < part ? left : part));
  const float4* g4 = reinterpret_cast<const float4*>(grad + begin);
  const float4* r4 = EF ? reinterpret_cast<const float4*>(residual + begin) : nullptr;
  float mn = INFINITY, mx = -INFINITY;
  const int quads = len >> 2;
  auto take = [&](int i, float4 g, float4 r) {
    if (EF) {
      g.x = hp_add(g.x, r.x); g.y = hp_add(g.y, r.y);
      g.z = hp_add(g.z, r.z); g.w = hp_add(g.w, r.w);
    }
    mn = fminf(mn, fminf(fminf(g.x, g.y), fminf(g.z, g.w)));
    mx = fmaxf(mx, fmaxf(fmaxf(g.x, g.y), fmaxf(g.z, g.w)));
    reinterpret_cast<float4*>(hold)[i] = g;
  };
  for (int q = tid; q < quads; q += 4 * kHoldThreads) {   // the last, partial round keeps its loads together too
    float4 g[4], r[4] = {};
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (q + u * kHoldThreads < quads) {
        g[u] = __ldg(g4 + q + u * kHoldThreads);
        if (EF) r[u] = r4[q + u * kHoldThreads];
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (q + u * kHoldThreads < quads) take(q + u * kHoldThreads, g[u], r[u]);
  }
  for (int e = 4 * quads + tid; e < len; e += kHoldThreads) {   // fewer than four
    const float v = EF ? hp_add(grad[begin + e], residual[begin + e]) : grad[begin + e];
    mn = fminf(mn, v);
    mx = fmaxf(mx, v);
  }
  if (!grid_minmax_all<kHoldThreads>(scratch, mn, mx, wait_ns, status, place)) {
    grid_leave(scratch, place);
    return;
  }
  const PushCursor cur{nullptr};
  if (tid == 0) {
    const float gap = tern_gap(mn, mx, BW);
    scale[0] = gap;
    scale[1] = tern_gap_inverse(gap);
    if (blockIdx.x == 0) put_header(dst, cur, n, BW, mn, mx);
  }
  __syncthreads();
  const float gap = scale[0], inv = scale[1];
  const int64_t byte0 = begin / DPB;                       // first payload byte of the part
  const int units = len / EPT;
  for (int u = tid; u < units; u += kHoldThreads) {
    float x[EPT], ef[EPT];
#pragma unroll
    for (int v = 0; v < EPT / 4; ++v) {
      const float4 h = reinterpret_cast<const float4*>(hold)[u * (EPT / 4) + v];
      x[4 * v] = h.x; x[4 * v + 1] = h.y; x[4 * v + 2] = h.z; x[4 * v + 3] = h.w;
    }
    const uint32_t b = tern_quant_unit<BW, EF>(x, byte0 + int64_t(u) * BPT, mn, inv, gap, random, seed, ef);
    if (EF) {
#pragma unroll
      for (int v = 0; v < EPT / 4; ++v)
        reinterpret_cast<float4*>(residual + begin)[u * (EPT / 4) + v] =
            make_float4(ef[4 * v], ef[4 * v + 1], ef[4 * v + 2], ef[4 * v + 3]);
    }
    hold_unit_bytes<BPT>(bytes_at + shift + u * BPT, b);   // shift is even
  }
  __syncthreads();
  hold_put(dst, kTernHeaderBytes, byte0, bytes_at, shift, units * BPT);
  if (tid == 32 && len > 0 && units * EPT < len)
    tern_leftover<BW, EF>(grad, residual, begin + int64_t(units) * EPT, n, mn, inv, gap, random, seed, dst, cur);
  grid_leave(scratch, place);
}

struct TernHeader {
  float mn, gap;
  int bw, ok;
};

__device__ __forceinline__ TernHeader read_header(const uint8_t* p, int64_t cap, int64_t n) {
  TernHeader h;
  h.bw = p[0];
  const int tail = p[1];
  uint32_t a = 0, b = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    a |= uint32_t(p[2 + k]) << (8 * k);
    b |= uint32_t(p[6 + k]) << (8 * k);
  }
  h.mn = __uint_as_float(a);
  h.ok = tern_bitwidth_ok(h.bw) && tern_payload_bytes(n, h.bw) <= cap && tail == tern_tail(n, h.bw);
  h.gap = h.ok ? tern_gap(h.mn, __uint_as_float(b), h.bw) : 0.f;
  return h;
}

// Headers of all payloads -> hdr (shared memory), their common bitwidth -> bw; false, with the status
// word set, when one of them does not fit.  BW > 0: the bitwidth they must have.  concat: payload r holds
// shard r only, possibly nothing.  Whole CTA.
template <int BW>
__device__ __forceinline__ bool read_headers(const UnpackSources& src, int64_t n, bool concat, TernHeader* hdr, int* status,
                                             int& bw) {
  __shared__ int all_ok;
  if (threadIdx.x == 0) all_ok = 1;
  __syncthreads();
  // Thread r reads header r.  The payload is selected and not branched to: a branch per rank would have the
  // ranks' loads, each a miss of every cache, wait for one another.
  const int r = int(threadIdx.x);
  if (r < src.world) {
    const int64_t count = concat ? shard_count(n, src.shard_elems, r) : n;
    if (count > 0) {
      hdr[r] = read_header(select_payload(src, r) + src.parity_off, select_payload_bytes(src, r), count);
      if (!hdr[r].ok) all_ok = 0;
    } else {
      hdr[r].ok = 1; hdr[r].bw = 0; hdr[r].mn = 0.f; hdr[r].gap = 0.f;
    }
  }
  __syncthreads();
  bw = BW;
  if (all_ok) {
    for (int q = 0; q < src.world; ++q) {  // every thread computes the same verdict
      if (hdr[q].bw == 0) continue;        // empty shard
      if (bw == 0) bw = hdr[q].bw;
      if (hdr[q].bw != bw) all_ok = 0;
    }
  }
  __syncthreads();
  if (all_ok && bw != 0) return true;
  if (!all_ok && blockIdx.x == 0 && threadIdx.x == 0 && status) atomicExch(status, int(kBadHeader));
  return false;
}

// Known bitwidth and 16-byte aligned dense arrays: index tables, or arithmetic at 8 bits.
template <int BW, bool APPLY, int WORLD>
__global__ void __launch_bounds__(index_threads(WORLD), index_ctas(WORLD))
tern_unpack_index_kernel(UnpackSources src, float* __restrict__ out, int64_t n, int add, float post_scale, SgdApply apply,
                         int* status, int align) {
  wait_for_previous();
  if (unpack_guarded(src)) return;
  resolve_epoch(src);
  extern __shared__ __align__(16) float smem[];
  __shared__ TernHeader hdr[kMaxWorld];
  const int64_t data_offset = kTernHeaderBytes + src.parity_off;
  int bw;
  if constexpr (BW == 8) {
    if (!read_headers<8>(src, n, false, hdr, status, bw)) return;
    float mn[WORLD], gap[WORLD];
#pragma unroll
    for (int r = 0; r < WORLD; ++r) {
      mn[r] = hdr[r].mn;
      gap[r] = hdr[r].gap;
    }
    unpack_bytes_body<APPLY, WORLD, false>(src, data_offset, align, out, n, add, post_scale, apply,
                                           [&](int r, uint32_t q) { return tern_dequant(q, gap[r], mn[r]); });
  } else {
    PayloadWords<WORLD> w;
    index_prefetch<BW, WORLD>(src, kTernHeaderBytes, n, align, w);
    if (!read_headers<BW>(src, n, false, hdr, status, bw)) return;
    build_index_tables<BW, WORLD, false, false>(
        smem, [&](int r, uint32_t q) { return tern_dequant(q, hdr[r].gap, hdr[r].mn); });
    __syncthreads();
    unpack_index_body<BW, APPLY, WORLD, false, false>(smem, w, 0u, src, data_offset, align, out, n, add, post_scale, apply);
  }
}

// Table-driven unpack of everything else (see unpack_lut.cuh).  All payloads of one call must carry the
// same bitwidth; it is read from the headers, so the host never has to look at a payload.  BW > 0
// compiles the decode loop for that bitwidth only (fewer registers, more resident CTAs); BW == 0
// dispatches on the header at run time for callers that do not know the bitwidth.
// CONCAT: concatenated shards (2 bits, aligned dense arrays); otherwise nibble or byte tables.
template <int BW, bool APPLY, bool CONCAT>
__global__ void __launch_bounds__(kUnpackThreads, CONCAT ? 4 : 1)
tern_unpack_lut_kernel(UnpackSources src, float* __restrict__ out, int64_t n, int add,
                       float post_scale, SgdApply apply, int* status) {
  if (unpack_guarded(src)) return;
  resolve_epoch(src);
  extern __shared__ __align__(16) float lut[];  // [world][256][dpb], byte-table path only
  constexpr bool nibbles = BW == 1 || BW == 2 || BW == 4;
  __shared__ __align__(128) float tab[nibbles ? kMaxWorld * 16 * (4 / (BW ? BW : 1)) : 1];
  __shared__ TernHeader hdr[kMaxWorld];
  uint32_t first[kMaxWorld];
  if constexpr (nibbles && !CONCAT) unpack_nibble_prefetch<BW>(src, kTernHeaderBytes, src.parity_off, n, first);
  int bw;
  if (!read_headers<BW>(src, n, CONCAT, hdr, status, bw)) return;
  const int64_t data_offset = kTernHeaderBytes + src.parity_off;
  if constexpr (nibbles) {
    // nibble tables (see unpack_lut.cuh): entry (rank, nibble, slot)
    constexpr int DPN = 4 / BW;
    for (int i = threadIdx.x; i < src.world * 16 * DPN; i += blockDim.x) {
      const int r = i / (16 * DPN), v = (i / DPN) & 15, j = i % DPN;
      tab[i] = tern_dequant((uint32_t(v) >> (BW * j)) & ((1u << BW) - 1u), hdr[r].gap, hdr[r].mn);
    }
    __syncthreads();
    if constexpr (CONCAT)
      unpack_concat_body<APPLY, false>(tab, src, data_offset, out, n, add, post_scale, apply);
    else
      unpack_nibble_body<BW, APPLY, false>(tab, first, src, data_offset, out, n, add, post_scale, apply);
    return;
  } else {
  const int dpb = 8 / bw;
  const uint32_t mask = (1u << bw) - 1u;
  for (int i = threadIdx.x; i < src.world * 256; i += blockDim.x) {
    const int r = i >> 8, v = i & 255;
    for (int j = 0; j < dpb; ++j)
      lut[(r * 256 + int(lut_row(uint32_t(v)))) * dpb + j] =
          tern_dequant((uint32_t(v) >> (bw * j)) & mask, hdr[r].gap, hdr[r].mn);
  }
  __syncthreads();
  if (BW > 0) {
    unpack_lut_body<8 / (BW > 0 ? BW : 1), APPLY>(lut, src, data_offset, out, n, add, post_scale, apply);
  } else {
    switch (bw) {
      case 1: unpack_lut_body<8, APPLY>(lut, src, data_offset, out, n, add, post_scale, apply); break;
      case 2: unpack_lut_body<4, APPLY>(lut, src, data_offset, out, n, add, post_scale, apply); break;
      case 4: unpack_lut_body<2, APPLY>(lut, src, data_offset, out, n, add, post_scale, apply); break;
      default: unpack_lut_body<1, APPLY>(lut, src, data_offset, out, n, add, post_scale, apply); break;
    }
  }
  }
}

template <int BW, bool APPLY, int WORLD>
cudaError_t launch_tern_index(const UnpackSources& src, float* out, int64_t n, int add, float post_scale,
                              const SgdApply& apply, int* status, cudaStream_t stream, bool overlap) {
  const int align = payload_alignment(src, kTernHeaderBytes);
  int grid = grid_for((n + 3) >> 2, index_threads(WORLD), 148 * 8);
  size_t smem = 0;
  if constexpr (BW != 8) {
    using L = IndexLayout<BW, WORLD, false, false>;
    smem = L::kBytes;
    grid = index_grid(n, IndexForm<BW>::kChunk, WORLD, smem);
    // with the static part, past the default limit; per device, and cheap: set on every launch rather than
    // remembered per process
    if (smem > 40 * 1024) {
      const cudaError_t e = cudaFuncSetAttribute(tern_unpack_index_kernel<BW, APPLY, WORLD>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
      if (e != cudaSuccess) return e;
    }
  }
  return launch_with(overlap, 1, tern_unpack_index_kernel<BW, APPLY, WORLD>, dim3(grid), dim3(index_threads(WORLD)), smem, stream, src,
                     out, n, add, post_scale, apply, status, align);
}

template <int BW, bool APPLY>
cudaError_t launch_tern_unpack(const UnpackSources& src, float* out, int64_t n, int add, float post_scale,
                               const SgdApply& apply, int* status, cudaStream_t stream, bool overlap) {
  bool aligned = aligned16(out);
  if (APPLY) aligned = aligned && aligned16(apply.param) && aligned16(apply.momentum);
  if constexpr (BW == 2) {
    if (src.shard_elems > 0) {
      const int grid = grid_for((n + 15) >> 4, kUnpackThreads, 148 * 4);
      tern_unpack_lut_kernel<2, APPLY, true><<<grid, kUnpackThreads, 0, stream>>>(src, out, n, add, post_scale, apply, status);
      return cudaGetLastError();
    }
  }
  if constexpr (BW > 0) {
    if (aligned) {
#define HP_INDEX(W) case W: return launch_tern_index<BW, APPLY, W>(src, out, n, add, post_scale, apply, status, stream, overlap)
      switch (src.world) {
        HP_INDEX(1); HP_INDEX(2); HP_INDEX(3); HP_INDEX(4); HP_INDEX(5); HP_INDEX(6); HP_INDEX(7); HP_INDEX(8);
        default: return cudaErrorInvalidValue;
      }
#undef HP_INDEX
    }
  }
  // table size: world x 256 x dpb floats; without a known bitwidth, room for 1-bit payloads (dpb = 8)
  const int dpb = BW > 0 ? 8 / BW : 8;
  const bool nibble = BW == 1 || BW == 2 || BW == 4;
  const size_t smem = nibble ? 0 : size_t(src.world) * 256 * dpb * sizeof(float);
  if (!nibble) {
    cudaError_t e = cudaFuncSetAttribute(tern_unpack_lut_kernel<BW, APPLY, false>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * 256 * 8 * 4);
    if (e != cudaSuccess) return e;
  }
  // a CTA decodes many groups so that building its tables stays small against the decode work
  const int64_t groups = (n + 4 * dpb - 1) / (4 * dpb);
  const int grid = grid_for(groups, kUnpackThreads, nibble ? 148 * 4 : 148 * 8);
  tern_unpack_lut_kernel<BW, APPLY, false><<<grid, kUnpackThreads, smem, stream>>>(src, out, n, add, post_scale, apply, status);
  return cudaGetLastError();
}

}  // namespace

size_t minmax_scratch_bytes() { return sizeof(MinMaxScratch); }

cudaError_t terngrad_compress(const float* grad, float* residual, int64_t n, int bitwidth,
                              int enable_random, uint64_t seed, const PushTargets& dst,
                              void* scratch, cudaStream_t stream, bool whole_gpu, int* status, uint64_t grid_wait_ns,
                              bool overlap) {
  if (n <= 0 || !tern_bitwidth_ok(bitwidth) || scratch == nullptr) return cudaErrorInvalidValue;
  auto* s = static_cast<MinMaxScratch*>(scratch);
  const bool ef = residual != nullptr;
  const bool vec = aligned16(grad) && (!ef || aligned16(residual));
  const int64_t S = dst.shard_elems;
  const int shift = chunk_shift(dst, kTernHeaderBytes);
  // scatter mode runs on the chunked path only (see tern_quant_kernel)
  if (S > 0 && (!vec || shift != 0 || S % 4096 != 0 || (n + S - 1) / S > dst.world)) return cudaErrorInvalidValue;
#define LAUNCH_FORMS(LAUNCH, BW)              \
  do {                                        \
    if (vec && ef) LAUNCH(BW, true, true);    \
    else if (vec) LAUNCH(BW, true, false);    \
    else if (ef) LAUNCH(BW, false, true);     \
    else LAUNCH(BW, false, false);            \
  } while (0)
#define LAUNCH_BITS(LAUNCH)                   \
  switch (bitwidth) {                         \
    case 1: LAUNCH_FORMS(LAUNCH, 1); break;   \
    case 2: LAUNCH_FORMS(LAUNCH, 2); break;   \
    case 4: LAUNCH_FORMS(LAUNCH, 4); break;   \
    default: LAUNCH_FORMS(LAUNCH, 8); break;  \
  }
  // a caller that has the GPU to itself, and a destination of this call's own: one launch where the tensor
  // fits (see tern_small_kernel and tern_hold_kernel)
  const bool own = hold_alone(whole_gpu, dst);
  if (own && n <= kSmallElems) {
#define LAUNCH_SMALL(BW, V, E) \
  return launch_with(overlap, 1, tern_small_kernel<BW, V, E>, dim3(kSmallCtas), dim3(kSmallThreads), 0, stream, grad, residual, n, \
                     enable_random, seed, dst)   /* its clusters are part of the kernel */
    LAUNCH_BITS(LAUNCH_SMALL);
#undef LAUNCH_SMALL
    return cudaErrorInvalidValue;
  }
  // 16-byte aligned inputs, and a part per SM that fits its shared memory: one read of them
  if (own && status != nullptr && vec && shift >= 0) {
    HoldPlan hold;
    cudaError_t e = hold_plan(n, bitwidth, hold);
    if (e != cudaSuccess) return e;
    if (hold.part > 0) {
#define LAUNCH_HOLD_AS(BW, E)                                                                                       \
  do {                                                                                                              \
    e = cudaFuncSetAttribute(tern_hold_kernel<BW, E>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(hold.smem)); \
    if (e != cudaSuccess) return e;                                                                                 \
    e = launch_resident(tern_hold_kernel<BW, E>, dim3(hold.ctas), dim3(kHoldThreads), hold.smem, stream, grad,      \
                        residual, n, hold.part, enable_random, seed, dst, s, shift, grid_wait_ns, status);          \
    if (e != cudaErrorCooperativeLaunchTooLarge) return e;                                                          \
    cudaGetLastError();   /* fewer SMs than the device has: the two launches below */                               \
  } while (0)
#define LAUNCH_HOLD(BW) \
  if (ef) LAUNCH_HOLD_AS(BW, true); else LAUNCH_HOLD_AS(BW, false)
      switch (bitwidth) {
        case 1: LAUNCH_HOLD(1); break;
        case 2: LAUNCH_HOLD(2); break;
        case 4: LAUNCH_HOLD(4); break;
        default: LAUNCH_HOLD(8); break;
      }
#undef LAUNCH_HOLD
#undef LAUNCH_HOLD_AS
    }
  }
  const int shards = S > 0 ? int((n + S - 1) / S) : 1;
  PushTargets hdr_dst = dst;
  hdr_dst.done = nullptr;  // only the quantising kernel publishes
  {
    const int64_t per = S > 0 ? (S < n ? S : n) : n;
    int gx = grid_for((per + 3) >> 2, kThreads, 148 * 4);
    if (shards > 1) gx = std::min(gx, std::max(1, (148 * 4 + shards - 1) / shards));
    const dim3 grid(gx, shards);
    auto minmax = vec ? (ef ? minmax_header_kernel<true, true> : minmax_header_kernel<true, false>)
                      : (ef ? minmax_header_kernel<false, true> : minmax_header_kernel<false, false>);
    const cudaError_t e = launch_with(overlap, 1, minmax, grid, dim3(kThreads), 0, stream, grad, residual, n, bitwidth, hdr_dst, s);
    if (e != cudaSuccess) return e;
  }
  {
    // chunked path with 16-byte stores once there is a chunk per warp of a half-filled GPU
    const int dpb = 8 / bitwidth;
    const int64_t chunks = n / (int64_t(kStageBytes) * dpb);
    const bool wide = vec && shift >= 0 && (S > 0 || chunks >= 148 * 2);
    const int threads = wide ? 128 : kThreads;
    const int grid = wide ? grid_for(chunks * 32, threads, 148 * 16)
                          : grid_for(n / (dpb > 4 ? dpb : 4), kThreads, 148 * 8);
    cudaError_t e = cudaSuccess;
#define LAUNCH_QUANT(BW, V, E)                                                                                   \
  e = launch_after(tern_quant_kernel<BW, V, E>, dim3(grid), dim3(threads), 0, stream, grad, residual, n,         \
                   enable_random, seed, dst, s, wide ? shift : -1)
    LAUNCH_BITS(LAUNCH_QUANT);
#undef LAUNCH_QUANT
    if (e != cudaSuccess) return e;
  }
#undef LAUNCH_BITS
#undef LAUNCH_FORMS
  return cudaGetLastError();
}

cudaError_t terngrad_unpack_accum(const UnpackSources& src, float* out, int64_t n, int add,
                                  float post_scale, const SgdApply& apply, int* status,
                                  cudaStream_t stream, int bitwidth_hint, bool overlap) {
  if (n <= 0 || src.world < 1 || src.world > kMaxWorld) return cudaErrorInvalidValue;
  if (bitwidth_hint != 0 && !tern_bitwidth_ok(bitwidth_hint)) return cudaErrorInvalidValue;
  if (src.shard_elems > 0) {
    // concatenated shards: 2-bit payloads and 16-byte aligned dense arrays only
    bool ok = bitwidth_hint == 2 && src.shard_elems % 2048 == 0 && aligned16(out) &&
              (n + src.shard_elems - 1) / src.shard_elems <= src.world;
    if (apply.param != nullptr) ok = ok && aligned16(apply.param) && aligned16(apply.momentum);
    if (!ok) return cudaErrorInvalidValue;
  }
  const bool ap = apply.param != nullptr;
#define HP_UNPACK(BW) \
  (ap ? launch_tern_unpack<BW, true>(src, out, n, add, post_scale, apply, status, stream, overlap) \
      : launch_tern_unpack<BW, false>(src, out, n, add, post_scale, apply, status, stream, overlap))
  switch (bitwidth_hint) {
    case 1: return HP_UNPACK(1);
    case 2: return HP_UNPACK(2);
    case 4: return HP_UNPACK(4);
    case 8: return HP_UNPACK(8);
    default: return HP_UNPACK(0);
  }
#undef HP_UNPACK
}

}  // namespace cuda
}  // namespace hipress
