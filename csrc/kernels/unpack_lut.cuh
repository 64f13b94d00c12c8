// One-pass decode + accumulate of up to 8 packed payloads through shared-memory tables.
//
// A payload byte holds DPB = 8/bitwidth quantised elements.  Instead of extracting and
// dequantising every field with integer and floating-point instructions (which made the first
// version of these kernels issue-bound at ~136 instructions per element for 8 ranks), each CTA
// first builds decode tables with the same contraction-free arithmetic as the CPU codec, and
// the main loop needs one 32-bit payload load per 4 bytes and rank plus table reads and adds.
//
// The decoded values of the ranks are summed in the canonical pairwise order (tree_sum in
// codec_math.h), so the result is bit-identical to the CPU codec on every replica.  Three table
// forms, fastest first:
//   index tables    bitwidths 1, 2, 4 and 16-byte aligned dense arrays: the fields of 8, 4 or 2 ranks
//                   make up one index, whose entry already holds those ranks' sum
//   nibble tables   bitwidths 1, 2, 4 at any alignment
//   byte tables     bitwidth 8 at any alignment, or unknown
// At 8 bits and with aligned dense arrays the levels are decoded arithmetically.
#pragma once
#include "../common/codec_math.h"
#include "kernels.h"
#include "p2p.cuh"

namespace hipress {
namespace cuda {

constexpr int kUnpackThreads = 256;

__device__ __forceinline__ uint32_t load_u32_any(const uint8_t* p) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  if ((a & 3) == 0) return *reinterpret_cast<const uint32_t*>(p);
  if ((a & 1) == 0)
    return uint32_t(reinterpret_cast<const uint16_t*>(p)[0]) | (uint32_t(reinterpret_cast<const uint16_t*>(p)[1]) << 16);
  return uint32_t(p[0]) | (uint32_t(p[1]) << 8) | (uint32_t(p[2]) << 16) | (uint32_t(p[3]) << 24);
}

__device__ __forceinline__ void sgd_update4(const SgdApply& a, int64_t i, const float* g) {
  const float4 p4 = *reinterpret_cast<const float4*>(a.param + i);
  float4 b4 = a.first_step ? make_float4(0, 0, 0, 0) : *reinterpret_cast<const float4*>(a.momentum + i);
  float p[4] = {p4.x, p4.y, p4.z, p4.w};
  float b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float d = g[k] + a.weight_decay * p[k];
    b[k] = a.first_step ? d : a.mu * b[k] + d;
    p[k] -= a.lr * b[k];
  }
  *reinterpret_cast<float4*>(a.momentum + i) = make_float4(b[0], b[1], b[2], b[3]);
  *reinterpret_cast<float4*>(a.param + i) = make_float4(p[0], p[1], p[2], p[3]);
}

// True when an earlier kernel of the step recorded a failure: the caller returns without writing.
__device__ __forceinline__ bool unpack_guarded(const UnpackSources& src) {
  return src.guard != nullptr && *reinterpret_cast<const volatile int*>(src.guard) != 0;
}

// payload[j] for a run-time j without indexing the kernel-parameter array dynamically (which
// would move the whole struct into local memory): a chain of selects over compile-time indices.
__device__ __forceinline__ const uint8_t* select_payload(const UnpackSources& src, int j) {
  const uint8_t* p = src.payload[0];
#pragma unroll
  for (int r = 1; r < kMaxWorld; ++r)
    if (r == j) p = src.payload[r];
  return p;
}
__device__ __forceinline__ int64_t select_payload_bytes(const UnpackSources& src, int j) {
  int64_t b = src.payload_bytes[0];
#pragma unroll
  for (int r = 1; r < kMaxWorld; ++r)
    if (r == j) b = src.payload_bytes[r];
  return b;
}

// Elements of shard j when a tensor of n elements is cut into shards of S.
__device__ __forceinline__ int64_t shard_count(int64_t n, int64_t S, int j) {
  const int64_t left = n - int64_t(j) * S;
  return left <= 0 ? 0 : (left < S ? left : S);
}

// Finish one group of 4 consecutive elements: accumulate mode, scale, store, fused update.
// The group lives at o[off .. off+3]; e is its index in the tensor (for the fused update).
template <bool APPLY>
__device__ __forceinline__ void unpack_finish4(float (&acc)[4], float* __restrict__ o, int off, int add,
                                               float post_scale, const SgdApply& apply, int64_t e) {
  if (add) {
    const float4 x = *reinterpret_cast<const float4*>(o + off);
    acc[0] = hp_add(acc[0], x.x); acc[1] = hp_add(acc[1], x.y);
    acc[2] = hp_add(acc[2], x.z); acc[3] = hp_add(acc[3], x.w);
  }
  if (post_scale != 1.0f) {
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[k] = hp_mul(acc[k], post_scale);
  }
  const bool clear = APPLY && apply.clear_grad;
  *reinterpret_cast<float4*>(o + off) =
      clear ? make_float4(0.f, 0.f, 0.f, 0.f) : make_float4(acc[0], acc[1], acc[2], acc[3]);
  if (APPLY) sgd_update4(apply, e, acc);
}
template <bool APPLY>
__device__ __forceinline__ void unpack_finish4(float (&acc)[4], float* __restrict__ out, int64_t e, int add,
                                               float post_scale, const SgdApply& apply) {
  unpack_finish4<APPLY>(acc, out + e, 0, add, post_scale, apply, e);
}
template <bool APPLY>
__device__ __forceinline__ void unpack_finish1(float acc, float* __restrict__ out, int64_t e, int add,
                                               float post_scale, const SgdApply& apply) {
  if (add) acc = hp_add(acc, out[e]);
  if (post_scale != 1.0f) acc = hp_mul(acc, post_scale);
  out[e] = (APPLY && apply.clear_grad) ? 0.f : acc;
  if (APPLY) sgd_update(apply, e, acc);
}

// Table row of byte value v.  Gradient payloads are dominated by a few byte values (fields
// near the middle levels); with rows stored in natural order those values fall on only four
// of the eight 16-byte bank groups and every table read is a multi-way bank conflict.  XOR-ing
// two higher bits into the low bits spreads them over all eight groups (a bijection on 0..255).
__device__ __forceinline__ uint32_t lut_row(uint32_t v) { return v ^ ((v >> 3) & 5u); }

// ---------------------------------------------------------------- byte tables
// lut: shared memory, entry (rank r, byte v, slot j) at lut[(r*256 + lut_row(v))*DPB + j].
// data_offset: bytes to skip at the start of each payload (header size + slot shift).
template <int DPB, bool APPLY>
__device__ __forceinline__ void unpack_lut_body(const float* lut, const UnpackSources& src, int64_t data_offset,
                                                float* __restrict__ out, int64_t n, int add,
                                                float post_scale, const SgdApply& apply) {
  constexpr int EPG = 4 * DPB;  // elements per group of 4 payload bytes
  constexpr int VW = DPB >= 4 ? 4 : DPB;  // values fetched per table read
  const int64_t full_groups = n / EPG;
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  const bool vec = ((reinterpret_cast<uintptr_t>(out) |
                     (APPLY ? (reinterpret_cast<uintptr_t>(apply.param) |
                               reinterpret_cast<uintptr_t>(apply.momentum)) : uintptr_t(0))) & 15) == 0;
  int64_t grp = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  // payload words of the group being decoded; the next group's words are requested before
  // the current ones are used, so their latency hides behind the decode
  uint32_t w[kMaxWorld];
#pragma unroll
  for (int r = 0; r < kMaxWorld; ++r)
    w[r] = (r < src.world && grp < full_groups) ? load_u32_any(src.payload[r] + data_offset + grp * 4) : 0u;
  for (; grp < full_groups; grp += stride) {
    const int64_t e0 = grp * EPG;
    const int64_t nxt = grp + stride;
    uint32_t wn[kMaxWorld];
#pragma unroll
    for (int r = 0; r < kMaxWorld; ++r)
      wn[r] = (r < src.world && nxt < full_groups) ? load_u32_any(src.payload[r] + data_offset + nxt * 4) : 0u;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
#pragma unroll
      for (int q = 0; q < DPB / VW; ++q) {
        float v[VW][kMaxWorld];
#pragma unroll
        for (int r = 0; r < kMaxWorld; ++r) {
          if (r < src.world) {
            const float* e = lut + (size_t(r) * 256 + lut_row((w[r] >> (8 * b)) & 255u)) * DPB + q * VW;
            if (VW == 4) {
              const float4 t = *reinterpret_cast<const float4*>(e);
              v[0][r] = t.x; v[1][r] = t.y; v[2][r] = t.z; v[3][r] = t.w;
            } else if (VW == 2) {
              const float2 t = *reinterpret_cast<const float2*>(e);
              v[0][r] = t.x; v[1][r] = t.y;
            } else {
              v[0][r] = e[0];
            }
          }
        }
        float acc[VW];
#pragma unroll
        for (int k = 0; k < VW; ++k) acc[k] = tree_sum(v[k], src.world);
        const int64_t e = e0 + b * DPB + q * VW;
        if (VW == 4 && vec) {
          if constexpr (VW == 4) unpack_finish4<APPLY>(acc, out, e, add, post_scale, apply);
        } else {
#pragma unroll
          for (int k = 0; k < VW; ++k) unpack_finish1<APPLY>(acc[k], out, e + k, add, post_scale, apply);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kMaxWorld; ++r) w[r] = wn[r];
  }
  // fewer than EPG leftover elements: one thread, element by element
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    for (int64_t e = full_groups * EPG; e < n; ++e) {
      float v[kMaxWorld];
#pragma unroll
      for (int r = 0; r < kMaxWorld; ++r) {
        if (r < src.world) {
          const uint32_t byte = src.payload[r][data_offset + e / DPB];
          v[r] = lut[(size_t(r) * 256 + lut_row(byte)) * DPB + int(e % DPB)];
        }
      }
      unpack_finish1<APPLY>(tree_sum(v, src.world), out, e, add, post_scale, apply);
    }
  }
}

// ---------------------------------------------------------------- nibble tables
// The byte table above costs one 16-byte shared-memory read per payload byte, and because a
// rank's table spans 4 KB, rows of different bytes collide on banks (measured: 2.2 wavefronts
// per quarter-warp read for 2-bit gradient payloads).  For bitwidths 1, 2 and 4 the table can
// instead be indexed by a 4-bit nibble: 16 rows of 4/BW floats.  At 2 bits a rank's table is
// exactly 128 bytes -- one row of all 32 banks -- so any two lanes either read the same row
// (a broadcast) or different banks: the reads are conflict free whatever the data.
//
// lut: entry (rank r, nibble v, slot j) at lut[(r*16 + v)*DPN + j], DPN = 4/BW (r = 0 when shared).
//
// The first payload words of a thread are requested by unpack_nibble_prefetch *before* the
// kernel reads headers and builds its tables, so that the DRAM latency of the first loads and
// the dependent loads of the prologue overlap instead of adding up.  A word is only requested
// when it lies inside the slot (payload_bytes), whatever the header will turn out to say.
// header_bytes: bytes before the packed data inside a slot; slot_shift: where this step's slot
// starts relative to src.payload[r] (the epoch-parity offset; 0 unless the epoch lives on the device).
template <int BW>
__device__ __forceinline__ void unpack_nibble_prefetch(const UnpackSources& src, int header_bytes,
                                                       int64_t slot_shift, int64_t n,
                                                       uint32_t (&w)[kMaxWorld]) {
  constexpr int EPG = 8 * (4 / BW);
  const int64_t grp = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
#pragma unroll
  for (int r = 0; r < kMaxWorld; ++r)
    w[r] = (r < src.world && grp < n / EPG && header_bytes + (grp + 1) * 4 <= src.payload_bytes[r])
               ? load_u32_any(src.payload[r] + slot_shift + header_bytes + grp * 4)
               : 0u;
}

// SHARED: all ranks decode through one table (TBQ); otherwise rank r's table starts 16 rows
// after rank r-1's.  w: the words unpack_nibble_prefetch returned for this thread.
template <int BW, bool APPLY, bool SHARED>
__device__ __forceinline__ void unpack_nibble_body(const float* lut, uint32_t (&w)[kMaxWorld],
                                                   const UnpackSources& src, int64_t data_offset,
                                                   float* __restrict__ out, int64_t n, int add,
                                                   float post_scale, const SgdApply& apply) {
  static_assert(BW == 1 || BW == 2 || BW == 4, "nibble tables cover bitwidths 1, 2 and 4");
  constexpr int DPN = 4 / BW;                                  // elements per nibble
  constexpr int EPG = 8 * DPN;                                 // elements per 32-bit payload word
  constexpr int ROW_SHIFT = DPN == 4 ? 4 : (DPN == 2 ? 3 : 2);  // log2(bytes per table row)
  constexpr int rank_stride = SHARED ? 0 : 16;
  const int64_t full_groups = n / EPG;
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  int64_t grp = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  for (; grp < full_groups; grp += stride) {
    const int64_t e0 = grp * EPG;
    const int64_t nxt = grp + stride;
    uint32_t wn[kMaxWorld];
#pragma unroll
    for (int r = 0; r < kMaxWorld; ++r)
      wn[r] = (r < src.world && nxt < full_groups) ? load_u32_any(src.payload[r] + data_offset + nxt * 4) : 0u;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      float v[DPN][kMaxWorld];
#pragma unroll
      for (int r = 0; r < kMaxWorld; ++r) {
        if (r < src.world) {
          const char* table = reinterpret_cast<const char*>(lut) + r * rank_stride * DPN * 4;
          // byte offset of the row of nibble k: ((w >> 4k) & 15) << ROW_SHIFT in one shift + mask
          const uint32_t off = (4 * k >= ROW_SHIFT ? (w[r] >> (4 * k - ROW_SHIFT)) : (w[r] << (ROW_SHIFT - 4 * k))) &
                               (15u << ROW_SHIFT);
          if (DPN == 4) {
            const float4 t = *reinterpret_cast<const float4*>(table + off);
            v[0][r] = t.x; v[1 % DPN][r] = t.y; v[2 % DPN][r] = t.z; v[3 % DPN][r] = t.w;
          } else if (DPN == 2) {
            const float2 t = *reinterpret_cast<const float2*>(table + off);
            v[0][r] = t.x; v[1 % DPN][r] = t.y;
          } else {
            v[0][r] = *reinterpret_cast<const float*>(table + off);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < DPN; ++j)
        unpack_finish1<APPLY>(tree_sum(v[j], src.world), out, e0 + k * DPN + j, add, post_scale, apply);
    }
#pragma unroll
    for (int r = 0; r < kMaxWorld; ++r) w[r] = wn[r];
  }
  // fewer than EPG leftover elements: one thread, element by element
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    constexpr int DPB = 8 / BW;
    for (int64_t e = full_groups * EPG; e < n; ++e) {
      const int in_byte = int(e % DPB);
      float v[kMaxWorld];
#pragma unroll
      for (int r = 0; r < kMaxWorld; ++r) {
        if (r < src.world) {
          const uint32_t byte = src.payload[r][data_offset + e / DPB];
          const uint32_t nib = (byte >> (4 * (in_byte / DPN))) & 15u;
          v[r] = lut[(size_t(r) * rank_stride + nib) * DPN + in_byte % DPN];
        }
      }
      unpack_finish1<APPLY>(tree_sum(v, src.world), out, e, add, post_scale, apply);
    }
  }
}

// ---------------------------------------------------------------- index tables: 1, 2 and 4 bits
// What bounds a decode of several payloads is not the dense store but the work per element and rank.
// Here one table read covers 8 / BW ranks of an element: the BW-bit fields of those ranks side by side
// are a byte, and row `byte` of the group's table holds their sum in the canonical order (the order
// adds neighbours first, so a group of 2, 4 or 8 ranks is a subtree of it).  Eight ranks at 2 bits are
// two reads and one add per element.  Every row is stored 32 times, once per bank: lane L reads its own
// column, so no read conflicts whatever the data is; the price is 32 KB per group, built once by each
// of the few resident CTAs.
//
// A lane loads 32 payload bits of each rank, turns the words of a group into one index byte per element
// (fields are exchanged between words, then bytes transposed), and writes those bytes to a buffer of
// its warp; the lanes read them back so that every dense access is a 512-byte run across the warp.
// The tables of two groups share rows of 256 bytes, 128 each: the address of an entry is then the index
// byte above the lane's column, which one byte permutation puts together.
// A table entry per pair of ranks and two elements, with bank conflicts and every index word moved by shuffle,
// is the alternative.  2 bits, eight payloads, 25 MB, in a chain of calls: 12.3 us; 17.2 with rows of 128 bytes, the
// fields moved one by one and the headers read one after another; (ncu, cold) 17.3 so, and 26.6 by pairs.
// Threads per CTA and CTAs per SM.  Eight payloads' tables and index buffers take 80 KB: two CTAs of 512
// threads that share them, because two of 256 leave four warps per scheduler, too few to cover the
// shared-memory latency (25 MB, compress and decode: 51.2 us against 43.0).  With one group of ranks three
// CTAs of 256 threads do.
__host__ __device__ constexpr int index_threads(int world) { return world > 4 ? 512 : 256; }
__host__ __device__ constexpr int index_ctas(int world) { return world > 4 ? 2 : 3; }

template <int BW>
struct IndexForm {
  static constexpr int kRanks = 8 / BW;        // ranks per group
  static constexpr int kElems = 32 / BW;       // elements per payload word = index bytes per lane and group
  static constexpr int kChunk = 32 * kElems;   // elements a warp decodes per iteration
  static constexpr int kDpb = 8 / BW;
};
// Sequential sums (the order of the ECQ codec: ascending ranks, one by one) read the first group's sum
// from its table and every later rank from a table of its own, all of them in the other half of its rows.
template <int BW, int WORLD, bool SHARED, bool SEQ>
struct IndexLayout {
  using F = IndexForm<BW>;
  static constexpr int kGroups = (WORLD + F::kRanks - 1) / F::kRanks;
  static constexpr int kFirst = WORLD < F::kRanks ? WORLD : F::kRanks;      // ranks of the first group
  static constexpr int kLast = WORLD - (kGroups - 1) * F::kRanks;            // ranks of the last one
  static constexpr int kFull = 1 << (BW * kFirst);                           // rows of a group but the last
  static constexpr int kTables = SHARED || SEQ ? 1 : kGroups;                // groups with a table of their own
  __host__ __device__ static constexpr int rows(int g) { return SHARED || g + 1 < kGroups ? kFull : 1 << (BW * kLast); }
  // bytes from row to row: the last of an odd number of groups has nothing to share its rows with
  __host__ __device__ static constexpr int stride(int g) { return kTables > 1 && g + 1 == kTables && g % 2 == 0 ? 128 : 256; }
  __host__ __device__ static constexpr int offset(int g) { return (g / 2) * kFull * 256 + (g % 2) * 128; }
  // SEQ: the tables of rank kFirst and on
  static constexpr int kSingles = SEQ ? (WORLD - kFirst) * (1 << BW) : 0;
  static_assert(kSingles <= kFull, "the other half of the rows holds them");
  __host__ __device__ static constexpr int single(int r) { return ((r - kFirst) << BW) * 256 + 128; }
  static constexpr int kTableBytes = offset(kTables - kTables % 2) + (kTables % 2) * rows(kTables - 1) * stride(kTables - 1);
  static constexpr int kStage = 32 * F::kElems * kGroups;                    // bytes per warp
  static constexpr size_t kBytes = size_t(kTableBytes) + size_t(index_threads(WORLD) / 32) * kStage;
};

// value(r, q): decoded value of level q of rank r.
template <int BW, int WORLD, bool SHARED, bool SEQ, typename Value>
__device__ __forceinline__ void build_index_tables(float* tables, Value value) {
  using L = IndexLayout<BW, WORLD, SHARED, SEQ>;
  constexpr int R = IndexForm<BW>::kRanks;
  constexpr uint32_t mask = (1u << BW) - 1u;
  // 32 copies; the lanes start at different columns, so that the stores spread over the banks
  auto put = [&](int at, float x) {
    float4* row = reinterpret_cast<float4*>(reinterpret_cast<char*>(tables) + at);
#pragma unroll
    for (int c = 0; c < 8; ++c) row[(c + threadIdx.x) & 7] = make_float4(x, x, x, x);
  };
#pragma unroll
  for (int g = 0; g < L::kTables; ++g) {
    const int ranks = WORLD - g * R < R ? WORLD - g * R : R;
    for (int i = threadIdx.x; i < L::rows(g); i += blockDim.x) {
      float v[R];
#pragma unroll
      for (int p = 0; p < R; ++p) v[p] = g * R + p < WORLD ? value(g * R + p, (uint32_t(i) >> (BW * p)) & mask) : 0.0f;
      if (SEQ) {
#pragma unroll
        for (int p = 1; p < R; ++p)
          if (p < ranks) v[0] = hp_add(v[0], v[p]);
      } else {
        tree_sum(v, ranks);
      }
      put(L::offset(g) + i * L::stride(g), v[0]);
    }
  }
  for (int i = threadIdx.x; i < L::kSingles; i += blockDim.x)
    put(L::single(L::kFirst) + i * 256, value(L::kFirst + (i >> BW), uint32_t(i) & mask));
}

// Index bytes of one group: u[] holds them in element order.  w: the payload words of the group's ranks.
template <int BW, int N>
__device__ __forceinline__ void index_bytes(const uint32_t (&w)[N], uint32_t (&u)[IndexForm<BW>::kElems / 4]) {
  constexpr int D = IndexForm<BW>::kDpb;
  uint32_t t[D];   // t[j], byte b: index of element b * D + j
  if constexpr (BW == 2 && N >= 3) {
    // the four words' fields as a 4 x 4 matrix in each byte, transposed in two steps of exchanges
    const uint32_t w3 = N == 4 ? w[N - 1] : 0u;
    const uint32_t a0 = (w[0] & 0x33333333u) | ((w[1] << 2) & 0xccccccccu), a1 = ((w[0] >> 2) & 0x33333333u) | (w[1] & 0xccccccccu);
    const uint32_t a2 = (w[2] & 0x33333333u) | ((w3 << 2) & 0xccccccccu), a3 = ((w[2] >> 2) & 0x33333333u) | (w3 & 0xccccccccu);
    t[0] = (a0 & 0x0f0f0f0fu) | ((a2 << 4) & 0xf0f0f0f0u);
    t[1] = (a1 & 0x0f0f0f0fu) | ((a3 << 4) & 0xf0f0f0f0u);
    t[2] = ((a0 >> 4) & 0x0f0f0f0fu) | (a2 & 0xf0f0f0f0u);
    t[3] = ((a1 >> 4) & 0x0f0f0f0fu) | (a3 & 0xf0f0f0f0u);
  } else {
    constexpr uint32_t field = BW == 4 ? 0x0f0f0f0fu : (BW == 2 ? 0x03030303u : 0x01010101u);
#pragma unroll
    for (int j = 0; j < D; ++j) {
      t[j] = 0;
#pragma unroll
      for (int p = 0; p < N; ++p) {
        const uint32_t moved = j >= p ? w[p] >> (BW * (j - p)) : w[p] << (BW * (p - j));
        t[j] |= moved & (field << (BW * p));
      }
    }
  }
  if constexpr (D == 2) {
    u[0] = __byte_perm(t[0], t[1], 0x5140);
    u[1] = __byte_perm(t[0], t[1], 0x7362);
  } else {
#pragma unroll
    for (int q = 0; q < D / 4; ++q) {
      const uint32_t a = __byte_perm(t[4 * q], t[4 * q + 1], 0x5140), b = __byte_perm(t[4 * q + 2], t[4 * q + 3], 0x5140);
      const uint32_t c = __byte_perm(t[4 * q], t[4 * q + 1], 0x7362), d = __byte_perm(t[4 * q + 2], t[4 * q + 3], 0x7362);
      u[0 * (D / 4) + q] = __byte_perm(a, b, 0x5410);
      u[1 * (D / 4) + q] = __byte_perm(a, b, 0x7632);
      u[2 * (D / 4) + q] = __byte_perm(c, d, 0x5410);
      u[3 * (D / 4) + q] = __byte_perm(c, d, 0x7632);
    }
  }
}

// Payload words in flight.  `align` says how every payload's packed data lies (payload_alignment): on
// 4-byte boundaries (the receive slots of the exchange), on 2-byte ones (behind a 10-byte header at the
// start of a tensor), or anyhow.  It is the same for the whole call, and the halves of a 2-byte aligned word
// are only put together where the word is used: a load that decides by its own address, and combines what
// it loaded, waits for memory once per rank instead of once for all.
template <int WORLD>
struct PayloadWords {
  uint32_t lo[WORLD], hi[WORLD];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int r = 0; r < WORLD; ++r) lo[r] = hi[r] = 0;
  }
  __device__ __forceinline__ void load(const UnpackSources& src, int64_t at, int align) {
    if (align == 4) {
#pragma unroll
      for (int r = 0; r < WORLD; ++r) {
        lo[r] = *reinterpret_cast<const uint32_t*>(src.payload[r] + at);
        hi[r] = 0;
      }
    } else if (align == 2) {
#pragma unroll
      for (int r = 0; r < WORLD; ++r) {
        const uint16_t* p = reinterpret_cast<const uint16_t*>(src.payload[r] + at);
        lo[r] = p[0];
        hi[r] = p[1];
      }
    } else {
#pragma unroll
      for (int r = 0; r < WORLD; ++r) {
        lo[r] = load_u32_any(src.payload[r] + at);
        hi[r] = 0;
      }
    }
  }
  __device__ __forceinline__ uint32_t word(int r) const { return lo[r] | (hi[r] << 16); }
};

// The first words of a thread, requested before the kernel reads headers and builds its tables.  A word
// is only requested when it lies inside the slot, whatever the header will turn out to say.
template <int BW, int WORLD>
__device__ __forceinline__ void index_prefetch(const UnpackSources& src, int header_bytes, int64_t n, int align,
                                               PayloadWords<WORLD>& w) {
  const int64_t warp = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t word = warp * 32 + (threadIdx.x & 31);
  bool ok = warp < n / IndexForm<BW>::kChunk;
#pragma unroll
  for (int r = 0; r < WORLD; ++r) ok = ok && header_bytes + (word + 1) * 4 <= src.payload_bytes[r];
  w.clear();
  if (ok) w.load(src, src.parity_off + header_bytes + word * 4, align);
}

// smem: tables, then the warps' index buffers.  pad: payload word of a rank that is not there in a
// SHARED table's last group (fields that decode to +0).
template <int BW, bool APPLY, int WORLD, bool SHARED, bool SEQ>
__device__ __forceinline__ void unpack_index_body(float* smem, PayloadWords<WORLD>& w, uint32_t pad, const UnpackSources& src,
                                                  int64_t data_offset, int align, float* __restrict__ out, int64_t n,
                                                  int add, float post_scale, const SgdApply& apply) {
  using F = IndexForm<BW>;
  using L = IndexLayout<BW, WORLD, SHARED, SEQ>;
  constexpr int R = F::kRanks, G = L::kGroups, V = F::kElems / 4;
  constexpr uint32_t mask = (1u << BW) - 1u;
  const int lane = threadIdx.x & 31;
  uint32_t* stage = reinterpret_cast<uint32_t*>(reinterpret_cast<char*>(smem) + L::kTableBytes) + (threadIdx.x >> 5) * (L::kStage / 4);
  const char* const table = reinterpret_cast<const char*>(smem);
  const uint32_t column = lane * 4;
  // four: per group, the index bytes of four elements; k: the element
  auto sum_of = [&](const uint32_t (&four)[G], int k) -> float {
    auto entry = [&](int g, int at) -> float {
      uint32_t off;
      if (L::stride(at) == 256) off = __byte_perm(four[g], column, 0x5504 | (k << 4));   // byte k, then the column
      else off = ((k == 0 ? four[g] << 7 : four[g] >> (8 * k - 7)) & 0x7f80u) | column;
      return *reinterpret_cast<const float*>(table + L::offset(at) + off);
    };
    if constexpr (SEQ) {
      float x = entry(0, 0);
#pragma unroll
      for (int r = L::kFirst; r < WORLD; ++r) {
        const int bit = 8 * k + BW * (r % R);   // of the rank's level, which goes to bit 8
        const uint32_t off = ((bit < 8 ? four[r / R] << (8 - bit) : four[r / R] >> (bit - 8)) & (mask << 8)) | column;
        x = hp_add(x, *reinterpret_cast<const float*>(table + L::single(r) + off));
      }
      return x;
    } else {
      float v[G];
#pragma unroll
      for (int g = 0; g < G; ++g) v[g] = entry(g, SHARED ? 0 : g);
      return tree_sum(v, G);
    }
  };
  const int64_t chunks = n / F::kChunk;
  const int64_t warps = int64_t(gridDim.x) * (blockDim.x >> 5);
  for (int64_t c = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); c < chunks; c += warps) {
#pragma unroll
    for (int g = 0; g < G; ++g) {
      uint32_t u[V];
      if (SHARED || g + 1 < G) {
        constexpr int N = SHARED && G > 1 ? R : L::kFirst;
        uint32_t x[N];
#pragma unroll
        for (int p = 0; p < N; ++p) x[p] = g * R + p < WORLD ? w.word((g * R + p) % WORLD) : pad;
        index_bytes<BW>(x, u);
      } else {
        uint32_t x[L::kLast];
#pragma unroll
        for (int p = 0; p < L::kLast; ++p) x[p] = w.word((g * R + p) % WORLD);
        index_bytes<BW>(x, u);
      }
      uint32_t* mine = stage + g * (8 * F::kElems) + lane * V;
      if constexpr (V == 2) {
        *reinterpret_cast<uint2*>(mine) = make_uint2(u[0], u[1]);
      } else {
#pragma unroll
        for (int q = 0; q < V / 4; ++q)
          reinterpret_cast<uint4*>(mine)[q] = make_uint4(u[4 * q], u[4 * q + 1], u[4 * q + 2], u[4 * q + 3]);
      }
    }
    if (c + warps < chunks) w.load(src, data_offset + ((c + warps) * 32 + lane) * 4, align);
    __syncwarp();
    float* const o = out + c * F::kChunk + lane * 4;
#pragma unroll
    for (int j = 0; j < V; ++j) {
      uint32_t four[G];
#pragma unroll
      for (int g = 0; g < G; ++g) four[g] = stage[g * (8 * F::kElems) + j * 32 + lane];
      float acc[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[k] = sum_of(four, k);
      unpack_finish4<APPLY>(acc, o, j * 128, add, post_scale, apply, c * F::kChunk + lane * 4 + j * 128);
    }
    __syncwarp();
  }
  // elements past the last complete chunk: block 0, element by element, through the same tables
  if (blockIdx.x == 0) {
    for (int64_t e = chunks * F::kChunk + threadIdx.x; e < n; e += blockDim.x) {
      const int sh = BW * int(e % F::kDpb);
      uint32_t byte[G];
#pragma unroll
      for (int g = 0; g < G; ++g) {
        byte[g] = 0;
#pragma unroll
        for (int p = 0; p < R; ++p) {
          const int r = g * R + p;
          uint32_t q = 0;
          if (r < WORLD) q = (uint32_t(src.payload[r % kMaxWorld][data_offset + e / F::kDpb]) >> sh) & mask;
          else if (SHARED && G > 1) q = pad & mask;
          byte[g] |= q << (BW * p);
        }
      }
      unpack_finish1<APPLY>(sum_of(byte, 0), out, e, add, post_scale, apply);
    }
  }
}

// ---------------------------------------------------------------- 8 bits
// A payload word is four elements: the lane that loads it stores them, and a level is decoded by its own
// two rounded operations (a table per rank would fill shared memory for no fewer instructions).
template <bool APPLY, int WORLD, bool SEQ, typename Value>
__device__ __forceinline__ void unpack_bytes_body(const UnpackSources& src, int64_t data_offset, int align,
                                                  float* __restrict__ out, int64_t n, int add, float post_scale,
                                                  const SgdApply& apply, Value value) {
  auto sum_of = [&](const uint32_t (&q)[WORLD]) -> float {
    float v[WORLD];
#pragma unroll
    for (int r = 0; r < WORLD; ++r) v[r] = value(r, q[r]);
    if constexpr (SEQ) {
#pragma unroll
      for (int r = 1; r < WORLD; ++r) v[0] = hp_add(v[0], v[r]);
      return v[0];
    } else {
      return tree_sum(v, WORLD);
    }
  };
  const int64_t words = n >> 2;
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  PayloadWords<WORLD> w;
  if (i < words) w.load(src, data_offset + i * 4, align);
  for (; i < words; i += stride) {
    uint32_t now[WORLD];
#pragma unroll
    for (int r = 0; r < WORLD; ++r) now[r] = w.word(r);
    if (i + stride < words) w.load(src, data_offset + (i + stride) * 4, align);
    float acc[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      uint32_t q[WORLD];
#pragma unroll
      for (int r = 0; r < WORLD; ++r) q[r] = (now[r] >> (8 * k)) & 255u;
      acc[k] = sum_of(q);
    }
    unpack_finish4<APPLY>(acc, out, i * 4, add, post_scale, apply);
  }
  if (blockIdx.x == 0 && threadIdx.x < (n & 3)) {
    const int64_t e = (words << 2) + threadIdx.x;
    uint32_t q[WORLD];
#pragma unroll
    for (int r = 0; r < WORLD; ++r) q[r] = src.payload[r][data_offset + e];
    unpack_finish1<APPLY>(sum_of(q), out, e, add, post_scale, apply);
  }
}

// 4, 2 or 1: the alignment of every payload's packed data (and, with slots double-buffered by parity, of the
// other slot's).
inline int payload_alignment(const UnpackSources& src, int header_bytes) {
  uintptr_t bits = uintptr_t(src.parity_stride);
  for (int r = 0; r < src.world; ++r) bits |= reinterpret_cast<uintptr_t>(src.payload[r] + header_bytes);
  return (bits & 3) == 0 ? 4 : ((bits & 1) == 0 ? 2 : 1);
}
// Resident CTAs of an index-table kernel: by shared memory and by registers (index_ctas).
inline int index_grid(int64_t n, int chunk, int world, size_t smem_bytes) {
  const int warps = index_threads(world) / 32;
  int64_t blocks = (n / chunk + warps - 1) / warps;
  int per_sm = int((size_t(227) * 1024) / (smem_bytes + 1024));
  per_sm = per_sm < 1 ? 1 : (per_sm > index_ctas(world) ? index_ctas(world) : per_sm);
  if (blocks > 148 * per_sm) blocks = 148 * per_sm;
  return blocks < 1 ? 1 : int(blocks);
}

// ---------------------------------------------------------------- concatenated shards, 2 bits
// Sharded exchange, last phase: payload[j] encodes shard j alone.  nib: [world or 1][16][2]
// nibble tables (rank j's at nib + j*32 floats; one table when SHARED).  Lane L decodes payload byte
// j*32 + L (j = 0..3) of the warp's 128-byte chunk; a 512-element chunk never straddles two shards
// (shard_elems % 2048 == 0).
// header_bytes + slot_shift: where the packed data starts inside payload[j].
template <bool APPLY, bool SHARED>
__device__ __forceinline__ void unpack_concat_body(const float* nib, const UnpackSources& src, int64_t data_offset,
                                                   float* __restrict__ out, int64_t n, int add,
                                                   float post_scale, const SgdApply& apply) {
  const int64_t S = src.shard_elems;
  const int64_t full_chunks = n / 512;
  const int lane = threadIdx.x & 31;
  const int64_t warps = int64_t(gridDim.x) * (blockDim.x >> 5);
  for (int64_t chunk = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); chunk < full_chunks;
       chunk += warps) {
    const int64_t e_chunk = chunk * 512;
    const int j = int(e_chunk / S);
    const uint8_t* p = select_payload(src, j) + data_offset + ((e_chunk - int64_t(j) * S) >> 2);
    const uint32_t word = *reinterpret_cast<const uint32_t*>(p + lane * 4);
    const char* table = reinterpret_cast<const char*>(nib) + (SHARED ? 0 : j * 128);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t wq = __shfl_sync(0xffffffffu, word, q * 8 + (lane >> 2));
      const uint32_t byte = (wq >> (8 * (lane & 3))) & 255u;
      const float2 lo = *reinterpret_cast<const float2*>(table + ((byte & 15u) << 3));
      const float2 hi = *reinterpret_cast<const float2*>(table + ((byte >> 4) << 3));
      float acc[4] = {lo.x, lo.y, hi.x, hi.y};
      unpack_finish4<APPLY>(acc, out, e_chunk + int64_t(q * 32 + lane) * 4, add, post_scale, apply);
    }
  }
  if (blockIdx.x == 0) {
    for (int64_t e = full_chunks * 512 + threadIdx.x; e < n; e += blockDim.x) {
      const int j = int(e / S);
      const int64_t le = e - int64_t(j) * S;
      const uint32_t byte = select_payload(src, j)[data_offset + (le >> 2)];
      const uint32_t nb = (byte >> (4 * ((le & 3) >> 1))) & 15u;
      unpack_finish1<APPLY>(nib[((SHARED ? 0 : j) * 16 + nb) * 2 + (le & 1)], out, e, add, post_scale, apply);
    }
  }
}

}  // namespace cuda
}  // namespace hipress
