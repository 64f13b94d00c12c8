// Sampled-threshold top-k sparsifier (GradDrop / DGC payloads) for sm_100a,
// with no host round-trip.
//
// The reference pipeline is transform(+) -> for_each(sample) -> sort -> D2H+sync
// -> copy_if (implicit sync) -> sort + truncate -> H2D+sync -> for_each(gather)
// (gd_body.h:121-229): four host synchronisations and two sorts.  Here:
//
//   sample      Draws the sample, stores every key (the order-preserving bits of |value|) and counts
//               the first of three digits (11 + 11 + 10 bits).
//   select      The k-th largest key of the sample: the CTAs pick the first digit's bin and collect the
//               few keys in it; the last CTA finds the threshold among those.
//   count       One pass: the codec's state update, the number of |R| > threshold, and a histogram of
//               those candidates above the threshold.
//   trim x2     Only when more than ceil(N*keep) candidates qualified (decided on the device; otherwise
//               the kernels return at once): the exact cut.  One pass over R; the second kernel only
//               has work when the cut lies more than a factor of two above the threshold.
//   write       Ordered compaction in one pass: indices ascending, values, residual zeroing, stored into every
//               destination (local and NVLink peers), then the completion flag.
//
// Content rule (identical to the CPU codec): keep |R[i]| > threshold in
// ascending index order; when over-selected keep the largest magnitudes, ties
// toward the lower index.
//
// Two forms of everything after the sampling.  The passes above ("scan form") read the whole
// tensor two or three times.  For small keep fractions (kListMaxKeep) the "list form" reads it ONCE:
//
//   count+collect  the one pass over the tensor.  It applies the codec's state update (R += G
//               for GradDrop; u = m*u + s*g, v += u and g = 0 for DGC with momentum correction;
//               nothing for plain DGC) and appends every candidate |value| > threshold, as
//               (index, value), to a per-warp list in index order.  A warp owns a contiguous
//               part of its CTA's chunk, so the lists, taken in order, are sorted by index.
//               Lists grow in blocks of 16 entries taken from a pool with one atomic.
//   cut         One CTA (eight for large selections): when more than ceil(N*keep) candidates qualified, the
//               exact cut, from counts that the collect pass has made of the candidates' magnitudes and
//               from the candidates themselves in the one bin that holds it.
//   emit        One warp per list: what each CTA's lists keep, where that starts (kept_before), then indices
//               and values to every destination, residual (and DGC's momentum u) cleared at the emitted
//               positions, and the completion flag.
//
// The kernels of a call overlap at their ends (launch.cuh): at 25 MB none but the pass over the tensor
// takes longer than the gap between two plain launches.
// Compress and decode, with the decode of that time, 64 MB, GradDrop at 0.1 %, four payloads: 112 us, and 129 as eight
// plain launches; 25 MB, DGC, eight payloads: 82 and 102.
//
// A sample of more than a hundredth of the elements does not fit the key array; its keys are then drawn
// again in each of three rounds, one per digit.  The pool is sized for many times the expected number of
// candidates (see list_plan); should it still run out, the candidates that did not fit stay in the residual
// and are sent in a later step (counted in SparseScratch::dropped).
#include "../common/codec_math.h"
#include "adamw.cuh"
#include "kernels.h"
#include "launch.cuh"
#include "p2p.cuh"
#include "unpack_lut.cuh"

#include <algorithm>
#include <cmath>

#include <cooperative_groups.h>

namespace hipress {
namespace cuda {

namespace {

namespace cg = cooperative_groups;

constexpr int kThreads = 256;
constexpr int kBins = 2048;
constexpr int kMaxBlocks = 148 * 4;
constexpr int kTile = kThreads * 4;  // elements per CTA iteration
constexpr int kMaxLists = kMaxBlocks * (kThreads / 32);
constexpr int kBlockEntries = 16;
constexpr unsigned int kNoBlock = 0xffffffffu;
// The list form serves keep fractions up to these, for tensors up to a size and larger ones.  Lists against scan,
// compress and decode: 1 M elements at 1 %, 55 us and 59; 6.5 M at 0.4 %, 68 and 82, at 1 %, 87 and 77; 33 M at 0.4 %, 248
// and 283, at 1 %, 360 and 274.  (The first has room for 1 % as one minus a drop ratio.)
constexpr double kListMaxKeepSmall = 0.0101, kListMaxKeep = 0.005;
constexpr int64_t kListSmall = int64_t(2) << 20;

constexpr int kFineBins = 512, kFineShift = 14;       // histogram above the threshold: one octave
constexpr int kExactBins = 1 << kFineShift;           // the keys of one of its bins
constexpr int kMaxSampleBlocks = kMaxBlocks;

struct SparseScratch {
  // Cleared by the first kernel of a call (clear_call_state).
  struct Call {
    unsigned int fine[kFineBins];      // candidates by (key - threshold) >> kFineShift; the last bin: all above
    unsigned int thist[3][kBins];      // digits of the candidates in that last bin; list form: [0], see far_bin
    unsigned int exact[kExactBins];    // keys inside the bin that holds the cut
    unsigned int ticket;               // write and emit kernels: chunks handed out
    unsigned int gave_up;              // a wait of theirs ran out (see kept_before)
    unsigned int trim_done[2];         // CTA arrivals of the trim kernels
    unsigned int t_prefix, t_rank;     // progress of the trim digits
    unsigned int clipped;              // the cut lies in the last fine bin
    unsigned int thr_key;              // threshold (key of a positive float)
    unsigned int cand;                 // candidates over the threshold
    unsigned int cut_key, ties_kept;   // final rule
    unsigned int pool_used;            // list form: blocks handed out
  } call;
  // Sampling: zero between calls.
  unsigned int shist[3][kBins];
  unsigned int s_prefix[3], s_rank[3];  // written by a round for the next
  unsigned int s_kept, s_done;
  unsigned int k;                       // elements emitted
  unsigned int dropped;                 // candidates that found no block (cumulative)
  unsigned int last_cand;               // candidates seen by the last call (metrics)
  unsigned int list_head[kMaxLists];    // first block of each warp's list, kNoBlock when empty
};

__device__ __forceinline__ void clear_call_state(SparseScratch* s) {
  static_assert(sizeof(SparseScratch::Call) % 4 == 0, "cleared word by word");
  unsigned int* w = reinterpret_cast<unsigned int*>(&s->call);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < int(sizeof(SparseScratch::Call) / 4); i += gridDim.x * blockDim.x)
    w[i] = 0u;
}

__device__ __forceinline__ int digit_of(uint32_t key, int round) {
  return round == 0 ? int(key >> 21) : round == 1 ? int((key >> 10) & 0x7ffu) : int(key & 0x3ffu);
}
__device__ __forceinline__ bool prefix_matches(uint32_t key, int round, uint32_t prefix) {
  return round == 0 ? true : round == 1 ? (key >> 21) == prefix : (key >> 10) == prefix;
}
__device__ __forceinline__ uint32_t extend_prefix(uint32_t prefix, int round, uint32_t digit) {
  return round == 0 ? digit : round == 1 ? (prefix << 11) | digit : (prefix << 10) | digit;
}

// Block-wide over kThreads threads: the bin holding the element of 0-indexed `rank` counted from the top
// bin down, and the rank inside that bin.  Every thread returns the same pair.  hist: BINS counters,
// 16-byte aligned, in shared or global memory.
template <int BINS>
__device__ __forceinline__ void pick_from_top(const unsigned int* hist, unsigned int rank, unsigned int& bin,
                                              unsigned int& rank_in_bin) {
  __shared__ unsigned int warp_sum[kThreads / 32];
  __shared__ unsigned int res[2];
  constexpr int PER = BINS / kThreads;
  static_assert(PER >= 4 ? PER % 4 == 0 : PER == 2, "a thread's bins are read in whole vectors");
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int base = BINS - (t + 1) * PER;   // this thread's bins, the highest last
  unsigned int sum = 0;
  if (PER >= 4) {
#pragma unroll 4
    for (int j = 0; j < PER / 4; ++j) {
      const uint4 v = *reinterpret_cast<const uint4*>(hist + base + 4 * j);
      sum += v.x + v.y + v.z + v.w;
    }
  } else {
    for (int j = 0; j < PER; ++j) sum += hist[base + j];
  }
  unsigned int inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned int a = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += a;
  }
  if (lane == 31) warp_sum[warp] = inc;
  if (t == 0) res[0] = res[1] = 0;
  __syncthreads();
  unsigned int before = inc - sum;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w)
    if (w < warp) before += warp_sum[w];
  if (rank >= before && rank - before < sum) {
    unsigned int run = before;
    for (int j = PER - 1; j >= 0; --j) {
      const unsigned int c = hist[base + j];
      if (rank - run < c) {
        res[0] = base + j;
        res[1] = rank - run;
        break;
      }
      run += c;
    }
  }
  __syncthreads();
  bin = res[0];
  rank_in_bin = res[1];
  __syncthreads();
}

// True in every thread of exactly one CTA: the last of the grid to get here; it sees what all others
// wrote before.  The counter is left at zero.
__device__ __forceinline__ bool last_cta(unsigned int* counter) {
  __shared__ bool is_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    is_last = atomicAdd(counter, 1u) == gridDim.x - 1;
    if (is_last) {
      *counter = 0u;
      __threadfence();
    }
  }
  __syncthreads();
  return is_last;
}

__device__ __forceinline__ void hist_flush(unsigned int* sh, unsigned int* gh) {
  __syncthreads();
  for (int i = threadIdx.x; i < kBins; i += kThreads) {
    const unsigned int v = sh[i];
    if (v) atomicAdd(gh + i, v);
  }
}

// Visit every element of [begin, end) once with f(value): 16-byte loads, four in flight per
// thread, scalar handling of an unaligned base or a ragged end.  `begin` is a multiple of the
// tile size, so the vector path applies whenever R itself is 16-byte aligned.
template <typename F>
__device__ __forceinline__ void for_each_value(const float* __restrict__ R, int64_t begin, int64_t end, F f) {
  if ((reinterpret_cast<uintptr_t>(R + begin) & 15) == 0) {
    const int64_t nvec = (end - begin) >> 2;
    const float4* v = reinterpret_cast<const float4*>(R + begin);
    int64_t i = threadIdx.x;
    for (; i + 3 * kThreads < nvec; i += 4 * kThreads) {
      const float4 a = v[i], b = v[i + kThreads], c = v[i + 2 * kThreads], d = v[i + 3 * kThreads];
      f(a.x); f(a.y); f(a.z); f(a.w);
      f(b.x); f(b.y); f(b.z); f(b.w);
      f(c.x); f(c.y); f(c.z); f(c.w);
      f(d.x); f(d.y); f(d.z); f(d.w);
    }
    for (; i < nvec; i += kThreads) {
      const float4 a = v[i];
      f(a.x); f(a.y); f(a.z); f(a.w);
    }
    for (int64_t j = begin + (nvec << 2) + threadIdx.x; j < end; j += kThreads) f(R[j]);
  } else {
    for (int64_t j = begin + threadIdx.x; j < end; j += kThreads) f(R[j]);
  }
}

// ---- the value the selection looks at, for one element, by mode
// mode 0: R as it is (plain DGC); mode 1: G + R (GradDrop's accumulation); mode 2: DGC with
// momentum correction, v + (m*u + s*g), rounded exactly as the collect pass rounds it.
struct SparseFuseDev {
  const float* grad;   // modes 1, 2
  float* u;            // mode 2: momentum
  float momentum;      // mode 2
  float clip;          // mode 2: > 0 = scale g by min(1, clip / |g|)
  const float* sumsq;  // mode 2 with clipping: |g|^2 of the bucket
  int zero_grad;       // mode 2: leave zeros in grad (the dense gradient is rebuilt from the payloads)
  int mode;
};
__device__ __forceinline__ float dgc_clip_scale(const SparseFuseDev& f) {
  if (f.mode != 2 || f.clip <= 0.f) return 1.0f;
  return fminf(1.0f, f.clip / (sqrtf(*f.sumsq) + 1e-6f));
}
__device__ __forceinline__ float dgc_new_u(float u, float g, float momentum, float scale) {
  return __fmaf_rn(momentum, u, __fmul_rn(scale, g));
}
__device__ __forceinline__ float fused_value(const SparseFuseDev& f, const float* R, uint32_t i, float scale) {
  if (f.mode == 0) return R[i];
  if (f.mode == 1) return hp_add(f.grad[i], R[i]);
  return __fadd_rn(R[i], dgc_new_u(f.u[i], f.grad[i], f.momentum, scale));
}

// ---- sampling
// Counts the digits of sampled keys: sampled magnitudes share their leading bits, so the lanes that hit
// the same bin are counted by one of them (one shared-memory atomic per bin and warp).  Whole warp;
// bin < 0: nothing to count.
__device__ __forceinline__ void count_digit(unsigned int* sh, int bin) {
  const unsigned int same = __match_any_sync(0xffffffffu, bin);
  if (bin >= 0 && int(threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&sh[bin], unsigned(__popc(same)));
}

// Round 0 stores every sample's key in `keys` when that is non-null (select_kernel goes on from there).
// Without the array each round draws the sample again and counts its own digit; the last CTA of round 2
// has the threshold.
template <int ROUND>
__global__ void __launch_bounds__(kThreads)
sample_round_kernel(SparseFuseDev fuse, const float* R, int64_t n,
                    int64_t sample_cnt, unsigned int rank0, uint64_t seed,
                    SparseScratch* s, uint32_t* keys, const uint32_t* epoch_dev) {
  wait_for_previous();
  let_next_start();
  if (ROUND == 0) clear_call_state(s);
  if (epoch_dev != nullptr) seed += uint64_t(*epoch_dev) * kEpochSeedStride;  // see PushTargets
  __shared__ __align__(16) unsigned int sh[kBins];
  for (int i = threadIdx.x; i < kBins; i += kThreads) sh[i] = 0;
  uint32_t prefix = 0;
  if (ROUND > 0) {
    const unsigned int rank = ROUND == 1 ? rank0 : s->s_rank[ROUND - 1];
    unsigned int bin, rin;
    pick_from_top<kBins>(s->shist[ROUND - 1], rank, bin, rin);
    prefix = extend_prefix(ROUND == 1 ? 0u : s->s_prefix[ROUND - 1], ROUND - 1, bin);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      // consumed by the next kernel in the stream
      s->s_prefix[ROUND] = prefix;
      s->s_rank[ROUND] = rin;
    }
  }
  __syncthreads();
  const float scale = dgc_clip_scale(fuse);
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  const int64_t padded = (sample_cnt + 31) & ~int64_t(31);   // whole warps iterate together
  for (int64_t x = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; x < padded; x += stride) {
    int bin = -1;
    if (x < sample_cnt) {
      const uint32_t idx = sparse_sample_index(seed, x, uint32_t(n));
      const uint32_t key = abs_key(fused_value(fuse, R, idx, scale));
      if (ROUND == 0 && keys != nullptr) keys[x] = key;
      if (prefix_matches(key, ROUND, prefix)) bin = digit_of(key, ROUND);
    }
    count_digit(sh, bin);
  }
  hist_flush(sh, s->shist[ROUND]);
  if (ROUND == 2) {
    if (!last_cta(&s->s_done)) return;
    unsigned int bin, rin;
    pick_from_top<kBins>(s->shist[2], s->s_rank[2], bin, rin);
    if (threadIdx.x == 0) s->call.thr_key = extend_prefix(s->s_prefix[2], 2, bin);
    for (int i = threadIdx.x; i < 3 * kBins; i += kThreads) (&s->shist[0][0])[i] = 0u;
  }
}

// The rest of the selection when the keys are stored: the keys in the first digit's bin (around the
// threshold of a 0.1 % selection, an eighth of an octave: hundreds of a 65,536-element sample) are
// collected in `kept`, and the last CTA finds the remaining digits among them.
__global__ void __launch_bounds__(kThreads)
select_kernel(int64_t sample_cnt, unsigned int rank0, SparseScratch* s, const uint32_t* keys, uint32_t* kept) {
  wait_for_previous();
  let_next_start();
  __shared__ __align__(16) unsigned int sh[kBins];
  unsigned int bin, rank;
  pick_from_top<kBins>(s->shist[0], rank0, bin, rank);
  uint32_t prefix = bin;
  __shared__ unsigned int mine[kThreads], held, place;
  const int64_t stride = int64_t(gridDim.x) * kThreads;
  for (int64_t x0 = int64_t(blockIdx.x) * kThreads; x0 < sample_cnt; x0 += stride) {
    const int64_t x = x0 + threadIdx.x;
    if (threadIdx.x == 0) held = 0;
    __syncthreads();
    const uint32_t key = x < sample_cnt ? keys[x] : 0u;
    if (x < sample_cnt && prefix_matches(key, 1, prefix)) mine[atomicAdd(&held, 1u)] = key;
    __syncthreads();
    if (threadIdx.x == 0 && held != 0) place = atomicAdd(&s->s_kept, held);   // one per CTA, not one per warp
    __syncthreads();
    if (threadIdx.x < held) kept[place + threadIdx.x] = mine[threadIdx.x];
    __syncthreads();   // the next step of a large sample resets `held`
  }
  if (!last_cta(&s->s_done)) return;
  const unsigned int count = *reinterpret_cast<volatile unsigned int*>(&s->s_kept);
#pragma unroll
  for (int round = 1; round < 3; ++round) {   // inside one bin of the first digit the rest spreads evenly
    for (int i = threadIdx.x; i < kBins; i += kThreads) sh[i] = 0;
    __syncthreads();
    for (unsigned int i = threadIdx.x; i < count; i += kThreads) {
      const uint32_t key = load_written(kept + i);
      if (prefix_matches(key, round, prefix)) atomicAdd(&sh[digit_of(key, round)], 1u);
    }
    __syncthreads();
    unsigned int rin;
    pick_from_top<kBins>(sh, rank, bin, rin);
    prefix = extend_prefix(prefix, round, bin);
    rank = rin;
  }
  if (threadIdx.x == 0) {
    s->call.thr_key = prefix;
    s->s_kept = 0u;
  }
  for (int i = threadIdx.x; i < kBins; i += kThreads) s->shist[0][i] = 0u;
}

constexpr int kWriteChunk = 4096;   // elements a CTA of write_kernel takes

// ---- scan form: the pass that updates the state, counts the candidates and files them by magnitude
// MODE = fuse.mode as a template parameter.  Candidates are filed by their distance from the threshold:
// the cut, when one is needed, lies a few per cent above the threshold, and its bin of this histogram
// holds few enough keys for the next kernel to count every key by itself.  What lies more than an octave
// above is filed by its first digit as well.
template <int MODE>
__global__ void __launch_bounds__(kThreads, 4)
count_kernel(SparseFuseDev fuse, float* R, int64_t n, int64_t chunk, SparseScratch* s, unsigned long long* state) {
  wait_for_previous();
  for (int64_t i = int64_t(blockIdx.x) * kThreads + threadIdx.x; i * kWriteChunk < n; i += int64_t(gridDim.x) * kThreads)
    state[i] = 0ull;   // of the write kernel
  constexpr int U = MODE == 2 ? 2 : 4;   // 16-byte loads of each array in flight per thread
  __shared__ unsigned int fine[kFineBins], coarse[kBins];
  __shared__ unsigned int blk_cnt;
  for (int i = threadIdx.x; i < kFineBins; i += kThreads) fine[i] = 0;
  for (int i = threadIdx.x; i < kBins; i += kThreads) coarse[i] = 0;
  if (threadIdx.x == 0) blk_cnt = 0;
  const uint32_t thr_key = s->call.thr_key;
  const float scale = MODE == 2 ? dgc_clip_scale(fuse) : 1.0f;
  __syncthreads();
  const int64_t begin = int64_t(blockIdx.x) * chunk;
  const int64_t end = begin + chunk < n ? begin + chunk : n;
  const float* grad = fuse.grad;
  float* gw = const_cast<float*>(fuse.grad);
  unsigned int mine = 0;
  auto file = [&](float r) {
    const uint32_t key = abs_key(r);
    if (key > thr_key) {
      ++mine;
      const uint32_t d = (key - thr_key) >> kFineShift;
      if (d < kFineBins - 1) {
        atomicAdd(&fine[d], 1u);
      } else {
        atomicAdd(&fine[kFineBins - 1], 1u);
        atomicAdd(&coarse[digit_of(key, 0)], 1u);
      }
    }
  };
  auto update = [&](float r, float g, float& u) -> float {
    if (MODE == 1) return hp_add(g, r);
    if (MODE == 2) {
      u = dgc_new_u(u, g, fuse.momentum, scale);
      return __fadd_rn(r, u);
    }
    return r;
  };
  uintptr_t bits = reinterpret_cast<uintptr_t>(R);
  if (MODE >= 1) bits |= reinterpret_cast<uintptr_t>(grad);
  if (MODE == 2) bits |= reinterpret_cast<uintptr_t>(fuse.u);
  int64_t rest = begin;
  if ((bits & 15) == 0 && (begin & 3) == 0) {
    const int64_t nv = (end - begin) >> 2;
    auto step = [&](int64_t e, float4 r4, float4 g4, float4 u4) {
      float r[4] = {r4.x, r4.y, r4.z, r4.w};
      const float g[4] = {g4.x, g4.y, g4.z, g4.w};
      float u[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) r[j] = update(r[j], g[j], u[j]);
      if (MODE >= 1) {
        *reinterpret_cast<float4*>(R + e) = make_float4(r[0], r[1], r[2], r[3]);
        if (MODE == 2) *reinterpret_cast<float4*>(fuse.u + e) = make_float4(u[0], u[1], u[2], u[3]);
        if (fuse.zero_grad) *reinterpret_cast<float4*>(gw + e) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) file(r[j]);
    };
    int64_t i = threadIdx.x;
    for (; i + (U - 1) * kThreads < nv; i += U * kThreads) {
      float4 r4[U], g4[U] = {}, u4[U] = {};
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const int64_t e = begin + 4 * (i + q * kThreads);
        r4[q] = *reinterpret_cast<const float4*>(R + e);
        if (MODE >= 1) g4[q] = *reinterpret_cast<const float4*>(grad + e);
        if (MODE == 2) u4[q] = *reinterpret_cast<const float4*>(fuse.u + e);
      }
#pragma unroll
      for (int q = 0; q < U; ++q) step(begin + 4 * (i + q * kThreads), r4[q], g4[q], u4[q]);
    }
    for (; i < nv; i += kThreads) {
      const int64_t e = begin + 4 * i;
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      step(e, *reinterpret_cast<const float4*>(R + e), MODE >= 1 ? *reinterpret_cast<const float4*>(grad + e) : zero,
           MODE == 2 ? *reinterpret_cast<const float4*>(fuse.u + e) : zero);
    }
    rest = begin + 4 * nv;
  }
  for (int64_t e = rest + threadIdx.x; e < end; e += kThreads) {
    float u = MODE == 2 ? fuse.u[e] : 0.f;
    const float r = update(R[e], MODE >= 1 ? grad[e] : 0.f, u);
    if (MODE >= 1) {
      R[e] = r;
      if (MODE == 2) fuse.u[e] = u;
      if (fuse.zero_grad) gw[e] = 0.f;
    }
    file(r);
  }
  let_next_start();
  for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
  if ((threadIdx.x & 31) == 0 && mine != 0) atomicAdd(&blk_cnt, mine);
  __syncthreads();
  for (int i = threadIdx.x; i < kFineBins; i += kThreads)
    if (fine[i]) atomicAdd(&s->call.fine[i], fine[i]);
  if (fine[kFineBins - 1]) hist_flush(coarse, s->call.thist[0]);
  if (threadIdx.x == 0) atomicAdd(&s->call.cand, blk_cnt);
}

// ---- where a chunk's entries start in the payload
// What each chunk keeps (elements above and at the cut) is published as soon as its CTA knows it, and what all
// chunks up to it keep once the CTA has added that up: a warp looks at the 32 chunks before, then at the 32 before
// those, until one has its sum.  (256 or 768 at a time are fewer steps, but what all CTAs poll slows the publishing:
// the write kernel's 18.1 us at 25 MB and 6.25 % are 20.2 and 22.6 so.)  Chunks are handed out by a ticket, so the ones waited for belong to
// CTAs that already run, and each publishes before it waits: the wait ends.  It is bounded all the same; a CTA
// whose wait runs out gets false, and must deliver and clear nothing.
// state: a word per chunk, zero before; the one word is the whole message.  Whole CTA of kThreads; every thread
// passes the chunk's own counts and gets those before it.
constexpr unsigned long long kCountReady = 1ull << 62, kSumReady = 2ull << 62, kReadyMask = 3ull << 62;
__device__ __forceinline__ unsigned long long pack_counts(unsigned int gt, unsigned int eq) {
  return (static_cast<unsigned long long>(gt) << 31) | eq;   // both below 2^31
}
__device__ __forceinline__ bool kept_before(unsigned long long* state, int block, unsigned int& gt, unsigned int& eq) {
  __shared__ unsigned int sum_gt, sum_eq;
  __shared__ bool in_time;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    if (lane == 0) atomicExch(&state[block], (block == 0 ? kSumReady : kCountReady) | pack_counts(gt, eq));
    unsigned int before_gt = 0, before_eq = 0;
    bool late = false;
    const uint64_t t0 = globaltimer_ns();
    for (int end = block; end > 0;) {   // lane L looks at chunk end - 1 - L
      const int b = end - 1 - lane;
      const unsigned long long w = b >= 0 ? *reinterpret_cast<volatile unsigned long long*>(&state[b]) : 0ull + kSumReady;
      const unsigned int sums = __ballot_sync(0xffffffffu, (w & kReadyMask) == kSumReady);
      const unsigned int missing = __ballot_sync(0xffffffffu, (w & kReadyMask) == 0ull);
      const unsigned int upto = sums == 0 ? 0xffffffffu : (2u << (__ffs(sums) - 1)) - 1u;   // lanes that count
      if ((missing & upto) != 0) {
        late = __any_sync(0xffffffffu, globaltimer_ns() - t0 > kGridWaitNs);   // the lanes need not agree on the time
        if (late) break;
        continue;
      }
      const bool counts = ((upto >> lane) & 1u) != 0;
      before_gt += __reduce_add_sync(0xffffffffu, counts ? unsigned((w & ~kReadyMask) >> 31) : 0u);
      before_eq += __reduce_add_sync(0xffffffffu, counts ? unsigned(w & 0x7fffffffull) : 0u);
      if (sums != 0) break;
      end -= 32;
    }
    if (lane == 0) {
      if (block != 0 && !late) atomicExch(&state[block], kSumReady | pack_counts(before_gt + gt, before_eq + eq));
      sum_gt = before_gt;
      sum_eq = before_eq;
      in_time = !late;
    }
  }
  __syncthreads();
  gt = sum_gt;
  eq = sum_eq;
  return in_time;
}

// ---- the exact cut (returns at once when not over-selected)
// ROUND 0: the keys in the cut's bin of the fine histogram, counted one by one; the last CTA has the cut.
// Should the cut lie in the histogram's last bin, this round counts the second digit of the keys there,
// and ROUND 1, which otherwise has nothing to do, the third.
template <int ROUND>
__global__ void __launch_bounds__(kThreads)
trim_kernel(const float* R, int64_t n, int64_t chunk, unsigned int expected, SparseScratch* s) {
  wait_for_previous();
  let_next_start();
  SparseScratch::Call& c = s->call;
  const uint32_t thr_key = c.thr_key;
  if (c.cand <= expected) {
    if (ROUND == 0 && blockIdx.x == 0 && threadIdx.x == 0) c.cut_key = thr_key;   // ties_kept stays 0
    return;
  }
  __shared__ __align__(16) unsigned int sh[kBins];
  const int64_t begin = int64_t(blockIdx.x) * chunk;
  const int64_t end = begin + chunk < n ? begin + chunk : n;
  unsigned int bin, rin;
  if (ROUND == 0) {
    pick_from_top<kFineBins>(c.fine, expected - 1, bin, rin);
    if (bin < kFineBins - 1) {
      const uint32_t base = thr_key + (bin << kFineShift);   // keys of the bin: base .. base + 2^14 - 1
      for_each_value(R, begin, end, [&](float x) {
        const uint32_t key = abs_key(x);
        if (key > thr_key && key - base < kExactBins) {
          // equal keys of a warp are counted by one lane: a tensor may hold one magnitude many times
          const unsigned int active = __activemask();
          const unsigned int same = __match_any_sync(active, key);
          if (int(threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&c.exact[key - base], unsigned(__popc(same)));
        }
      });
      if (!last_cta(&c.trim_done[0])) return;
      pick_from_top<kExactBins>(c.exact, rin, bin, rin);
      if (threadIdx.x == 0) {
        c.cut_key = base + bin;
        c.ties_kept = rin + 1;
      }
      return;
    }
  } else if (c.clipped == 0) {
    return;
  }
  const unsigned int rank = ROUND == 0 ? expected - 1 : c.t_rank;
  pick_from_top<kBins>(c.thist[ROUND], rank, bin, rin);
  const uint32_t prefix = extend_prefix(ROUND == 0 ? 0u : c.t_prefix, ROUND, bin);
  for (int i = threadIdx.x; i < kBins; i += kThreads) sh[i] = 0;
  __syncthreads();
  for_each_value(R, begin, end, [&](float x) {
    const uint32_t key = abs_key(x);
    if (key > thr_key && ((key - thr_key) >> kFineShift) >= kFineBins - 1 && prefix_matches(key, ROUND + 1, prefix))
      atomicAdd(&sh[digit_of(key, ROUND + 1)], 1u);
  });
  hist_flush(sh, c.thist[ROUND + 1]);
  if (!last_cta(&c.trim_done[ROUND])) return;
  if (ROUND == 0) {
    if (threadIdx.x == 0) {
      c.clipped = 1u;
      c.t_prefix = prefix;
      c.t_rank = rin;
    }
  } else {
    unsigned int low, in_low;
    pick_from_top<kBins>(c.thist[2], rin, low, in_low);
    if (threadIdx.x == 0) {
      c.cut_key = extend_prefix(prefix, 2, low);
      c.ties_kept = in_low + 1;
    }
  }
}

// ---- ordered compaction and delivery
// Output order is index order; position of an element = (elements above the cut before it) +
// min(ties kept, elements equal to the cut before it).  A CTA takes a chunk of 4,096 elements, counts what it
// keeps, and gets its starting place from kept_before; a CTA whose wait there runs out records kGridWait, delivers
// nothing and clears nothing, and the payload's flag is not published.
// What bounds it is instructions, not memory: a test, a position and two clearing stores for each of the 16
// elements of a lane are a thousand of them a warp.  A lane therefore holds its elements' tests as the bits of a mask
// and their values in shared memory; one scan over the warp places all of them, and the few that are kept are
// listed there in order, so that the stores to the payload (which loop over the destinations) and the clearing
// ones are made by full warps.
// 25 MB, 6.25 % kept, in a chain of calls: 18.1 us; 28.4 with a position and stores of its own for each element,
// chunks too large for the registers, which are walked twice, and starting places added up over all chunks.
__global__ void __launch_bounds__(kThreads)
write_kernel(float* R, float* u_mask, float* sumsq_to_clear, int64_t n, unsigned int expected, PushTargets dst, SparseScratch* s,
             unsigned long long* state, int* status) {
  wait_for_previous();
  resolve_epoch(dst);
  constexpr int kWarps = kThreads / 32;
  constexpr int kSteps = 4;                        // 16-byte words of a lane: element j * 128 + lane * 4 + i of the warp
  constexpr int kWarpElems = kSteps * 128;
  static_assert(kWarps * kWarpElems == kWriteChunk, "one chunk per CTA");
  __shared__ unsigned int warp_gt[kWarps], warp_eq[kWarps];
  __shared__ __align__(16) float values[kWarps][kWarpElems];
  __shared__ uint16_t kept[kWarps][kWarpElems];    // places among the warp's elements
  __shared__ int ticket;
  if (threadIdx.x == 0) ticket = int(atomicAdd(&s->call.ticket, 1u));
  const uint32_t cut = s->call.cut_key;
  const unsigned int ties = s->call.ties_kept;
  const unsigned int cand = s->call.cand;
  const unsigned int k_total = cand < expected ? cand : expected;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  const int block = ticket;
  if (block == 0 && threadIdx.x == 0) {
    s->k = k_total;
    s->last_cand = cand;
    const uint32_t total = 4u + 8u * k_total;
    uint8_t header[4];
    for (int i = 0; i < 4; ++i) header[i] = uint8_t(total >> (8 * i));
    push_bytes(dst, 0, header, 4);
    if (sumsq_to_clear != nullptr) *sumsq_to_clear = 0.f;
  }
  const int64_t wbegin = int64_t(block) * kWriteChunk + warp * kWarpElems;   // the warp's elements, clipped at n
  float v[kSteps][4];
  if ((reinterpret_cast<uintptr_t>(R) & 15) == 0 && wbegin + kWarpElems <= n) {
#pragma unroll
    for (int j = 0; j < kSteps; ++j) {
      const float4 q = *reinterpret_cast<const float4*>(R + wbegin + j * 128 + lane * 4);
      v[j][0] = q.x; v[j][1] = q.y; v[j][2] = q.z; v[j][3] = q.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < kSteps; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int64_t e = wbegin + j * 128 + lane * 4 + i;
        v[j][i] = e < n ? R[e] : 0.0f;
      }
  }
  // Bit 4 * j + i: the element is above the cut, or at it.  A place past the end holds zero, whose key is above no cut;
  // it equals the cut only where the cut is zero, and then nothing at the cut is kept: a candidate is above a
  // threshold that is not negative.
  uint32_t above = 0, at_cut = 0;
#pragma unroll
  for (int j = 0; j < kSteps; ++j) {
    *reinterpret_cast<float4*>(&values[warp][j * 128 + lane * 4]) = make_float4(v[j][0], v[j][1], v[j][2], v[j][3]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      above |= abs_key(v[j][i]) > cut ? 1u << (4 * j + i) : 0u;
      at_cut |= abs_key(v[j][i]) == cut ? 1u << (4 * j + i) : 0u;
    }
  }
  const unsigned int my_gt = __reduce_add_sync(0xffffffffu, unsigned(__popc(above)));
  const unsigned int my_eq = __reduce_add_sync(0xffffffffu, unsigned(__popc(at_cut)));
  if (lane == 0) {
    warp_gt[warp] = my_gt;
    warp_eq[warp] = my_eq;
  }
  __syncthreads();
  unsigned int run_gt = 0, run_eq = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    run_gt += warp_gt[w];
    run_eq += warp_eq[w];
  }
  if (!kept_before(state, block, run_gt, run_eq)) {
    if (threadIdx.x == 0) {
      s->call.gave_up = 1u;
      if (status != nullptr) atomicExch(status, int(kGridWait));
    }
    publish_when_grid_done(dst, &s->call.gave_up);
    return;
  }
  for (int w = 0; w < warp; ++w) {
    run_gt += warp_gt[w];
    run_eq += warp_eq[w];
  }
  // Of a mask, per step: how many bits the steps and lanes before this lane's hold.  A byte per step (128 at most).
  auto bits_before = [&](uint32_t mask, unsigned int (&before)[kSteps]) {
    uint32_t mine = 0;
#pragma unroll
    for (int j = 0; j < kSteps; ++j) mine |= unsigned(__popc((mask >> (4 * j)) & 15u)) << (8 * j);
    uint32_t inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += x;
    }
    const uint32_t totals = __shfl_sync(0xffffffffu, inc, 31);
    unsigned int run = 0;
#pragma unroll
    for (int j = 0; j < kSteps; ++j) {
      before[j] = run + (((inc - mine) >> (8 * j)) & 255u);
      run += (totals >> (8 * j)) & 255u;
    }
    return run;
  };
  if (my_gt != 0 || (ties > run_eq && my_eq != 0)) {
    unsigned int run_kept = run_gt + (run_eq < ties ? run_eq : ties);
    uint32_t keep = above;
    unsigned int before[kSteps];
    if (my_eq != 0 && run_eq < ties) {   // ties are kept from the lower index on
      bits_before(at_cut, before);
#pragma unroll
      for (int j = 0; j < kSteps; ++j) {
        unsigned int rank = run_eq + before[j];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t bit = at_cut & (1u << (4 * j + i));
          if (bit != 0 && rank++ < ties) keep |= bit;
        }
      }
    }
    const unsigned int held = bits_before(keep, before);
#pragma unroll
    for (int j = 0; j < kSteps; ++j) {
      unsigned int at = before[j];
      for (uint32_t bits = (keep >> (4 * j)) & 15u; bits != 0; bits &= bits - 1)
        kept[warp][at++] = uint16_t(j * 128 + lane * 4 + __ffs(bits) - 1);
    }
    __syncwarp();
    for (unsigned int i = lane; i < held; i += 32) {
      const unsigned int pos = run_kept + i;
      if (pos < k_total) {
        const int place = kept[warp][i];
        const int64_t e = wbegin + place;
        push_u32(dst, 4 + 4 * int64_t(pos), uint32_t(e));
        push_u32(dst, 4 + 4 * int64_t(k_total) + 4 * int64_t(pos), __float_as_uint(values[warp][place]));
        R[e] = 0.0f;
        if (u_mask != nullptr) u_mask[e] = 0.0f;   // DGC's momentum factor masking
      }
    }
  }
  publish_when_grid_done(dst, &s->call.gave_up);
}

__global__ void __launch_bounds__(kThreads)
scatter_kernel(const uint8_t* __restrict__ payload, int64_t cap, float* __restrict__ out, int64_t n,
               float post_scale, int* status, const uint32_t* epoch_dev, int64_t parity_stride,
               const int* guard) {
  if (status_guarded(guard)) return;
  if (epoch_dev != nullptr && (*epoch_dev & 1u)) payload += parity_stride;  // see UnpackSources
  uint32_t total = 0;
  for (int k = 0; k < 4; ++k) total |= uint32_t(payload[k]) << (8 * k);
  if (total < 4 || int64_t(total) > cap) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && status) atomicExch(status, int(kPayloadBounds));
    return;
  }
  const int64_t k = (int64_t(total) - 4) / 8;
  const uint32_t* idx = reinterpret_cast<const uint32_t*>(payload + 4);
  const uint32_t* val = reinterpret_cast<const uint32_t*>(payload + 4 + 4 * k);
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  for (int64_t x = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; x < k; x += stride) {
    const uint32_t i = idx[x];
    if (int64_t(i) >= n) {
      if (status) atomicExch(status, int(kPayloadBounds));
      continue;
    }
    float v = __uint_as_float(val[x]);
    if (post_scale != 1.0f) v = hp_mul(v, post_scale);
    // indices are unique inside one payload: a plain read-modify-write is race free
    out[i] = hp_add(out[i], v);
  }
}

// ================================================================ list form
// Pool of list blocks, behind the sample keys in the scratch: block b holds count[b] (index,
// value bits) pairs in entry[b * 16 ..] and continues in block next[b].
struct ListPool {
  unsigned int* count;
  unsigned int* next;
  uint2* entry;
  uint32_t* dense;        // the candidates' keys once more, densely packed in no particular order
  unsigned int capacity;  // blocks
};

// Cursor of a warp's list; only lane 0's copy is used, but for the last two.
struct ListCursor {
  unsigned int block = kNoBlock, fill = 0, lost = 0, total = 0;
  bool exhausted = false;
  unsigned int seen = 0;   // candidates, the same in all lanes
  uint32_t key = 0;        // of candidate number `lane`
};
// Bin of a candidate by its distance from the threshold: 2,048 bins of 4,096 keys, one octave, the last bin
// for all above.
constexpr int kFar = 12;   // log2 of the keys per bin
__device__ __forceinline__ int far_bin(uint32_t key, uint32_t thr_key) {
  const uint32_t d = (key - thr_key) >> kFar;
  return int(d < kBins - 1 ? d : kBins - 1);
}

// Appends this step's candidates of the calling warp to the warp's list, in lane order and,
// within a lane, element order.  count: candidates of this lane (0..4); idx / val: their
// indices and values.  Candidates are rare (0.1 % of the elements), so the entries are handed
// to lane 0 by shuffle and appended one at a time; a list grows by one block of the pool when
// its last block is full.  Each is counted in the bin that the cut is looked for in.
__device__ __forceinline__ void list_append(SparseScratch* s, const ListPool& pool, int list, int lane, uint32_t thr_key,
                                            unsigned int count, const uint32_t (&idx)[4], const float (&val)[4],
                                            ListCursor& cur) {
  unsigned int mask = __ballot_sync(0xffffffffu, count != 0);
  while (mask != 0) {
    const int src = __ffs(mask) - 1;
    mask &= mask - 1;
    const unsigned int c = __shfl_sync(0xffffffffu, count, src);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t i = __shfl_sync(0xffffffffu, idx[j], src);
      const float v = __shfl_sync(0xffffffffu, val[j], src);
      if (j < int(c) && cur.seen++ == unsigned(lane)) cur.key = abs_key(v);
      if (lane != 0 || j >= int(c)) continue;
      if (cur.exhausted) {
        ++cur.lost;
        continue;
      }
      if (cur.block == kNoBlock || cur.fill == kBlockEntries) {
        const unsigned int id = atomicAdd(&s->call.pool_used, 1u);
        if (id >= pool.capacity) {
          cur.exhausted = true;
          ++cur.lost;
          continue;
        }
        pool.count[id] = 0;
        pool.next[id] = kNoBlock;
        if (cur.block == kNoBlock) s->list_head[list] = id;
        else pool.next[cur.block] = id;
        cur.block = id;
        cur.fill = 0;
      }
      pool.entry[size_t(cur.block) * kBlockEntries + cur.fill] = make_uint2(i, __float_as_uint(v));
      pool.count[cur.block] = ++cur.fill;
      atomicAdd(&s->call.thist[0][far_bin(abs_key(v), thr_key)], 1u);
      ++cur.total;
    }
  }
}

// ---- the one pass over the tensor
// MODE = fuse.mode as a template parameter (no registers for arrays a mode does not read); four
// CTAs per SM, so that the whole grid of 4 x 148 CTAs is resident at once.
template <int MODE>
__global__ void __launch_bounds__(kThreads, 4)
collect_kernel(SparseFuseDev fuse, float* R, int64_t n, int64_t chunk, SparseScratch* s, ListPool pool,
               unsigned long long* state) {
  wait_for_previous();
  if (threadIdx.x == 0) state[blockIdx.x] = 0ull;   // of the emit kernel
  fuse.mode = MODE;
  constexpr int kWarps = kThreads / 32;
  constexpr int U = MODE == 2 ? 2 : 4;   // steps whose loads are issued together
  const uint32_t thr_key = s->call.thr_key;
  const float scale = dgc_clip_scale(fuse);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int list = blockIdx.x * kWarps + warp;
  const int64_t begin = int64_t(blockIdx.x) * chunk;
  const int64_t end = begin + chunk < n ? begin + chunk : n;
  // warp ranges: multiples of 128 elements so that every step is 32 lanes x 4 elements
  int64_t wlen = (end - begin + kWarps - 1) / kWarps;
  wlen = (wlen + 127) / 128 * 128;
  const int64_t wbegin = begin + warp * wlen < end ? begin + warp * wlen : end;
  const int64_t wend = wbegin + wlen < end ? wbegin + wlen : end;
  uintptr_t bits = reinterpret_cast<uintptr_t>(R);
  if (MODE >= 1) bits |= reinterpret_cast<uintptr_t>(fuse.grad);
  if (MODE == 2) bits |= reinterpret_cast<uintptr_t>(fuse.u);
  const bool vec_ok = (bits & 15) == 0 && (begin & 3) == 0;
  float* gw = const_cast<float*>(fuse.grad);   // mode 2 leaves zeros behind

  ListCursor cur;
  if (lane == 0) s->list_head[list] = kNoBlock;

  // state update + candidate test of the 4 elements at e0 (e0 + 3 < wend, 16-byte aligned)
  auto step4 = [&](int64_t e0, float4 r4, float4 g4, float4 u4, uint32_t (&idx)[4], float (&val)[4]) -> unsigned int {
    float r[4] = {r4.x, r4.y, r4.z, r4.w};
    if (MODE == 1) {
      const float g[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) r[j] = hp_add(g[j], r[j]);
      *reinterpret_cast<float4*>(R + e0) = make_float4(r[0], r[1], r[2], r[3]);
      if (fuse.zero_grad) *reinterpret_cast<float4*>(gw + e0) = make_float4(0.f, 0.f, 0.f, 0.f);
    } else if (MODE == 2) {
      const float g[4] = {g4.x, g4.y, g4.z, g4.w};
      float u[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        u[j] = dgc_new_u(u[j], g[j], fuse.momentum, scale);
        r[j] = __fadd_rn(r[j], u[j]);
      }
      *reinterpret_cast<float4*>(fuse.u + e0) = make_float4(u[0], u[1], u[2], u[3]);
      *reinterpret_cast<float4*>(R + e0) = make_float4(r[0], r[1], r[2], r[3]);
      if (fuse.zero_grad) *reinterpret_cast<float4*>(gw + e0) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    unsigned int count = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (abs_key(r[j]) > thr_key) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {   // compile-time indices keep idx / val in registers
          if (c == int(count)) {
            idx[c] = uint32_t(e0 + j);
            val[c] = r[j];
          }
        }
        ++count;
      }
    }
    return count;
  };

  int64_t base = wbegin;
  if (vec_ok) {
    // U steps per iteration with their loads issued together
    for (; base + U * 128 <= wend; base += U * 128) {
      float4 r4[U], g4[MODE >= 1 ? U : 1] = {}, u4[MODE == 2 ? U : 1] = {};
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const int64_t e0 = base + q * 128 + lane * 4;
        r4[q] = *reinterpret_cast<const float4*>(R + e0);
        if (MODE >= 1) g4[MODE >= 1 ? q : 0] = *reinterpret_cast<const float4*>(fuse.grad + e0);
        if (MODE == 2) u4[MODE == 2 ? q : 0] = *reinterpret_cast<const float4*>(fuse.u + e0);
      }
#pragma unroll
      for (int q = 0; q < U; ++q) {
        uint32_t idx[4] = {0u, 0u, 0u, 0u};
        float val[4] = {0.f, 0.f, 0.f, 0.f};
        const unsigned int count = step4(base + q * 128 + lane * 4, r4[q], g4[MODE >= 1 ? q : 0], u4[MODE == 2 ? q : 0], idx, val);
        if (__ballot_sync(0xffffffffu, count != 0) != 0) list_append(s, pool, list, lane, thr_key, count, idx, val, cur);
      }
    }
  }
  // the rest of the warp's range, element by element within steps of 128
  for (; base < wend; base += 128) {
    uint32_t idx[4] = {0u, 0u, 0u, 0u};
    float val[4] = {0.f, 0.f, 0.f, 0.f};
    unsigned int count = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t e = base + lane * 4 + j;
      if (e < wend) {
        float r = R[e];
        if (MODE == 1) {
          r = hp_add(fuse.grad[e], r);
          R[e] = r;
          if (fuse.zero_grad) gw[e] = 0.f;
        } else if (MODE == 2) {
          const float u = dgc_new_u(fuse.u[e], fuse.grad[e], fuse.momentum, scale);
          r = __fadd_rn(r, u);
          fuse.u[e] = u;
          R[e] = r;
          if (fuse.zero_grad) gw[e] = 0.f;
        }
        if (abs_key(r) > thr_key) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (c == int(count)) {
              idx[c] = uint32_t(e);
              val[c] = r;
            }
          }
          ++count;
        }
      }
    }
    if (__ballot_sync(0xffffffffu, count != 0) != 0) list_append(s, pool, list, lane, thr_key, count, idx, val, cur);
  }
  let_next_start();
  // The cut kernel wants all candidate keys in one flat array (a sweep over the half-empty list blocks cost it
  // 70 us).  Each warp copies its own to a range that it reserves with one atomic: the lanes hold the first 32, and
  // the rest is read back from the list.
  if (lane == 0 && cur.lost != 0) atomicAdd(&s->dropped, cur.lost);
  const unsigned int total = __shfl_sync(0xffffffffu, cur.total, 0);
  if (total != 0) {
    unsigned int base = 0;
    if (lane == 0) base = atomicAdd(&s->call.cand, total);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (total <= 32u) {   // the first `total` candidates found room, any others none
      if (lane < int(total)) pool.dense[base + lane] = cur.key;
      return;
    }
    __syncwarp();   // lane 0's list writes are visible to the other lanes
    unsigned int done = 0;
    for (unsigned int b = s->list_head[list]; b != kNoBlock && b < pool.capacity; b = pool.next[b]) {
      const unsigned int c = pool.count[b];
      if (lane < int(c)) pool.dense[base + done + lane] = pool.entry[size_t(b) * kBlockEntries + lane].y & 0x7fffffffu;
      done += c;
    }
  }
}

// ---- the exact cut among the candidates
// The collect pass has counted the candidates by their distance from the threshold, in bins of 4,096 keys.  The
// bin that holds the cut follows from those counts, and one pass over the candidates counts the keys of that bin one
// by one: on ordinary data some hundred of 17,000.  The leading bits of the keys themselves are nearly all the same,
// which costs either colliding atomics or a match instruction per warp; their three digits are counted only
// when the cut lies in the last bin, more than an octave above the threshold.
// CTAS = 1, or a cluster of eight that share the candidates and count in the first CTA's memory.
// The kernel behind starts at once: its walk over the lists needs nothing from here.
// 17,000 candidates of 64 MB: 5 us behind the collect pass; 15 with all keys brought to shared memory, three rounds of counting, and a
// count of what each CTA's lists keep.
constexpr int kCutThreads = 1024;
constexpr int kCutCluster = 8;
constexpr int kCutBins = 1 << kFar;
constexpr int64_t kCutOneCta = 40 * 1024;   // selections up to this are one CTA's work

// Exclusive scan over kCutThreads values, one per thread; total: their sum.  ws: 33 words of shared memory.
__device__ __forceinline__ unsigned int exclusive_scan_1024(unsigned int v, unsigned int* ws, unsigned int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned int inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned int a = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += a;
  }
  __syncthreads();
  if (lane == 31) ws[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const unsigned int x = ws[lane];
    unsigned int sx = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned int a = __shfl_up_sync(0xffffffffu, sx, o);
      if (lane >= o) sx += a;
    }
    ws[lane] = sx - x;
    if (lane == 31) ws[32] = sx;
  }
  __syncthreads();
  total = ws[32];
  return ws[warp] + inc - v;
}

// The bin that holds the element of 0-indexed `rank` from the top, and the rank inside it.  c: this thread's PER
// bins, highest first; thread t has those from (1,024 - t) * PER - 1 down.  Whole CTA.
template <int PER>
__device__ __forceinline__ uint32_t cut_pick(const unsigned int (&c)[PER], unsigned int& rank, unsigned int* ws, unsigned int* res) {
  unsigned int mine = 0, unused;
#pragma unroll
  for (int j = 0; j < PER; ++j) mine += c[j];
  const unsigned int before = exclusive_scan_1024(mine, ws, unused);
  if (rank >= before && rank - before < mine) {
    unsigned int run = before;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      if (rank >= run && rank - run < c[j]) {
        res[0] = unsigned((kCutThreads - int(threadIdx.x)) * PER - 1 - j);
        res[1] = rank - run;
      }
      run += c[j];
    }
  }
  __syncthreads();
  const uint32_t bin = res[0];
  rank = res[1];
  __syncthreads();
  return bin;
}

template <int CTAS>
__global__ void __launch_bounds__(kCutThreads, 1)
cut_kernel(unsigned int expected, PushTargets dst, SparseScratch* s, ListPool pool, float* sumsq_to_clear) {
  wait_for_previous();
  let_next_start();   // behind the wait: what the collect pass wrote is complete
  resolve_epoch(dst);
  constexpr int kAhead = 8;             // keys of a thread in flight
  __shared__ unsigned int sh[kCutBins];
  __shared__ unsigned int ws[33], res[2];
  const int t = threadIdx.x;
  const int part = CTAS > 1 ? int(blockIdx.x) : 0;
  uint32_t key[kAhead];
  if (CTAS == 1) {   // the first ones, whether or not there are that many: the array is longer
#pragma unroll
    for (int u = 0; u < kAhead; ++u) key[u] = pool.dense[u * kCutThreads + t];
  }
  const uint2 top = *reinterpret_cast<const uint2*>(&s->call.thist[0][kBins - 2 - 2 * t]);
  const unsigned int cand = s->call.cand;
  const uint32_t thr = s->call.thr_key;
  const unsigned int share = (cand + CTAS - 1) / CTAS;
  const unsigned int first = share * part < cand ? share * part : cand;
  const unsigned int count = first + share < cand ? share : cand - first;
  for (int i = t; i < kCutBins; i += kCutThreads) sh[i] = 0;
  if (t == 0) res[0] = res[1] = 0;
  uint32_t cut = thr;
  unsigned int ties = 0;
  if (cand > expected) {   // the same in every CTA
    unsigned int rank = expected - 1;   // 0-based from the top
    const unsigned int far_counts[2] = {top.y, top.x};
    const uint32_t far = cut_pick<2>(far_counts, rank, ws, res);
    unsigned int* counts = sh;          // the cluster counts in its first CTA
    if constexpr (CTAS > 1) {
      cg::this_cluster().sync();        // cleared
      counts = cg::this_cluster().map_shared_rank(sh, 0);
    }
    if (far < kBins - 1) {
      const uint32_t base = thr + (far << kFar);
      for (unsigned int i0 = 0; i0 < count; i0 += kCutThreads * kAhead) {
        if (CTAS > 1 || i0 != 0) {
#pragma unroll
          for (int u = 0; u < kAhead; ++u) {
            const unsigned int i = i0 + u * kCutThreads + t;
            key[u] = i < count ? pool.dense[first + i] : 0u;
          }
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
          if (i0 + u * kCutThreads + t < count && key[u] - base < unsigned(kCutBins)) atomicAdd(&counts[key[u] - base], 1u);
      }
      if constexpr (CTAS > 1) cg::this_cluster().sync();
      else __syncthreads();
      if (part == 0) {
        unsigned int c[kCutBins / kCutThreads];
        const int hi = (kCutThreads - t) * (kCutBins / kCutThreads) - 1;
#pragma unroll
        for (int j = 0; j < kCutBins / kCutThreads; ++j) c[j] = sh[hi - j];
        cut = base + cut_pick<kCutBins / kCutThreads>(c, rank, ws, res);
      }
    } else {
      rank = expected - 1;
      uint32_t prefix = 0;
      for (int round = 0; round < 3; ++round) {
        const unsigned int count_padded = (count + 31u) & ~31u;   // whole warps iterate together
        for (unsigned int i = t; i < count_padded; i += kCutThreads) {
          const uint32_t k = i < count ? pool.dense[first + i] : 0u;
          count_digit(counts, i < count && prefix_matches(k, round, prefix) ? digit_of(k, round) : -1);
        }
        if constexpr (CTAS > 1) cg::this_cluster().sync();
        else __syncthreads();
        const unsigned int c[2] = {counts[kBins - 1 - 2 * t], counts[kBins - 2 - 2 * t]};
        const uint32_t bin = cut_pick<2>(c, rank, ws, res);
        prefix = extend_prefix(prefix, round, bin);
        if constexpr (CTAS > 1) cg::this_cluster().sync();   // read by every CTA
        if (part == 0)
          for (int i = t; i < kBins; i += kCutThreads) sh[i] = 0;
        if (t == 0) res[0] = res[1] = 0;
        if constexpr (CTAS > 1) cg::this_cluster().sync();
        else __syncthreads();
      }
      cut = prefix;
    }
    ties = rank + 1;
  }
  if (part == 0 && t == 0) {
    const unsigned int k = cand < expected ? cand : expected;
    s->call.cut_key = cut;
    s->call.ties_kept = ties;
    s->k = k;
    s->last_cand = cand;
    const uint32_t total = 4u + 8u * k;
    uint8_t header[4];
    for (int i = 0; i < 4; ++i) header[i] = uint8_t(total >> (8 * i));
    push_bytes(dst, 0, header, 4);
    if (sumsq_to_clear != nullptr) *sumsq_to_clear = 0.f;
  }
  if constexpr (CTAS > 1) cg::this_cluster().sync();   // nobody leaves while its memory is used
}

// ---- one warp per list: deliver, clear the emitted positions, publish
// A CTA takes the eight lists of one CTA of the collect pass, in the order of their indices (see kept_before).
// The lists were complete before the kernel before this one began to look at them, and are brought in while it
// works; only the cut is waited for.
__global__ void __launch_bounds__(kThreads)
emit_kernel(float* R, float* u_mask, unsigned int expected, PushTargets dst, SparseScratch* s, ListPool pool,
            unsigned long long* state, int* status) {
  constexpr int kWarps = kThreads / 32;
  __shared__ unsigned int w_gt[kWarps], w_eq[kWarps];
  __shared__ int ticket;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) ticket = int(atomicAdd(&s->call.ticket, 1u));
  __syncthreads();
  const int block = ticket;
  const unsigned int head = s->list_head[block * kWarps + warp];
  // the list's first block; most lists have one
  unsigned int first_count = 0, first_next = kNoBlock;
  uint2 first_entry = make_uint2(0u, 0u);
  if (head < pool.capacity) {   // kNoBlock is not
    first_count = pool.count[head];
    first_next = pool.next[head];
    if (lane < kBlockEntries) first_entry = pool.entry[size_t(head) * kBlockEntries + lane];
  }
  wait_for_previous();
  resolve_epoch(dst);
  const uint32_t cut = s->call.cut_key;
  const unsigned int ties = s->call.ties_kept, cand = s->call.cand;
  const unsigned int k_total = cand < expected ? cand : expected;
  // calls f(entry, whether this lane has one) for the list's entries, a block at a time
  auto walk = [&](auto f) {
    if (head >= pool.capacity) return;
    f(first_entry, lane < int(first_count));
    for (unsigned int b = first_next; b < pool.capacity; b = pool.next[b]) {
      const unsigned int c = pool.count[b];
      uint2 en = make_uint2(0u, 0u);
      if (lane < int(c)) en = pool.entry[size_t(b) * kBlockEntries + lane];
      f(en, lane < int(c));
    }
  };
  unsigned int gt = 0, eq = 0;
  walk([&](uint2 en, bool has) {
    const uint32_t key = en.y & 0x7fffffffu;
    gt += __popc(__ballot_sync(0xffffffffu, has && key > cut));
    eq += __popc(__ballot_sync(0xffffffffu, has && key == cut));
  });
  if (lane == 0) {
    w_gt[warp] = gt;
    w_eq[warp] = eq;
  }
  __syncthreads();
  unsigned int run_gt = 0, run_eq = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    run_gt += w_gt[w];
    run_eq += w_eq[w];
  }
  if (!kept_before(state, block, run_gt, run_eq)) {
    if (threadIdx.x == 0) {
      s->call.gave_up = 1u;
      if (status != nullptr) atomicExch(status, int(kGridWait));
    }
    publish_when_grid_done(dst, &s->call.gave_up);
    return;
  }
  for (int w = 0; w < warp; ++w) {
    run_gt += w_gt[w];
    run_eq += w_eq[w];
  }
  walk([&](uint2 en, bool has) {
    const uint32_t key = en.y & 0x7fffffffu;
    const bool above = has && key > cut, at = has && key == cut;
    const unsigned int ma = __ballot_sync(0xffffffffu, above), me = __ballot_sync(0xffffffffu, at);
    const unsigned int lt = (1u << lane) - 1u;
    const unsigned int gt_before = run_gt + __popc(ma & lt), eq_before = run_eq + __popc(me & lt);
    if (above || (at && eq_before < ties)) {
      const unsigned int pos = gt_before + (eq_before < ties ? eq_before : ties);
      if (pos < k_total) {
        push_u32(dst, 4 + 4 * int64_t(pos), en.x);
        push_u32(dst, 4 + 4 * int64_t(k_total) + 4 * int64_t(pos), en.y);
        R[en.x] = 0.0f;
        if (u_mask != nullptr) u_mask[en.x] = 0.0f;
      }
    }
    run_gt += __popc(ma);
    run_eq += __popc(me);
  });
  publish_when_grid_done(dst, &s->call.gave_up);
}

// ================================================================ one-pass decode
// All payloads into a dense tensor that is written from scratch: a CTA owns a tile of the tensor and adds the
// payloads' entries of that range, rank after rank, in shared memory.  The indices of a payload ascend (the
// content rule above), so a tile's entries are found by a search: one warp per rank.
//
// What bounds it: the dense store, and a chain of dependent loads.  The chain is two long: the payload's
// header together with the probes of the search, whose places follow from the slot's size; then the entries
// of a window that certainly holds the tile's and a few of its neighbours', which are passed over.  Searching
// on until the tile's ends are known exactly costs one to three loads more.  Where a tile holds few entries its
// zeros are stored before the search ends, and the few sums afterwards, so that the store and the chain overlap
// (SPARSE).
// 25 MB at 0.1 %, eight payloads, in a chain of calls: 10.0 us, 17.4 with exact ends and the tile stored at the
// end; 64 MB, four payloads: 18.4 and 25.9.
//
// A payload whose indices do not ascend is still decoded: the tiles' windows begin where a boundary's search
// ended, the same place for the tile before, so the pieces from one beginning to the next cover the payload;
// each tile compares the neighbouring indices of its piece.  One that finds a descent raises `redo`, and the
// kernel behind decodes everything again without assuming an order.  Where there is none, every probe said the
// truth and the windows are right.  An index past the end is reported by the tile whose piece holds it.
constexpr int kDenseTile = 8192;   // elements: 32 KB, six CTAs per SM
constexpr int kBriefWindow = 64;   // entries of a rank that its warp holds in registers, two per lane
constexpr double kSparseTile = 24; // evenly spread entries of a tile up to which SPARSE is taken

// The window of a tile in one rank's payload: entries outside [begin, end) lie outside the tile, and
// [begin, own_end) is the piece whose order this tile checks.
struct TileWindow {
  uint32_t begin, own_end, end;
};
// The first probes of a search for both ends of a tile: positions around the place that evenly spread indices
// would give, two square roots of the expected count to either side, and what was read there.
struct TileProbes {
  int64_t at[2];
  uint32_t found[2];
};
__device__ __forceinline__ int64_t probe_step(uint32_t guess) { return 1 + int64_t(sqrtf(float(guess)) * 0.125f); }
// guess: entries that fit the slot; no position from there on is read, whatever the header will say.
__device__ __forceinline__ void first_probes(const uint32_t* idx, uint32_t guess, float inv_n,
                                             const int64_t (&x)[2], int lane, TileProbes& p) {
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    p.at[t] = int64_t(float(x[t]) * inv_n * float(guess)) + int64_t(lane - 16) * probe_step(guess);
    p.found[t] = p.at[t] >= 0 && p.at[t] < int64_t(guess) ? idx[p.at[t]] : 0u;
  }
}
// Whole warp.  For each end x the first position whose index is not below it lies between two places that
// depend on x, k and the payload alone; they are brought within `slack` of one another, 32 ways at a time.
__device__ __forceinline__ TileWindow tile_window(const uint32_t* idx, uint32_t k, uint32_t guess,
                                                  const TileProbes& p, const int64_t (&x)[2], uint32_t slack, int lane) {
  uint32_t a[2], len[2];
  const int64_t step0 = probe_step(guess);
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const bool below = p.at[t] < 0 || (p.at[t] < int64_t(k) && int64_t(p.found[t]) < x[t]);
    const int hits = __popc(__ballot_sync(0xffffffffu, below));
    const int64_t lowest = __shfl_sync(0xffffffffu, p.at[t], 0);
    int64_t lo = hits == 0 ? 0 : lowest + int64_t(hits - 1) * step0 + 1;   // past the last probe below x
    int64_t hi = hits == 32 ? int64_t(k) : lowest + int64_t(hits) * step0; // the first one that is not
    lo = lo < 0 ? 0 : (lo > int64_t(k) ? int64_t(k) : lo);
    hi = hi < lo ? lo : (hi > int64_t(k) ? int64_t(k) : hi);
    a[t] = uint32_t(lo);
    len[t] = uint32_t(hi - lo);
  }
  while (len[0] > slack || len[1] > slack) {
    uint32_t step[2];
    bool below[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      step[t] = (len[t] + 31) / 32;
      const uint64_t at = uint64_t(a[t]) + uint64_t(lane + 1) * step[t] - 1;
      below[t] = len[t] > slack && at < uint64_t(a[t]) + len[t] && int64_t(idx[at]) < x[t];
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const uint32_t hits = uint32_t(__popc(__ballot_sync(0xffffffffu, below[t])));
      if (len[t] <= slack) continue;
      const uint32_t rest = len[t] - hits * step[t];   // hits * step <= len: every hit lies inside
      a[t] += hits * step[t];
      len[t] = rest < step[t] - 1 ? rest : step[t] - 1;   // the probe after the last hit is not below x
    }
  }
  return {a[0], a[1], a[1] + len[1]};
}

// Entries of a payload, 0 with the status word set when the header does not fit the slot.
__device__ __forceinline__ uint32_t payload_entries(const uint8_t* payload, int64_t cap, int* status, bool report) {
  const uint32_t total = *reinterpret_cast<const uint32_t*>(payload);
  if (total >= 4 && int64_t(total) <= cap) return (total - 4) / 8;
  if (report && status != nullptr) atomicExch(status, int(kPayloadBounds));
  return 0;
}

struct TilePlan {
  int tile;         // elements
  uint32_t slack;   // see tile_window
  float inv_n;
};

// The tile [lo, lo + len) of this CTA, decoded into buf (its float4s are whole), or with SPARSE into memory at
// o; vec: o is 16-byte aligned.  False in the threads that saw a descent.  Ends with a barrier, except where it
// has stored everything itself.
template <bool SPARSE>
__device__ __forceinline__ bool decode_tile(const UnpackSources& src, int64_t n, const TilePlan& plan, int64_t lo, int len,
                                            float post_scale, int* status, float* buf, float* o, bool vec) {
  __shared__ TileWindow windows[kMaxWorld];
  __shared__ uint32_t entries[kMaxWorld];
  __shared__ int list_at[kMaxWorld][kBriefWindow];     // place in the tile, or negative
  __shared__ float list_value[kMaxWorld][kBriefWindow];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool first = blockIdx.x == 0, last = blockIdx.x == gridDim.x - 1;
  const int64_t ends[2] = {lo, lo + plan.tile};
  bool bad = false;
  uint32_t k = 0, guess = 0;
  const uint32_t* idx = nullptr;
  TileProbes probes{};
#pragma unroll
  for (int r = 0; r < kMaxWorld; ++r) {   // compile-time index into src; one warp per rank
    if (r == warp && r < src.world) {
      const uint8_t* payload = src.payload[r] + src.parity_off;
      const int64_t fit = (src.payload_bytes[r] - 4) / 8;
      guess = uint32_t(fit < 0 ? 0 : fit);
      idx = reinterpret_cast<const uint32_t*>(payload + 4);
      first_probes(idx, guess, plan.inv_n, ends, lane, probes);
      k = payload_entries(payload, src.payload_bytes[r], status, first && lane == 0);
    }
  }
  auto clear_buf = [&]() {
    for (int i = tid; i < (len + 3) / 4; i += kThreads) reinterpret_cast<float4*>(buf)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  };
  if (SPARSE) {
    const int quads = vec ? len >> 2 : 0;
    for (int i = tid; i < quads; i += kThreads) reinterpret_cast<float4*>(o)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = 4 * quads + tid; i < len; i += kThreads) o[i] = 0.f;
  } else {
    clear_buf();
  }
  // An entry that was read at e: its place in the tile, or negative.
  auto place = [&](uint32_t i, uint32_t next, uint32_t e, uint32_t total, const TileWindow& w) -> int {
    if (e < w.own_end) {
      if (e + 1 < total && next < i) bad = true;
      if (int64_t(i) >= n && status != nullptr) atomicExch(status, int(kPayloadBounds));
    }
    const int64_t at = int64_t(i) - lo;
    return at >= 0 && at < len ? int(at) : -1;
  };
  auto scaled = [&](float v) { return post_scale != 1.0f ? hp_mul(v, post_scale) : v; };
  int at[2] = {-1, -1};
  bool brief = true;
  if (warp < src.world) {
    TileWindow w = tile_window(idx, k, guess, probes, ends, plan.slack, lane);
    if (first) w.begin = 0;
    if (last) w.own_end = w.end = k;
    brief = w.end <= w.begin || w.end - w.begin <= kBriefWindow;
    if (brief) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const uint32_t e = w.begin + lane + 32 * q;
        float v = 0.f;
        if (e < w.end) {
          const uint32_t i = idx[e], next = e + 1 < k ? idx[e + 1] : 0u;
          v = __uint_as_float(idx[k + e]);
          at[q] = place(i, next, e, k, w);
        }
        if (SPARSE && at[q] >= 0) buf[at[q]] = 0.f;
        list_at[warp][lane + 32 * q] = at[q];
        list_value[warp][lane + 32 * q] = scaled(v);
      }
    }
    if (lane == 0) {
      windows[warp] = w;
      entries[warp] = k;
    }
  }
  if (__syncthreads_and(brief)) {
    if (warp == 0) {
      // ranks one after another, the indices inside a payload are unique
#pragma unroll
      for (int r = 0; r < kMaxWorld; ++r) {
        if (r < src.world) {
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int here = list_at[r][lane + 32 * q];
            if (here >= 0) buf[here] = hp_add(buf[here], list_value[r][lane + 32 * q]);
          }
          __syncwarp();
        }
      }
    }
    __syncthreads();
    if (SPARSE) {   // over the zeros stored before the barriers
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (at[q] >= 0) o[at[q]] = buf[at[q]];
    }
    return !bad;
  }
  if (SPARSE) {   // more entries than expected: the tile is put together here and stored over the zeros
    clear_buf();
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < kMaxWorld; ++r) {
    if (r < src.world) {
      const uint32_t* from = reinterpret_cast<const uint32_t*>(src.payload[r] + src.parity_off + 4);
      const uint32_t total = entries[r];
      const TileWindow w = windows[r];
      auto add_entry = [&](uint32_t i, uint32_t next, float v, uint32_t e) {
        const int here = place(i, next, e, total, w);
        if (here >= 0) buf[here] = hp_add(buf[here], scaled(v));
      };
      // four entries in flight per thread: at a quarter of the elements a tile holds 2,048 per rank
      uint32_t e = w.begin + tid;
      for (; int64_t(e) + 3 * kThreads < int64_t(w.end); e += 4 * kThreads) {
        uint32_t i[4], next[4];
        float v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t x = e + u * kThreads;
          i[u] = from[x];
          next[u] = x + 1 < total ? from[x + 1] : 0u;
          v[u] = __uint_as_float(from[total + x]);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) add_entry(i[u], next[u], v[u], e + u * kThreads);
      }
      for (; e < w.end; e += kThreads) add_entry(from[e], e + 1 < total ? from[e + 1] : 0u, __uint_as_float(from[total + e]), e);
      __syncthreads();
    }
  }
  if (SPARSE) {
    const int quads = vec ? len >> 2 : 0;
    for (int i = tid; i < quads; i += kThreads) reinterpret_cast<float4*>(o)[i] = reinterpret_cast<const float4*>(buf)[i];
    for (int i = 4 * quads + tid; i < len; i += kThreads) o[i] = buf[i];
  }
  return !bad;
}

template <bool SPARSE, bool VEC>
__global__ void __launch_bounds__(kThreads, 6)
dense_tile_kernel(UnpackSources src, float* __restrict__ out, int64_t n, TilePlan plan, float post_scale, int* status,
                  unsigned int* redo) {
  __shared__ __align__(16) float buf[kDenseTile];
  wait_for_previous();
  let_next_start();
  const int tid = threadIdx.x;
  const int64_t lo = int64_t(blockIdx.x) * plan.tile;
  const int len = int(lo + plan.tile < n ? plan.tile : n - lo);
  float* o = out + lo;
  if (!decode_tile<SPARSE>(src, n, plan, lo, len, post_scale, status, buf, o, VEC)) *redo = 1u;
  if (SPARSE) return;
  const int quads = VEC ? len >> 2 : 0;
  for (int i = tid; i < quads; i += kThreads) reinterpret_cast<float4*>(o)[i] = reinterpret_cast<const float4*>(buf)[i];
  for (int i = 4 * quads + tid; i < len; i += kThreads) o[i] = buf[i];
}

// ---- decode and optimizer step in one pass
// When nobody keeps the dense gradient, the tile goes straight into the update of its parameters: the
// gradient is neither written nor read (4 of AdamW's 28 bytes per element) nor cleared afterwards, and
// one pass takes the place of a scatter per rank, the dense update and the clearing pass.
// Receive half of a 128 MB bucket at 0.1 %, by the host's clock: AdamW with eight payloads 204 us, 249 with the
// scatters, the dense update and the clearing pass; with one payload 187 and 192.  SGD: 135 and 220, 121 and 165.
// An update cannot be taken back, so the payloads are looked at first: sparse_check_kernel records any
// index that does not ascend or lies outside, and the update kernel returns on a recorded failure, as the
// dense ones do.  OPT: 0 = SGD with momentum, 1 = AdamW.
__global__ void __launch_bounds__(kThreads)
sparse_check_kernel(UnpackSources src, int64_t n, int* status) {
  let_next_start();
  if (status_guarded(src.guard)) return;
  resolve_epoch(src);
  const int r = blockIdx.y;
  const uint8_t* payload = select_payload(src, r) + src.parity_off;
  const uint32_t k = payload_entries(payload, select_payload_bytes(src, r), status, threadIdx.x == 0);
  const uint32_t* idx = reinterpret_cast<const uint32_t*>(payload + 4);
  bool bad = false;
  for (uint32_t e = blockIdx.x * kThreads + threadIdx.x; e < k; e += gridDim.x * kThreads) {
    const uint32_t i = idx[e];
    bad = bad || int64_t(i) >= n || (e > 0 && idx[e - 1] >= i);
  }
  if (bad) atomicExch(status, int(kPayloadBounds));
}

template <int OPT>
__global__ void __launch_bounds__(kThreads, 4)
sparse_apply_kernel(UnpackSources src, int64_t n, TilePlan plan, float post_scale, SgdApply sgd, AdamWApply adamw, int vec,
                    const int* guard, int* status) {
  __shared__ __align__(16) float buf[kDenseTile];
  wait_for_previous();
  if (status_guarded(guard)) return;
  resolve_epoch(src);
  float bc1 = 0.f, rsqrt_bc2 = 0.f;
  if (OPT == 1) adamw_bias(adamw, bc1, rsqrt_bc2);
  const int tid = threadIdx.x;
  const int64_t lo = int64_t(blockIdx.x) * plan.tile;
  const int len = int(lo + plan.tile < n ? plan.tile : n - lo);
  decode_tile<false>(src, n, plan, lo, len, post_scale, status, buf, nullptr, false);
  const int quads = vec ? len >> 2 : 0;
#pragma unroll 2
  for (int i = tid; i < quads; i += kThreads) {
    const float4 g = reinterpret_cast<const float4*>(buf)[i];
    if (OPT == 1) {
      adamw_four(adamw, bc1, rsqrt_bc2, (lo >> 2) + i, g);
    } else {
      const float g4[4] = {g.x, g.y, g.z, g.w};
      sgd_update4(sgd, lo + 4 * i, g4);
    }
  }
  for (int i = 4 * quads + tid; i < len; i += kThreads) {
    if (OPT == 1) adamw_at(adamw, bc1, rsqrt_bc2, lo + i, buf[i]);
    else sgd_update(sgd, lo + i, buf[i]);
  }
}

// Decode without an assumption on the order of the indices; returns at once unless a tile asked for
// it.  A CTA owns a range of the tensor and looks through all entries for those in its range.
// redo[0] the request, redo[1] CTAs done; both are left at zero.
constexpr int kRedoThreads = 1024;
__global__ void __launch_bounds__(kRedoThreads)
dense_redo_kernel(UnpackSources src, float* __restrict__ out, int64_t n, float post_scale, unsigned int* redo) {
  wait_for_previous();
  if (*reinterpret_cast<volatile unsigned int*>(redo) == 0u) return;
  const int64_t span = (n + gridDim.x - 1) / gridDim.x;
  const int64_t lo = int64_t(blockIdx.x) * span, hi = lo + span < n ? lo + span : n;
  for (int64_t i = lo + threadIdx.x; i < hi; i += kRedoThreads) out[i] = 0.0f;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kMaxWorld; ++r) {
    if (r < src.world) {
      const uint32_t k = payload_entries(src.payload[r], src.payload_bytes[r], nullptr, false);
      const uint32_t* idx = reinterpret_cast<const uint32_t*>(src.payload[r] + 4);
      for (uint32_t e = threadIdx.x; e < k; e += kRedoThreads) {
        const int64_t i = idx[e];
        if (i >= lo && i < hi) {
          float v = __uint_as_float(idx[k + e]);
          if (post_scale != 1.0f) v = hp_mul(v, post_scale);
          out[i] = hp_add(out[i], v);
        }
      }
      __syncthreads();
    }
  }
  if (threadIdx.x == 0) {
    if (atomicAdd(redo + 1, 1u) == gridDim.x - 1) {   // every CTA has read the request
      redo[0] = 0u;
      redo[1] = 0u;
    }
  }
}

struct Plan {
  int blocks;
  int64_t chunk;
};
inline Plan plan_for(int64_t n) {
  int64_t blocks = (n + kTile - 1) / kTile;
  if (blocks > kMaxBlocks) blocks = kMaxBlocks;
  if (blocks < 1) blocks = 1;
  int64_t chunk = (n + blocks - 1) / blocks;
  chunk = (chunk + kTile - 1) / kTile * kTile;
  blocks = (n + chunk - 1) / chunk;
  return {int(blocks), chunk};
}

}  // namespace

namespace {

// Layout of the scratch behind SparseScratch: sample keys, the pool of list blocks, the states of kept_before.  All
// are sized from n alone, so that one allocation serves every keep fraction and sample rate a
// caller may pick later; a call whose sample or expected candidate count does not fit takes the
// scan form, which needs neither.
struct ListPlan {
  int64_t key_capacity;    // sample keys, and as many places for the ones select_kernel keeps
  int64_t pool_blocks;
  size_t keys_offset, pool_offset, state_offset, total_bytes;
};
inline ListPlan list_plan(int64_t n) {
  ListPlan p;
  p.key_capacity = n / 100 + 1024;
  // candidates: 6 % of n (six times the largest expectation the list form serves) plus a floor
  // that covers thresholds drawn from a handful of samples, plus one partly filled block per list
  const int64_t entries = n / 100 * 6 + 65536;
  p.pool_blocks = entries / kBlockEntries + kMaxLists;
  p.keys_offset = (sizeof(SparseScratch) + 255) / 256 * 256;
  p.pool_offset = (p.keys_offset + size_t(p.key_capacity) * 8 + 255) / 256 * 256;
  // count[blocks], next[blocks], entry[blocks][16], dense[blocks * 16]
  p.state_offset = (p.pool_offset + size_t(p.pool_blocks) * (8 + kBlockEntries * (sizeof(uint2) + 4)) + 512 + 7) / 8 * 8;
  p.total_bytes = p.state_offset + size_t((n + kWriteChunk - 1) / kWriteChunk + kMaxBlocks) * 8;   // kept_before's states
  return p;
}

}  // namespace

size_t sparse_scratch_bytes(int64_t n) { return list_plan(n < 1 ? 1 : n).total_bytes; }

cudaError_t sparse_compress_fused(const SparseFuse& fuse, float* R, int64_t n, double sample_rate,
                                  double keep_fraction, uint64_t seed, const PushTargets& dst, void* scratch,
                                  cudaStream_t stream, int* status, int* launches) {
  if (n <= 0 || n > 0x7fffffff || scratch == nullptr || R == nullptr) return cudaErrorInvalidValue;
  if (fuse.mode < 0 || fuse.mode > 2 || (fuse.mode >= 1 && fuse.grad == nullptr) || (fuse.mode == 2 && fuse.u == nullptr))
    return cudaErrorInvalidValue;
  for (int p = 0; p < dst.world; ++p)
    if (reinterpret_cast<uintptr_t>(dst.payload[p]) & 3) return cudaErrorInvalidValue;
  auto* s = static_cast<SparseScratch*>(scratch);
  const Plan pl = plan_for(n);
  int64_t expected = sparse_expected_k(n, keep_fraction);
  if (expected > n) expected = n;
  const int64_t sample_cnt = sparse_sample_count(n, sample_rate);
  int64_t rank0 = sparse_threshold_rank(sample_cnt, keep_fraction);
  if (sample_cnt > 0 && rank0 > sample_cnt - 1) rank0 = sample_cnt - 1;
  const ListPlan lp = list_plan(n);
  SparseFuseDev f{fuse.grad, fuse.u, fuse.momentum, fuse.clip, fuse.sumsq, fuse.zero_grad, fuse.mode};
  uint32_t* keys = sample_cnt <= lp.key_capacity
                       ? reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(scratch) + lp.keys_offset) : nullptr;
  // the list form: small keep fractions, and a pool that holds the candidates with a wide
  // margin: their number is about n (rank0+1) / (samples+1) with a relative spread of
  // 1 / sqrt(rank0+1); without sampling every non-zero element is a candidate
  bool lists = keep_fraction <= (n <= kListSmall ? kListMaxKeepSmall : kListMaxKeep) && sample_cnt > 0;
  if (lists) {
    const double mean = double(n) * double(rank0 + 1) / double(sample_cnt + 1);
    const double need = mean * (1.0 + 40.0 / std::sqrt(double(rank0 + 1)));
    lists = need <= double(lp.pool_blocks - kMaxLists) * kBlockEntries;
  }
  if (fuse.mode == 2 && fuse.clip > 0.f) {
    if (fuse.sumsq == nullptr) return cudaErrorInvalidValue;
    const cudaError_t err = dgc_sumsq(fuse.grad, n, const_cast<float*>(fuse.sumsq), stream);
    if (err != cudaSuccess) return err;
  }
  cudaError_t e = cudaSuccess;
  const dim3 block(kThreads);
  float* const sumsq = fuse.mode == 2 && fuse.clip > 0.f ? const_cast<float*>(fuse.sumsq) : nullptr;
  if (sample_cnt > 0) {
    int64_t sb = (sample_cnt + kThreads - 1) / kThreads;
    if (sb > kMaxSampleBlocks) sb = kMaxSampleBlocks;
    const dim3 grid = dim3(unsigned(sb));
    // the first kernel of the chain, unless the gradient's norm was taken before it
    e = launch_with(sumsq != nullptr, 1, sample_round_kernel<0>, grid, block, 0, stream, f, R, n, sample_cnt,
                    unsigned(rank0), seed, s, keys, dst.epoch_dev);
    if (keys != nullptr) {
      if (e == cudaSuccess)
        e = launch_after(select_kernel, grid, block, 0, stream, sample_cnt, unsigned(rank0), s, keys, keys + lp.key_capacity);
    } else {
      if (e == cudaSuccess)
        e = launch_after(sample_round_kernel<1>, grid, block, 0, stream, f, R, n, sample_cnt, unsigned(rank0), seed, s, keys,
                         dst.epoch_dev);
      if (e == cudaSuccess)
        e = launch_after(sample_round_kernel<2>, grid, block, 0, stream, f, R, n, sample_cnt, unsigned(rank0), seed, s, keys,
                         dst.epoch_dev);
    }
  } else {
    e = cudaMemsetAsync(&s->call, 0, sizeof(s->call), stream);   // every non-zero element is a candidate
  }
  if (e != cudaSuccess) return e;
  if (launches != nullptr)   // the norm; the sample and its selection; the list form's kernels or the scan form's
    *launches += (sumsq != nullptr ? 1 : 0) + (sample_cnt > 0 ? (keys != nullptr ? 2 : 3) : 0) + (lists ? 3 : 4);
  const dim3 grid = dim3(unsigned(pl.blocks));
  float* const u_mask = fuse.mode == 2 ? fuse.u : nullptr;
  auto* state = reinterpret_cast<unsigned long long*>(static_cast<uint8_t*>(scratch) + lp.state_offset);
  if (lists) {
    PushTargets hdr = dst;
    hdr.done = nullptr;
    uint8_t* pool_base = static_cast<uint8_t*>(scratch) + lp.pool_offset;
    ListPool pool;
    pool.capacity = static_cast<unsigned int>(lp.pool_blocks);
    pool.count = reinterpret_cast<unsigned int*>(pool_base);
    pool.next = pool.count + lp.pool_blocks;
    pool.entry = reinterpret_cast<uint2*>((reinterpret_cast<uintptr_t>(pool.next + lp.pool_blocks) + 127) & ~uintptr_t(127));
    pool.dense = reinterpret_cast<uint32_t*>(pool.entry + size_t(lp.pool_blocks) * kBlockEntries);
    auto collect = fuse.mode == 2 ? collect_kernel<2> : (fuse.mode == 1 ? collect_kernel<1> : collect_kernel<0>);
    e = launch_after(collect, grid, block, 0, stream, f, R, n, pl.chunk, s, pool, state);   // lists: there was a sample
    if (e != cudaSuccess) return e;
    const bool one = expected <= kCutOneCta;
    const int ctas = one ? 1 : kCutCluster;
    e = launch_with(true, ctas, one ? cut_kernel<1> : cut_kernel<kCutCluster>, dim3(unsigned(ctas)), dim3(kCutThreads), 0, stream,
                    unsigned(expected), hdr, s, pool, sumsq);
    if (e != cudaSuccess) return e;
    return launch_after(emit_kernel, grid, block, 0, stream, R, u_mask, unsigned(expected), dst, s, pool, state, status);
  }
  // scan form
  auto count = fuse.mode == 2 ? count_kernel<2> : (fuse.mode == 1 ? count_kernel<1> : count_kernel<0>);
  e = launch_with(sample_cnt > 0, 1, count, grid, block, 0, stream, f, R, n, pl.chunk, s, state);
  if (e == cudaSuccess)
    e = launch_after(trim_kernel<0>, grid, block, 0, stream, static_cast<const float*>(R), n, pl.chunk, unsigned(expected), s);
  if (e == cudaSuccess)
    e = launch_after(trim_kernel<1>, grid, block, 0, stream, static_cast<const float*>(R), n, pl.chunk, unsigned(expected), s);
  if (e != cudaSuccess) return e;
  return launch_after(write_kernel, dim3(unsigned((n + kWriteChunk - 1) / kWriteChunk)), block, 0, stream, R, u_mask, sumsq,
                      n, unsigned(expected), dst, s, state, status);
}

cudaError_t sparse_compress(const float* grad, float* R, int64_t n, double sample_rate,
                            double keep_fraction, uint64_t seed, int accumulate,
                            const PushTargets& dst, void* scratch, cudaStream_t stream, int* status) {
  SparseFuse fuse;
  fuse.mode = accumulate ? 1 : 0;
  fuse.grad = accumulate ? grad : nullptr;
  return sparse_compress_fused(fuse, R, n, sample_rate, keep_fraction, seed, dst, scratch, stream, status);
}

// Counters of the last compress call that used `scratch`: {elements emitted, candidates over the
// sampled threshold (list form; 0 otherwise), threshold as the bit pattern of a float, candidates
// dropped so far because the pool was full}.  Copied to the host on `stream`.
cudaError_t sparse_read_stats(const void* scratch, unsigned int* host4, cudaStream_t stream) {
  const auto* s = static_cast<const SparseScratch*>(scratch);
  cudaError_t e = cudaMemcpyAsync(host4 + 0, &s->k, 4, cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(host4 + 1, &s->last_cand, 4, cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(host4 + 2, &s->call.thr_key, 4, cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(host4 + 3, &s->dropped, 4, cudaMemcpyDeviceToHost, stream);
  return e;
}

namespace {
// Tiles of 8,192 elements, smaller ones while they would not cover every SM four times.  per_tile: entries of
// the fullest slot that a tile would hold if they were evenly spread.
inline TilePlan tile_plan(const UnpackSources& src, int64_t n, double& per_tile) {
  const int64_t tile = std::min<int64_t>(std::max<int64_t>((n / (148 * 4) + 1023) / 1024 * 1024, 1024), kDenseTile);
  int64_t fit = 0;
  for (int r = 0; r < src.world; ++r) fit = std::max<int64_t>(fit, (src.payload_bytes[r] - 4) / 8);
  per_tile = double(fit) * double(tile) / double(n);
  // a window may be that much longer than the tile's entries at either end
  return {int(tile), uint32_t(16 + std::min(per_tile, double(tile)) / 4), 1.0f / float(n)};
}
}  // namespace

cudaError_t sparse_apply(const UnpackSources& src, int64_t n, float post_scale, const SgdApply* sgd,
                         const AdamWApply* adamw, int* status, cudaStream_t stream) {
  if (n <= 0 || n > 0x7fffffff || src.world < 1 || src.world > kMaxWorld || status == nullptr ||
      (sgd != nullptr) == (adamw != nullptr))
    return cudaErrorInvalidValue;
  int64_t kmax = 1;
  for (int r = 0; r < src.world; ++r) {
    if ((reinterpret_cast<uintptr_t>(src.payload[r]) | uintptr_t(src.parity_stride)) & 3) return cudaErrorInvalidValue;
    kmax = std::max<int64_t>(kmax, (src.payload_bytes[r] - 4) / 8);
  }
  const int64_t check_blocks = std::min<int64_t>((kmax + kThreads - 1) / kThreads, 148);
  sparse_check_kernel<<<dim3(unsigned(check_blocks), unsigned(src.world)), kThreads, 0, stream>>>(src, n, status);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  double per_tile;
  const TilePlan plan = tile_plan(src, n, per_tile);
  const dim3 grid = dim3(unsigned((n + plan.tile - 1) / plan.tile)), block(kThreads);
  if (adamw != nullptr) {
    if (!adamw->param || !adamw->exp_avg || !adamw->exp_avg_sq || adamw->step < 1) return cudaErrorInvalidValue;
    const int vec = al(adamw->param) && al(adamw->exp_avg) && al(adamw->exp_avg_sq) ? 1 : 0;
    return launch_after(sparse_apply_kernel<1>, grid, block, 0, stream, src, n, plan, post_scale, SgdApply{}, *adamw, vec,
                        static_cast<const int*>(status), status);
  }
  if (!sgd->param || !sgd->momentum) return cudaErrorInvalidValue;
  const int vec = al(sgd->param) && al(sgd->momentum) ? 1 : 0;
  return launch_after(sparse_apply_kernel<0>, grid, block, 0, stream, src, n, plan, post_scale, *sgd, AdamWApply{}, vec,
                      static_cast<const int*>(status), status);
}

cudaError_t sparse_unpack_accum(const UnpackSources& src, float* out, int64_t n, int add,
                                float post_scale, int* status, cudaStream_t stream, unsigned int* redo, bool overlap) {
  if (n <= 0 || src.world < 1 || src.world > kMaxWorld) return cudaErrorInvalidValue;
  if (!add && redo != nullptr && n <= 0x7fffffff && src.epoch_dev == nullptr && src.guard == nullptr) {
    for (int r = 0; r < src.world; ++r)
      if (reinterpret_cast<uintptr_t>(src.payload[r]) & 3) return cudaErrorInvalidValue;
    double per_tile;
    const TilePlan plan = tile_plan(src, n, per_tile);
    const unsigned blocks = unsigned((n + plan.tile - 1) / plan.tile);
    const bool vec = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    // few entries: the window of nearly every tile fits a warp's registers (see decode_tile)
    const bool sparse = per_tile <= kSparseTile;
    auto kernel = sparse ? (vec ? dense_tile_kernel<true, true> : dense_tile_kernel<true, false>)
                         : (vec ? dense_tile_kernel<false, true> : dense_tile_kernel<false, false>);
    const cudaError_t e = launch_with(overlap, 1, kernel, dim3(blocks), dim3(kThreads), 0, stream, src, out, n, plan, post_scale,
                                      status, redo);
    if (e != cudaSuccess) return e;
    return launch_after(dense_redo_kernel, dim3(148), dim3(kRedoThreads), 0, stream, src, out, n, post_scale, redo);
  }
  if (!add) {
    cudaError_t e = cudaMemsetAsync(out, 0, size_t(n) * sizeof(float), stream);
    if (e != cudaSuccess) return e;
  }
  for (int r = 0; r < src.world; ++r) {
    if (reinterpret_cast<uintptr_t>(src.payload[r]) & 3) return cudaErrorInvalidValue;
    // worst-case k is bounded by the slot capacity
    const int64_t kmax = (src.payload_bytes[r] - 4) / 8;
    int64_t blocks = (kmax + kThreads - 1) / kThreads;
    if (blocks < 1) blocks = 1;
    if (blocks > 148 * 8) blocks = 148 * 8;
    scatter_kernel<<<int(blocks), kThreads, 0, stream>>>(src.payload[r], src.payload_bytes[r], out,
                                                        n, post_scale, status, src.epoch_dev,
                                                        src.parity_stride, src.guard);
  }
  return cudaGetLastError();
}

}  // namespace cuda
}  // namespace hipress
