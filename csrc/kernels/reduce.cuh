// Grid-wide min/max (and abs-max) reduction without a host round-trip.
//
// Each CTA reduces its grid-stride share and writes one partial pair; the last
// CTA to finish (elected through a counter) folds the partials and calls a
// finaliser that turns the extremes into header bytes and scale factors on the
// device.  The reference does this with thrust::minmax_element, two 4-byte
// device-to-host copies and a stream synchronise per batch
// (terngrad_body.h:186-195).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.h"
#include "launch.cuh"
#include "p2p.cuh"

namespace hipress {
namespace cuda {

constexpr int kReduceMaxBlocks = 1024;
constexpr int kResidentMaxBlocks = 256;   // CTAs of grid_minmax_all, one per SM

struct MinMaxScratch {
  unsigned int counter;  // zero between launches
  unsigned int left;     // zero between launches
  float mn, mx;    // result
  float inv, gap;  // compress-side scale and decode-side step
  float partial_min[kReduceMaxBlocks];
  float partial_max[kReduceMaxBlocks];
  unsigned long long extremes[kResidentMaxBlocks];   // zero between launches
  unsigned long long of_all;   // zero between launches
};
static_assert(sizeof(MinMaxScratch) <= 12288, "the place of the next state in a stream's scratch");

__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide reduction of (mn, mx); result valid in thread 0.
template <int THREADS>
__device__ __forceinline__ void block_minmax(float& mn, float& mx) {
  __shared__ float smin[THREADS / 32];
  __shared__ float smax[THREADS / 32];
  mn = warp_min(mn);
  mx = warp_max(mx);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    smin[warp] = mn;
    smax[warp] = mx;
  }
  __syncthreads();
  if (warp == 0) {
    mn = lane < THREADS / 32 ? smin[lane] : smin[0];
    mx = lane < THREADS / 32 ? smax[lane] : smax[0];
    mn = warp_min(mn);
    mx = warp_max(mx);
  }
  __syncthreads();
}

// Extremes over a grid whose CTAs are all resident (launch_resident): every thread of every CTA gets them.
// A CTA's extremes are one 64-bit word, which is zero until they are there: what says that they have arrived is what
// carries them, so that no fence and no counter stand between the store and the look.  CTA 0 collects the words and
// stores the extremes of all in one more, at which the others look.  25 MB, from the last CTA's arrival until all have
// them: 1.9 us; 3.2 with partials, a fence, a counter, a fence, the partials' loads and a reduction over the CTA.
// TernGrad of 25 MB and the decode of eight payloads: 35.3 and 36.7 us; 38.9 with all CTAs looking at all words, which
// holds the stores up, and 38.0 with a pause between their looks.
// The words' places are taken by a counter (grid_arrive, early in the kernel, where nobody waits for it).  The wait
// is bounded; when it runs out (a CTA that is resident arrives, so it does not) the CTA returns false after
// recording it in *status.  Every CTA arrives once and leaves once, whatever it saw, and the last one to leave makes
// the state ready for the next launch (grid_leave, at the end of the kernel; nobody waits for the counter of that
// either).  No fence goes before: what the last one resets was read, and acted upon, by the warp that leaves.
struct GridPlace {
  unsigned int arrived = 0, left = 0;   // thread 0's
};
__device__ __forceinline__ void grid_arrive(MinMaxScratch* s, GridPlace& place) {
  if (threadIdx.x == 0) place.arrived = atomicAdd(&s->counter, 1u);
}
template <int THREADS>
__device__ __forceinline__ bool grid_minmax_all(MinMaxScratch* s, float& mn, float& mx, uint64_t wait_ns, int* status,
                                                GridPlace& place) {
  constexpr int kWarps = THREADS / 32, kWords = kResidentMaxBlocks / 32;
  static_assert(kWarps <= 32, "one lane per warp");
  __shared__ float smin[kWarps], smax[kWarps];
  __shared__ float res[2];
  __shared__ bool arrived;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  mn = warp_min(mn);
  mx = warp_max(mx);
  if (lane == 0) {
    smin[warp] = mn;
    smax[warp] = mx;
  }
  __syncthreads();
  if (warp == 0) {
    mn = warp_min(smin[lane < kWarps ? lane : 0]);
    mx = warp_max(smax[lane < kWarps ? lane : 0]);
    // zero stands for "not there": the maximum's bits are turned over, and a maximum that is no NaN leaves a one there
    const unsigned long long mine = (unsigned long long)(~__float_as_uint(mx)) << 32 | __float_as_uint(mn);
    if (lane == 0 && place.arrived < gridDim.x)
      asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(&s->extremes[place.arrived]), "l"(mine) : "memory");
    const uint64_t t0 = globaltimer_ns();
    bool all = false;
    unsigned long long of_all = 0;
    if (blockIdx.x == 0) {
      unsigned long long w[kWords];
#pragma unroll
      for (int k = 0; k < kWords; ++k) w[k] = k * 32 + lane < int(gridDim.x) ? 0 : 1;
      for (unsigned int i = 1; !all; ++i) {
        bool here = true;
#pragma unroll
        for (int k = 0; k < kWords; ++k)
          if (w[k] == 0)
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w[k]) : "l"(&s->extremes[k * 32 + lane]) : "memory");
#pragma unroll
        for (int k = 0; k < kWords; ++k) here = here && w[k] != 0;
        all = __all_sync(0xffffffffu, here);
        if ((i & 63u) == 0 && __any_sync(0xffffffffu, globaltimer_ns() - t0 > wait_ns)) break;
      }
      mn = INFINITY;
      mx = -INFINITY;
#pragma unroll
      for (int k = 0; k < kWords; ++k) {
        if (k * 32 + lane < int(gridDim.x)) {
          mn = fminf(mn, __uint_as_float(uint32_t(w[k])));
          mx = fmaxf(mx, __uint_as_float(~uint32_t(w[k] >> 32)));
        }
      }
      mn = warp_min(mn);
      mx = warp_max(mx);
      of_all = (unsigned long long)(~__float_as_uint(mx)) << 32 | __float_as_uint(mn);
      if (lane == 0 && all) asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(&s->of_all), "l"(of_all) : "memory");
    } else if (lane == 0) {
      for (unsigned int i = 1; !all; ++i) {
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(of_all) : "l"(&s->of_all) : "memory");
        all = of_all != 0;
        if ((i & 63u) == 0 && globaltimer_ns() - t0 > wait_ns) break;
      }
      mn = __uint_as_float(uint32_t(of_all));
      mx = __uint_as_float(~uint32_t(of_all >> 32));
    }
    if (lane == 0) {
      if (!all) atomicExch(status, int(kGridWait));
      arrived = all;
      res[0] = mn;
      res[1] = mx;
      place.left = atomicAdd(&s->left, 1u);
    }
  }
  __syncthreads();
  mn = res[0];
  mx = res[1];
  return arrived;
}
__device__ __forceinline__ void grid_leave(MinMaxScratch* s, const GridPlace& place) {
  if (threadIdx.x >= 32 || __shfl_sync(0xffffffffu, place.left, 0) != gridDim.x - 1) return;
  for (int i = threadIdx.x; i < int(gridDim.x); i += 32) s->extremes[i] = 0;
  if (threadIdx.x == 0) {
    s->counter = 0u;
    s->left = 0u;
    s->of_all = 0;
  }
}

// Returns true in every thread of exactly one CTA: the last to arrive.  Before
// returning true the partials of all CTAs are visible to the caller.
template <int THREADS>
__device__ __forceinline__ bool grid_minmax_last_block(MinMaxScratch* s, float mn, float mx,
                                                       float& out_mn, float& out_mx) {
  __shared__ bool is_last;
  block_minmax<THREADS>(mn, mx);
  if (threadIdx.x == 0) {
    s->partial_min[blockIdx.x] = mn;
    s->partial_max[blockIdx.x] = mx;
    __threadfence();
    const unsigned int prev = atomicAdd(&s->counter, 1u);
    is_last = (prev == gridDim.x - 1);
  }
  __syncthreads();
  if (!is_last) return false;
  __threadfence();
  float a = INFINITY, b = -INFINITY;
  for (int i = threadIdx.x; i < int(gridDim.x); i += THREADS) {
    a = fminf(a, reinterpret_cast<volatile float*>(s->partial_min)[i]);
    b = fmaxf(b, reinterpret_cast<volatile float*>(s->partial_max)[i]);
  }
  block_minmax<THREADS>(a, b);
  __shared__ float res[2];
  if (threadIdx.x == 0) {
    res[0] = a;
    res[1] = b;
    s->counter = 0u;
  }
  __syncthreads();
  out_mn = res[0];
  out_mx = res[1];
  return true;
}

}  // namespace cuda
}  // namespace hipress
