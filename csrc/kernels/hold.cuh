// Quantisers that read their inputs once: one CTA per SM keeps its part of the tensor in shared memory, the CTAs
// exchange their extremes (grid_minmax_all), and quantise from there (tern_hold_kernel, ecq_hold_kernel).
#pragma once
#include "kernels.h"
#include "launch.cuh"
#include "p2p.cuh"
#include "reduce.cuh"

namespace hipress {
namespace cuda {

constexpr int kHoldThreads = 1024;
constexpr size_t kHoldBytes = 208 * 1024;    // of fp32 values per CTA
constexpr size_t kHoldSmem = 224 * 1024;     // with the payload bytes

// A CTA's part: a multiple of 512 elements, so that the parts' payload bytes start equally far past a
// 16-byte boundary (64 bytes at 1 bit) and their units are whole.  part == 0: the tensor does not fit.
struct HoldPlan {
  int64_t part = 0;
  unsigned ctas = 0;
  size_t smem = 0;
};
inline cudaError_t hold_plan(int64_t n, int bitwidth, HoldPlan& p) {
  int device = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return e;
  if (sms > kResidentMaxBlocks) sms = kResidentMaxBlocks;
  const int64_t part = ((n + sms - 1) / sms + 511) / 512 * 512;
  p.smem = size_t(part) * sizeof(float) + size_t(part * bitwidth / 8) + 32;
  if (size_t(part) * sizeof(float) > kHoldBytes || p.smem > kHoldSmem) return cudaSuccess;
  p.part = part;
  p.ctas = unsigned((n + part - 1) / part);
  return cudaSuccess;
}
// The caller has the GPU to itself and the payload goes to one destination of this call's own.
inline bool hold_alone(bool whole_gpu, const PushTargets& dst) {
  return whole_gpu && dst.shard_elems == 0 && dst.world == 1 && dst.done == nullptr && dst.guard == nullptr &&
         dst.epoch_dev == nullptr && dst.remote == 0 && dst.mc == nullptr;
}

// The payload bytes of one unit into the CTA's buffer; the address is even, BPT is 1, 2 or 4.
template <int BPT>
__device__ __forceinline__ void hold_unit_bytes(uint8_t* at, uint32_t bytes) {
  if (BPT == 1) {
    *at = uint8_t(bytes);
  } else {
#pragma unroll
    for (int h = 0; h < BPT / 2; ++h) reinterpret_cast<uint16_t*>(at)[h] = uint16_t(bytes >> (16 * h));
  }
}
// `count` payload bytes that lie at bytes_at + shift, to byte `first` of the packed data: 16-byte words of the
// destination, the first and the last one by bytes.  The CTA's first 32 threads do the latter.
__device__ __forceinline__ void hold_put(const PushTargets& dst, int header_bytes, int64_t first, const uint8_t* bytes_at, int shift,
                                         int count) {
  const PushCursor cur{nullptr};
  const int tid = threadIdx.x;
  const int64_t to = header_bytes + first - shift;
  const int words = (shift + count) >> 4;                  // words that end inside the part
  for (int w = tid + (shift != 0 ? 1 : 0); w < words; w += kHoldThreads)
    put_u128(dst, cur, to + 16 * w, reinterpret_cast<const uint4*>(bytes_at)[w]);
  const int head_end = shift == 0 ? 0 : (16 < shift + count ? 16 : shift + count);
  const int tail_begin = words * 16 > head_end ? words * 16 : head_end;
  if (tid < 16) {
    if (tid >= shift && tid < head_end) put_u8(dst, cur, to + tid, bytes_at[tid]);
  } else if (tid < 32) {
    const int at = tail_begin + tid - 16;
    if (at >= shift && at < shift + count) put_u8(dst, cur, to + at, bytes_at[at]);
  }
}

}  // namespace cuda
}  // namespace hipress
