// Launches whose start overlaps the end of the kernel before them in the stream (programmatic
// dependent launch).  A chain of short kernels otherwise pays, between any two of them, the drain
// of one and the ramp-up of the next.
//
// Rules the kernels here follow.  A kernel launched by launch_after() calls wait_for_previous()
// before it touches what the kernel before it wrote; the wait covers that whole kernel, so a chain is
// ordered exactly as plain launches are.  What a kernel reads through the read-only path (__ldg, const
// __restrict__) was complete before the chain began: such a load may be moved above the wait.  The kernel
// before it calls let_next_start() (its result is only about when the next one is brought in, never about
// what it may read), and a long one only when its work is nearly done: CTAs that wait hold registers and
// shared memory which kernels of other streams, the backward pass above all, could use.
// The first kernel of a chain may be launched so as well, behind whatever the stream holds (`overlap` in kernels.h):
// it waits before it touches anything and reads through ordinary loads.  A kernel of somebody else's that
// never lets the next one start has then ended, and what is saved is the launch behind it, about a microsecond;
// behind anything but a kernel the launch is a plain one.  The calls of ops.cpp ask for it, except while a graph
// is recorded, where the stream may depend on several nodes, and except for the sparse compressors: their grids
// are one CTA for each place on the chip, and what is brought in while the kernel ahead still holds some of them is
// spread unevenly (64 MB, GradDrop: 97 us plain and 117 so).
// ECQ, 25 MB: 40.7 us a pass, 39.0 so; PowerSGD, 4096 x 4096: 107.9 and 100.3; TernGrad, 9.4 MB: 14.4 and 13.0.
#pragma once
#include <cuda_runtime.h>

namespace hipress {
namespace cuda {

__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Loads past L1 of what another CTA or the kernel before has just written.  Unlike __ldcg, which the
// compiler may move freely, these keep their place behind the wait, the flag or the counter that they follow.
__device__ __forceinline__ float2 load_written(const float2* p) {
  float2 v;
  asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float load_written(const float* p) {
  float v;
  asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned int load_written(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.global.cg.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// A kernel whose CTAs wait for one another: all of them are resident at once, or the launch fails.
template <typename... Params, typename... Args>
cudaError_t launch_resident(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// overlap: start while the kernel before is still running.  cluster: CTAs per cluster (1: none).
template <typename... Params, typename... Args>
cudaError_t launch_with(bool overlap, int cluster, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                        cudaStream_t stream, Args... args) {
  cudaLaunchAttribute attr[2]{};
  unsigned count = 0;
  if (overlap) {
    attr[count].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[count++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    attr[count].id = cudaLaunchAttributeClusterDimension;
    attr[count].val.clusterDim.x = unsigned(cluster);
    attr[count].val.clusterDim.y = attr[count].val.clusterDim.z = 1;
    ++count;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = count;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}
template <typename... Params, typename... Args>
cudaError_t launch_after(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                         Args... args) {
  return launch_with(true, 1, kernel, grid, block, smem, stream, args...);
}

}  // namespace cuda
}  // namespace hipress
