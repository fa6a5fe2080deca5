// Programmatic dependent launch for the kernels of the pipelines: a kernel
// launched with launch_dependent is set up and starts as soon as the last CTA
// of the kernel before it on the stream has left, instead of after that
// kernel's completion has gone through the stream.  It may read only its
// parameters and the context's constant tables until grid_wait() returns:
// then the kernel before it has completed and its writes are visible.  Every
// thread that touches memory which kernels write calls it first, and reads
// that memory with plain loads, never through __ldg, whose loads the compiler
// may move above the wait.
//
// One multiplication at level 22 (5 kernels) 98.8 -> 85.4 us, at level 7
// 55.4 -> 43.5.  No kernel lets its successor start earlier
// (griddepcontrol.launch_dependents): CTAs that arrive while others still run
// fill the free SMs unevenly, and the same calls took 87 to 102 and 48 to 71
// us, differently from run to run.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace chd {

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
inline void launch_dependent(void (*kern)(P...), dim3 grid, int block, size_t smem, cudaStream_t s, A &&...args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

// Launch parameters travel with every launch: a call on one ciphertext fills
// a few of a batch's descriptors.  18 KiB for them cost no time on the GPU but
// 1 us and more of the host's per launch.  Host time of a call, enqueued
// among others, in whole and in small batches: a plaintext product and rescale
// at level 5 19.6 and 15.1 us, one polynomial of 24 primes forward and inverse
// 22.1 and 16.2, one multiplication at level 22 22.9 and 18.0.  The GPU needs
// 16.3, 19.6 and 84.5 us for them, so the first two had waited for the host
// (20.4 and 22.9 us a call).
constexpr int kFewRows = 64, kFewJobs = 8;

}  // namespace chd
