// xg_launch.cuh — launches that follow one another closely.
//
// A kernel launched with programmatic stream serialization starts its blocks
// as the last blocks of the kernel ahead of it in the stream leave, and opens
// with await_previous() for that kernel's memory: the launch costs its
// blocks' start, but not the gap before them (2 to 3.5 us each between small
// dependent kernels: a 1,000-stage chain's transient of 141 Newton iterations
// 21.2 to 17.7 ms).  What another kernel wrote is never read through
// __restrict__ or __ldg there, whose loads may be taken for constant over the
// kernel's life; what no kernel writes (schedules, patterns) may be read
// before the wait.  Every thread waits, so a kernel that has ended has seen
// all those ahead of it end.
#pragma once

#include <cuda_runtime.h>

#include "xg_internal.h"

namespace xg {

__device__ __forceinline__ void await_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launches a kernel that opens with await_previous; cluster > 0: in clusters
// of so many blocks.
template <class... P, class... A>
inline cudaError_t launch_close(void (*fn)(P...), int64_t grid, int threads, size_t smem, int cluster, cudaStream_t s,
                                A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(grid));
  cfg.blockDim = dim3(unsigned(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = unsigned(cluster);
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = cluster > 0 ? 2 : 1;
  count_launches(1);
  return cudaLaunchKernelEx(&cfg, fn, P(args)...);
}

}  // namespace xg
