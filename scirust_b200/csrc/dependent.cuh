// Programmatic dependent launch of the kernels that follow one another in a decode step.
//
// A kernel launched with the stream-serialization attribute may start while its predecessor in the stream still runs:
// as soon as every CTA of the predecessor has called pdl_trigger() or exited, and there is room on an SM. What does not
// depend on the predecessor (barrier set-up, tensor memory, bringing weights into L2) runs at once; pdl_wait() returns
// when the predecessor has completed and its writes are visible, and precedes every read and every write of global
// memory. Both are no-ops in a kernel that was launched without the attribute.
//
// Ahead of the wait, memory is only touched by L2 prefetches. L2 is where all SMs' reads and writes meet, so a prefetch
// cannot hand a stale value to a later load, and it is safe even where the predecessor writes the prefetched bytes.
//
// Rules for a kernel that triggers before it ends: every CTA waits (so that its completion implies that of all its
// predecessors); tensor memory is allocated before the trigger (a dependent CTA on the same SM could otherwise take the
// columns that this one still needs, and wait for it); pointers to what a predecessor may write are not __restrict__
// (such loads count as invariant and may be moved ahead of the wait).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace sb {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Brings one box of a 2-D tensor map into L2. The part of the box outside the tensor is skipped.
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* m, int c0, int c1) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(m)),
               "r"(c0), "r"(c1)
               : "memory");
}

bool dependent_launches();   // decode.cu: sb_set_pdl

// `dependent` false: plain stream order. cluster_y > 1: clusters of that many CTAs along the grid's y.
template <typename... KArgs, typename... Args>
static cudaError_t launch_dep_cluster(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                      int cluster_y, bool dependent, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = s;
  cudaLaunchAttribute at[2];
  int n = 0;
  if (dependent && dependent_launches()) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster_y > 1) {
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = 1; at[n].val.clusterDim.y = cluster_y; at[n++].val.clusterDim.z = 1;
  }
  cfg.attrs = at;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

template <typename... KArgs, typename... Args>
static cudaError_t launch_dep(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
  return launch_dep_cluster(kern, grid, block, smem, s, 1, true, args...);
}

}  // namespace sb
