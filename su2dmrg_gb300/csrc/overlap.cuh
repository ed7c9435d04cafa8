// Launches whose start overlaps the end of the kernel before them in the stream
// (programmatic dependent launch).  A kernel launched by launch_overlapped may
// start once every CTA of its predecessor has called dependents_may_start() or
// ended; it waits in wait_for_predecessor() until the predecessor has completed
// and its writes are visible.  Between the two it may read what no kernel
// writes (work lists) and nothing else.
//
// Every CTA calls wait_for_predecessor() before it ends, so that a kernel's
// completion implies that of all before it.  The wait returns a zero the
// compiler does not know, and pointers to data that kernels write get it added
// (after_wait): their loads cannot then be moved above the wait.  Such data is
// read with plain loads only: a read-only one (__ldg) asks that nothing writes
// the data while the reading grid exists, and this grid exists while its
// predecessor still writes.
//
// What it saves is the gap between kernels, launch latency and prologue: an
// application at D = 40 (two FP64 launches) takes 9 us instead of 14, at D =
// 200 (six split launches) 48 instead of 61, at D = 777 237 instead of 260.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace su2g {

__device__ __forceinline__ void dependents_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ int64_t wait_for_predecessor() {
  int64_t zero;
  asm volatile("griddepcontrol.wait;\n mov.b64 %0, 0;" : "=l"(zero)::"memory");
  return zero;
}
template <class T>
__device__ __forceinline__ T* after_wait(T* p, int64_t zero) {
  return p + zero;
}
// cluster: CTAs of a cluster along x (0: none)
template <class... P, class... A>
cudaError_t launch_overlapped(void (*kernel)(P...), dim3 grid, int threads, size_t smem, int cluster,
                              cudaStream_t stream, A... args) {
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 0 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, (P)args...);
}

}  // namespace su2g
