// Programmatic dependent launch for kernels that follow one another on a stream: the next kernel's CTAs come up (barriers,
// TMEM, shared memory) while the last CTAs of the one before still run, and pdlWait() holds every thread until that kernel
// has finished and its writes are visible.  A kernel launched with launchPdl calls pdlWait() before its first access to
// global memory, reads and writes alike; behind anything but a kernel that calls pdlRelease() the wait is an ordinary
// stream dependency.
//
// The pointer parameters of such a kernel carry no __restrict__: what they point to may still be written, by the kernel
// before, while this one is resident.  For a `const ... __restrict__` pointer the compiler may use the non-coherent load
// path, which is for memory that nobody writes while the kernel lives, and may move a load across the wait.
//
// A kernel that allocates TMEM calls pdlRelease() after its allocation: a successor that allocated first would hold the
// columns while it waits for this kernel, which waits for the columns.
#pragma once
#include <cuda_runtime.h>

namespace fcxpdl {

__device__ __forceinline__ void pdlRelease() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdlWait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// `cluster`: CTAs per cluster, or {0, 0, 0} for a kernel that has none or sets its own.
template <typename... Params, typename... Args>
inline cudaError_t launchPdlAttr(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, dim3 cluster, cudaStream_t s, Args &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster.x;
  attr[1].val.clusterDim.y = cluster.y;
  attr[1].val.clusterDim.z = cluster.z;
  cfg.attrs = attr;
  cfg.numAttrs = cluster.x ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

template <typename... Params, typename... Args>
inline cudaError_t launchPdl(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args &&...args) {
  return launchPdlAttr(kernel, grid, block, smem, dim3(0, 0, 0), s, static_cast<Args &&>(args)...);
}

template <typename... Params, typename... Args>
inline cudaError_t launchPdlCluster(void (*kernel)(Params...), dim3 grid, dim3 block, dim3 cluster, cudaStream_t s, Args &&...args) {
  return launchPdlAttr(kernel, grid, block, 0, cluster, s, static_cast<Args &&>(args)...);
}

}  // namespace fcxpdl
