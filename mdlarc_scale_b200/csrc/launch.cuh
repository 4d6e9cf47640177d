// Kernel launch helper: every kernel of the library is launched through arcb_launch(), which adds the
// programmatic-stream-serialization attribute when programmatic dependent launch is enabled.
//
// Protocol inside the kernels (common.cuh): pdl_launch_dependents() at entry lets the NEXT kernel in
// the stream (or captured graph) be scheduled as soon as every block of this one is resident, so its
// launch latency and its prologue (barrier initialisation, tensor-memory allocation, descriptor
// prefetch) overlap this kernel's tail; pdl_wait() returns only when the PREVIOUS kernel has
// completed and its writes are visible, and every kernel calls it before its first access to global
// memory other than its own parameters.  Because a grid completes only after the blocks that did its
// work have passed their own wait, completion is transitive along the stream: passing the wait on
// kernel N-1 implies kernels N-2, N-3, ... have completed too.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <utility>

bool arcb_pdl_enabled();
void arcb_pdl_set(bool on);
// Launches made by this thread while suppressed carry no programmatic attribute (used around the
// event-record nodes of the decode graph: a programmatic edge must join two kernel nodes).
void arcb_pdl_suppress(bool on);
bool arcb_pdl_suppressed();

// `cluster` > 1: CTAs x, x + 1, ... of the grid form clusters of that many (the kernel carries no cluster size of its own).
template <typename... KArgs, typename... Args>
inline cudaError_t arcb_launch_cluster(void (*kernel)(KArgs...), int cluster, dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                       Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  if (arcb_pdl_enabled() && !arcb_pdl_suppressed()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = n ? attr : nullptr;
  cfg.numAttrs = n;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
  if (e != cudaSuccess) cudaGetLastError();   // reported through the return value; do not leave it for the next API call
  return e;
}

template <typename... KArgs, typename... Args>
inline cudaError_t arcb_launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                               Args&&... args) {
  return arcb_launch_cluster(kernel, 1, grid, block, smem, stream, std::forward<Args>(args)...);
}

// Shared-memory opt-in of a kernel that needs more than the default 48 KB, at its first launch on a device (`done`: a bit each):
// doing it for all forms when an engine is created loads kernels that most programs never use (0.3 ms each).
template <typename K>
inline cudaError_t arcb_opt_in_smem(K kernel, int bytes, std::atomic<unsigned long long>& done) {
  if (bytes <= 48 * 1024) return cudaSuccess;
  int dev = 0;
  const unsigned long long bit = cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 ? 1ull << dev : 0;   // 0: every launch
  if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
  return e;
}
