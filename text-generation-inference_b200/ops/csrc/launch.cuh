// Kernel launch helper with optional programmatic dependent launch (PDL).
//
// A decode step is several hundred short kernels replayed from a CUDA graph.  With PDL a kernel is
// launched with the "programmatic stream serialization" attribute and starts with `pdl_wait()`, which
// blocks until the kernels it depends on have completed and flushed their memory; its launch and what it does before
// that overlap with their ends.  Nothing is read or written before `pdl_wait()`, so stream-order semantics are preserved (but for
// settled weights, see `pdl_release`).
//
// The attribute is always set on GEMMs that fetch settled weights; `TGI_B200_PDL=1` sets it on all launches, which gains next to
// nothing inside a graph, where launch gaps are already small.  Steps on B200 without / with it, us: 8B bf16 19 sequences
// 2185 / 2179, 201 sequences 5458 / 5453, 70B fp8 256 sequences 4403 / 4404 (8 layers), 8B 4-bit 12 sequences 1784 / 1769;
// over two GPUs, where kernels wait for the other rank's, it cost 2 to 3 % (70B fp8 34.8 / 35.4 ms, 8B 10.4 / 10.7).  Hence off by default.
// Without the attribute the device-side calls do nothing.
#pragma once
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>

namespace tgi {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Kernels trigger their dependents implicitly, when they end: with a trigger at entry everywhere the early CTAs take SM slots from
// later waves of the running kernel (a step of 19 sequences on an 8B model 2255 -> 2427 us).  This is the explicit trigger of the
// short kernels that a decode step's GEMMs follow (norm, activation, quantisation, decode attention): such a GEMM may be launched so
// that it fetches settled weights meanwhile (`launch_after`), and its CTAs take nothing that these kernels' later CTAs need, since all
// of those have started when the trigger takes effect.  Comes after `pdl_wait()`, so that what runs ahead of its own wait runs after
// everything but its direct predecessor.
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

inline bool pdl_enabled() {
  static const bool on = [] {
    const char* v = std::getenv("TGI_B200_PDL");
    return v != nullptr && std::strcmp(v, "1") == 0;
  }();
  return on;
}

// `early`: the kernel may be placed when all CTAs of its predecessor have triggered or ended; it calls `pdl_wait()` before it
// touches anything that the predecessor reads or writes.
template <typename... Params, typename... Args>
inline cudaError_t launch_after(bool early, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                          Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

template <typename... Params, typename... Args>
inline cudaError_t launch(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  return launch_after(pdl_enabled(), kernel, grid, block, smem, stream, args...);
}

// `launch_after` with an optional thread-block cluster of `cluster_x` CTAs along x (1 = no cluster attribute).
template <typename... Params, typename... Args>
inline cudaError_t launch_cluster_after(bool early, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                  int cluster_x, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (cluster_x > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster_x;
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (early) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

}  // namespace tgi
