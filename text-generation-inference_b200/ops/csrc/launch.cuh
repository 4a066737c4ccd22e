// Kernel launch helper with optional programmatic dependent launch (PDL).
//
// A decode step is several hundred short kernels replayed from a CUDA graph.  With PDL a kernel is
// launched with the "programmatic stream serialization" attribute and starts with `pdl_wait()` (which
// blocks until the kernels it depends on have completed and flushed their memory) followed by
// `pdl_trigger()`, so the next kernel's CTAs can be placed on the SMs while this one is still
// running.  Nothing is read or written before `pdl_wait()`, so stream-order semantics are preserved (but for settled weights,
// see `pdl_release`).
//
// Measured on B200 (CUDA-graph decode step): Llama-3-70B fp8 at TP=1 56.6 ms with PDL against 56.4 ms
// without, TP=2 35.4 against 34.8 ms, Llama-3-8B bf16 at TP=2 10.7 against 10.4 ms.  Inside a graph the
// launch gaps are already small and the early-placed CTAs only take resources, so the attribute is
// OFF by default; `TGI_B200_PDL=1` switches it on (the device-side calls are no-ops without it).
#pragma once
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>

namespace tgi {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Early trigger: lets the dependent grid be placed while this one still runs.  Measured slower (the early CTAs
// take SM slots from later waves of the running kernel), so by default the trigger is the implicit one at CTA
// exit and only the launch latency and the prologue of the next kernel overlap with this kernel's tail.
__device__ __forceinline__ void pdl_trigger() {
#ifdef TGI_PDL_EARLY_TRIGGER
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#endif
}

// The trigger of the short kernels that a decode step's GEMMs follow (norm, activation, quantisation, decode attention): such a
// GEMM may be launched so that it fetches settled weights meanwhile (`launch_after`), and its CTAs take nothing that these
// kernels' later CTAs need, since all of those have started when the trigger takes effect.  Comes after `pdl_wait()`, so that what
// runs ahead of its own wait runs after everything but its direct predecessor.
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
