// Programmatic dependent launch: a kernel launched with the stream-serialisation attribute may
// start while the kernel before it in the stream is still running. Its threads run up to
// `pdl_wait()`, which returns once every earlier kernel of the stream has finished and its
// writes are visible; what comes before the wait (barrier and TMEM set-up, tensor-map
// prefetch, loads of weights that no kernel writes) overlaps the earlier kernel's tail, and
// the launch latency disappears behind it. `pdl_trigger()` tells the scheduler that the next
// kernel of the stream may be placed; it is issued as early as the rules allow because the next
// kernel protects itself with its own wait.
//
// Rules every kernel launched through `launch_pdl` follows:
//   * no global write and no read of data another kernel produces before `pdl_wait()`. What a copy of the
//     host's has written ahead of the step's first kernel (an attention work list) and parameters may be
//     read: copies signal nothing early, so no kernel after one starts before it is done. A kernel of
//     this library must not write either: a kernel two places further on could read too soon;
//   * every thread that touches such data executes `pdl_wait()` first, and no block leaves before one of its
//     threads has (a kernel that has finished says that those before it have);
//   * `pdl_trigger()` comes behind the barrier that follows `tcgen05.alloc`. The allocation waits without a
//     limit. A block of the next kernel that shares the SM could otherwise take the columns first and then
//     wait for this kernel, which waits for them.
// A kernel launched without the attribute sees both instructions as no-ops, and a kernel
// launched with a plain <<<>>> after one of these waits for its full completion as usual.
#pragma once

#include <cuda_runtime.h>

#include <cstdlib>
#include <utility>

namespace ab200 {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// AB200_PDL=1 or 0 says so; otherwise on in a process that is the only rank. On one GPU, steps in us without
// and with: a text of 50 tokens embedded 910 and 719, decode of one request 579 and 558, of 128 requests 1485
// and 1469, drafts 876 and 863, 1024 short texts 12705 and 12210. With kernels that stored more, the serving
// benchmark on two GPUs lost 1 %: several ranks keep ordinary stream order. Without the attribute the two
// griddepcontrol instructions are no-ops.
inline bool pdl_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("AB200_PDL");
    if (e != nullptr) return e[0] == '1';
    const char* ranks = std::getenv("WORLD_SIZE");
    return ranks == nullptr || std::atoi(ranks) <= 1;
  }();
  return on;
}

// `cluster_x` > 1 launches thread-block clusters of that many consecutive blocks (grid.x must
// be a multiple of it).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl_cluster(void (*kernel)(KArgs...), dim3 grid, dim3 block,
                                      size_t smem, cudaStream_t stream, unsigned cluster_x,
                                      Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cluster_x > 1) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster_x;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(std::forward<Args>(args))...);
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                              cudaStream_t stream, Args&&... args) {
  return launch_pdl_cluster(kernel, grid, block, smem, stream, 1u, std::forward<Args>(args)...);
}

}  // namespace ab200
