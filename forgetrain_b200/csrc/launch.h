// Launch with programmatic stream serialization: the grid may start while the kernel in front of
// it on the stream is still finishing, as soon as every CTA of that one has run pdl_trigger() (or
// exited). Launch latency, barrier set-up, the TMEM allocation and the descriptor fetches then
// overlap the other kernel's tail instead of following it.
//
// Rule for every kernel launched this way: each thread calls pdl_wait() (ptx.cuh) before its
// first access to global memory. The wait returns when the kernel in front has COMPLETED, and
// that one has waited for its own predecessor in the same way, so the order of all memory accesses
// on the stream is what it is without overlap. Kernels that wait for other ranks (comm.cu,
// gemm_tp_sm100.cu) are launched plainly and never trigger: nothing may hold an SM behind them.
//
// Back-to-back launches of a one-tile GEMM: 4.3 us apart without, 3.25 us with it. Training steps: 8B
// geometry, 1 x 4096 tokens, 38.2 -> 37.3 ms; 0.5B, 3 x 1280 tokens, 18.1 -> 17.5 ms.
#pragma once
#include <cuda_runtime.h>

namespace ft {

template <class... P, class... A>
inline cudaError_t launch_pdl_cluster(void (*kernel)(P...), int cluster, int grid, int block,
                                      size_t smem, cudaStream_t st, const A&... args) {
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <class... P, class... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), int grid, int block, size_t smem,
                              cudaStream_t st, const A&... args) {
  return launch_pdl_cluster(kernel, 1, grid, block, smem, st, args...);
}

}  // namespace ft
