// Launches with programmatic stream serialization: the grid is scheduled as the last CTAs of
// the kernel before it leave, and waits for that kernel's memory before it touches any. What
// it saves is the gap between dependent launches, a microsecond or so, a good part of the time
// at small bonds: U(1) DMRG call 26.7 -> 23.5 ms, QR of 1024 x 512 4.85 -> 4.29 ms, H_eff at
// bonds 250 x 256 135 -> 119 us. No kernel lets its successor in earlier: CTAs that wait where
// others still run end up stacked on the SMs that had room first (H_eff 135 -> 160 us, DMMA
// GEMM of bond 64 30 -> 45 us with the trigger at the start of every kernel).
// Every kernel launched through here calls grid_wait() first thing in every thread that
// reads or writes global memory, and never exits without it: then the completion of a grid
// implies that of all grids before it in the stream. Kernels launched otherwise keep the
// full dependency on both sides.
#pragma once

#include <cuda_runtime.h>
#include <utility>

namespace ptn {

// waits for the grids this one depends on
__device__ __forceinline__ void grid_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

struct LaunchShape {
  dim3 grid, block;
  size_t smem;
  dim3 cluster{0, 0, 0};   // 0: no cluster
};

template <typename... P, typename... A>
cudaError_t launch_shape(void (*kernel)(P...), const LaunchShape& s, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = s.grid;
  cfg.blockDim = s.block;
  cfg.dynamicSmemBytes = s.smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = s.cluster.x;
  attr[1].val.clusterDim.y = s.cluster.y;
  attr[1].val.clusterDim.z = s.cluster.z;
  cfg.attrs = attr;
  cfg.numAttrs = s.cluster.x != 0 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <typename... P, typename... A>
cudaError_t launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                   A... args) {
  return launch_shape(kernel, LaunchShape{grid, block, smem}, st, args...);
}

}  // namespace ptn
