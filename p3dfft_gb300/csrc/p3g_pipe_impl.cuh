// Launchers of the pipelined kernels: one translation unit per path and
// direction (the unrolled codelets dominate the build time).
#pragma once

#include <utility>

#include "p3g_pipe.cuh"

namespace p3g {

// Launch with programmatic stream serialization: the kernel may start while
// the one before it in the stream still runs, and waits (pass_begin) before it
// touches anything that kernel reads or writes.  Only for passes of few tiles
// per group, whose start is a good part of their time: the long binary32
// passes ran 4-8 % slower with it (1024^3 forward 6.28 -> 6.57 ms).
constexpr int kOverlapTiles = 16;
template <class... Params, class... Args>
cudaError_t launch_pass(void (*kernel)(Params...), const PipeCommon& pc, int grid, int threads, size_t smem,
                        cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = (long long)pc.ntiles <= (long long)kOverlapTiles * grid * pc.groups ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

template <class P, int DIR>
cudaError_t launch_strided_pipe(const CUtensorMap* map, const CUtensorMap* omap, const SPipeParams& p,
                                const float4* tw, TileMode mode, int threads, size_t smem, int grid,
                                cudaStream_t st) {
  auto kernel = k_strided_pipe<P, DIR, kTileGeneral>;
  if (mode == kTileFull) kernel = k_strided_pipe<P, DIR, kTileFull>;
  if (mode == kTileSmall) kernel = k_strided_pipe<P, DIR, kTileSmall>;
  if constexpr (!P::kF64) {
    if (mode == kTileFullWide) kernel = k_strided_pipe<P, DIR, kTileFullWide>;
  }
  const cudaError_t e = opt_in_smem((const void*)kernel, 227 * 1024);
  if (e != cudaSuccess) return e;
  return launch_pass(kernel, p.c, grid, threads, smem, st, *map, *omap, p, tw);
}

template <class P, bool R2C>
cudaError_t launch_x_pipe(const XPipeParams& p, const float4* tw, TileMode mode, int threads,
                          size_t smem, int grid, cudaStream_t st) {
  auto kernel = k_x_pipe<P, R2C, kTileGeneral>;
  if (mode == kTileSmall) kernel = k_x_pipe<P, R2C, kTileSmall>;
  constexpr TileMode kFull = P::kF64 ? kTileFull : kTileFullWide;  // the unguarded form that size_x gives
  if (mode == kFull) kernel = k_x_pipe<P, R2C, kFull>;
  const cudaError_t e = opt_in_smem((const void*)kernel, 227 * 1024);
  if (e != cudaSuccess) return e;
  return launch_pass(kernel, p.c, grid, threads, smem, st, p, tw);
}

#define P3G_X_INSTANTIATE(P, R2C)                                                                              \
  template cudaError_t launch_x_pipe<P, R2C>(const XPipeParams&, const float4*, TileMode, int, \
                                             size_t, int, cudaStream_t);
#define P3G_STRIDED_INSTANTIATE(P, DIR)                                                                       \
  template cudaError_t launch_strided_pipe<P, DIR>(const CUtensorMap*, const CUtensorMap*, const SPipeParams&, \
                                                   const float4*, TileMode, int, size_t, int,    \
                                                   cudaStream_t);

}  // namespace p3g
