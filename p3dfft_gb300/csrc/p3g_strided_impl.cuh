// Launchers of the strided pipelined kernels: one translation unit per path
// and direction (the unrolled codelets dominate the build time).
#pragma once

#include "p3g_pipe.cuh"

namespace p3g {

template <class P, int DIR>
cudaError_t launch_strided_pipe(const CUtensorMap* map, const CUtensorMap* omap, const SPipeParams& p,
                                const StagePlan* sp, const float4* tw, StridedMode mode, int threads, size_t smem, int grid,
                                cudaStream_t st) {
  auto kernel = k_strided_pipe<P, DIR, kStridedGeneral>;
  if (mode == kStridedFull) kernel = k_strided_pipe<P, DIR, kStridedFull>;
  if (mode == kStridedSmall) kernel = k_strided_pipe<P, DIR, kStridedSmall>;
  if constexpr (!P::kF64) {
    if (mode == kStridedFullWide) kernel = k_strided_pipe<P, DIR, kStridedFullWide>;
  }
  const cudaError_t e = opt_in_smem((const void*)kernel, 227 * 1024);
  if (e != cudaSuccess) return e;
  kernel<<<grid, threads, smem, st>>>(*map, *omap, p, sp, tw);
  return cudaGetLastError();
}

#define P3G_STRIDED_INSTANTIATE(P, DIR)                                                                       \
  template cudaError_t launch_strided_pipe<P, DIR>(const CUtensorMap*, const CUtensorMap*, const SPipeParams&, \
                                                   const StagePlan*, const float4*, StridedMode, int, size_t, int,    \
                                                   cudaStream_t);

}  // namespace p3g
