// Batch kernel for the F32 path with 256-thread CTAs,
// plans without 6- and 7-point stages.
#include "p3g_batch_kernels.cuh"

namespace p3g {
P3G_BATCH_INSTANTIATE(PathF32, 256, false)
}  // namespace p3g
