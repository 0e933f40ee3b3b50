// Strided Y/Z pass kernels, F32 path, forward sign.
#include "p3g_pipe_impl.cuh"

namespace p3g {
P3G_STRIDED_INSTANTIATE(PathF32, -1)
}  // namespace p3g
