// X r2c pass kernels, F32 path.
#include "p3g_pipe_impl.cuh"

namespace p3g {
P3G_X_INSTANTIATE(PathF32, true)
}  // namespace p3g
