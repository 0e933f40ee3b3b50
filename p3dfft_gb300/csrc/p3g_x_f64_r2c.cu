// X r2c pass kernels, F64 path.
#include "p3g_pipe_impl.cuh"

namespace p3g {
P3G_X_INSTANTIATE(PathF64, true)
}  // namespace p3g
