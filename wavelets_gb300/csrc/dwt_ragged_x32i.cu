// Register passes (dwt_strided.cuh): x passes of 32-bit integer rows of lengths without a kernel of their own.
#include "dwt_strided.cuh"

namespace wl {
WL_RAGGED_LAUNCH(strided_x_i32, int32_t, kSource)
WL_RAGGED_LAUNCH(strided_x_inv_i32, int32_t, kOutput)
}  // namespace wl
