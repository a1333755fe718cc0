// Register passes (dwt_strided.cuh): x passes of 32-bit integer rows.
#include "dwt_strided.cuh"

namespace wl {
WL_STRIDED_LAUNCH(strided_x_i32, int32_t, kSource)
WL_STRIDED_LAUNCH(strided_x_inv_i32, int32_t, kOutput)
}  // namespace wl
