// Register passes (dwt_strided.cuh): x passes of 8-bit rows of lengths without a kernel of their own.
#include "dwt_strided.cuh"

namespace wl {
WL_RAGGED_LAUNCH(strided_x_u8, uint8_t, kSource)
WL_RAGGED_LAUNCH(strided_x_inv_u8, uint8_t, kOutput)
}  // namespace wl
