// Register passes (dwt_strided.cuh): x passes of 16-bit rows of lengths without a kernel of their own.
#include "dwt_strided.cuh"

namespace wl {
WL_RAGGED_LAUNCH(strided_x_u16, uint16_t, kSource)
WL_RAGGED_LAUNCH(strided_x_inv_u16, uint16_t, kOutput)
}  // namespace wl
