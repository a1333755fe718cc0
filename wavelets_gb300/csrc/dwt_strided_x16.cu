// Register passes (dwt_strided.cuh): x passes of 16-bit rows.
#include "dwt_strided.cuh"

namespace wl {
WL_STRIDED_LAUNCH(strided_x_u16, uint16_t, kSource)
WL_STRIDED_LAUNCH(strided_x_inv_u16, uint16_t, kOutput)
}  // namespace wl
