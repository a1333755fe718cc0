// Register passes (dwt_strided.cuh): x passes of float rows of lengths without a kernel of their own.
#include "dwt_strided.cuh"

namespace wl {
WL_RAGGED_LAUNCH(strided_x_f32, float, kSource)
WL_RAGGED_LAUNCH(strided_x_inv_f32, float, kOutput)
}  // namespace wl
