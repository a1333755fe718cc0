// Register passes (dwt_strided.cuh): x passes of float rows.
#include "dwt_strided.cuh"

namespace wl {
WL_STRIDED_LAUNCH(strided_x_f32, float, kSource)
WL_STRIDED_LAUNCH(strided_x_inv_f32, float, kOutput)
}  // namespace wl
