// Register passes (dwt_strided.cuh): the y passes of lengths without a kernel of their own.
#include "dwt_strided.cuh"

namespace wl {
WL_RAGGED_LAUNCH(strided_y, float, kStrided)
WL_RAGGED_LAUNCH(strided_y_inv, float, kStridedInv)
}  // namespace wl
