// Register passes (dwt_strided.cuh): the y passes.
#include "dwt_strided.cuh"

namespace wl {
WL_STRIDED_LAUNCH(strided_y, float, kStrided)
WL_STRIDED_LAUNCH(strided_y_inv, float, kStridedInv)
}  // namespace wl
