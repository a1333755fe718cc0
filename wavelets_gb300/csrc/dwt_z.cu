// Register passes (dwt_strided.cuh): the z passes without the select statistics.
#include "dwt_strided.cuh"

namespace wl {
void strided_z(const PassDesc *p, const int *tp, int n, int blocks, int L, cudaStream_t s) {
  launch_z<false, false>(p, tp, n, blocks, L, s);
}
}  // namespace wl
