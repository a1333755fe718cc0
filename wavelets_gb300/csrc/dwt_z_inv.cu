// Register passes (dwt_strided.cuh): the inverse z passes.
#include "dwt_strided.cuh"

namespace wl {
void strided_z_inv(const PassDesc *p, const int *tp, int n, int blocks, int L, cudaStream_t s) {
  launch_z<true, false>(p, tp, n, blocks, L, s);
}
}  // namespace wl
