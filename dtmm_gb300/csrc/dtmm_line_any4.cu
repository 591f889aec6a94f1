// Fixed-point row passes of run-time lengths, 4 components (dtmm_linekern.cuh):
// the sides without kernels of their own, and complex operator records.
#include "dtmm_linekern.cuh"

namespace dtmm {

template <bool REAL>
static cudaError_t row_of(const LineLaunch& L, const RowParams& p, const Grid& g, const void* U, void* X) {
  return L.maxl <= 16 ? row_line_launch<4, REAL, 16, 0, 0>(L, p, g, U, X) : row_line_launch<4, REAL, 32, 0, 0>(L, p, g, U, X);
}

cudaError_t row_line_any4(bool real, const LineLaunch& L, const RowParams& p, const Grid& g, const void* U, void* X) {
  return real ? row_of<true>(L, p, g, U, X) : row_of<false>(L, p, g, U, X);
}

}  // namespace dtmm
