// complex64 row passes of run-time lengths (instantiations; dtmm_linef.cuh).
#include "dtmm_linef.cuh"

namespace dtmm {

template <int C, bool REAL>
static cudaError_t row_of(const LineLaunch& L, const RowParams& p, const Grid& g, const void* U, void* X) {
  if (L.maxl <= 16)
    return line_launch(k_row_linef<C, REAL, 16, 0, 0>, L, p, g, L.geom, L.lim, (const cpx<float>*)U, (cpx<float>*)X);
  return line_launch(k_row_linef<C, REAL, 32, 0, 0>, L, p, g, L.geom, L.lim, (const cpx<float>*)U, (cpx<float>*)X);
}

cudaError_t row_linef(int C, bool real, const LineLaunch& L, const RowParams& p, const Grid& g, const void* U, void* X) {
  if (real) {
#define DTMM_LINEF_ROW(A, B) \
  if (L.geom.n1 == A && L.geom.n2 == B) return row_linef_##A##_##B(C, L, p, g, U, X);
    DTMM_LINEF_SIDES(DTMM_LINEF_ROW)
#undef DTMM_LINEF_ROW
  }
  if (C == 4) return real ? row_of<4, true>(L, p, g, U, X) : row_of<4, false>(L, p, g, U, X);
  return real ? row_of<2, true>(L, p, g, U, X) : row_of<2, false>(L, p, g, U, X);
}

}  // namespace dtmm
