// complex64 column passes and plain row transforms of run-time lengths
// (instantiations; dtmm_linef.cuh).
#include "dtmm_linef.cuh"

namespace dtmm {

cudaError_t col_linef(const LineLaunch& L, const ColParams& p, const Grid& g, const void* in, void* out) {
#define DTMM_LINEF_COL(A, B) \
  if (L.geom.n1 == A && L.geom.n2 == B) return col_linef_##A##_##B(L, p, g, in, out);
  DTMM_LINEF_SIDES(DTMM_LINEF_COL)
#undef DTMM_LINEF_COL
  if (L.maxl <= 16)
    return line_launch(k_col_linef<16, 0, 0>, L, p, g, L.geom, L.lim, (const cpx<float>*)in, (cpx<float>*)out);
  return line_launch(k_col_linef<32, 0, 0>, L, p, g, L.geom, L.lim, (const cpx<float>*)in, (cpx<float>*)out);
}

cudaError_t rows_linef(const LineLaunch& L, const void* src, void* dst, int nlines, int W, bool inv, const void* tw,
                       double scale, int lpb) {
  return line_launch(L.maxl <= 16 ? k_rows_linef<16> : k_rows_linef<32>, L, (const cpx<float>*)src, (cpx<float>*)dst, nlines,
                     W, L.geom, (int)inv, (const cpx<float>*)tw, (float)scale, lpb);
}

}  // namespace dtmm
