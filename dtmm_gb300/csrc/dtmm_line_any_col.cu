// Fixed-point column passes and plain row transforms of run-time lengths
// (dtmm_linekern.cuh).
#include "dtmm_linekern.cuh"

namespace dtmm {

cudaError_t col_line_any(const LineLaunch& L, const ColParams& p, const Grid& g, const void* in, void* out) {
  return L.maxl <= 16 ? col_line_launch<16, 0, 0>(L, p, g, in, out) : col_line_launch<32, 0, 0>(L, p, g, in, out);
}

cudaError_t rows_line(const LineLaunch& L, const void* src, void* dst, int nlines, int W, bool inv, const void* tw,
                      double scale, int lpb) {
  return line_launch(L.maxl <= 16 ? k_rows_line<16> : k_rows_line<32>, L, (const cpx<double>*)src, (cpx<double>*)dst, nlines,
                     W, L.geom, (int)inv, (const cpx<double>*)tw, scale, lpb);
}

}  // namespace dtmm
