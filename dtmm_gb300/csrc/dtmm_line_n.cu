// Fixed-point line passes of sides 432, 448, 480 (instantiations; the kernels are in
// dtmm_linekern.cuh).
#include "dtmm_linekern.cuh"

namespace dtmm {

DTMM_LINE_DEFINE(18, 24)
DTMM_LINE_DEFINE(16, 28)
DTMM_LINE_DEFINE(20, 24)

}  // namespace dtmm
