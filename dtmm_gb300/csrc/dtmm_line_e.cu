// Fixed-point line passes of sides 48, 50, 60, 72, 75, 90 (instantiations; the kernels are in
// dtmm_linekern.cuh).
#include "dtmm_linekern.cuh"

namespace dtmm {

DTMM_LINE_DEFINE(6, 8)
DTMM_LINE_DEFINE(5, 10)
DTMM_LINE_DEFINE(6, 10)
DTMM_LINE_DEFINE(8, 9)
DTMM_LINE_DEFINE(5, 15)
DTMM_LINE_DEFINE(9, 10)

}  // namespace dtmm
