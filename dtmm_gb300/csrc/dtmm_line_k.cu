// Fixed-point line passes of sides 45, 63, 110, 125, 220 (instantiations; the kernels are in
// dtmm_linekern.cuh).
#include "dtmm_linekern.cuh"

namespace dtmm {

DTMM_LINE_DEFINE(5, 9)
DTMM_LINE_DEFINE(7, 9)
DTMM_LINE_DEFINE(10, 11)
DTMM_LINE_DEFINE(5, 25)
DTMM_LINE_DEFINE(11, 20)

}  // namespace dtmm
