// Fixed-point line passes of sides 175, 250, 350 (instantiations; the kernels are in
// dtmm_linekern.cuh).
#include "dtmm_linekern.cuh"

namespace dtmm {

DTMM_LINE_DEFINE(7, 25)
DTMM_LINE_DEFINE(10, 25)
DTMM_LINE_DEFINE(14, 25)

}  // namespace dtmm
