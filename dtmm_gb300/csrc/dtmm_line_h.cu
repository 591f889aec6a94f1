// Fixed-point line passes of sides 200, 270, 280, 288 (instantiations; the kernels are in
// dtmm_linekern.cuh).
#include "dtmm_linekern.cuh"

namespace dtmm {

DTMM_LINE_DEFINE(10, 20)
DTMM_LINE_DEFINE(15, 18)
DTMM_LINE_DEFINE(14, 20)
DTMM_LINE_DEFINE(16, 18)

}  // namespace dtmm
