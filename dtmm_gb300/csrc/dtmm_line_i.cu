// Fixed-point line passes of sides 300, 320, 400 (instantiations; the kernels are in
// dtmm_linekern.cuh).
#include "dtmm_linekern.cuh"

namespace dtmm {

DTMM_LINE_DEFINE(15, 20)
DTMM_LINE_DEFINE(16, 20)
DTMM_LINE_DEFINE(20, 20)

}  // namespace dtmm
