// Fixed-point line passes of sides 225, 240, 256 (instantiations; the kernels are in
// dtmm_linekern.cuh).
#include "dtmm_linekern.cuh"

namespace dtmm {

DTMM_LINE_DEFINE(15, 15)
DTMM_LINE_DEFINE(15, 16)
DTMM_LINE_DEFINE(16, 16)

}  // namespace dtmm
