// Fixed-point line passes of sides 112, 135, 140, 168 (instantiations; the kernels are in
// dtmm_linekern.cuh).
#include "dtmm_linekern.cuh"

namespace dtmm {

DTMM_LINE_DEFINE(8, 14)
DTMM_LINE_DEFINE(9, 15)
DTMM_LINE_DEFINE(10, 14)
DTMM_LINE_DEFINE(12, 14)

}  // namespace dtmm
