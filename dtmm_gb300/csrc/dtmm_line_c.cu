// Fixed-point line passes of sides 144, 180, 192 (instantiations; the kernels are in
// dtmm_linekern.cuh).
#include "dtmm_linekern.cuh"

namespace dtmm {

DTMM_LINE_DEFINE(12, 12)
DTMM_LINE_DEFINE(12, 15)
DTMM_LINE_DEFINE(12, 16)

}  // namespace dtmm
