// Fixed-point line passes of sides 196, 210, 224 (instantiations; the kernels are in
// dtmm_linekern.cuh).
#include "dtmm_linekern.cuh"

namespace dtmm {

DTMM_LINE_DEFINE(14, 14)
DTMM_LINE_DEFINE(14, 15)
DTMM_LINE_DEFINE(14, 16)

}  // namespace dtmm
