// Fixed-point line passes of sides 384, 512, 640 (instantiations; the kernels are in
// dtmm_linekern.cuh).
#include "dtmm_linekern.cuh"

namespace dtmm {

DTMM_LINE_DEFINE(16, 24)
DTMM_LINE_DEFINE(16, 32)
DTMM_LINE_DEFINE(20, 32)

}  // namespace dtmm
