// Fixed-point line passes of sides 64, 80, 96, 128 (instantiations; the kernels are in
// dtmm_linekern.cuh).
#include "dtmm_linekern.cuh"

namespace dtmm {

DTMM_LINE_DEFINE(8, 8)
DTMM_LINE_DEFINE(8, 10)
DTMM_LINE_DEFINE(8, 12)
DTMM_LINE_DEFINE(8, 16)

}  // namespace dtmm
