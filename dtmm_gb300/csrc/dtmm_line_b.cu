// Fixed-point line passes of sides 100, 120, 150, 160 (instantiations; the kernels are in
// dtmm_linekern.cuh).
#include "dtmm_linekern.cuh"

namespace dtmm {

DTMM_LINE_DEFINE(10, 10)
DTMM_LINE_DEFINE(10, 12)
DTMM_LINE_DEFINE(10, 15)
DTMM_LINE_DEFINE(10, 16)

}  // namespace dtmm
