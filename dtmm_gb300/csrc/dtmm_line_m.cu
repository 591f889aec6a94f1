// Fixed-point line passes of sides 330, 336, 352, 360 (instantiations; the kernels are in
// dtmm_linekern.cuh).
#include "dtmm_linekern.cuh"

namespace dtmm {

DTMM_LINE_DEFINE(15, 22)
DTMM_LINE_DEFINE(16, 21)
DTMM_LINE_DEFINE(16, 22)
DTMM_LINE_DEFINE(18, 20)

}  // namespace dtmm
