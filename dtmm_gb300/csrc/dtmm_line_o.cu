// Fixed-point line passes of sides 1024 (instantiations; the kernels are in
// dtmm_linekern.cuh).
#include "dtmm_linekern.cuh"

namespace dtmm {

DTMM_LINE_DEFINE(32, 32)

}  // namespace dtmm
