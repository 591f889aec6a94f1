// complex64 line passes of sides 100, 110, 120, 125, 135, 140, 150, 168
// (instantiations; dtmm_linef.cuh).
#include "dtmm_linef.cuh"

namespace dtmm {

DTMM_LINEF_DEFINE(10, 10)
DTMM_LINEF_DEFINE(10, 11)
DTMM_LINEF_DEFINE(10, 12)
DTMM_LINEF_DEFINE(5, 25)
DTMM_LINEF_DEFINE(9, 15)
DTMM_LINEF_DEFINE(10, 14)
DTMM_LINEF_DEFINE(10, 15)
DTMM_LINEF_DEFINE(12, 14)

}  // namespace dtmm
