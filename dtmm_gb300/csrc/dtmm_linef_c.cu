// complex64 line passes of sides 175, 180, 196, 200, 210, 220, 225, 250
// (instantiations; dtmm_linef.cuh).
#include "dtmm_linef.cuh"

namespace dtmm {

DTMM_LINEF_DEFINE(7, 25)
DTMM_LINEF_DEFINE(12, 15)
DTMM_LINEF_DEFINE(14, 14)
DTMM_LINEF_DEFINE(10, 20)
DTMM_LINEF_DEFINE(14, 15)
DTMM_LINEF_DEFINE(11, 20)
DTMM_LINEF_DEFINE(15, 15)
DTMM_LINEF_DEFINE(10, 25)

}  // namespace dtmm
