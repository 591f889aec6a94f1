// complex64 line passes of sides 45, 48, 50, 60, 63, 72, 75, 90
// (instantiations; dtmm_linef.cuh).
#include "dtmm_linef.cuh"

namespace dtmm {

DTMM_LINEF_DEFINE(5, 9)
DTMM_LINEF_DEFINE(6, 8)
DTMM_LINEF_DEFINE(5, 10)
DTMM_LINEF_DEFINE(6, 10)
DTMM_LINEF_DEFINE(7, 9)
DTMM_LINEF_DEFINE(8, 9)
DTMM_LINEF_DEFINE(5, 15)
DTMM_LINEF_DEFINE(9, 10)

}  // namespace dtmm
