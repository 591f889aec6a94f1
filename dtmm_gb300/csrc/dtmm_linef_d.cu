// complex64 line passes of sides 270, 280, 300, 330, 350, 352, 360
// (instantiations; dtmm_linef.cuh).
#include "dtmm_linef.cuh"

namespace dtmm {

DTMM_LINEF_DEFINE(15, 18)
DTMM_LINEF_DEFINE(14, 20)
DTMM_LINEF_DEFINE(15, 20)
DTMM_LINEF_DEFINE(15, 22)
DTMM_LINEF_DEFINE(14, 25)
DTMM_LINEF_DEFINE(16, 22)
DTMM_LINEF_DEFINE(18, 20)

}  // namespace dtmm
