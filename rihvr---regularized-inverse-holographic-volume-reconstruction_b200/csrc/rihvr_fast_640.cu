// Line FFT passes of the plane sides 640, 2304.
#include "rihvr_fast.cuh"

namespace rihvr {

RIHVR_FAST_SIDE(, 640)
RIHVR_FAST_SIDE(, 2304)

}  // namespace rihvr
