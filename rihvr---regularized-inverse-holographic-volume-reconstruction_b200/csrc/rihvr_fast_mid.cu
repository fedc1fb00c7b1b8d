// Line FFT passes of the plane sides 384, 512.
#include "rihvr_fast.cuh"

namespace rihvr {

RIHVR_FAST_SIDE(, 384)
RIHVR_FAST_SIDE(, 512)

}  // namespace rihvr
