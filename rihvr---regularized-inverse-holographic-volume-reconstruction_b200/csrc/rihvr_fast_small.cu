// Line FFT passes of the plane sides 32, 48, 64, 128, 256.
#include "rihvr_fast.cuh"

namespace rihvr {

RIHVR_FAST_SIDE(, 32)
RIHVR_FAST_SIDE(, 48)
RIHVR_FAST_SIDE(, 64)
RIHVR_FAST_SIDE(, 128)
RIHVR_FAST_SIDE(, 256)

}  // namespace rihvr
