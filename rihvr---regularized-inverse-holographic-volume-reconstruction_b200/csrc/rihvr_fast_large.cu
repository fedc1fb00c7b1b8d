// Line FFT passes of the plane sides 768, 1024.
#include "rihvr_fast.cuh"

namespace rihvr {

RIHVR_FAST_SIDE(, 768)
RIHVR_FAST_SIDE(, 1024)

}  // namespace rihvr
