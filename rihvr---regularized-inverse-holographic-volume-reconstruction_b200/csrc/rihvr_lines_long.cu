// The line FFT kernels with 24 elements a thread (rihvr_line_fft.cuh).
#include "rihvr_line_fft.cuh"

namespace rihvr {
namespace lines {

const LineKernels& long_kernels() {
  static const LineKernels k = make_kernels<kElemsLong>();
  return k;
}

}  // namespace lines
}  // namespace rihvr
