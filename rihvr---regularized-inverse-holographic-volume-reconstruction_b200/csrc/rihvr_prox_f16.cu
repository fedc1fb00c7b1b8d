// The 2-D total-variation prox with F16 storage.
#include "rihvr_prox.cuh"

namespace rihvr {

template cudaError_t prox_tv2d_stored<__half2>(const ProxArgs&, int*, cudaStream_t);

}  // namespace rihvr
