// The 2-D total-variation prox with F32 storage.
#include "rihvr_prox.cuh"

namespace rihvr {

template cudaError_t prox_tv2d_stored<float2>(const ProxArgs&, int*, cudaStream_t);

}  // namespace rihvr
