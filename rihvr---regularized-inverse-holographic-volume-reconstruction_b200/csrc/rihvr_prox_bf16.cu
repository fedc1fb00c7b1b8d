// The 2-D total-variation prox with BF16 storage.
#include "rihvr_prox.cuh"

namespace rihvr {

template cudaError_t prox_tv2d_stored<__nv_bfloat162>(const ProxArgs&, int*, cudaStream_t);

}  // namespace rihvr
