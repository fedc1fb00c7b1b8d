// Dispatch of the 2-D total-variation prox (mode 7) over the storage types and
// the prox of mode 5 (sparsity alone), with the sums of the line search, the
// restart test and the objective.
#include <algorithm>

#include "rihvr_device.cuh"
#include "rihvr_kernels.cuh"
#include "rihvr_launch.cuh"
#include "rihvr_prox.cuh"

namespace rihvr {

extern template cudaError_t prox_tv2d_stored<float2>(const ProxArgs&, int*, cudaStream_t);
extern template cudaError_t prox_tv2d_stored<__nv_bfloat162>(const ProxArgs&, int*, cudaStream_t);
extern template cudaError_t prox_tv2d_stored<__half2>(const ProxArgs&, int*, cudaStream_t);

size_t max_partial_blocks(int W, int H, int Nz) {
  // the tiled TV prox with the largest halo it accepts (n_tv <= 20)
  const int h = 21, VW = TV_EW - 2 * h, VH = TV_EH - 2 * h;
  const size_t tv = (size_t)((W + VW - 1) / VW) * ((H + VH - 1) / VH) * Nz;
  // the streaming TV prox with its narrowest strips (n_tv = 10) and the most
  // runs per plane (64), one block per run
  using Sh = TvwShape<kStripNtvMax, 2>;
  const size_t strip = (size_t)((W + Sh::VW - 1) / Sh::VW) * (size_t)std::min(64, H) * Nz;
  const size_t flat = 4096;
  return std::max(std::max(tv, strip), flat);
}

cudaError_t launch_prox_tv2d(int storage, const ProxArgs& a, int* nblocks_out, cudaStream_t st) {
  switch (storage) {
    case STORE_BF16: return prox_tv2d_stored<__nv_bfloat162>(a, nblocks_out, st);
    case STORE_F16: return prox_tv2d_stored<__half2>(a, nblocks_out, st);
    default: return prox_tv2d_stored<float2>(a, nblocks_out, st);
  }
}

// ---------------------------------------------------------------------------
// Elementwise prox (mode 5): proximalL1, sparse_compressive_holo.cu:3274-3392,
// p = shrink(x - t g, t l1), plus the same sums (TV terms absent).
// ---------------------------------------------------------------------------

template <typename ST>
__global__ void __launch_bounds__(FLAT_THREADS) k_prox_l1(ProxArgs a0) {
  const ProxArgs a = resolve_scalars(a0);
  const size_t HW = (size_t)a.W * a.H, n = HW * a.Nz;
  const ST* P = static_cast<const ST*>(a.P);
  const ST* Pp = static_cast<const ST*>(a.Pprev);
  ST* Pn = static_cast<ST*>(a.Pnew);
  double acc[kNumSums];
#pragma unroll
  for (int k = 0; k < kNumSums; ++k) acc[k] = 0.0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float2 y0 = Store<ST>::ld(P + i), pp = Store<ST>::ld(Pp + i), g = a.G[i];
    const float2 x = make_float2(fmaf(a.beta, y0.x - pp.x, y0.x), fmaf(a.beta, y0.y - pp.y, y0.y));
    const float2 xh = make_float2(fmaf(-a.t, g.x, x.x), fmaf(-a.t, g.y, x.y));
    const float2 p = shrink(xh, a.thr, a.faithful);
    Store<ST>::st(Pn + i, p);
    const float2 d = csub(p, x);
    acc[SUM_LIM1] += (double)(d.x * g.x) + (double)(d.y * g.y);
    acc[SUM_LIM2] += (double)cabs2(d);
    float wr, wi;
    restart_w(i % HW, a.faithful, &wr, &wi);
    const float2 u = csub(x, p), v = csub(p, y0);
    acc[SUM_RS] += (double)(wr * u.x * v.x) + (double)(wi * u.y * v.y);
    if (a.want_norms) {
      acc[SUM_L1P] += (double)norm_sqrt(cabs2(p));
      acc[SUM_L1X] += (double)norm_sqrt(cabs2(x));
    }
  }
  block_write_sums<FLAT_THREADS>(acc, a.partials, blockIdx.x);
}

cudaError_t launch_prox_l1(int storage, const ProxArgs& a, int* nblocks_out, cudaStream_t st) {
  const int blocks = flat_blocks((size_t)a.W * a.H * a.Nz);
  *nblocks_out = blocks;
  switch (storage) {
    case STORE_BF16:
      k_prox_l1<__nv_bfloat162><<<blocks, FLAT_THREADS, 0, st>>>(a);
      break;
    case STORE_F16:
      k_prox_l1<__half2><<<blocks, FLAT_THREADS, 0, st>>>(a);
      break;
    default:
      k_prox_l1<float2><<<blocks, FLAT_THREADS, 0, st>>>(a);
  }
  return cudaGetLastError();
}

}  // namespace rihvr
