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
  // the 3-D TV prox's finish pass, a block a 64 x 8 tile at least: more than the
  // others on one tall plane (4200 blocks at 588 x 3360)
  return std::max({tv, strip, flat, prox6_partial_blocks(W, H, Nz)});
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

//
// Bound by memory (24 + s bytes a voxel).  A thread takes two adjacent voxels
// at a time (16-byte loads of FP32 storage; rows are of even length, so a pair
// lies in one row) and keeps its place in the plane by addition: one 64-bit
// modulo a voxel, for the restart weights, had cost as much as the loads
// (371 us at 512 x 512 x 200, FP32 with norms; 310 us here, 5.4 TB/s).
template <typename ST, bool NORMS>
__global__ void __launch_bounds__(FLAT_THREADS) k_prox_l1(ProxArgs a0) {
  const ProxArgs a = resolve_scalars(a0);
  const unsigned hw2 = (unsigned)a.W * (unsigned)a.H / 2;  // pairs of a plane
  const size_t n2 = (size_t)hw2 * a.Nz;
  const ST* P = static_cast<const ST*>(a.P);
  const ST* Pp = static_cast<const ST*>(a.Pprev);
  ST* Pn = static_cast<ST*>(a.Pnew);
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const unsigned step = (unsigned)(stride % hw2);
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned e2 = (unsigned)(i % hw2);  // pair within its plane
  double acc[kNumSums];
#pragma unroll
  for (int k = 0; k < kNumSums; ++k) acc[k] = 0.0;
#pragma unroll 2
  for (; i < n2; i += stride) {
    float2 y0[2], pp[2], g[2], p[2];
    Pair<ST>::ld(P + 2 * i, y0[0], y0[1]);
    Pair<ST>::ld(Pp + 2 * i, pp[0], pp[1]);
    Pair<float2>::ld(a.G + 2 * i, g[0], g[1]);
    float wr, wi;
    restart_w(2 * e2, a.faithful, &wr, &wi);  // an even place: both voxels are in the same 512
    e2 += step;
    if (e2 >= hw2) e2 -= hw2;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float2 x =
          make_float2(fmaf(a.beta, y0[c].x - pp[c].x, y0[c].x), fmaf(a.beta, y0[c].y - pp[c].y, y0[c].y));
      const float2 xh = make_float2(fmaf(-a.t, g[c].x, x.x), fmaf(-a.t, g[c].y, x.y));
      p[c] = shrink(xh, a.thr, a.faithful);
      const float2 d = csub(p[c], x);
      acc[SUM_LIM1] += (double)(d.x * g[c].x) + (double)(d.y * g[c].y);
      acc[SUM_LIM2] += (double)cabs2(d);
      const float2 u = csub(x, p[c]), v = csub(p[c], y0[c]);
      acc[SUM_RS] += (double)(wr * u.x * v.x) + (double)(wi * u.y * v.y);
      if (NORMS) {
        acc[SUM_L1P] += (double)norm_sqrt(cabs2(p[c]));
        acc[SUM_L1X] += (double)norm_sqrt(cabs2(x));
      }
    }
    Raw2<ST>::st(Pn + 2 * i, p[0], p[1]);
  }
  block_write_sums<FLAT_THREADS>(acc, a.partials, blockIdx.x);
}

template <typename ST>
static void prox_l1_launch(const ProxArgs& a, int blocks, cudaStream_t st) {
  if (a.want_norms) k_prox_l1<ST, true><<<blocks, FLAT_THREADS, 0, st>>>(a);
  else k_prox_l1<ST, false><<<blocks, FLAT_THREADS, 0, st>>>(a);
}

cudaError_t launch_prox_l1(int storage, const ProxArgs& a, int* nblocks_out, cudaStream_t st) {
  const int blocks = flat_blocks((size_t)a.W * a.H * a.Nz / 2);
  *nblocks_out = blocks;
  switch (storage) {
    case STORE_BF16: prox_l1_launch<__nv_bfloat162>(a, blocks, st); break;
    case STORE_F16: prox_l1_launch<__half2>(a, blocks, st); break;
    default: prox_l1_launch<float2>(a, blocks, st);
  }
  return cudaGetLastError();
}

}  // namespace rihvr
