// 3-D fused lasso prox (mode 6).
#include "rihvr_device.cuh"
#include "rihvr_kernels.cuh"
#include "rihvr_launch.cuh"

namespace rihvr {

// ---------------------------------------------------------------------------
// 3-D fused lasso (mode 6): proximalFusedLasso (:3422-3475) with
// totalVariationProjection (:3832-4018): half threshold, n_tv unnormalised dual
// steps over the whole volume (periodic in x, y, z; the projection is disabled
// at :3964), final estimate, half threshold.
// ---------------------------------------------------------------------------
template <typename ST>
__global__ void k_prox6_init(ProxArgs a, float2* __restrict__ X1) {
  const size_t n = (size_t)a.W * a.H * a.Nz;
  const ST* P = static_cast<const ST*>(a.P);
  const ST* Pp = static_cast<const ST*>(a.Pprev);
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float2 x = xval(P, Pp, a.beta, i), g = a.G[i];
    const float2 xh = make_float2(fmaf(-a.t, g.x, x.x), fmaf(-a.t, g.y, x.y));
    X1[i] = shrink(xh, 0.5f * a.thr, a.faithful);
  }
}

cudaError_t launch_prox6_init(int storage, const ProxArgs& a, float2* X1, cudaStream_t st) {
  const int blocks = flat_blocks((size_t)a.W * a.H * a.Nz);
  switch (storage) {
    case STORE_BF16:
      k_prox6_init<__nv_bfloat162><<<blocks, FLAT_THREADS, 0, st>>>(a, X1);
      break;
    case STORE_F16:
      k_prox6_init<__half2><<<blocks, FLAT_THREADS, 0, st>>>(a, X1);
      break;
    default:
      k_prox6_init<float2><<<blocks, FLAT_THREADS, 0, st>>>(a, X1);
  }
  return cudaGetLastError();
}

__global__ void k_tv3_estimate(const float2* __restrict__ X1, const float2* __restrict__ gx,
                               const float2* __restrict__ gy, const float2* __restrict__ gz, float2* __restrict__ Y,
                               int W, int H, int Nz, float mu) {
  const size_t HW = (size_t)W * H, n = HW * Nz;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int z = (int)(i / HW);
    const size_t e = i - (size_t)z * HW;
    const int yy = (int)(e / W), xx = (int)(e - (size_t)yy * W);
    const int xp = xx < W - 1 ? xx + 1 : 0, yp = yy < H - 1 ? yy + 1 : 0, zp = z < Nz - 1 ? z + 1 : 0;
    const float2 d1 = csub(gx[(size_t)z * HW + (size_t)yy * W + xp], gx[i]);
    const float2 d2 = csub(gy[(size_t)z * HW + (size_t)yp * W + xx], gy[i]);
    const float2 d3 = csub(gz[(size_t)zp * HW + e], gz[i]);
    const float2 dv = cadd(cadd(d1, d2), d3);
    Y[i] = make_float2(fmaf(-mu, dv.x, X1[i].x), fmaf(-mu, dv.y, X1[i].y));
  }
}

cudaError_t launch_tv3_estimate(const float2* X1, const float2* gx, const float2* gy, const float2* gz, float2* Y,
                                int W, int H, int Nz, float mu, cudaStream_t st) {
  k_tv3_estimate<<<flat_blocks((size_t)W * H * Nz), FLAT_THREADS, 0, st>>>(X1, gx, gy, gz, Y, W, H, Nz, mu);
  return cudaGetLastError();
}

__global__ void k_tv3_dual(const float2* __restrict__ Y, float2* gx, float2* gy, float2* gz, int W, int H, int Nz,
                           float s) {
  const size_t HW = (size_t)W * H, n = HW * Nz;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int z = (int)(i / HW);
    const size_t e = i - (size_t)z * HW;
    const int yy = (int)(e / W), xx = (int)(e - (size_t)yy * W);
    const int xm = xx > 0 ? xx - 1 : W - 1, ym = yy > 0 ? yy - 1 : H - 1, zm = z > 0 ? z - 1 : Nz - 1;
    const float2 yv = Y[i];
    const float2 a1 = csub(Y[(size_t)z * HW + (size_t)yy * W + xm], yv);
    const float2 a2 = csub(Y[(size_t)z * HW + (size_t)ym * W + xx], yv);
    const float2 a3 = csub(Y[(size_t)zm * HW + e], yv);
    gx[i] = make_float2(fmaf(s, a1.x, gx[i].x), fmaf(s, a1.y, gx[i].y));
    gy[i] = make_float2(fmaf(s, a2.x, gy[i].x), fmaf(s, a2.y, gy[i].y));
    gz[i] = make_float2(fmaf(s, a3.x, gz[i].x), fmaf(s, a3.y, gz[i].y));
  }
}

cudaError_t launch_tv3_dual(const float2* Y, float2* gx, float2* gy, float2* gz, int W, int H, int Nz, float s,
                            cudaStream_t st) {
  k_tv3_dual<<<flat_blocks((size_t)W * H * Nz), FLAT_THREADS, 0, st>>>(Y, gx, gy, gz, W, H, Nz, s);
  return cudaGetLastError();
}

template <typename ST>
__global__ void __launch_bounds__(FLAT_THREADS) k_prox6_finish(ProxArgs a, const float2* __restrict__ Y) {
  const int W = a.W, H = a.H, Nz = a.Nz;
  const size_t HW = (size_t)W * H, n = HW * Nz;
  const ST* P = static_cast<const ST*>(a.P);
  const ST* Pp = static_cast<const ST*>(a.Pprev);
  ST* Pn = static_cast<ST*>(a.Pnew);
  const float T = 0.5f * a.thr;
  double acc[kNumSums];
#pragma unroll
  for (int k = 0; k < kNumSums; ++k) acc[k] = 0.0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int z = (int)(i / HW);
    const size_t e = i - (size_t)z * HW;
    const int yy = (int)(e / W), xx = (int)(e - (size_t)yy * W);
    const float2 p = shrink(Y[i], T, a.faithful);
    Store<ST>::st(Pn + i, p);
    const float2 y0 = Store<ST>::ld(P + i);
    const float2 x = xval(P, Pp, a.beta, i), g = a.G[i];
    const float2 d = csub(p, x);
    acc[SUM_LIM1] += (double)(d.x * g.x) + (double)(d.y * g.y);
    acc[SUM_LIM2] += (double)cabs2(d);
    float wr, wi;
    restart_w(e, a.faithful, &wr, &wi);
    const float2 u = csub(x, p), v = csub(p, y0);
    acc[SUM_RS] += (double)(wr * u.x * v.x) + (double)(wi * u.y * v.y);
    if (a.want_norms) {
      const int xm = xx > 0 ? xx - 1 : W - 1, ym = yy > 0 ? yy - 1 : H - 1, zm = z > 0 ? z - 1 : Nz - 1;
      const size_t il = (size_t)z * HW + (size_t)yy * W + xm, iu = (size_t)z * HW + (size_t)ym * W + xx,
                   ib = (size_t)zm * HW + e;
      const float2 pl = shrink(Y[il], T, a.faithful), pu = shrink(Y[iu], T, a.faithful),
                   pb = shrink(Y[ib], T, a.faithful);
      acc[SUM_L1P] += (double)norm_sqrt(cabs2(p));
      acc[SUM_TVP] += (double)norm_sqrt(cabs2(csub(pl, p)) + cabs2(csub(pu, p)) + cabs2(csub(pb, p)));
      const float2 xl = xval(P, Pp, a.beta, il), xu = xval(P, Pp, a.beta, iu), xb = xval(P, Pp, a.beta, ib);
      acc[SUM_L1X] += (double)norm_sqrt(cabs2(x));
      acc[SUM_TVX] += (double)norm_sqrt(cabs2(csub(xl, x)) + cabs2(csub(xu, x)) + cabs2(csub(xb, x)));
    }
  }
  block_write_sums<FLAT_THREADS>(acc, a.partials, blockIdx.x);
}

cudaError_t launch_prox6_finish(int storage, const ProxArgs& a, const float2* Y, int* nblocks_out, cudaStream_t st) {
  const int blocks = flat_blocks((size_t)a.W * a.H * a.Nz);
  *nblocks_out = blocks;
  switch (storage) {
    case STORE_BF16:
      k_prox6_finish<__nv_bfloat162><<<blocks, FLAT_THREADS, 0, st>>>(a, Y);
      break;
    case STORE_F16:
      k_prox6_finish<__half2><<<blocks, FLAT_THREADS, 0, st>>>(a, Y);
      break;
    default:
      k_prox6_finish<float2><<<blocks, FLAT_THREADS, 0, st>>>(a, Y);
  }
  return cudaGetLastError();
}

}  // namespace rihvr
