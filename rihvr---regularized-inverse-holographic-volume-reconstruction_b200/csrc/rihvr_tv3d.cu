// 3-D fused lasso (mode 6): proximalFusedLasso (sparse_compressive_holo.cu:
// 3422-3475) with totalVariationProjection (:3832-4018): half threshold, n_tv
// dual steps over the whole volume (periodic in x, y, z), final estimate, half
// threshold.
//
// The reference disables the projection of the dual (:3964), so its step is
// linear and the dual drops out.  With g the dual, L = div grad, X1 the
// thresholded input and y_k = X1 - mu div g_k the estimate before step k:
//   g_{k+1} = g_k + s grad y_k   =>   y_{k+1} = y_k - mu s L y_k,
// L y = 6 y - (sum of the six neighbours).  n_tv applications of one 7-point
// stencil to X1 give the estimate, with one volume in and one out instead of
// four in and three out for each step (the dual form moved 96 bytes a voxel
// and step, a stencil pass 16).  At 256 x 256 x 100 with 5 steps the prox took
// 817 us in the dual form and 207 us here.
#include <algorithm>
#include <cmath>
#include <utility>

#include "rihvr_device.cuh"
#include "rihvr_kernels.cuh"
#include "rihvr_launch.cuh"

namespace rihvr {

// ---------------------------------------------------------------------------
// half threshold of the gradient step, two voxels a thread
// ---------------------------------------------------------------------------
template <typename ST>
__global__ void __launch_bounds__(FLAT_THREADS) k_prox6_init(ProxArgs a0, float2* __restrict__ X1) {
  const ProxArgs a = resolve_scalars(a0);
  const size_t n2 = (size_t)a.W * a.H * a.Nz / 2;  // W is even
  const ST* P = static_cast<const ST*>(a.P);
  const ST* Pp = static_cast<const ST*>(a.Pprev);
  const float T = 0.5f * a.thr;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += (size_t)gridDim.x * blockDim.x) {
    float2 p[2], q[2], g[2], v[2];
    Pair<ST>::ld(P + 2 * i, p[0], p[1]);
    Pair<ST>::ld(Pp + 2 * i, q[0], q[1]);
    Pair<float2>::ld(a.G + 2 * i, g[0], g[1]);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float2 x = make_float2(fmaf(a.beta, p[c].x - q[c].x, p[c].x), fmaf(a.beta, p[c].y - q[c].y, p[c].y));
      v[c] = shrink(make_float2(fmaf(-a.t, g[c].x, x.x), fmaf(-a.t, g[c].y, x.y)), T, a.faithful);
    }
    reinterpret_cast<float4*>(X1)[i] = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
  }
}

cudaError_t launch_prox6_init(int storage, const ProxArgs& a, float2* X1, cudaStream_t st) {
  const int blocks = flat_blocks((size_t)a.W * a.H * a.Nz / 2);
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

// ---------------------------------------------------------------------------
// T stencil steps in one pass over the volume.  A block owns a tile of 64 x EY
// columns (with a recomputed halo of T on every side, rounded up to even in x
// so that a lane's two columns stay 16-byte aligned) and walks a run of planes;
// the T steps are pipelined one plane apart: when plane k arrives, step 1
// makes plane k - 1, step 2 plane k - 2 and so on.  A thread holds two columns
// of R rows and, for every step, the last two planes of its input in registers;
// x neighbours move by shuffles, and only the first and last row of a warp's
// rows cross warps, through double-buffered shared memory, with one barrier a
// plane.  A run starts T planes early (periodic), so its outputs are exact.
// ---------------------------------------------------------------------------
template <int T>
struct Tv3Shape {
  static constexpr int HX = (T + 1) / 2 * 2;   // x halo
  static constexpr int R = T >= 3 ? 2 : 4;     // rows a thread
  static constexpr int NW = T >= 3 ? 16 : 8;   // warps, stacked in y
  static constexpr int EY = NW * R;
  static constexpr int VX = 64 - 2 * HX, VY = EY - 2 * T;
  static constexpr int THREADS = 32 * NW;
  static constexpr int MINB = T >= 3 ? 1 : 2;
  static constexpr size_t SMEM = sizeof(float4) * 2 * T * NW * 2 * 32;
};

struct Tv3Grid {
  int W, H, Nz, seg_len;
};

__device__ __forceinline__ float2 stencil7(float2 y, float2 xl, float2 xr, float2 yu, float2 yd, float2 zm, float2 zp,
                                           float2 c2) {
  const float2 s = f2add(f2add(f2add(xl, xr), f2add(yu, yd)), f2add(zm, zp));
  return f2fma(c2, f2fma(make_float2(-6.f, -6.f), y, s), y);
}

template <int T>
__global__ void __launch_bounds__(Tv3Shape<T>::THREADS, Tv3Shape<T>::MINB)
    k_tv3_steps(const float2* __restrict__ in, float2* __restrict__ out, Tv3Grid gr, float mu0, float s0,
                const float* __restrict__ dscal) {
  using Sh = Tv3Shape<T>;
  constexpr int R = Sh::R, NW = Sh::NW;
  // first and last row of every warp's current plane, per parity and step
  extern __shared__ float4 tv3_edge[];
  auto& edge = *reinterpret_cast<float4(*)[2][T][NW][2][32]>(tv3_edge);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int W = gr.W, H = gr.H, Nz = gr.Nz;
  const float mu = dscal ? __ldg(dscal + 2) : mu0, s = dscal ? __ldg(dscal + 3) : s0;
  const float c = mu * s;
  const float2 c2 = make_float2(c, c);
  const int cu = (int)blockIdx.x * Sh::VX - Sh::HX + 2 * lane;  // unwrapped first column (even)
  const int gc = ((cu % W) + W) % W;                            // even, as W is
  const int ru = (int)blockIdx.y * Sh::VY - T + w * R;          // unwrapped first row
  const bool lane_ok = 2 * lane >= Sh::HX && 2 * lane < Sh::HX + Sh::VX && cu < W;
  const int z0 = (int)blockIdx.z * gr.seg_len, z1 = min(Nz, z0 + gr.seg_len);
  const size_t HW = (size_t)H * W;
  unsigned off[R];  // a thread's rows within a plane
  bool row_ok[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int y = ru + r;
    off[r] = (unsigned)(((y % H) + H) % H) * (unsigned)W + (unsigned)gc;
    row_ok[r] = lane_ok && w * R + r >= T && w * R + r < T + Sh::VY && y < H;
  }
  const float2 zero = make_float2(0.f, 0.f);
  float2 prev[T][R][2], cur[T][R][2];
#pragma unroll
  for (int L = 0; L < T; ++L)
#pragma unroll
    for (int r = 0; r < R; ++r) prev[L][r][0] = prev[L][r][1] = cur[L][r][0] = cur[L][r][1] = zero;
  for (int e = threadIdx.x; e < T * NW * 2 * 32; e += Sh::THREADS) (&edge[1][0][0][0][0])[e] = make_float4(0.f, 0.f, 0.f, 0.f);

  int zl = ((z0 - T) % Nz + Nz) % Nz;  // plane being loaded
  float4 nx[R];
#pragma unroll
  for (int r = 0; r < R; ++r) nx[r] = __ldg(reinterpret_cast<const float4*>(in + (size_t)zl * HW + off[r]));
  __syncthreads();
  const int steps = z1 - z0 + 2 * T;
#pragma unroll 1
  for (int i = 0; i < steps; ++i) {
    float2 nw[R][2];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      nw[r][0] = make_float2(nx[r].x, nx[r].y);
      nw[r][1] = make_float2(nx[r].z, nx[r].w);
    }
    if (i + 1 < steps) {
      zl = zl + 1 == Nz ? 0 : zl + 1;
#pragma unroll
      for (int r = 0; r < R; ++r) nx[r] = __ldg(reinterpret_cast<const float4*>(in + (size_t)zl * HW + off[r]));
    }
    const int rd = (i + 1) & 1, wr = i & 1;
#pragma unroll
    for (int L = 0; L < T; ++L) {
      // nw: step L's newest plane (its input for L = 0); cur and prev the two before it
      edge[wr][L][w][0][lane] = make_float4(nw[0][0].x, nw[0][0].y, nw[0][1].x, nw[0][1].y);
      edge[wr][L][w][1][lane] = make_float4(nw[R - 1][0].x, nw[R - 1][0].y, nw[R - 1][1].x, nw[R - 1][1].y);
      // the rows above and below this warp's on plane cur (halo rows at the tile's edges: value irrelevant)
      const float4 ua = edge[rd][L][w > 0 ? w - 1 : 0][1][lane], da = edge[rd][L][w + 1 < NW ? w + 1 : w][0][lane];
      const float2 up[2] = {make_float2(ua.x, ua.y), make_float2(ua.z, ua.w)};
      const float2 dn[2] = {make_float2(da.x, da.y), make_float2(da.z, da.w)};
      float2 y[R][2];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float2 l = shfl_up2(cur[L][r][1]), rt = shfl_down2(cur[L][r][0]);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const float2 yu = r > 0 ? cur[L][r > 0 ? r - 1 : 0][k] : up[k];
          const float2 yd = r + 1 < R ? cur[L][r + 1 < R ? r + 1 : 0][k] : dn[k];
          y[r][k] = stencil7(cur[L][r][k], k ? cur[L][r][0] : l, k ? rt : cur[L][r][1], yu, yd, prev[L][r][k],
                             nw[r][k], c2);
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          prev[L][r][k] = cur[L][r][k];
          cur[L][r][k] = nw[r][k];
          nw[r][k] = y[r][k];
        }
    }
    if (i >= 2 * T) {
      float2* o = out + (size_t)(z0 + i - 2 * T) * HW;
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (row_ok[r])
          *reinterpret_cast<float4*>(o + off[r]) = make_float4(nw[r][0].x, nw[r][0].y, nw[r][1].x, nw[r][1].y);
    }
    __syncthreads();
  }
}

template <int T>
static cudaError_t tv3_steps_launch(const float2* in, float2* out, const ProxArgs& a, cudaStream_t st) {
  using Sh = Tv3Shape<T>;
  const int bx = (a.W + Sh::VX - 1) / Sh::VX, by = (a.H + Sh::VY - 1) / Sh::VY;
  // runs of planes: whole waves of resident blocks against the 2 T planes each run reads early
  const double slots = (double)num_sms() * Sh::MINB;
  int nseg = 1;
  double best = 1e300;
  for (int n = 1; n <= a.Nz && n <= 64; ++n) {
    const int len = (a.Nz + n - 1) / n;
    const double cost = std::max(1.0, std::ceil((double)bx * by * n / slots)) * (len + 2 * T + 1);
    if (cost < best * 0.999) {
      best = cost;
      nseg = n;
    }
  }
  Tv3Grid g{a.W, a.H, a.Nz, (a.Nz + nseg - 1) / nseg};
  nseg = (a.Nz + g.seg_len - 1) / g.seg_len;
  if (by > 65535) return cudaErrorInvalidConfiguration;
  cudaError_t e = allow_smem(k_tv3_steps<T>, Sh::SMEM);
  if (e != cudaSuccess) return e;
  k_tv3_steps<T><<<dim3(bx, by, nseg), Sh::THREADS, Sh::SMEM, st>>>(in, out, g, a.mu, a.s, a.dscal);
  return cudaGetLastError();
}

// n_tv stencil steps from X1; `other` is a second volume.  *result: the one of
// the two that holds the estimate.
cudaError_t launch_tv3(const ProxArgs& a, float2* X1, float2* other, const float2** result, int* launches,
                       cudaStream_t st) {
  float2 *src = X1, *dst = other;
  int left = a.n_tv;
  *launches = 0;
  while (left > 0) {
    const int T = left == 4 ? 2 : std::min(left, 3);  // 4 as 2 + 2 instead of 3 + 1
    cudaError_t e = T == 3   ? tv3_steps_launch<3>(src, dst, a, st)
                    : T == 2 ? tv3_steps_launch<2>(src, dst, a, st)
                             : tv3_steps_launch<1>(src, dst, a, st);
    if (e != cudaSuccess) return e;
    ++*launches;
    left -= T;
    std::swap(src, dst);
  }
  *result = src;
  return cudaSuccess;
}

// ---------------------------------------------------------------------------
// half threshold of the estimate, P_new and the sums.  A block of 8 rows of 64
// columns walks a run of planes, so that the plane before it (which the 3-D TV
// norms need) is at hand; left neighbours move by shuffles, upper ones come
// from the caches.
//
// What bounds it: latency.  A plane's loads are issued while the plane before
// is worked on, as stored (a conversion would wait for them); with the loads of
// each plane after the last one's sums, 256 x 256 x 100 took 96 us with the norm
// terms, 67 us so (40 us at the memory's rate).
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 momentum(float2 p, float2 q, float beta) {
  return make_float2(fmaf(beta, p.x - q.x, p.x), fmaf(beta, p.y - q.y, p.y));
}

// two voxels of Y, P and Pprev as stored
template <typename ST>
struct Raw6 {
  float4 y;
  typename Raw2<ST>::T p, q;
  __device__ __forceinline__ void ld(const float2* Y, const ST* P, const ST* Pp, size_t i) {
    y = Raw2<float2>::ld(Y + i);
    p = Raw2<ST>::ld(P + i);
    q = Raw2<ST>::ld(Pp + i);
  }
  // the thresholded estimate v, the momentum point x and P itself
  __device__ __forceinline__ void get(float T, float beta, int faithful, float2 (&v)[2], float2 (&x)[2],
                                      float2 (&pv)[2]) const {
    float2 qv[2];
    Raw2<float2>::cvt(y, v[0], v[1]);
    Raw2<ST>::cvt(p, pv[0], pv[1]);
    Raw2<ST>::cvt(q, qv[0], qv[1]);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      v[c] = shrink(v[c], T, faithful);
      x[c] = momentum(pv[c], qv[c], beta);
    }
  }
};

template <typename ST, bool NORMS>
__global__ void __launch_bounds__(FLAT_THREADS) k_prox6_finish(ProxArgs a0, const float2* __restrict__ Y,
                                                              int seg_len) {
  const ProxArgs a = resolve_scalars(a0);
  const int W = a.W, H = a.H, Nz = a.Nz;
  const size_t HW = (size_t)W * H;
  const ST* P = static_cast<const ST*>(a.P);
  const ST* Pp = static_cast<const ST*>(a.Pprev);
  ST* Pn = static_cast<ST*>(a.Pnew);
  const float T = 0.5f * a.thr;
  const int lane = threadIdx.x & 31;
  const int xx = ((int)blockIdx.x * 32 + lane) * 2, yy = (int)blockIdx.y * 8 + (threadIdx.x >> 5);
  const int z0 = (int)blockIdx.z * seg_len, z1 = min(Nz, z0 + seg_len);
  const bool ok = xx < W && yy < H;
  const size_t e = ok ? (size_t)yy * W + xx : 0;
  // the column left of the block's and the row above
  const size_t el = ok ? (size_t)yy * W + (xx > 0 ? xx - 1 : W - 1) : 0;
  const size_t eu = ok ? (size_t)(yy > 0 ? yy - 1 : H - 1) * W + xx : 0;
  float wr, wi;
  restart_w(e, a.faithful, &wr, &wi);  // e is even: both columns are in the same 512
  double acc[kNumSums];
#pragma unroll
  for (int k = 0; k < kNumSums; ++k) acc[k] = 0.0;
  float2 pb[2], xb[2];  // p and x on the plane before
  if (NORMS) {
    Raw6<ST> r;
    float2 t[2];
    r.ld(Y, P, Pp, (size_t)(z0 > 0 ? z0 - 1 : Nz - 1) * HW + e);
    r.get(T, a.beta, a.faithful, pb, xb, t);
  }
  // the plane to come, as stored: this pair, the one above and lane 0's left neighbour
  Raw6<ST> rc, ru;
  float4 rg;
  float2 ly;
  ST lp, lq;
  auto request = [&](int z) {
    const size_t zo = (size_t)z * HW;
    rc.ld(Y, P, Pp, zo + e);
    rg = Raw2<float2>::ld(a.G + zo + e);
    if (NORMS) {
      ru.ld(Y, P, Pp, zo + eu);
      if (lane == 0) {
        ly = Y[zo + el];
        lp = P[zo + el];
        lq = Pp[zo + el];
      }
    }
  };
  if (z0 < z1) request(z0);
#pragma unroll 1
  for (int z = z0; z < z1; ++z) {
    float2 p[2], x[2], y0[2], g[2], pu[2], xu[2], pl[2], xl[2];
    rc.get(T, a.beta, a.faithful, p, x, y0);
    Raw2<float2>::cvt(rg, g[0], g[1]);
    if (NORMS) {
      float2 t[2];
      ru.get(T, a.beta, a.faithful, pu, xu, t);
      pl[1] = p[0];
      xl[1] = x[0];
      pl[0] = shfl_up2(p[1]);
      xl[0] = shfl_up2(x[1]);
      if (lane == 0) {
        pl[0] = shrink(ly, T, a.faithful);
        xl[0] = momentum(Store<ST>::ld(&lp), Store<ST>::ld(&lq), a.beta);
      }
    }
    if (z + 1 < z1) request(z + 1);
    if (ok) {
      Raw2<ST>::st(Pn + (size_t)z * HW + e, p[0], p[1]);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float2 d = csub(p[c], x[c]);
        acc[SUM_LIM1] += (double)(d.x * g[c].x) + (double)(d.y * g[c].y);
        acc[SUM_LIM2] += (double)cabs2(d);
        const float2 u = csub(x[c], p[c]), v = csub(p[c], y0[c]);
        acc[SUM_RS] += (double)(wr * u.x * v.x) + (double)(wi * u.y * v.y);
        if (NORMS) {
          acc[SUM_L1P] += (double)norm_sqrt(cabs2(p[c]));
          acc[SUM_TVP] += (double)norm_sqrt(cabs2(csub(pl[c], p[c])) + cabs2(csub(pu[c], p[c])) +
                                            cabs2(csub(pb[c], p[c])));
          acc[SUM_L1X] += (double)norm_sqrt(cabs2(x[c]));
          acc[SUM_TVX] += (double)norm_sqrt(cabs2(csub(xl[c], x[c])) + cabs2(csub(xu[c], x[c])) +
                                            cabs2(csub(xb[c], x[c])));
        }
      }
    }
    if (NORMS) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        pb[c] = p[c];
        xb[c] = x[c];
      }
    }
  }
  block_write_sums<FLAT_THREADS>(acc, a.partials, (int)((blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x));
}

// Blocks of the finish pass: 64 x 8 tiles and runs of planes, about eight blocks an SM,
// one run of planes a block.
struct FinishGrid {
  int bx, by, nseg, len;  // len: planes a run
  long long blocks() const { return (long long)bx * by * nseg; }
};
static FinishGrid finish_grid(int W, int H, int Nz) {
  FinishGrid g;
  g.bx = (W / 2 + 31) / 32;
  g.by = (H + 7) / 8;
  const long long tiles = (long long)g.bx * g.by;
  const long long nseg = std::max(1LL, std::min<long long>(Nz, (8LL * num_sms() + tiles - 1) / tiles));
  g.len = (int)((Nz + nseg - 1) / nseg);
  g.nseg = (Nz + g.len - 1) / g.len;
  return g;
}

size_t prox6_partial_blocks(int W, int H, int Nz) { return (size_t)finish_grid(W, H, Nz).blocks(); }

template <typename ST>
static cudaError_t prox6_finish_launch(const ProxArgs& a, const float2* Y, int* nblocks_out, cudaStream_t st) {
  const FinishGrid g = finish_grid(a.W, a.H, a.Nz);
  const long long blocks = g.blocks();
  if (g.by > 65535 || g.nseg > 65535 || blocks > a.partial_cap || blocks > 0x7fffffffLL)
    return cudaErrorInvalidConfiguration;
  *nblocks_out = (int)blocks;
  const dim3 grid((unsigned)g.bx, (unsigned)g.by, (unsigned)g.nseg);
  if (a.want_norms) k_prox6_finish<ST, true><<<grid, FLAT_THREADS, 0, st>>>(a, Y, g.len);
  else k_prox6_finish<ST, false><<<grid, FLAT_THREADS, 0, st>>>(a, Y, g.len);
  return cudaGetLastError();
}

cudaError_t launch_prox6_finish(int storage, const ProxArgs& a, const float2* Y, int* nblocks_out, cudaStream_t st) {
  switch (storage) {
    case STORE_BF16: return prox6_finish_launch<__nv_bfloat162>(a, Y, nblocks_out, st);
    case STORE_F16: return prox6_finish_launch<__half2>(a, Y, nblocks_out, st);
    default: return prox6_finish_launch<float2>(a, Y, nblocks_out, st);
  }
}

}  // namespace rihvr
