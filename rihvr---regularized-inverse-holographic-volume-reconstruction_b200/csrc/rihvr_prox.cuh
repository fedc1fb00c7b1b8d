// The 2-D total-variation prox (mode 7) as templates over the storage type;
// compiled per type in rihvr_prox_*.cu, dispatched in rihvr_prox.cu.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "rihvr_device.cuh"
#include "rihvr_kernels.cuh"
#include "rihvr_launch.cuh"

namespace rihvr {

// ---------------------------------------------------------------------------
// Fused 2-D TV prox (mode 7): proximalFusedLasso2d, sparse_compressive_holo.cu:
// 3652-3732 with kernels :3478-3597.  Per plane tile, with the momentum point
// formed on the fly:
//   x = P + beta (P - Pprev);  xh = x - t g
//   gx = gy = 0; n_tv times: y = xh - mu div(g);  g = (g + s grad y)/max(1, |.|)
//   y = xh - mu div(g);  p = shrink(y, thr)
// div uses forward periodic differences, grad backward periodic differences and
// the projection norm is taken over the four real components (Jacobi updates,
// as the reference's two kernels per iteration).
//
// Layout: a block holds a 64 x 64 tile (columns x rows) with a recomputed halo
// of n_tv + 1 pixels on every side, which makes the interior exact.  Warp w owns
// rows [8w, 8w+8); lane l owns columns 2l and 2l+1.  The Chambolle state (xh, gx,
// gy) stays in registers; each TV iteration sweeps a thread's 8 rows top to
// bottom so that y is only ever live for one row, right neighbours of gx and
// left neighbours of y move by warp shuffles, and only the first/last row of
// each warp's run crosses warps, through double-buffered shared memory (one
// barrier per iteration).  The row above a run is recomputed from the published
// last row of the warp above instead of being waited for.
// The final sweep also accumulates the line-search sums, the restart statistic
// and (optionally) the L1/TV norms of p and x.
// ---------------------------------------------------------------------------
constexpr int TV_CPL = 2;                  // columns per lane
constexpr int TV_EW = 32 * TV_CPL;         // tile width incl. halo
constexpr int TV_R = 8;                    // rows per thread
constexpr int TV_NW = 8;                   // warps, stacked vertically
constexpr int TV_EH = TV_NW * TV_R;        // tile height incl. halo
constexpr int TV_THREADS = 32 * TV_NW;
constexpr int TV_BND = TV_NW * TV_EW;      // one boundary row per warp
constexpr size_t TV_SMEM = sizeof(float2) * (2 * TV_EH * TV_EW + 3 * 2 * TV_BND + TV_BND);

// y = xh - mu ((gxr - gx) + (gyd - gy)), packed: nmu = (-mu, -mu)
__device__ __forceinline__ float2 tv_estimate(float2 xh, float2 gx, float2 gxr, float2 gy, float2 gyd, float2 nmu) {
  return f2fma(nmu, f2add(f2sub(gxr, gx), f2sub(gyd, gy)), xh);
}

// hardware reciprocal square root.  The flush-to-zero form is one instruction;
// the other one scales subnormal inputs before and after.  The projection only
// uses min(1, rsqrt(n2)), which is 1 for every subnormal n2 and for 0 either way
// (the same bits).  1024 x 1024 x 1000, 5 iterations: 9.42 ms instead of 9.73;
// with the norms' square roots 1.04 instead of 1.13 ms at 1280 x 1024 x 64.
__device__ __forceinline__ float rsqrt_approx(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// g = P(g + s grad y) for one pixel: px = gx + s (yl - y), py = gy + s (yu - y),
// divided by max(1, |(px, py)|) over the four real components.
__device__ __forceinline__ void tv_dual(float2& gx, float2& gy, float2 y, float2 yl, float2 yu, float2 s2) {
  const float2 px = f2fma(s2, f2sub(yl, y), gx);
  const float2 py = f2fma(s2, f2sub(yu, y), gy);
  const float2 q = f2fma(py, py, f2mul(px, px));
  const float n2 = q.x + q.y;
  // 1 / max(1, sqrt(n2)) as min(1, rsqrt(n2)): one instruction instead of a
  // compare and a select (n2 = 0 gives rsqrt = inf, hence 1)
  const float sc = fminf(1.f, rsqrt_approx(n2));
  const float2 sc2 = make_float2(sc, sc);
  gx = f2mul(px, sc2);
  gy = f2mul(py, sc2);
}

// wrap an index that lies within one period of [0, n)
__device__ __forceinline__ int wrap1(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

template <typename ST>
__global__ void __launch_bounds__(TV_THREADS, 2) k_prox_tv2d(ProxArgs a0) {
  const ProxArgs a = resolve_scalars(a0);
  static_assert(TV_CPL == 2, "paired loads assume two columns per lane");
  extern __shared__ float2 smem[];
  float2* s_g = smem;                      // [EH][EW] gradient at load
  float2* s_P = s_g + TV_EH * TV_EW;       // [EH][EW] P at load
  float2* s_gyf = s_P + TV_EH * TV_EW;     // [2][NW][EW] first-row gy of each run
  float2* s_gxl = s_gyf + 2 * TV_BND;      // [2][NW][EW] last-row gx
  float2* s_gyl = s_gxl + 2 * TV_BND;      // [2][NW][EW] last-row gy
  float2* s_xhl = s_gyl + 2 * TV_BND;      // [NW][EW]   last-row xh
  const int W = a.W, H = a.H;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int h = a.n_tv + 1, VW = TV_EW - 2 * h, VH = TV_EH - 2 * h;
  const int ox = blockIdx.x * VW - h, oy = blockIdx.y * VH - h;
  const size_t plane = (size_t)blockIdx.z * W * H;
  const ST* P = static_cast<const ST*>(a.P) + plane;
  const ST* Pp = static_cast<const ST*>(a.Pprev) + plane;
  const float2* G = a.G + plane;
  const float t = a.t, beta = a.beta;
  const float2 nmu = make_float2(-a.mu, -a.mu), s2 = make_float2(a.s, a.s);
  const int col0 = lane * TV_CPL;
  // tiles are at most one period outside the plane when it is at least as
  // large as a tile; smaller planes wrap several times
  const bool small = (W < TV_EW) || (H < TV_EH);
  // adjacent column pairs are contiguous and 16-byte aligned when the tile
  // origin is even (the plane side is even)
  const bool paired = !small && ((ox & 1) == 0);

  float2 xh[TV_R][TV_CPL], gx[TV_R][TV_CPL], gy[TV_R][TV_CPL];
  int gc[TV_CPL];
#pragma unroll
  for (int c = 0; c < TV_CPL; ++c) gc[c] = small ? ((ox + col0 + c) % W + W) % W : wrap1(ox + col0 + c, W);
#pragma unroll
  for (int i = 0; i < TV_R; ++i) {
    const int row = w * TV_R + i;
    const int gr = small ? ((oy + row) % H + H) % H : wrap1(oy + row, H);
    const size_t rbase = (size_t)gr * W;
    float2 p[TV_CPL], pp[TV_CPL], g[TV_CPL];
    if (paired) {
      Pair<ST>::ld(P + rbase + gc[0], p[0], p[1]);
      Pair<ST>::ld(Pp + rbase + gc[0], pp[0], pp[1]);
      Pair<float2>::ld(G + rbase + gc[0], g[0], g[1]);
    } else {
#pragma unroll
      for (int c = 0; c < TV_CPL; ++c) {
        p[c] = Store<ST>::ld(P + rbase + gc[c]);
        pp[c] = Store<ST>::ld(Pp + rbase + gc[c]);
        g[c] = G[rbase + gc[c]];
      }
    }
#pragma unroll
    for (int c = 0; c < TV_CPL; ++c) {
      const float2 x = f2fma(make_float2(beta, beta), f2sub(p[c], pp[c]), p[c]);
      xh[i][c] = f2fma(make_float2(-t, -t), g[c], x);
      gx[i][c] = make_float2(0.f, 0.f);
      gy[i][c] = make_float2(0.f, 0.f);
    }
    *reinterpret_cast<float4*>(s_g + row * TV_EW + col0) = make_float4(g[0].x, g[0].y, g[1].x, g[1].y);
    *reinterpret_cast<float4*>(s_P + row * TV_EW + col0) = make_float4(p[0].x, p[0].y, p[1].x, p[1].y);
  }
#pragma unroll
  for (int c = 0; c < TV_CPL; ++c) s_xhl[w * TV_EW + col0 + c] = xh[TV_R - 1][c];

  for (int k = 0; k < a.n_tv; ++k) {
    float2* gyf = s_gyf + (k & 1) * TV_BND;
    float2* gxl = s_gxl + (k & 1) * TV_BND;
    float2* gyl = s_gyl + (k & 1) * TV_BND;
#pragma unroll
    for (int c = 0; c < TV_CPL; ++c) {
      gyf[w * TV_EW + col0 + c] = gy[0][c];
      gxl[w * TV_EW + col0 + c] = gx[TV_R - 1][c];
      gyl[w * TV_EW + col0 + c] = gy[TV_R - 1][c];
    }
    __syncthreads();
    // y of the row above this run, recomputed from the published last row of warp w-1
    float2 yu[TV_CPL];
#pragma unroll
    for (int c = 0; c < TV_CPL; ++c) {
      yu[c] = make_float2(0.f, 0.f);  // top halo rows: value irrelevant
      if (w > 0) {
        const int col = col0 + c, b = (w - 1) * TV_EW;
        const float2 gxu = gxl[b + col], gyu = gyl[b + col];
        const float2 gxru = (col + 1 < TV_EW) ? gxl[b + col + 1] : gxu;
        yu[c] = tv_estimate(s_xhl[b + col], gxu, gxru, gyu, gy[0][c], nmu);
      }
    }
#pragma unroll
    for (int i = 0; i < TV_R; ++i) {
      float2 gxr[TV_CPL], gyd[TV_CPL], y[TV_CPL], yl[TV_CPL];
#pragma unroll
      for (int c = 0; c < TV_CPL - 1; ++c) gxr[c] = gx[i][c + 1];
      gxr[TV_CPL - 1] = shfl_down2(gx[i][0]);  // lane 31 gets its own (halo column)
#pragma unroll
      for (int c = 0; c < TV_CPL; ++c) {
        if (i < TV_R - 1) gyd[c] = gy[i + 1][c];
        else gyd[c] = (w < TV_NW - 1) ? gyf[(w + 1) * TV_EW + col0 + c] : gy[i][c];
        y[c] = tv_estimate(xh[i][c], gx[i][c], gxr[c], gy[i][c], gyd[c], nmu);
      }
      yl[0] = shfl_up2(y[TV_CPL - 1]);  // lane 0 gets its own (halo column)
#pragma unroll
      for (int c = 1; c < TV_CPL; ++c) yl[c] = y[c - 1];
#pragma unroll
      for (int c = 0; c < TV_CPL; ++c) {
        tv_dual(gx[i][c], gy[i][c], y[c], yl[c], yu[c], s2);
        yu[c] = y[c];
      }
    }
  }

  // final estimate and shrink: p replaces gx in registers
  {
    float2* gyf = s_gyf + (a.n_tv & 1) * TV_BND;
#pragma unroll
    for (int c = 0; c < TV_CPL; ++c) gyf[w * TV_EW + col0 + c] = gy[0][c];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TV_R; ++i) {
      float2 gxr[TV_CPL];
#pragma unroll
      for (int c = 0; c < TV_CPL - 1; ++c) gxr[c] = gx[i][c + 1];
      gxr[TV_CPL - 1] = shfl_down2(gx[i][0]);
#pragma unroll
      for (int c = 0; c < TV_CPL; ++c) {
        float2 gyd;
        if (i < TV_R - 1) gyd = gy[i + 1][c];
        else gyd = (w < TV_NW - 1) ? gyf[(w + 1) * TV_EW + col0 + c] : gy[i][c];
        const float2 y = tv_estimate(xh[i][c], gx[i][c], gxr[c], gy[i][c], gyd, nmu);
        gx[i][c] = shrink(y, a.thr, a.faithful);
      }
    }
  }
  // last-row p and x of each run for the TV norms of the run below
  float2* pl_last = s_gxl;  // reused: no TV reads remain
  float2* xl_last = s_gyl;
  const float2 t2 = make_float2(t, t);
  if (a.want_norms) {
#pragma unroll
    for (int c = 0; c < TV_CPL; ++c) {
      const int col = col0 + c;
      const float2 g = s_g[(w * TV_R + TV_R - 1) * TV_EW + col];
      pl_last[w * TV_EW + col] = gx[TV_R - 1][c];
      xl_last[w * TV_EW + col] = f2fma(t2, g, xh[TV_R - 1][c]);
    }
  }
  __syncthreads();

  // per-thread FP32 partials over at most 16 pixels, FP64 from there on
  float acc[kNumSums];
#pragma unroll
  for (int k = 0; k < kNumSums; ++k) acc[k] = 0.f;
  ST* Pn = static_cast<ST*>(a.Pnew) + plane;
  float2 pu[TV_CPL], xu[TV_CPL];
#pragma unroll
  for (int c = 0; c < TV_CPL; ++c) {
    pu[c] = make_float2(0.f, 0.f);
    xu[c] = make_float2(0.f, 0.f);
    if (w > 0 && a.want_norms) {
      pu[c] = pl_last[(w - 1) * TV_EW + col0 + c];
      xu[c] = xl_last[(w - 1) * TV_EW + col0 + c];
    }
  }
#pragma unroll
  for (int i = 0; i < TV_R; ++i) {
    const int row = w * TV_R + i;
    const int grow = oy + row;
    const bool row_ok = row >= h && row < h + VH && grow < H;
    float2 x[TV_CPL], pl[TV_CPL], xl[TV_CPL], g[TV_CPL], y0[TV_CPL];
    {
      const float4 gv = *reinterpret_cast<const float4*>(s_g + row * TV_EW + col0);
      const float4 pv = *reinterpret_cast<const float4*>(s_P + row * TV_EW + col0);
      g[0] = make_float2(gv.x, gv.y);
      g[1] = make_float2(gv.z, gv.w);
      y0[0] = make_float2(pv.x, pv.y);
      y0[1] = make_float2(pv.z, pv.w);
    }
#pragma unroll
    for (int c = 0; c < TV_CPL; ++c) x[c] = f2fma(t2, g[c], xh[i][c]);
    pl[0] = shfl_up2(gx[i][TV_CPL - 1]);
    xl[0] = shfl_up2(x[TV_CPL - 1]);
#pragma unroll
    for (int c = 1; c < TV_CPL; ++c) {
      pl[c] = gx[i][c - 1];
      xl[c] = x[c - 1];
    }
#pragma unroll
    for (int c = 0; c < TV_CPL; ++c) {
      const int col = col0 + c, gcl = ox + col;
      const float2 p = gx[i][c];
      if (row_ok && col >= h && col < h + VW && gcl < W) {
        const size_t e = (size_t)grow * W + gcl;
        Store<ST>::st(Pn + e, p);
        const float2 d = f2sub(p, x[c]);
        const float2 dg = f2mul(d, g[c]);
        acc[SUM_LIM1] += dg.x + dg.y;
        acc[SUM_LIM2] += cabs2(d);
        float wr, wi;
        restart_w(e, a.faithful, &wr, &wi);
        const float2 uv = f2mul(f2sub(x[c], p), f2sub(p, y0[c]));
        acc[SUM_RS] += fmaf(wr, uv.x, wi * uv.y);
        if (a.want_norms) {
          acc[SUM_L1P] += norm_sqrt(cabs2(p));
          acc[SUM_TVP] += norm_sqrt(cabs2(f2sub(pl[c], p)) + cabs2(f2sub(pu[c], p)));
          acc[SUM_L1X] += norm_sqrt(cabs2(x[c]));
          acc[SUM_TVX] += norm_sqrt(cabs2(f2sub(xl[c], x[c])) + cabs2(f2sub(xu[c], x[c])));
        }
      }
      pu[c] = p;
      xu[c] = x[c];
    }
  }
  double dacc[kNumSums];
#pragma unroll
  for (int k = 0; k < kNumSums; ++k) dacc[k] = (double)acc[k];
  const int blk = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  block_write_sums<TV_THREADS>(dacc, a.partials, blk);
}

struct TvsGrid {
  int nstrips, nseg, seg_len;
};

// ---------------------------------------------------------------------------
// Streaming form of the same prox (1 <= n_tv <= 10), the default.  The tiled
// kernel above recomputes a halo of n_tv + 1 rows and columns around every
// 64 x 64 tile, so a third of its work is thrown away, and it needs a block
// barrier per TV iteration.  Here a lane owns CPL adjacent columns and a warp a
// strip of 32 CPL columns with an x halo of HX (n_tv + 1 rounded up to a
// multiple of CPL) on each side; the warp walks a run of rows with the n_tv
// Chambolle iterations pipelined one row apart: at the step that loads row j,
// iteration k updates row j - k from iteration k-1's rows j-k (kept from the
// previous step) and j-k+1 (produced this step), and the final estimate and
// shrink produce row j - n_tv - 1.  A run starts 2 (n_tv + 1) rows early
// (periodic wrap) so that its first output row is exact, which removes the y
// halo.  Warps are independent and exchange x neighbours by shuffles only.
//
// Per lane, the state is one row of (gx, gy) and one row of y per iteration in
// registers.  Rows arrive one step ahead by cp.async into a per-lane ring of D
// rows in shared memory holding (raw Pprev, overwritten by xh), G and raw P;
// each lane reads back only what it copied, so no barrier is involved.
// Iteration 1 starts from g = 0, where the estimate is xh itself.  The
// arithmetic is the tiled kernel's operation for operation, so P_new has the
// same bits; the sums differ only in summation order.
//
// The step loop is unrolled by four (by two it needs 10% more instructions; by
// eight the loop body outgrows the instruction cache).  With a step count that
// is not a multiple of the unroll factor, unrolled builds gave the last row of a
// run 1 ulp away from the tiled kernel, so runs start up to three rows earlier
// and every run has a multiple of four steps.
// ---------------------------------------------------------------------------
template <int NTV, int CPL>
struct TvwShape {
  static constexpr int h = NTV + 1;
  static constexpr int AL = CPL < 2 ? 2 : CPL;
  static constexpr int HX = (h + AL - 1) / AL * AL;   // keeps each lane's columns aligned
  static constexpr int SW = 32 * CPL;                 // strip width
  static constexpr int VW = SW - 2 * HX;              // valid columns per strip
  static constexpr int D = (h + 2 <= 8) ? 8 : 16;     // rows in use: h + 1, plus one landing
  static constexpr int F4 = CPL / 2;                  // float4 per array per lane row (FP32)
  static constexpr int SLOT = 3 * F4 * 32;            // float4 per ring slot, whole warp
  // Two warps per block.  Without the objective's norm terms and with the
  // 8-row ring (n_tv <= 5), the kernel fits 128 registers with at most a few
  // bytes of spill, and 8 blocks (16 warps) share an SM; the norm terms need
  // about 160 registers, which caps them at 6 blocks (12 warps).  At
  // 1024 x 1024 x 1000 (n_tv = 5, no norm terms) a launch took 10.42 ms with
  // 4-warp blocks at 12 warps per SM, 9.5 ms with 2-warp blocks at 16 (9.1 ms
  // now).  Four columns a lane (strips of 128, a tenth fewer columns computed
  // twice, 8 warps per SM at 221 registers, no spills) took 12.1 ms unrolled by
  // four and 10.6 ms by two.
  static constexpr int NW = 2;
  static constexpr size_t SMEM = sizeof(float4) * (size_t)SLOT * D * NW;
  static_assert(CPL == 2 || CPL == 4, "columns per lane");
  static_assert(VW > 0, "halo wider than the strip");
};

// Blocks per SM the register allocation targets (__launch_bounds__).  At 7
// two-warp blocks ptxas caps the kernel at 128 registers (8 blocks then fit,
// as registers are split per scheduler); asking for 8 gives the same cap with
// ten times the spill.
template <int NTV, bool NORMS>
constexpr int tvw_minb() {
  return TvwShape<NTV, 2>::D == 8 ? (NORMS ? 6 : 7) : 4;
}

// copy CPL complex values in storage type (16-byte aligned source for
// CPL * sizeof(ST) >= 16, else 8-byte aligned) to shared memory
template <typename ST, int CPL>
__device__ __forceinline__ void cp_async_run(float4* smem, const ST* gmem) {
  constexpr int BYTES = CPL * (int)sizeof(ST);
  if constexpr (BYTES >= 16) {
#pragma unroll
    for (int k = 0; k < BYTES / 16; ++k) {
      const unsigned d = (unsigned)__cvta_generic_to_shared(smem + k * 32);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d),
                   "l"(reinterpret_cast<const char*>(gmem) + 16 * k)
                   : "memory");
    }
  } else {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(gmem) : "memory");
  }
}

// CPL complex values of storage type ST from their ring copy (16-byte pieces
// 32 float4 apart)
template <typename ST, int CPL>
__device__ __forceinline__ void ring_vals(const float4* e, float2 (&v)[CPL]) {
  if constexpr (sizeof(ST) == 8) {
#pragma unroll
    for (int k = 0; k < CPL / 2; ++k) {
      const float4 f = e[k * 32];
      v[2 * k] = make_float2(f.x, f.y);
      v[2 * k + 1] = make_float2(f.z, f.w);
    }
  } else {
#pragma unroll
    for (int k = 0; k < (CPL + 3) / 4; ++k) {
      const float4 f = e[k * 32];
      const unsigned u[4] = {__float_as_uint(f.x), __float_as_uint(f.y), __float_as_uint(f.z), __float_as_uint(f.w)};
#pragma unroll
      for (int j = 0; j < 4 && 4 * k + j < CPL; ++j) {
        float2 a, b;
        Raw2<ST>::cvt(make_uint2(u[j], 0u), a, b);
        v[4 * k + j] = a;
      }
    }
  }
}

template <typename ST, int CPL>
__device__ __forceinline__ void store_run(ST* p, const float2 (&v)[CPL]) {
#pragma unroll
  for (int c = 0; c < CPL; c += 2) Raw2<ST>::st(p + c, v[c], v[c + 1]);
}

template <typename ST, int NTV, bool NORMS, int CPL = 2, int NW = TvwShape<NTV, CPL>::NW,
          int MINB = tvw_minb<NTV, NORMS>(), int PART = 0>
__global__ void __launch_bounds__(32 * NW, MINB) k_prox_tv2d_strip(ProxArgs a0, TvsGrid gr) {
  const ProxArgs a = resolve_scalars(a0);
  using Sh = TvwShape<NTV, CPL>;
  constexpr int h = Sh::h, HX = Sh::HX, VW = Sh::VW, D = Sh::D, F4 = Sh::F4;
  constexpr int UNR = 4;          // steps of an unrolled loop body
  constexpr int QS = F4 * 32;     // float4 between the arrays of a slot
  constexpr int SL = 3 * QS;      // float4 per slot
  static_assert(PART == 0 || CPL == 2, "the two-part forms move a lane's two columns as one float4");
  extern __shared__ float4 tvw_ring[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  float4* ring = tvw_ring + (size_t)w * SL * D + lane;
  // second part: 2 rows of the stored duals (gx pair, gy pair) after the warps' rings
  float4* gring = tvw_ring + (size_t)NW * SL * D + (size_t)w * 2 * 32 * 2 + lane;
  const int W = a.W, H = a.H;
  const long long work = (long long)blockIdx.x * NW + w;
  const long long nwork = (long long)gr.nstrips * gr.nseg * a.Nz;

  // the FP64 sums are touched every eighth row: in shared memory they cost no
  // registers, which the loop is short of
  constexpr int NS = NORMS ? kNumSums : SUM_RS + 1;  // sums this kernel accumulates
  __shared__ double dsum[NS][32 * NW];
#pragma unroll
  for (int k = 0; k < NS; ++k) dsum[k][threadIdx.x] = 0.0;

  if (work < nwork) {
    const int strip = (int)(work % gr.nstrips);
    const long long rest = work / gr.nstrips;
    const int seg = (int)(rest % gr.nseg);
    const size_t plane = (size_t)(rest / gr.nseg) * W * H;
    const ST* P = static_cast<const ST*>(a.P) + plane;
    const ST* Pp = static_cast<const ST*>(a.Pprev) + plane;
    const float2* G = a.G + plane;
    ST* Pn = static_cast<ST*>(a.Pnew) + plane;
    const float t = a.t, beta = a.beta;
    const float2 nmu = make_float2(-a.mu, -a.mu), s2 = make_float2(a.s, a.s);
    const float2 bb = make_float2(beta, beta), nt2 = make_float2(-t, -t);
    const float2 z2 = make_float2(0.f, 0.f);
    const float thr = a.thr;
    const int faithful = a.faithful;

    const int cu = strip * VW - HX + CPL * lane;   // first column of this lane, unwrapped
    const int gc = ((cu % W) + W) % W;             // a multiple of CPL; W is one too
    const bool lane_ok = (CPL * lane >= HX) && (CPL * lane < HX + VW) && (cu < W);
    const int r0 = seg * gr.seg_len;
    const int r1 = min(H, r0 + gr.seg_len);
    // runs start up to UNR - 1 rows earlier so that the step count is a
    // multiple of the unroll factor
    const int pad = (UNR - ((r1 - r0 + 2 * h) % UNR)) % UNR;
    const int nsteps = (r1 - r0) + 2 * h + pad;
    // the warm-up may reach back more than one plane height on short planes
    int lrow = ((r0 - h - pad) % H + H) % H;
    int orow = ((r0 - 2 * h - pad) % H + H) % H;

    // Ring slots are read as rows above r0 - h before any copy lands there;
    // those rows only feed rows above r0, which are not written.
    // the first part's duals on row `off` (second part): a 2-row ring, so
    // the copy for the next step is issued once this step has read its rows
    auto request_g = [&](size_t off, int step) {
      if constexpr (PART == 2) {
        float4* gslot = gring + (step & 1) * 2 * 32;
        cp_async_run<float2, CPL>(gslot, a.gdx + plane + off);
        cp_async_run<float2, CPL>(gslot + 32, a.gdy + plane + off);
        cp_async_commit();
      }
    };
    size_t goff = 0;  // row offset of the last main-ring request
    auto request = [&](float4* e) {
      const size_t off = (size_t)lrow * W + gc;
      cp_async_run<ST, CPL>(e, Pp + off);
      cp_async_run<float2, CPL>(e + QS, G + off);
      cp_async_run<ST, CPL>(e + 2 * QS, P + off);
      cp_async_commit();
      goff = off;
      lrow = (lrow + 1 == H) ? 0 : lrow + 1;
    };
    request(ring);
    request_g(goff, 0);

    float2 gX[NTV][CPL], gY[NTV][CPL], yU[NTV][CPL];
#pragma unroll
    for (int k = 0; k < NTV; ++k)
#pragma unroll
      for (int c = 0; c < CPL; ++c) gX[k][c] = gY[k][c] = yU[k][c] = z2;
    float2 pu[CPL], xu[CPL];
#pragma unroll
    for (int c = 0; c < CPL; ++c) pu[c] = xu[c] = z2;
    float acc[kNumSums];
#pragma unroll
    for (int k = 0; k < kNumSums; ++k) acc[k] = 0.f;

    // The ring in groups of UNR slots, rotated once a loop body: the slot `back`
    // steps behind step u of the body is a group's offset plus a constant, where
    // a slot from the step's number took a mask and a multiply for each of the
    // 10 or so slots a step touches (1024 x 1024 x 1000, no norms: 9.42 ms with
    // that, 9.1 ms so, with the FP64 sums in shared memory; 1280 x 1024 x 64 with
    // norms: 1.04 and 0.99 ms).
    int grp[D / UNR];
#pragma unroll
    for (int k = 0; k < D / UNR; ++k) grp[k] = k * UNR * SL;
    auto slot_of = [&](int u, int back) -> float4* {
      const int s = (u - back + 2 * D) % D;
      return ring + grp[s / UNR] + (s % UNR) * SL;
    };
#pragma unroll 1
    for (int i0 = 0; i0 < nsteps; i0 += UNR) {
#pragma unroll
      for (int u = 0; u < UNR; ++u) {
        const int i = i0 + u;
        cp_async_wait<0>();
        // stage 0: xh = P + beta (P - Pprev) - t G replaces Pprev in the slot
        {
          float4* e = slot_of(u, 0);
          float2 p[CPL], q[CPL], g[CPL];
          ring_vals<ST, CPL>(e + 2 * QS, p);
          ring_vals<ST, CPL>(e, q);
          ring_vals<float2, CPL>(e + QS, g);
#pragma unroll
          for (int k = 0; k < F4; ++k) {
            const float2 xa = f2fma(nt2, g[2 * k], f2fma(bb, f2sub(p[2 * k], q[2 * k]), p[2 * k]));
            const float2 xb = f2fma(nt2, g[2 * k + 1], f2fma(bb, f2sub(p[2 * k + 1], q[2 * k + 1]), p[2 * k + 1]));
            e[k * 32] = make_float4(xa.x, xa.y, xb.x, xb.y);
          }
        }
        if (i + 1 < nsteps) request(slot_of(u, -1));

        float2 ny[CPL];   // gy of the iteration before, on the row below
        // iteration 1 on row j-1: g^0 = 0, so the estimate is xh itself; in the
        // second part g^0 is the first part's dual, loaded with the rows
        {
          float2 y[CPL], yl[CPL], g0x[CPL], g0y[CPL];
          ring_vals<float2, CPL>(slot_of(u, 1), y);
          if constexpr (PART == 2) {
            float2 g1y[CPL], gxr[CPL];
            const float4* gp = gring + ((u + 1) & 1) * 2 * 32;  // row j-1 (steps of even i0 + u at 0)
            const float4* gq = gring + (u & 1) * 2 * 32;        // row j
            ring_vals<float2, CPL>(gp, g0x);
            ring_vals<float2, CPL>(gp + 32, g0y);
            ring_vals<float2, CPL>(gq + 32, g1y);
#pragma unroll
            for (int c = 0; c < CPL - 1; ++c) gxr[c] = g0x[c + 1];
            gxr[CPL - 1] = shfl_down2(g0x[0]);
#pragma unroll
            for (int c = 0; c < CPL; ++c) y[c] = tv_estimate(y[c], g0x[c], gxr[c], g0y[c], g1y[c], nmu);
            // row j-1's values have been used, so its slot is free: the next
            // step's row goes there
            if (i + 1 < nsteps) request_g(goff, i + 1);
          } else {
#pragma unroll
            for (int c = 0; c < CPL; ++c) g0x[c] = g0y[c] = z2;
          }
          yl[0] = shfl_up2(y[CPL - 1]);
#pragma unroll
          for (int c = 1; c < CPL; ++c) yl[c] = y[c - 1];
#pragma unroll
          for (int c = 0; c < CPL; ++c) {
            float2 gx = g0x[c], gy = g0y[c];
            tv_dual(gx, gy, y[c], yl[c], yU[0][c], s2);
            yU[0][c] = y[c];
            ny[c] = gy;
            // the new row replaces the one above it, which moves to (y, yl)
            const float2 ogx = gX[0][c], ogy = gY[0][c];
            gX[0][c] = gx;
            gY[0][c] = gy;
            y[c] = ogx;
            yl[c] = ogy;
          }
          // from here (y, yl) carry the previous iteration's (gx, gy) on the
          // row the next stage works on
#pragma unroll
          for (int L = 1; L <= NTV; ++L) {
            // stage L+1 (iteration L+1, or the final stage when L == NTV) on row j-1-L
            const float4* e = slot_of(u, 1 + L);
            float2 xh[CPL];
            ring_vals<float2, CPL>(e, xh);
            float2 gxr[CPL], yy[CPL];
#pragma unroll
            for (int c = 0; c < CPL - 1; ++c) gxr[c] = y[c + 1];
            gxr[CPL - 1] = shfl_down2(y[0]);
#pragma unroll
            for (int c = 0; c < CPL; ++c) yy[c] = tv_estimate(xh[c], y[c], gxr[c], yl[c], ny[c], nmu);
            if (L < NTV) {
              float2 yls[CPL];
              yls[0] = shfl_up2(yy[CPL - 1]);
#pragma unroll
              for (int c = 1; c < CPL; ++c) yls[c] = yy[c - 1];
#pragma unroll
              for (int c = 0; c < CPL; ++c) {
                float2 gx = y[c], gy = yl[c];
                tv_dual(gx, gy, yy[c], yls[c], yU[L][c], s2);
                yU[L][c] = yy[c];
                ny[c] = gy;
                const float2 ogx = gX[L][c], ogy = gY[L][c];
                gX[L][c] = gx;
                gY[L][c] = gy;
                y[c] = ogx;
                yl[c] = ogy;
              }
            } else if constexpr (PART == 1) {
              // first part: (y, yl) hold this kernel's last dual on row j - h; it
              // goes to memory for the second part instead of the estimate
              if (i >= 2 * h + pad && lane_ok) {
                const size_t eo = plane + (size_t)orow * W + gc;
                *reinterpret_cast<float4*>(a.gdx + eo) = make_float4(y[0].x, y[0].y, y[1].x, y[1].y);
                *reinterpret_cast<float4*>(a.gdy + eo) = make_float4(yl[0].x, yl[0].y, yl[1].x, yl[1].y);
              }
            } else {
              // final stage: p = shrink(estimate) on row j - h, then the sums
              float2 p[CPL], x[CPL], g[CPL], y0[CPL];
              ring_vals<float2, CPL>(e + QS, g);
              ring_vals<ST, CPL>(e + 2 * QS, y0);
#pragma unroll
              for (int c = 0; c < CPL; ++c) {
                p[c] = shrink(yy[c], thr, faithful);
                x[c] = make_float2(fmaf(t, g[c].x, xh[c].x), fmaf(t, g[c].y, xh[c].y));
              }
              if (i >= 2 * h + pad) {  // row orow is exact
                float2 pl0 = z2, xl0 = z2;
                if (NORMS) {
                  pl0 = shfl_up2(p[CPL - 1]);
                  xl0 = shfl_up2(x[CPL - 1]);
                }
                if (lane_ok) {
                  const size_t eo = (size_t)orow * W + gc;
                  store_run<ST, CPL>(Pn + eo, p);
                  float wr, wi;
                  restart_w(eo, faithful, &wr, &wi);
#pragma unroll
                  for (int c = 0; c < CPL; ++c) {
                    const float2 d = f2sub(p[c], x[c]);
                    acc[SUM_LIM1] = fmaf(d.x, g[c].x, fmaf(d.y, g[c].y, acc[SUM_LIM1]));
                    acc[SUM_LIM2] = fmaf(d.x, d.x, fmaf(d.y, d.y, acc[SUM_LIM2]));
                    const float2 dv = f2mul(d, f2sub(p[c], y0[c]));  // (x - p)(p - y0) with the sign turned
                    acc[SUM_RS] = fmaf(-wr, dv.x, fmaf(-wi, dv.y, acc[SUM_RS]));
                    if (NORMS) {
                      const float2 pl = c ? p[c - 1] : pl0, xl = c ? x[c - 1] : xl0;
                      acc[SUM_L1P] += norm_sqrt(cabs2(p[c]));
                      acc[SUM_TVP] += norm_sqrt(cabs2(f2sub(pl, p[c])) + cabs2(f2sub(pu[c], p[c])));
                      acc[SUM_L1X] += norm_sqrt(cabs2(x[c]));
                      acc[SUM_TVX] += norm_sqrt(cabs2(f2sub(xl, x[c])) + cabs2(f2sub(xu[c], x[c])));
                    }
                  }
                }
                if (((i - 2 * h - pad) & 7) == 7) {  // FP32 partials over at most 8 rows
#pragma unroll
                  for (int k = 0; k < NS; ++k) {
                    dsum[k][threadIdx.x] += (double)acc[k];
                    acc[k] = 0.f;
                  }
                }
              }
              if (NORMS) {
#pragma unroll
                for (int c = 0; c < CPL; ++c) {
                  pu[c] = p[c];
                  xu[c] = x[c];
                }
              }
            }
          }
        }
        orow = (orow + 1 == H) ? 0 : orow + 1;
      }
      const int g0 = grp[0];
#pragma unroll
      for (int k = 0; k + 1 < D / UNR; ++k) grp[k] = grp[k + 1];
      grp[D / UNR - 1] = g0;
    }
    cp_async_wait<0>();
#pragma unroll
    for (int k = 0; k < NS; ++k) dsum[k][threadIdx.x] += (double)acc[k];
  }
  if constexpr (PART != 1) {
    double dacc[kNumSums];
#pragma unroll
    for (int k = 0; k < kNumSums; ++k) dacc[k] = k < NS ? dsum[k < NS ? k : 0][threadIdx.x] : 0.0;
    block_write_sums<32 * NW>(dacc, a.partials, blockIdx.x);
  }
}

// Runs per plane: enough warps for several full waves, while keeping the
// warm-up rows of each run small against the run length.
inline TvsGrid tvs_grid(int W, int H, int Nz, int VW, int warps_per_sm, int warm) {
  TvsGrid g;
  g.nstrips = (W + VW - 1) / VW;
  const double slots = (double)num_sms() * warps_per_sm;  // resident warps
  double best = 1e300;
  g.nseg = 1;
  for (int ns = 1; ns <= 64 && ns <= H; ++ns) {
    const int len = (H + ns - 1) / ns;
    if (ns > 1 && len < 2 * warm) break;
    const double runs = (double)g.nstrips * ns * Nz;
    const double waves = std::ceil(runs / slots);
    const double cost = waves * (len + warm);  // steps on the critical path
    if (cost < best * 0.999) {
      best = cost;
      g.nseg = ns;
    }
  }
  g.seg_len = (H + g.nseg - 1) / g.nseg;
  g.nseg = (H + g.seg_len - 1) / g.seg_len;
  return g;
}

// Warps a block of the streaming prox: 2 (built in), or 4 when the tuning
// asks for it (tv_kernel 3) and the 8-row ring applies (n_tv <= 5), where
// three 4-warp blocks (12 warps) share an SM at up to 168 registers.
template <int NTV, bool NORMS, int NW>
constexpr int tvw_minb_nw() {
  return NW == 2 ? tvw_minb<NTV, NORMS>() : 3;
}

template <typename ST, int NTV, bool NORMS, int NW, int PART = 0>
static cudaError_t strip_launch_nw(const ProxArgs& a, int* nblocks_out, cudaStream_t st) {
  using Sh = TvwShape<NTV, 2>;
  constexpr int MINB = tvw_minb_nw<NTV, NORMS, NW>();
  // one ring a warp, and for the second part a 4-row ring of the stored duals
  constexpr size_t SMEM = Sh::SMEM / Sh::NW * NW + (PART == 2 ? (size_t)NW * 2 * 32 * 2 * sizeof(float4) : 0);
  auto kern = k_prox_tv2d_strip<ST, NTV, NORMS, 2, NW, MINB, PART>;
  cudaError_t e = allow_smem(kern, SMEM);
  if (e != cudaSuccess) return e;
  // resident blocks per SM, for the choice of runs per plane
  static const int resident = [kern] {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kern, 32 * NW, SMEM) != cudaSuccess || b <= 0) {
      cudaGetLastError();
      b = MINB;
    }
    return b;
  }();
  TvsGrid g = tvs_grid(a.W, a.H, a.Nz, Sh::VW, NW * resident, 2 * Sh::h + 3);
  if (a.tv_nseg > 0) {  // tuned number of runs per plane
    g.seg_len = (a.H + min(a.tv_nseg, a.H) - 1) / min(a.tv_nseg, a.H);
    g.nseg = (a.H + g.seg_len - 1) / g.seg_len;
  }
  const long long runs = (long long)g.nstrips * g.nseg * a.Nz;
  const long long blocks = (runs + NW - 1) / NW;
  if (blocks > 0x7fffffffLL || blocks > a.partial_cap) return cudaErrorInvalidConfiguration;
  *nblocks_out = (int)blocks;
  kern<<<(unsigned)blocks, 32 * NW, SMEM, st>>>(a, g);
  return cudaGetLastError();
}

template <typename ST, int NTV, bool NORMS>
static cudaError_t strip_launch_n(const ProxArgs& a, int* nblocks_out, cudaStream_t st) {
  if constexpr (TvwShape<NTV, 2>::D == 8) {
    if (a.tv_kernel == 3) return strip_launch_nw<ST, NTV, NORMS, 4>(a, nblocks_out, st);
  }
  return strip_launch_nw<ST, NTV, NORMS, 2>(a, nblocks_out, st);
}

template <typename ST, int NTV>
static cudaError_t strip_launch(const ProxArgs& a, int* nblocks_out, cudaStream_t st) {
  return a.want_norms ? strip_launch_n<ST, NTV, true>(a, nblocks_out, st)
                      : strip_launch_n<ST, NTV, false>(a, nblocks_out, st);
}

// n_tv = K1 + K2 Chambolle iterations as two streaming launches: the first
// runs iterations 1..K1 and stores the dual (gx, gy) of every voxel (gx in
// a.gdx, gy in a.gdy, FP32 complex); the second starts from that dual, runs
// iterations K1+1..n_tv, the estimate, the shrink and the sums.  Each launch
// needs an x halo of K + 1 columns instead of n_tv + 1 and the 8-row ring, so
// at n_tv = 10 a 64-column strip keeps 52 valid columns instead of 40 and 16
// warps share an SM instead of 8.  The arithmetic is the single pass's, in the
// same order, and the dual goes through memory unrounded, so P_new has the
// same bits; only the second launch writes block partials.
template <typename ST, int K1, int K2>
static cudaError_t strip_launch_split(const ProxArgs& a, int* nblocks_out, cudaStream_t st) {
  int nb1 = 0;
  cudaError_t e = strip_launch_nw<ST, K1, false, 2, 1>(a, &nb1, st);
  if (e != cudaSuccess) return e;
  return a.want_norms ? strip_launch_nw<ST, K2, true, 2, 2>(a, nblocks_out, st)
                      : strip_launch_nw<ST, K2, false, 2, 2>(a, nblocks_out, st);
}

template <typename ST>
static cudaError_t strip_dispatch(const ProxArgs& a, int* nb, cudaStream_t st) {
  if (a.gdx && a.gdy && a.tv_kernel != 4) {  // two launches for more than 5 iterations
    switch (a.n_tv) {
      case 6: return strip_launch_split<ST, 3, 3>(a, nb, st);
      case 7: return strip_launch_split<ST, 3, 4>(a, nb, st);
      case 8: return strip_launch_split<ST, 4, 4>(a, nb, st);
      case 9: return strip_launch_split<ST, 4, 5>(a, nb, st);
      case 10: return strip_launch_split<ST, 5, 5>(a, nb, st);
      default: break;
    }
  }
  switch (a.n_tv) {
    case 1: return strip_launch<ST, 1>(a, nb, st);
    case 2: return strip_launch<ST, 2>(a, nb, st);
    case 3: return strip_launch<ST, 3>(a, nb, st);
    case 4: return strip_launch<ST, 4>(a, nb, st);
    case 5: return strip_launch<ST, 5>(a, nb, st);
    case 6: return strip_launch<ST, 6>(a, nb, st);
    case 7: return strip_launch<ST, 7>(a, nb, st);
    case 8: return strip_launch<ST, 8>(a, nb, st);
    case 9: return strip_launch<ST, 9>(a, nb, st);
    case 10: return strip_launch<ST, 10>(a, nb, st);
    default: return cudaErrorInvalidValue;
  }
}
constexpr int kStripNtvMax = 10;

// RIHVR_TV_KERNEL=tiles forces the tiled kernel (comparison and fallback);
// read once per process.
inline bool tv_stream_enabled() {
  static const bool on = [] {
    const char* v = std::getenv("RIHVR_TV_KERNEL");
    return !(v && std::strcmp(v, "tiles") == 0);
  }();
  return on;
}
// RIHVR_TV_KERNEL=strip4 (4-warp blocks) or strip1 (one launch for 6-10
// iterations) as tv_kernel 3 or 4; 0 when unset
inline int tv_kernel_forced() {
  static const int k = [] {
    const char* v = std::getenv("RIHVR_TV_KERNEL");
    if (v && std::strcmp(v, "strip4") == 0) return 3;
    if (v && std::strcmp(v, "strip1") == 0) return 4;
    return 0;
  }();
  return k;
}

inline void tv_grid(const ProxArgs& a, dim3* g) {
  const int h = a.n_tv + 1;
  const int VW = TV_EW - 2 * h, VH = TV_EH - 2 * h;
  *g = dim3((a.W + VW - 1) / VW, (a.H + VH - 1) / VH, a.Nz);
}


template <typename ST>
cudaError_t prox_tv2d_stored(const ProxArgs& a, int* nblocks_out, cudaStream_t st) {
  if (a.n_tv < 0 || a.n_tv > 20) return cudaErrorInvalidValue;
  if (a.n_tv >= 1 && a.n_tv <= kStripNtvMax && a.tv_kernel != 1 && tv_stream_enabled()) {
    ProxArgs b = a;
    if (tv_kernel_forced()) b.tv_kernel = tv_kernel_forced();
    return strip_dispatch<ST>(b, nblocks_out, st);
  }
  dim3 g;
  tv_grid(a, &g);
  *nblocks_out = (int)(g.x * g.y * g.z);
  const cudaError_t e = allow_smem(k_prox_tv2d<ST>, TV_SMEM);
  if (e != cudaSuccess) return e;
  k_prox_tv2d<ST><<<g, TV_THREADS, TV_SMEM, st>>>(a);
  return cudaGetLastError();
}

}  // namespace rihvr
