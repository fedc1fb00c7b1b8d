// Weight gradient of the warm-start network's 3x3x3 convolutions:
//   dW[co][k][ci] += sum_v dY[v][co] X[v + off_k][ci],   k = 27 taps.
//
// A GEMM with the voxels as its long dimension.  A block walks bricks of
// BZ x BY x BX voxels; for each it stages dY and the halo of X (16 input
// channels) once, rounded to BF16 as the forward convolution rounds its
// operands, and all 27 taps read their shifted windows of that halo.  Its nine
// warps take the nine (dz, dy) pairs, three dx taps each; the partial sums of
// a warp's 3 taps x Cout x 16 stay in FP32 registers over all of the block's
// bricks and reach memory as one atomic add each at the end.  The tensor core's
// own accumulation truncates, so a chain of MMAs ends after at most 16 steps
// (256 voxels) in a rounded FP32 add to a second set of registers; at 64 output
// channels, where these do not fit, a block takes two small bricks and ends.
// (One chain over a block's bricks left the gradients 1.5e-5 off.)  Both operands
// lie voxel by voxel, so the fragments of mma.sync m16n8k16 (M = output
// channels, N = input channels, K = 16 voxels of an x-row) come through
// ldmatrix.trans, without a transposed copy.
//
// What bounds it: shared-memory reads of the fragments (4 ldmatrix.x4 for 6
// MMAs at 16 output channels).  The form before it gave every tap and slice a
// grid of its own, which staged every voxel of X and dY 27 times through
// scalar transposing stores and added its sums by atomics every 1024 voxels: the
// gradients of a 32 x 128 x 128 volume took 16.2 ms with it, 2.3 ms with this one
// (a 16 -> 16 layer at full size 53 us).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "rihvr_unet_tc.cuh"

namespace rihvr {
namespace unet {

namespace {

constexpr int kWgWarps = 9, kWgThreads = 32 * kWgWarps;

template <int COT, int BZ, int BY, int BX>
struct WgShape {
  static constexpr int CO = 16 * COT;
  static constexpr int HZ = BZ + 2, HY = BY + 2, HX = BX + 2;
  static constexpr int HALO = HZ * HY * HX, VOX = BZ * BY * BX;
  static constexpr size_t SMEM = sizeof(__nv_bfloat16) * (16 * (size_t)HALO + (size_t)CO * VOX);
};

__device__ __forceinline__ unsigned pack2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const unsigned*>(&v);
}
__device__ __forceinline__ uint4 pack8(const float* p) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  return make_uint4(pack2(a.x, a.y), pack2(a.z, a.w), pack2(b.x, b.y), pack2(b.z, b.w));
}

// 16-byte chunk c of row r of an array of CH chunks a row, swizzled so that
// the same chunk of 8 consecutive rows covers the 32 banks once
template <int CH>
__device__ __forceinline__ int chunk_at(int r, int c) {
  if constexpr (CH == 2) return r * 2 + (c ^ ((r >> 2) & 1));
  else if constexpr (CH == 4) return r * 4 + (c ^ ((r >> 1) & 3));
  else return r * 8 + (c ^ (r & 7));
}

__device__ __forceinline__ void ldmatrix_x4_trans(unsigned (&v)[4], const void* row) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(row);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"(a)
               : "memory");
}

__device__ __forceinline__ void mma_16816(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int COT, int BZ, int BY, int BX>
__global__ void __launch_bounds__(kWgThreads)
    k_wgrad(const float* __restrict__ X, int Cin, const float* __restrict__ dY, float* __restrict__ dW, int D, int H,
            int W, int bricks) {
  using Sh = WgShape<COT, BZ, BY, BX>;
  constexpr int CO = Sh::CO, CH = 2 * COT;
  extern __shared__ __align__(16) uint4 wsm[];
  uint4* const Xs = wsm;                 // [HALO][2 chunks]
  uint4* const Ys = wsm + 2 * Sh::HALO;  // [VOX][CH chunks]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int dz = warp / 3, dy = warp % 3;  // halo offsets 0..2
  const int s = blockIdx.y;                // slice of 16 input channels
  const int nbx = (W + BX - 1) / BX, nby = (H + BY - 1) / BY;
  // fragment addresses: matrix m of an x4 load is read by lanes 8 m .. 8 m + 7, one row each
  const int mr = lane & 7, m = lane >> 3;
  const int a_vox = mr + (m >> 1) * 8, a_chunk = m & 1;  // A: (voxels, co) quarters
  const int b_vox = mr + (m & 1) * 8, b_chunk = m >> 1;  // B: (voxels, ci) quarters
  constexpr bool SUMS = COT <= 2;  // a second set of registers takes the chains' results
  constexpr int ROWS = 16 * 16 / BX < BZ * BY ? 16 * 16 / BX : BZ * BY;  // x-rows of a chain
  static_assert(BZ * BY % ROWS == 0, "whole chains");
  float acc[3][COT][2][4], sum[SUMS ? 3 : 1][SUMS ? COT : 1][2][4];
  auto each = [&](auto fn) {
#pragma unroll
    for (int t = 0; t < 3; ++t)
#pragma unroll
      for (int i = 0; i < COT; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int h = 0; h < 4; ++h) fn(t, i, j, h);
  };
  each([&](int t, int i, int j, int h) {
    acc[t][i][j][h] = 0.f;
    if constexpr (SUMS) sum[t][i][j][h] = 0.f;
  });
#pragma unroll 1
  for (int b = blockIdx.x; b < bricks; b += gridDim.x) {
    const int x0 = (b % nbx) * BX, y0 = ((b / nbx) % nby) * BY, z0 = (b / (nbx * nby)) * BZ;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    for (int e = threadIdx.x; e < 2 * Sh::HALO; e += kWgThreads) {
      const int h = e >> 1, c = e & 1;
      const int hx = h % Sh::HX, hy = (h / Sh::HX) % Sh::HY, hz = h / (Sh::HX * Sh::HY);
      const int x = x0 + hx - 1, y = y0 + hy - 1, z = z0 + hz - 1;
      const bool in = x >= 0 && x < W && y >= 0 && y < H && z >= 0 && z < D;
      Xs[chunk_at<2>(h, c)] =
          in ? pack8(X + (((size_t)z * H + y) * W + x) * Cin + s * 16 + c * 8) : zero;
    }
    for (int e = threadIdx.x; e < CH * Sh::VOX; e += kWgThreads) {
      const int v = e / CH, c = e % CH;
      const int x = x0 + v % BX, y = y0 + (v / BX) % BY, z = z0 + v / (BX * BY);
      Ys[chunk_at<CH>(v, c)] =
          (x < W && y < H && z < D) ? pack8(dY + (((size_t)z * H + y) * W + x) * CO + c * 8) : zero;
    }
    __syncthreads();
#pragma unroll 1
    for (int row = 0; row < BZ * BY; ++row) {
      if constexpr (SUMS) {
        if (row % ROWS == 0)
          each([&](int t, int i, int j, int h) {
            sum[t][i][j][h] += acc[t][i][j][h];
            acc[t][i][j][h] = 0.f;
          });
      }
      const int rz = row / BY, ry = row % BY;
      const int hrow = ((rz + dz) * Sh::HY + ry + dy) * Sh::HX;  // halo voxel left of the row (dx = 0)
#pragma unroll
      for (int xs = 0; xs < BX; xs += 16) {
        unsigned a[COT][4];
#pragma unroll
        for (int i = 0; i < COT; ++i)
          ldmatrix_x4_trans(a[i], Ys + chunk_at<CH>(row * BX + xs + a_vox, 2 * i + a_chunk));
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          unsigned q[4];
          ldmatrix_x4_trans(q, Xs + chunk_at<2>(hrow + xs + t + b_vox, b_chunk));
#pragma unroll
          for (int i = 0; i < COT; ++i) {
            mma_16816(acc[t][i][0], a[i], q[0], q[1]);
            mma_16816(acc[t][i][1], a[i], q[2], q[3]);
          }
        }
      }
    }
    __syncthreads();
  }
  if constexpr (SUMS) each([&](int t, int i, int j, int h) { acc[t][i][j][h] += sum[t][i][j][h]; });
  const int g = lane >> 2, t4 = lane & 3;
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const int k = (dz * 3 + dy) * 3 + t;
#pragma unroll
    for (int i = 0; i < COT; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float* d = dW + ((size_t)(i * 16 + g + h * 8) * 27 + k) * Cin + s * 16 + j * 8 + 2 * t4;
          atomicAdd(d, acc[t][i][j][2 * h]);
          atomicAdd(d + 1, acc[t][i][j][2 * h + 1]);
        }
  }
}

template <int COT, int BZ, int BY, int BX>
cudaError_t wgrad_launch(const float* X, int Cin, const float* dY, float* dW, int D, int H, int W, int blocks_max,
                         cudaStream_t st) {
  using Sh = WgShape<COT, BZ, BY, BX>;
  const cudaError_t e = cudaFuncSetAttribute(k_wgrad<COT, BZ, BY, BX>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)Sh::SMEM);
  if (e != cudaSuccess) return e;
  const long long bricks = (long long)((W + BX - 1) / BX) * ((H + BY - 1) / BY) * ((D + BZ - 1) / BZ);
  if (bricks > 0x7fffffffLL) return cudaErrorInvalidValue;
  const int slices = Cin / 16;
  // a block's walk over the bricks, or, without the second registers, two of them
  const int gx = COT <= 2 ? (int)std::min<long long>(bricks, std::max(1, blocks_max / slices))
                          : (int)((bricks + 1) / 2);
  k_wgrad<COT, BZ, BY, BX><<<dim3(gx, slices), kWgThreads, Sh::SMEM, st>>>(X, Cin, dY, dW, D, H, W, (int)bricks);
  return cudaGetLastError();
}

template <int COT>
cudaError_t wgrad_pick(const float* X, int Cin, const float* dY, float* dW, int D, int H, int W, cudaStream_t st) {
  constexpr int kSms = 148;
  // large bricks read 2 halo voxels of X for each of their own, small ones
  // 3.4; they are taken where they still give every SM a block
  if constexpr (COT <= 2) {
    const long long large = (long long)((W + 31) / 32) * ((H + 7) / 8) * ((D + 3) / 4) * (Cin / 16);
    if (large >= kSms) return wgrad_launch<COT, 4, 8, 32>(X, Cin, dY, dW, D, H, W, 2 * kSms, st);
  }
  return wgrad_launch<COT, 2, 4, 16>(X, Cin, dY, dW, D, H, W, 4 * kSms, st);
}

}  // namespace

cudaError_t conv3_wgrad(const float* X, int Cin, const float* dY, int Cout, float* dW, int D, int H, int W,
                        cudaStream_t st) {
  if (Cin % 16 != 0) return cudaErrorInvalidValue;
  switch (Cout) {
    case 16: return wgrad_pick<1>(X, Cin, dY, dW, D, H, W, st);
    case 32: return wgrad_pick<2>(X, Cin, dY, dW, D, H, W, st);
    case 64: return wgrad_pick<4>(X, Cin, dY, dW, D, H, W, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace unet
}  // namespace rihvr
