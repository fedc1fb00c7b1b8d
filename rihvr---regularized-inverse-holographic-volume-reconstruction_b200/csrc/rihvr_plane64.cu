// Spectrum of a real plane in FP64, rounded once to FP32.
//
// The residual of every iteration is the estimate's spectrum minus the measured
// hologram's.  The latter is the same in all of them, so its rounding does not
// average out over a solve as that of the transforms in the loop does: from FP32
// transforms (2e-7 of the hologram) it left the volume 5 to 20 % farther from a
// solve in 64 bits than a residual formed in space.  It is made once a hologram,
// so the two passes can be in FP64.
//
// A block transforms two lines (one, where two do not fit shared memory) of any
// supported side: Stockham stages of radix 4, 2, 3, 5 and 7 between two buffers,
// with the twiddles in a shared table.  What bounds it: latency (a few waves of
// blocks, one or two an SM, a barrier a stage).  A hologram's two passes take 10 us
// more than FP32 ones at side 512, 33 at 1024 and 245 at 2304; one line a block, 512
// threads or a table made from fewer sincos did not shorten them.
#include "rihvr_device.cuh"
#include "rihvr_kernels.cuh"
#include "rihvr_launch.cuh"

namespace rihvr {

namespace {

constexpr int kThreads = 256, kMaxStages = 12;

struct Plan64 {
  int n, stages;
  int r[kMaxStages];
};

bool plan64(int n, Plan64* p) {
  p->n = n;
  p->stages = 0;
  for (int r : {4, 2, 3, 5, 7})
    while (n % r == 0) {
      if (p->stages == kMaxStages) return false;
      p->r[p->stages++] = r;
      n /= r;
    }
  return n == 1;
}

size_t smem64(int n, int lines) { return sizeof(double2) * ((size_t)n + 2 * (size_t)n * lines); }

__device__ __forceinline__ double2 add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 mul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}

// One stage over the block's lines, element i of line c at [i * lines + c]; ns is the
// product of the radices before it.
template <int R>
__device__ __forceinline__ void stage64(const double2* in, double2* out, const double2* tw, int n, int ns, int lines) {
  const int m = n / R, step = m / ns;  // twiddle exponent of one step of k
  for (int b = threadIdx.x; b < m * lines; b += kThreads) {
    const int j = b / lines, c = b - j * lines, k = j % ns;
    double2 a[R], x[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      a[r] = in[(j + r * m) * lines + c];
      if (r > 0) a[r] = mul(a[r], tw[k * r * step]);
    }
    if constexpr (R == 4) {
      const double2 s = add(a[0], a[2]), d = sub(a[0], a[2]), t = add(a[1], a[3]), e = sub(a[1], a[3]);
      x[0] = add(s, t);
      x[1] = make_double2(d.x + e.y, d.y - e.x);
      x[2] = sub(s, t);
      x[3] = make_double2(d.x - e.y, d.y + e.x);
    } else {
#pragma unroll
      for (int q = 0; q < R; ++q) {
        x[q] = a[0];
#pragma unroll
        for (int r = 1; r < R; ++r) x[q] = add(x[q], mul(a[r], tw[q * r % R * m]));
      }
    }
    const int o = (j - k) * R + k;
#pragma unroll
    for (int q = 0; q < R; ++q) out[(o + q * ns) * lines + c] = x[q];
  }
}

// ROWS: lines of the real plane `src` into dst; else columns of it, rounded to FP32.
template <bool ROWS>
__global__ void __launch_bounds__(kThreads)
    k_plane64(const __grid_constant__ Plan64 p, const void* __restrict__ src, void* __restrict__ dst, int W, int lines) {
  extern __shared__ __align__(16) double2 sm64[];
  const int n = p.n, first = blockIdx.x * lines, total = n * lines;
  double2* const tw = sm64;
  double2 *in = sm64 + n, *out = in + total;
  for (int i = threadIdx.x; i < n; i += kThreads) {
    double s, c;
    sincospi(-2.0 * i / n, &s, &c);
    tw[i] = make_double2(c, s);
  }
  for (int e = threadIdx.x; e < total; e += kThreads) {
    if constexpr (ROWS) {
      const int c = e / n, i = e - c * n;
      in[i * lines + c] = make_double2(static_cast<const float*>(src)[(size_t)(first + c) * W + i], 0.0);
    } else {
      const int i = e / lines, c = e - i * lines;
      in[e] = static_cast<const double2*>(src)[(size_t)i * W + first + c];
    }
  }
  __syncthreads();
  for (int i = 0, ns = 1; i < p.stages; ns *= p.r[i++]) {
    switch (p.r[i]) {
      case 2: stage64<2>(in, out, tw, n, ns, lines); break;
      case 3: stage64<3>(in, out, tw, n, ns, lines); break;
      case 4: stage64<4>(in, out, tw, n, ns, lines); break;
      case 5: stage64<5>(in, out, tw, n, ns, lines); break;
      default: stage64<7>(in, out, tw, n, ns, lines); break;
    }
    __syncthreads();
    double2* const t = in;
    in = out;
    out = t;
  }
  for (int e = threadIdx.x; e < total; e += kThreads) {
    if constexpr (ROWS) {
      const int c = e / n, i = e - c * n;
      static_cast<double2*>(dst)[(size_t)(first + c) * W + i] = in[i * lines + c];
    } else {
      const int i = e / lines, c = e - i * lines;
      static_cast<float2*>(dst)[(size_t)i * W + first + c] = make_float2((float)in[e].x, (float)in[e].y);
    }
  }
}

template <bool ROWS>
cudaError_t pass64(const void* src, void* dst, int W, int H, cudaStream_t st) {
  Plan64 p;
  if (!plan64(ROWS ? W : H, &p)) return cudaErrorInvalidValue;
  // both sides are even; 227 KB hold two lines of up to 2905 elements, and one of 4096
  const int lines = smem64(p.n, 2) <= 227 * 1024 ? 2 : 1;
  const size_t smem = smem64(p.n, lines);
  const cudaError_t e = allow_smem(k_plane64<ROWS>, smem);
  if (e != cudaSuccess) return e;
  k_plane64<ROWS><<<(ROWS ? H : W) / lines, kThreads, smem, st>>>(p, src, dst, W, lines);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_plane_spectrum(const float* src, double2* work, float2* dst, int W, int H, cudaStream_t st) {
  const cudaError_t e = pass64<true>(src, work, W, H, st);
  return e != cudaSuccess ? e : pass64<false>(work, dst, W, H, st);
}

}  // namespace rihvr
