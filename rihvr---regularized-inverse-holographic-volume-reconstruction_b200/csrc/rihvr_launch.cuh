// Launch helpers and device pieces shared by the kernel files of the
// reconstruction path: SM count, shared-memory opt-in, block sums, the shrink
// and the restart weights.
#pragma once
#include <atomic>

#include "rihvr_device.cuh"
#include "rihvr_kernels.cuh"

namespace rihvr {

// SM count of the current device, cached per device ordinal.  Worker threads of
// a frame batch and callers on other host threads read it concurrently, so the
// cache entries are atomics (a racing first fill writes the same value twice).
constexpr int kSmCacheDevices = 64;
inline std::atomic<int> g_num_sms[kSmCacheDevices];
inline int num_sms() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
  std::atomic<int>* slot = (dev >= 0 && dev < kSmCacheDevices) ? &g_num_sms[dev] : nullptr;
  int n = slot ? slot->load(std::memory_order_relaxed) : 0;
  if (n <= 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    if (slot) slot->store(n, std::memory_order_relaxed);
  }
  return n;
}

template <typename K>
inline cudaError_t allow_smem(K kernel, size_t bytes) {
  // dynamic plus static shared memory above 48 KB needs the opt-in
  if (bytes + 4096 <= 48 * 1024) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

constexpr int FLAT_THREADS = 256;

// blocks of a flat grid-stride launch over n elements
inline int flat_blocks(size_t n) {
  size_t b = (n + FLAT_THREADS - 1) / FLAT_THREADS;
  size_t cap = (size_t)8 * num_sms();
  return (int)(b < cap ? (b > 0 ? b : 1) : cap);
}


// ---------------------------------------------------------------------------
// block reduction of kNumSums doubles into partials[block]
// ---------------------------------------------------------------------------
template <int NT>
__device__ __forceinline__ void block_write_sums(double (&acc)[kNumSums], double* partials, int block) {
  __shared__ double red[NT / 32][kNumSums];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < kNumSums; ++k) {
    double v = warp_sum(acc[k]);
    if (lane == 0) red[wid][k] = v;
  }
  __syncthreads();
  if (threadIdx.x < kNumSums) {
    double s = 0;
    for (int w = 0; w < NT / 32; ++w) s += red[w][threadIdx.x];
    partials[(size_t)block * kNumSums + threadIdx.x] = s;
  }
}

// A sum finished by the block that ends last: partials[block] = this block's
// sum; the last one to arrive adds them up in a fixed order into
// sums[SUM_RR] (the other sums of the slot become 0) and leaves the counter at
// 0 for the next launch.  Saves the one or two reduction launches that would
// follow a small kernel.  No block waits for another.
template <int NT>
__device__ __forceinline__ void last_block_rr(double acc, double* partials, double* sums, unsigned* counter) {
  __shared__ double red[NT / 32];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double v = warp_sum(acc);
  if (lane == 0) red[wid] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0;
    for (int w = 0; w < NT / 32; ++w) s += red[w];
    partials[blockIdx.x] = s;
    __threadfence();
    last = atomicInc(counter, gridDim.x - 1) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double t = 0;
  for (unsigned b = threadIdx.x; b < gridDim.x; b += NT) t += __ldcg(partials + b);
  t = warp_sum(t);
  __syncthreads();
  if (lane == 0) red[wid] = t;
  __syncthreads();
  if (threadIdx.x < kNumSums) {
    double s = 0;
    if (threadIdx.x == SUM_RR)
      for (int w = 0; w < NT / 32; ++w) s += red[w];
    sums[threadIdx.x] = s;
  }
}

// Restart statistic weights: sparse_fistaRestart_kernel<512> (RIHVR
// sparse_compressive_holo.cu:4393-4432) overwrites the second element's real
// product with its imaginary one and re-adds the first element's imaginary
// product (:4411-4413): within each 1024-element chunk of a plane, elements
// 0..511 count Re + 2 Im and elements 512..1023 count Im only.
__device__ __forceinline__ void restart_w(size_t e, int faithful, float* wr, float* wi) {
  if (!faithful) {
    *wr = 1.f;
    *wi = 1.f;
  } else if ((e & 1023u) < 512u) {
    *wr = 1.f;
    *wi = 2.f;
  } else {
    *wr = 0.f;
    *wi = 1.f;
  }
}

// Soft thresholds: block_soft_threshold_kernel (sparse_compressive_holo.cu:
// 3065-3110) shrinks Re and Im separately; the non-faithful variant shrinks
// the complex modulus.
__device__ __forceinline__ float2 shrink(float2 v, float T, int faithful) {
  if (T <= 0.f) return v;
  if (faithful) {
    const float mr = fabsf(v.x) - T, mi = fabsf(v.y) - T;
    return make_float2(mr > 0.f ? copysignf(mr, v.x) : 0.f, mi > 0.f ? copysignf(mi, v.y) : 0.f);
  }
  const float a = sqrtf(v.x * v.x + v.y * v.y);
  if (a <= T) return make_float2(0.f, 0.f);
  const float f = (a - T) / a;
  return make_float2(v.x * f, v.y * f);
}

__device__ __forceinline__ float cabs2(float2 a) { return a.x * a.x + a.y * a.y; }

// The prox arguments with the step and momentum scalars taken from their
// device copy when one is given (captured launches, see ProxArgs::dscal).
__device__ __forceinline__ ProxArgs resolve_scalars(const ProxArgs& a0) {
  ProxArgs a = a0;
  if (a0.dscal) {
    a.beta = __ldg(a0.dscal + 0);
    a.t = __ldg(a0.dscal + 1);
    a.mu = __ldg(a0.dscal + 2);
    a.s = __ldg(a0.dscal + 3);
    a.thr = __ldg(a0.dscal + 4);
  }
  return a;
}

// Square roots of the objective's norm terms (L1 and TV sums) use the
// hardware approximation in its flush-to-zero form (one instruction; a
// magnitude below 1.1e-19 counts as 0): they only feed the reported objective,
// summed over millions of voxels in FP64.
__device__ __forceinline__ float norm_sqrt(float q) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(q));
  return r;
}

__device__ __forceinline__ float2 shfl_down2(float2 v) {
  return make_float2(__shfl_down_sync(0xffffffffu, v.x, 1), __shfl_down_sync(0xffffffffu, v.y, 1));
}
__device__ __forceinline__ float2 shfl_up2(float2 v) {
  return make_float2(__shfl_up_sync(0xffffffffu, v.x, 1), __shfl_up_sync(0xffffffffu, v.y, 1));
}

template <typename ST>
struct Pair;  // two adjacent complex values in storage layout
template <>
struct Pair<float2> {
  using T = float4;
  static __device__ __forceinline__ void ld(const float2* p, float2& a, float2& b) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    a = make_float2(v.x, v.y);
    b = make_float2(v.z, v.w);
  }
};
template <>
struct Pair<__nv_bfloat162> {
  static __device__ __forceinline__ void ld(const __nv_bfloat162* p, float2& a, float2& b) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x));
    b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
  }
};
template <>
struct Pair<__half2> {
  static __device__ __forceinline__ void ld(const __half2* p, float2& a, float2& b) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    a = __half22float2(*reinterpret_cast<const __half2*>(&v.x));
    b = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
  }
};

template <typename ST>
struct Raw2;  // two adjacent complex values as loaded from storage
template <>
struct Raw2<float2> {
  using T = float4;
  static __device__ __forceinline__ T ld(const float2* p) { return *reinterpret_cast<const float4*>(p); }
  static __device__ __forceinline__ void cvt(T v, float2& a, float2& b) {
    a = make_float2(v.x, v.y);
    b = make_float2(v.z, v.w);
  }
  static __device__ __forceinline__ void st(float2* p, float2 a, float2 b) {
    *reinterpret_cast<float4*>(p) = make_float4(a.x, a.y, b.x, b.y);
  }
};
template <>
struct Raw2<__nv_bfloat162> {
  using T = uint2;
  static __device__ __forceinline__ T ld(const __nv_bfloat162* p) { return *reinterpret_cast<const uint2*>(p); }
  static __device__ __forceinline__ void cvt(T v, float2& a, float2& b) {
    a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x));
    b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
  }
  static __device__ __forceinline__ void st(__nv_bfloat162* p, float2 a, float2 b) {
    const __nv_bfloat162 u = __float22bfloat162_rn(a), v = __float22bfloat162_rn(b);
    *reinterpret_cast<uint2*>(p) =
        make_uint2(*reinterpret_cast<const unsigned*>(&u), *reinterpret_cast<const unsigned*>(&v));
  }
};
template <>
struct Raw2<__half2> {
  using T = uint2;
  static __device__ __forceinline__ T ld(const __half2* p) { return *reinterpret_cast<const uint2*>(p); }
  static __device__ __forceinline__ void cvt(T v, float2& a, float2& b) {
    a = __half22float2(*reinterpret_cast<const __half2*>(&v.x));
    b = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
  }
  static __device__ __forceinline__ void st(__half2* p, float2 a, float2 b) {
    const __half2 u = __float22half2_rn(a), v = __float22half2_rn(b);
    *reinterpret_cast<uint2*>(p) =
        make_uint2(*reinterpret_cast<const unsigned*>(&u), *reinterpret_cast<const unsigned*>(&v));
  }
};

// 16-byte asynchronous global -> shared copies (Ampere+ cp.async, L2 only)
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N_>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N_) : "memory");
}

// element of kind IN (compile time) as a complex value
template <int IN>
__device__ __forceinline__ float2 load_as(const void* p, size_t i) {
  if constexpr (IN == ELEM_R32) return make_float2(static_cast<const float*>(p)[i], 0.f);
  else if constexpr (IN == ELEM_STORE_BF16) return Store<__nv_bfloat162>::ld(static_cast<const __nv_bfloat162*>(p) + i);
  else if constexpr (IN == ELEM_STORE_F16) return Store<__half2>::ld(static_cast<const __half2*>(p) + i);
  else return static_cast<const float2*>(p)[i];
}

// keep the compiler from moving memory accesses across this point
__device__ __forceinline__ void sched_fence() { asm volatile("" ::: "memory"); }

}  // namespace rihvr
