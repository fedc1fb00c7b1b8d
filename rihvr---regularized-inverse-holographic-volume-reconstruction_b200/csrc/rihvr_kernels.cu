// sm_100a kernels of the reconstruction hot path.
//
// Operator structure (RIHVR src/core/sparse_compressive_holo.cu:1935-2077 forward,
// src/core/sparse_gradient.cu:47-165 adjoint), restated by linearity:
//   forward  d   = Re( F^-1 sum_z H'_z F(x_z) ),  H'_z = exp(i z c(f))
//   adjoint  g_z = F^-1( conj(H'_z) F(r) )
// with c(f) = 2 pi / lambda (sqrt(1 - (lambda f)^2) - 1).  The per-plane carrier
// factor exp(-+ i 2 pi z / lambda) that the reference applies separately is folded
// into H'_z.  The 2-D DFT of a plane is a row pass plus a column pass; the column
// passes carry the transfer-function multiply (regenerated from an FP64 table of
// c/(2 pi) per frequency, phase reduced mod 1 turn in FP64) and, for the forward
// operator, the sum over z, so the Nz transformed planes never go back to memory.
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <utility>

#include "rihvr_device.cuh"
#include "rihvr_kernels.cuh"
#include "rihvr_launch.cuh"
#include "rihvr_fast.cuh"
#include "rihvr_lines.cuh"

namespace rihvr {

// the sides' passes are compiled in rihvr_fast_*.cu
#define RIHVR_SIDE(NN) RIHVR_FAST_SIDE(extern, NN)
RIHVR_FOR_EACH_SIZE(RIHVR_SIDE)
#undef RIHVR_SIDE

bool line_size_supported(int n) {
  switch (n) {
#define RIHVR_CASE(NN) case NN:
    RIHVR_FOR_EACH_SIZE(RIHVR_CASE)
#undef RIHVR_CASE
    return true;
    default:
      return false;
  }
}

static cudaError_t launch_rows_fast(int inverse, int in_kind, const void* in, int out_kind, void* out, int W,
                                    long long nlines, float scale, cudaStream_t st) {
  switch (W) {
#define RIHVR_CASE(NN) \
  case NN:             \
    return rows_n<NN>(inverse, in_kind, in, out_kind, out, nlines, scale, st);
    RIHVR_FOR_EACH_SIZE(RIHVR_CASE)
#undef RIHVR_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

bool adj_recurrence_supported(int W, int H, int rec_mode) {
  switch (H) {
  // rectangular planes: the TMA-fed forms only, which need a column block's width (adj_col_n)
#define RIHVR_CASE(NN)                                                                         \
  case NN:                                                                                     \
    return W != NN && (rec_mode == 1 || W < ColLayout<NN>::CC) ? false                         \
           : rec_mode == 3                                     ? kTableCols<NN>                \
                                                               : (kHoistTw<NN> && (NN % ColLayout<NN>::CC == 0));
    RIHVR_FOR_EACH_SIZE(RIHVR_CASE)
#undef RIHVR_CASE
    default:
      return false;
  }
}

static cudaError_t launch_adj_col_fast(const float2* Rs, const double* cturn, const double* zlist, float2* U, int W,
                                      int H, int z0, int z1, cudaStream_t st, int chunks_hint, double dz_uniform,
                                      int rec_mode) {
  switch (H) {
#define RIHVR_CASE(NN) \
  case NN:             \
    return adj_col_n<NN>(Rs, cturn, zlist, U, W, z0, z1, st, chunks_hint, dz_uniform, rec_mode);
    RIHVR_FOR_EACH_SIZE(RIHVR_CASE)
#undef RIHVR_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

// Z-chunks of the forward column pass.  The cost of a count, in planes of one
// block: waves of resident blocks times (planes a chunk + what a block spends
// before its first plane: the twiddle table and the rotations, about three
// planes), plus the partial spectra, written and summed once a chunk.  At
// 1024 x 1024 x 1000 this takes 5 chunks (three waves of 200 planes) where
// 4 blocks an SM took 3 (1.7 waves of 334): 1.87 ms instead of 2.06; 384 x 384 x
// 40: 34 instead of 51 us (27 since the rotations come from a table).
static int fwd_col_chunks_fast(int W, int H, int Nz) {
  int cc = 8, resident = 2;
  switch (H) {
#define RIHVR_CASE(NN)                                                                       \
  case NN:                                                                                   \
    cc = ColLayout<NN>::CC;                                                                  \
    resident = kTableCols<NN> ? col3_minb<NN>() : 2;                                         \
    break;
    RIHVR_FOR_EACH_SIZE(RIHVR_CASE)
#undef RIHVR_CASE
    default:
      break;
  }
  const int strips = (W + cc - 1) / cc;
  const double slots = (double)num_sms() * resident;
  // bytes a block streams a plane, at its share of the pass's rate, against
  // the plane of partial sums of the whole chip
  const double per_chunk = 2.0 * (double)W / cc / slots;
  int best = 1;
  double least = 1e300;
  for (int ch = 1; ch <= 16 && ch <= Nz; ++ch) {
    const int zpb = (Nz + ch - 1) / ch, used = (Nz + zpb - 1) / zpb;
    if (used != ch) continue;  // the same chunk length with fewer chunks has been looked at
    const double cost = std::ceil(strips * ch / slots) * (zpb + 3) + ch * per_chunk;
    if (cost < least * 0.999) {
      least = cost;
      best = ch;
    }
  }
  return best;
}

// The adjoint column pass's built-in variant for evenly spaced planes: the
// recurrence where a block walks enough planes to pay for its rotations (a
// block's first plane costs about two more), with the twiddles kept in
// registers, or from the table for lines of 48 elements a thread: 0.92 instead
// of 1.17 ms at 2304 x 2304 x 48, 125 instead of 130 us at 512 x 512 x 200.
int adj_col_builtin(int W, int H, int Nz) {
  int cc = 8;
  switch (H) {
#define RIHVR_CASE(NN) \
  case NN:             \
    cc = ColLayout<NN>::CC; break;
    RIHVR_FOR_EACH_SIZE(RIHVR_CASE)
#undef RIHVR_CASE
    default:
      return 0;
  }
  const int strips = (W + cc - 1) / cc;
  if ((long long)Nz * strips < 4LL * 8 * num_sms()) return 0;
  return adj_recurrence_supported(W, H, 2) ? 2 : adj_recurrence_supported(W, H, 3) ? 3 : 0;
}

bool fwd_horner_supported(int W, int H, int horner_mode) {
  switch (H) {
  // rectangular planes: the TMA-fed form only, which needs a column block's width (fwd_col_n)
#define RIHVR_CASE(NN)                                                                    \
  case NN:                                                                                \
    return W != NN && (horner_mode != 3 || W < ColLayout<NN>::CC) ? false                 \
           : horner_mode >= 2                                     ? kTableCols<NN>        \
                                                                  : (ColLayout<NN>::STAGE && LineCfg<NN>::EXACT);
    RIHVR_FOR_EACH_SIZE(RIHVR_CASE)
#undef RIHVR_CASE
    default:
      return false;
  }
}

static cudaError_t launch_fwd_col_fast(const float2* T, const double* cturn, const double* zlist, float2* Spart,
                                      int W, int H, int z0, int z1, int nchunks, cudaStream_t st, int horner_mode,
                                      const HornerTable& table) {
  switch (H) {
#define RIHVR_CASE(NN) \
  case NN:             \
    return fwd_col_n<NN>(T, cturn, zlist, Spart, W, z0, z1, nchunks, st, horner_mode, table);
    RIHVR_FOR_EACH_SIZE(RIHVR_CASE)
#undef RIHVR_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

// HornerTable of the spacing dz: d is D = H'_dz rounded to FP32, drift D / d - 1 times
// kHornerDriftScale
__global__ void __launch_bounds__(FLAT_THREADS) k_horner_table(const double* __restrict__ cturn, double dz,
                                                               float2* __restrict__ d, __half2* __restrict__ drift,
                                                               long long n) {
  for (long long i = (long long)blockIdx.x * FLAT_THREADS + threadIdx.x; i < n; i += (long long)gridDim.x * FLAT_THREADS) {
    double u = dz * cturn[i], s, c;
    u -= rint(u);
    sincospi(2.0 * u, &s, &c);
    const float2 r = make_float2((float)c, (float)s);
    const float2 e = cmulc(make_float2((float)(c - (double)r.x), (float)(s - (double)r.y)), r);  // |r| = 1
    d[i] = r;
    drift[i] = __float22half2_rn(cscale(e, kHornerDriftScale));
  }
}

cudaError_t launch_horner_table(const double* cturn, double dz, float2* d, __half2* drift, long long n,
                                cudaStream_t st) {
  k_horner_table<<<flat_blocks((size_t)n), FLAT_THREADS, 0, st>>>(cturn, dz, d, drift, n);
  return cudaGetLastError();
}

static cudaError_t launch_plane_col_fast(int inverse, const float2* in, float2* out, int W, int H, float scale,
                                        cudaStream_t st) {
  switch (H) {
#define RIHVR_CASE(NN) \
  case NN:             \
    return plane_col_n<NN>(inverse, in, out, W, scale, st);
    RIHVR_FOR_EACH_SIZE(RIHVR_CASE)
#undef RIHVR_CASE
    default:
      return cudaErrorInvalidValue;
  }
}

// ---------------------------------------------------------------------------
// sum of partial spectra (fixed order: deterministic)
// ---------------------------------------------------------------------------
__global__ void k_sum_chunks(const float2* __restrict__ Spart, int nchunks, float2* __restrict__ S, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    float2 a = Spart[i];
    for (int k = 1; k < nchunks; ++k) a = cadd(a, Spart[(size_t)k * n + i]);
    S[i] = a;
  }
}

cudaError_t launch_sum_chunks(const float2* Spart, int nchunks, float2* S, long long n, cudaStream_t st) {
  int blocks = (int)((n + 255) / 256);
  if (blocks > 4 * num_sms()) blocks = 4 * num_sms();
  k_sum_chunks<<<blocks, 256, 0, st>>>(Spart, nchunks, S, n);
  return cudaGetLastError();
}

struct SlabSources {
  const float2* p[kMaxSlabs];
};

__global__ void k_sum_slabs(SlabSources s, int n, float2* __restrict__ dst, long long count) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (long long)gridDim.x * blockDim.x) {
    float2 a = s.p[0][i];
    for (int k = 1; k < n; ++k) a = cadd(a, s.p[k][i]);
    dst[i] = a;
  }
}

cudaError_t launch_sum_slabs(const float2* const* src, int n, float2* dst, long long count, cudaStream_t st) {
  if (n < 1 || n > kMaxSlabs) return cudaErrorInvalidValue;
  SlabSources s{};
  for (int k = 0; k < n; ++k) s.p[k] = src[k];
  int blocks = (int)((count + 255) / 256);
  if (blocks > 4 * num_sms()) blocks = 4 * num_sms();
  k_sum_slabs<<<blocks, 256, 0, st>>>(s, n, dst, count);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// reduction of block partials in two fixed-shape stages (deterministic):
// stage 1 sums contiguous slices of the partials, stage 2 sums the slices.
// ---------------------------------------------------------------------------
constexpr int RED_THREADS = 256;
constexpr int RED_SLICES = 512;

template <int NT>
__global__ void __launch_bounds__(NT) k_reduce_stage(const double* __restrict__ in, int n, int per_block,
                                                     double* __restrict__ out) {
  __shared__ double red[NT / 32][kNumSums];
  const int b0 = blockIdx.x * per_block, b1 = min(n, b0 + per_block);
  // thread j handles slot j % kNumSums of rows b0 + j / kNumSums, strided
  const int slot = threadIdx.x % kNumSums, lane_row = threadIdx.x / kNumSums;
  constexpr int ROWS_PER_PASS = NT / kNumSums;
  double v = 0.0;
  for (int b = b0 + lane_row; b < b1; b += ROWS_PER_PASS) v += in[(size_t)b * kNumSums + slot];
  // gather per-slot sums: rows of the same slot are kNumSums lanes apart
#pragma unroll
  for (int o = 16; o >= kNumSums; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane < kNumSums) red[wid][lane] = v;
  __syncthreads();
  if (threadIdx.x < kNumSums) {
    double s = 0.0;
    for (int w = 0; w < NT / 32; ++w) s += red[w][threadIdx.x];
    out[(size_t)blockIdx.x * kNumSums + threadIdx.x] = s;
  }
}

cudaError_t launch_reduce_partials(const double* partials, int nblocks, double* scratch, double* out,
                                   cudaStream_t st) {
  if (nblocks <= RED_THREADS) {
    k_reduce_stage<RED_THREADS><<<1, RED_THREADS, 0, st>>>(partials, nblocks, nblocks, out);
    return cudaGetLastError();
  }
  if (nblocks <= kReduceOneLaunch) {  // 16 rows a thread at most: shorter than a second launch
    k_reduce_stage<1024><<<1, 1024, 0, st>>>(partials, nblocks, nblocks, out);
    return cudaGetLastError();
  }
  const int per = (nblocks + RED_SLICES - 1) / RED_SLICES;
  const int slices = (nblocks + per - 1) / per;
  k_reduce_stage<RED_THREADS><<<slices, RED_THREADS, 0, st>>>(partials, nblocks, per, scratch);
  k_reduce_stage<RED_THREADS><<<1, RED_THREADS, 0, st>>>(scratch, slices, slices, out);
  return cudaGetLastError();
}

size_t reduce_scratch_doubles() { return (size_t)RED_SLICES * kNumSums; }

// ---------------------------------------------------------------------------
// plane-level kernels
// ---------------------------------------------------------------------------
// d = Re(c); sum (d - b)^2.  back_propagate_finish_kernel (:1918-1933) keeps
// only the real part; calcResidual (:2676-2723) forms r = estimate - measured.
__global__ void __launch_bounds__(FLAT_THREADS) k_finish_forward(const float2* __restrict__ c,
                                                                 const float* __restrict__ b,
                                                                 float* __restrict__ dnew, long long n,
                                                                 double* partials) {
  double acc[kNumSums];
#pragma unroll
  for (int k = 0; k < kNumSums; ++k) acc[k] = 0.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float d = c[i].x;
    dnew[i] = d;
    const float r = d - b[i];
    acc[SUM_RR] += (double)r * (double)r;
  }
  block_write_sums<FLAT_THREADS>(acc, partials, blockIdx.x);
}

cudaError_t launch_finish_forward(const float2* c, const float* b, float* dnew, long long n, double* partials,
                                  int* nblocks_out, cudaStream_t st) {
  const int blocks = flat_blocks((size_t)n);
  *nblocks_out = blocks;
  k_finish_forward<<<blocks, FLAT_THREADS, 0, st>>>(c, b, dnew, n, partials);
  return cudaGetLastError();
}

// Counter-based uniform fill in [-1, 1) for both parts of a complex volume
// (splitmix64 of the seed and the element index), so that a host model can
// regenerate exactly the same start vector.
__device__ __forceinline__ unsigned long long splitmix64(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ float unit_from_bits(unsigned long long r) {
  // top 24 bits -> [0, 1), then [-1, 1): exact in float
  return (float)(r >> 40) * (1.0f / 16777216.0f) * 2.0f - 1.0f;
}
__global__ void __launch_bounds__(FLAT_THREADS) k_fill_uniform_c(float2* __restrict__ x, long long n,
                                                                 unsigned long long seed) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const unsigned long long k = seed * 0x100000001B3ull + 2ull * (unsigned long long)i;
    x[i] = make_float2(unit_from_bits(splitmix64(k)), unit_from_bits(splitmix64(k + 1)));
  }
}

cudaError_t launch_fill_uniform_c(float2* x, long long n, unsigned long long seed, cudaStream_t st) {
  k_fill_uniform_c<<<flat_blocks((size_t)n), FLAT_THREADS, 0, st>>>(x, n, seed);
  return cudaGetLastError();
}

// sum x^2 over n floats in FP64 (the SUM_RR entry of the block partials)
__global__ void __launch_bounds__(FLAT_THREADS) k_sumsq(const float* __restrict__ x, long long n, double* partials) {
  double acc[kNumSums];
#pragma unroll
  for (int k = 0; k < kNumSums; ++k) acc[k] = 0.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double v = x[i];
    acc[SUM_RR] += v * v;
  }
  block_write_sums<FLAT_THREADS>(acc, partials, blockIdx.x);
}

cudaError_t launch_sumsq(const float* x, long long n, double* partials, int* nblocks_out, cudaStream_t st) {
  const int blocks = flat_blocks((size_t)n);
  *nblocks_out = blocks;
  k_sumsq<<<blocks, FLAT_THREADS, 0, st>>>(x, n, partials);
  return cudaGetLastError();
}

// Momentum in hologram space (:480-498, fistaUpdate on holograms :4599-4642):
// dX = d + beta (d - dY0); dY0 = d; r = dX - b.
__global__ void __launch_bounds__(FLAT_THREADS) k_holo_momentum(const float* __restrict__ dnew, float* dY0,
                                                                float* __restrict__ dX, const float* __restrict__ b,
                                                                float* __restrict__ r, float beta0, long long n,
                                                                double* partials, const float* __restrict__ dbeta) {
  const float beta = dbeta ? __ldg(dbeta) : beta0;  // device copy for captured launches
  double acc[kNumSums];
#pragma unroll
  for (int k = 0; k < kNumSums; ++k) acc[k] = 0.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float d = dnew[i], d0 = dY0[i];
    const float x = fmaf(beta, d - d0, d);
    dX[i] = x;
    dY0[i] = d;
    const float rr = x - b[i];
    r[i] = rr;
    acc[SUM_RR] += (double)rr * (double)rr;
  }
  block_write_sums<FLAT_THREADS>(acc, partials, blockIdx.x);
}

cudaError_t launch_holo_momentum(const float* dnew, float* dY0, float* dX, const float* b, float* r, float beta,
                                 long long n, double* partials, int* nblocks_out, cudaStream_t st,
                                 const float* dbeta) {
  const int blocks = flat_blocks((size_t)n);
  *nblocks_out = blocks;
  k_holo_momentum<<<blocks, FLAT_THREADS, 0, st>>>(dnew, dY0, dX, b, r, beta, n, partials, dbeta);
  return cudaGetLastError();
}

// A small frame's iteration is a chain of short launches, and one plane fills
// few SMs: the two inverse and two forward passes of the hologram, its pointwise
// steps and their reductions were ten launches and a third of an iteration at
// 128 x 128 x 32 (38 of 118 us; 54 of 276 at 384 x 384 x 40).  These two are
// what is left of them in the loop.  The sum of the z-chunks' spectra is bound by
// latency: one part after another took 15 us at
// 16 parts, and the steps of an iteration 25 us at 128 x 128 x 32 (22 us now)
// and 29 us at 384 x 384 x 40 (26 us now).
__global__ void __launch_bounds__(FLAT_THREADS) k_spec_residual(const float2* __restrict__ parts, int nparts,
                                                                const float2* __restrict__ Bh,
                                                                float2* __restrict__ Dn, int W, int H, SpecSums s) {
  const size_t HW = (size_t)W * H;
  const unsigned half = (unsigned)(H / 2 + 1) * (unsigned)W;  // H is even
  double acc = 0.0;
  for (unsigned i = blockIdx.x * FLAT_THREADS + threadIdx.x; i < half; i += gridDim.x * FLAT_THREADS) {
    const unsigned y = i / (unsigned)W, x = i - y * (unsigned)W;
    const unsigned p = (y ? H - y : 0) * (unsigned)W + (x ? W - x : 0);  // the element at -f
    float2 a = parts[i], b = parts[p];
    // eight parts' loads in flight, added in order
    for (int k0 = 1; k0 < nparts; k0 += 8) {
      float2 va[8], vb[8];
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k0 + k < nparts) {
          va[k] = parts[(k0 + k) * HW + i];
          vb[k] = parts[(k0 + k) * HW + p];
        }
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k0 + k < nparts) {
          a = cadd(a, va[k]);
          b = cadd(b, vb[k]);
        }
    }
    const float2 d = make_float2(0.5f * (a.x + b.x), 0.5f * (a.y - b.y));
    const bool pair = y > 0 && y < (unsigned)H / 2;  // else the partner's own thread writes it
    Dn[i] = d;
    if (pair) Dn[p] = make_float2(d.x, -d.y);
    if (Bh) {
      const float2 e = csub(d, Bh[i]);
      const double q = (double)e.x * (double)e.x + (double)e.y * (double)e.y;
      acc += pair ? 2.0 * q : q;
    }
  }
  if (Bh) last_block_rr<FLAT_THREADS>(acc / (double)HW, s.partials, s.sums, s.counter);
}

cudaError_t launch_spec_residual(const float2* parts, int nparts, const float2* Bh, float2* Dn, int W, int H,
                                 const SpecSums& s, cudaStream_t st) {
  k_spec_residual<<<flat_blocks((size_t)(H / 2 + 1) * W), FLAT_THREADS, 0, st>>>(parts, nparts, Bh, Dn, W, H, s);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(FLAT_THREADS) k_spec_momentum(const float2* __restrict__ Dn, float2* D0,
                                                                float2* __restrict__ DX,
                                                                const float2* __restrict__ Bh,
                                                                float2* __restrict__ Rs, float beta0,
                                                                const float* __restrict__ dbeta, long long n,
                                                                float scale, SpecSums s) {
  const float beta = dbeta ? __ldg(dbeta) : beta0;  // device copy for captured launches
  double acc = 0.0;
  for (long long i = (long long)blockIdx.x * FLAT_THREADS + threadIdx.x; i < n; i += (long long)gridDim.x * FLAT_THREADS) {
    const float2 d = Dn[i], d0 = D0[i];
    const float2 x = make_float2(fmaf(beta, d.x - d0.x, d.x), fmaf(beta, d.y - d0.y, d.y));
    DX[i] = x;
    D0[i] = d;
    const float2 e = csub(x, Bh[i]);
    Rs[i] = cscale(e, scale);
    acc += (double)e.x * (double)e.x + (double)e.y * (double)e.y;
  }
  last_block_rr<FLAT_THREADS>(acc / (double)n, s.partials, s.sums, s.counter);
}

cudaError_t launch_spec_momentum(const float2* Dn, float2* D0, float2* DX, const float2* Bh, float2* Rs, float beta,
                                 const float* dbeta, long long n, const SpecSums& s, cudaStream_t st) {
  k_spec_momentum<<<flat_blocks((size_t)n), FLAT_THREADS, 0, st>>>(Dn, D0, DX, Bh, Rs, beta, dbeta, n,
                                                                  1.0f / (float)n, s);
  return cudaGetLastError();
}

__global__ void k_spec_pair(const float2* __restrict__ D0, const float2* __restrict__ DX, float2* __restrict__ out,
                            long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float2 a = D0[i], b = DX[i];
    out[i] = make_float2(a.x - b.y, a.y + b.x);
  }
}

cudaError_t launch_spec_pair(const float2* D0, const float2* DX, float2* out, long long n, cudaStream_t st) {
  k_spec_pair<<<flat_blocks((size_t)n), FLAT_THREADS, 0, st>>>(D0, DX, out, n);
  return cudaGetLastError();
}

__global__ void k_spec_fields(const float2* __restrict__ in, const float* __restrict__ b, float* __restrict__ d0,
                              float* __restrict__ d1, float* __restrict__ dX, float* __restrict__ r, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float2 v = in[i];
    d0[i] = v.x;
    d1[i] = v.x;
    dX[i] = v.y;
    r[i] = v.y - b[i];
  }
}

cudaError_t launch_spec_fields(const float2* in, const float* b, float* d0, float* d1, float* dX, float* r, long long n,
                               cudaStream_t st) {
  k_spec_fields<<<flat_blocks((size_t)n), FLAT_THREADS, 0, st>>>(in, b, d0, d1, dX, r, n);
  return cudaGetLastError();
}

// L1 and TV norms of the momentum point x = P + beta (P - Pprev):
// calcL1NormComplex (sparse_volume.cu:194-235), calcTVNorm2d (:365-446),
// calcTVNorm (:240-363, periodic in z).

template <typename ST>
__global__ void __launch_bounds__(FLAT_THREADS) k_momentum_norms(const ST* __restrict__ P, const ST* __restrict__ Pp,
                                                                 float beta, int W, int H, int Nz, int mode,
                                                                 double* partials) {
  double acc[kNumSums];
#pragma unroll
  for (int k = 0; k < kNumSums; ++k) acc[k] = 0.0;
  const size_t HW = (size_t)W * H, n = HW * Nz;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int z = (int)(i / HW);
    const size_t e = i - (size_t)z * HW;
    const int yy = (int)(e / W), xx = (int)(e - (size_t)yy * W);
    const float2 x = xval(P, Pp, beta, i);
    acc[SUM_L1X] += (double)norm_sqrt(cabs2(x));
    acc[SUM_LIM1] += (x.x != 0.f || x.y != 0.f) ? 1.0 : 0.0;  // non-zero voxels
    if (mode == 7 || mode == 6) {
      const int xm = xx > 0 ? xx - 1 : W - 1, ym = yy > 0 ? yy - 1 : H - 1;
      const float2 xl = xval(P, Pp, beta, (size_t)z * HW + (size_t)yy * W + xm);
      const float2 xu = xval(P, Pp, beta, (size_t)z * HW + (size_t)ym * W + xx);
      float q = cabs2(csub(xl, x)) + cabs2(csub(xu, x));
      if (mode == 6) {
        const int zm = z > 0 ? z - 1 : Nz - 1;
        q += cabs2(csub(xval(P, Pp, beta, (size_t)zm * HW + e), x));
      }
      acc[SUM_TVX] += (double)norm_sqrt(q);
    }
  }
  block_write_sums<FLAT_THREADS>(acc, partials, blockIdx.x);
}

cudaError_t launch_momentum_norms(int storage, const void* P, const void* Pprev, float beta, int W, int H, int Nz,
                                  int mode, double* partials, int* nblocks_out, cudaStream_t st) {
  const int blocks = flat_blocks((size_t)W * H * Nz);
  *nblocks_out = blocks;
  switch (storage) {
    case STORE_BF16:
      k_momentum_norms<__nv_bfloat162><<<blocks, FLAT_THREADS, 0, st>>>(
          (const __nv_bfloat162*)P, (const __nv_bfloat162*)Pprev, beta, W, H, Nz, mode, partials);
      break;
    case STORE_F16:
      k_momentum_norms<__half2><<<blocks, FLAT_THREADS, 0, st>>>((const __half2*)P, (const __half2*)Pprev, beta, W,
                                                                  H, Nz, mode, partials);
      break;
    default:
      k_momentum_norms<float2><<<blocks, FLAT_THREADS, 0, st>>>((const float2*)P, (const float2*)Pprev, beta, W, H,
                                                                 Nz, mode, partials);
  }
  return cudaGetLastError();
}

template <typename ST>
__global__ void k_materialize_x(const ST* __restrict__ P, const ST* __restrict__ Pp, float beta, float2* out,
                                long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = xval(P, Pp, beta, (size_t)i);
}

cudaError_t launch_materialize_x(int storage, const void* P, const void* Pprev, float beta, float2* out, long long n,
                                 cudaStream_t st) {
  const int blocks = flat_blocks((size_t)n);
  switch (storage) {
    case STORE_BF16:
      k_materialize_x<<<blocks, FLAT_THREADS, 0, st>>>((const __nv_bfloat162*)P, (const __nv_bfloat162*)Pprev, beta,
                                                       out, n);
      break;
    case STORE_F16:
      k_materialize_x<<<blocks, FLAT_THREADS, 0, st>>>((const __half2*)P, (const __half2*)Pprev, beta, out, n);
      break;
    default:
      k_materialize_x<<<blocks, FLAT_THREADS, 0, st>>>((const float2*)P, (const float2*)Pprev, beta, out, n);
  }
  return cudaGetLastError();
}

template <typename ST>
__global__ void k_store_volume(const float2* __restrict__ in, ST* __restrict__ out, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    Store<ST>::st(out + i, in[i]);
}

cudaError_t launch_store_volume(int storage, const float2* in, void* out, long long n, cudaStream_t st) {
  const int blocks = flat_blocks((size_t)n);
  switch (storage) {
    case STORE_BF16:
      k_store_volume<<<blocks, FLAT_THREADS, 0, st>>>(in, (__nv_bfloat162*)out, n);
      break;
    case STORE_F16:
      k_store_volume<<<blocks, FLAT_THREADS, 0, st>>>(in, (__half2*)out, n);
      break;
    default:
      k_store_volume<<<blocks, FLAT_THREADS, 0, st>>>(in, (float2*)out, n);
  }
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// dispatch: sides with a register-resident split take the passes above, the
// others the line passes of rihvr_lines.cu; rows by the width, columns by the
// height, each for itself
// ---------------------------------------------------------------------------
int fwd_col_chunks(int W, int H, int Nz) {
  return line_size_supported(H) ? fwd_col_chunks_fast(W, H, Nz) : line_fwd_col_chunks(W, H, Nz);
}

cudaError_t launch_rows(int inverse, int in_kind, const void* in, int out_kind, void* out, int W, long long nlines,
                        float scale, cudaStream_t st) {
  return line_size_supported(W) ? launch_rows_fast(inverse, in_kind, in, out_kind, out, W, nlines, scale, st)
                                : launch_line_rows(inverse, in_kind, in, out_kind, out, W, nlines, scale, st);
}

cudaError_t launch_adj_col(const float2* Rs, const double* cturn, const double* zlist, float2* U, int W, int H,
                           int z0, int z1, cudaStream_t st, int chunks_hint, double dz_uniform, int rec_mode) {
  return line_size_supported(H)
             ? launch_adj_col_fast(Rs, cturn, zlist, U, W, H, z0, z1, st, chunks_hint, dz_uniform, rec_mode)
             : launch_line_adj_col(Rs, cturn, zlist, U, W, H, z0, z1, st, chunks_hint);
}

static __device__ unsigned g_col_wait_timeouts;

unsigned* col_timeout_counter() {
  static std::atomic<unsigned*> ptr[kSmCacheDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  std::atomic<unsigned*>* slot = (dev >= 0 && dev < kSmCacheDevices) ? &ptr[dev] : nullptr;
  unsigned* p = slot ? slot->load(std::memory_order_relaxed) : nullptr;
  if (!p) {
    void* v = nullptr;
    if (cudaGetSymbolAddress(&v, g_col_wait_timeouts) != cudaSuccess) return nullptr;
    p = static_cast<unsigned*>(v);
    if (slot) slot->store(p, std::memory_order_relaxed);
  }
  return p;
}

cudaError_t col_wait_timeouts(cudaStream_t st, unsigned* count) {
  unsigned zero = 0;
  cudaError_t e = cudaMemcpyFromSymbolAsync(count, g_col_wait_timeouts, sizeof(unsigned), 0, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess && *count) e = cudaMemcpyToSymbolAsync(g_col_wait_timeouts, &zero, sizeof(unsigned), 0,
                                                              cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess && *count) e = cudaStreamSynchronize(st);
  return e;
}

cudaError_t launch_fwd_col(const float2* T, const double* cturn, const double* zlist, float2* Spart, int W, int H,
                           int z0, int z1, int nchunks, cudaStream_t st, int horner_mode, const HornerTable& table) {
  return line_size_supported(H)
             ? launch_fwd_col_fast(T, cturn, zlist, Spart, W, H, z0, z1, nchunks, st, horner_mode, table)
             : launch_line_fwd_col(T, cturn, zlist, Spart, W, H, z0, z1, nchunks, st);
}

cudaError_t launch_plane_col(int inverse, const float2* in, float2* out, int W, int H, float scale,
                             cudaStream_t st) {
  return line_size_supported(H) ? launch_plane_col_fast(inverse, in, out, W, H, scale, st)
                                : launch_line_plane_col(inverse, in, out, W, H, scale, st);
}

}  // namespace rihvr
