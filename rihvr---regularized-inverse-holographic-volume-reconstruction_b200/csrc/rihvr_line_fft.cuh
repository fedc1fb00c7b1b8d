// Kernels of the line FFT passes, as templates on the elements a thread holds:
// rihvr_lines.cu has the shorter form and the launchers, rihvr_lines_long.cu the
// longer one (each takes minutes to compile).
#pragma once
#include "rihvr_device.cuh"
#include "rihvr_kernels.cuh"
#include "rihvr_launch.cuh"

namespace rihvr {
namespace lines {

constexpr int kMaxSide = 4096;
constexpr int kMaxStages = 6;
// Elements a thread holds at a time.  16 give the shorter blocks; the sides
// above 2400 whose shortest plan holds one butterfly of radix 9 or 10 a thread
// (2430, 3000, 4050 and 21 more) would need more threads than a block has for
// one row or two columns, and take 24.
constexpr int kElems = 16, kElemsLong = 24;
constexpr int kRowThreadsMax = 256, kColThreadsMax = 512;
constexpr int kRowElems = 1536;        // elements of a row block's lines (blocks of 3 to 4 warps, five an SM)
constexpr int kRowLinesMax = 128, kColsMax = 16;

// one stage of radix r: m = n / r butterflies a line, ns the product of the radices before it
struct LStage {
  int r, m, ns, tstep;         // tstep = n / (ns r): twiddle exponent of one step of k
  int m_over_ns;               // m / ns of the second stage
  unsigned magic_m, magic_ns;  // ceil(2^32 / d): b / d = umulhi(b, magic) for b d < 2^32
};
struct LPlan {
  int n, nst;
  LStage s[kMaxStages];
};

// elements a thread holds of radix-r butterflies
constexpr int butterflies(int r, int e) { return e / r > 0 ? e / r : 1; }

// Places of a line's elements in the shared copy.  The first stage stores its
// output r of butterfly j at r P + j, P = n / R_0 padded to an odd number, so
// that lanes (consecutive j) write consecutive places; the second stage reads
// element i of the sorted order at (i % R_0) P + i / R_0, which for its inputs
// j + r m is linear in r too (R_0 divides m).  From the second stage on the
// outputs lie in sorted order.  Every access of a butterfly is then a base and
// a stride.  (Sorted places with one element of padding every 16 took an add
// and a shift more for every access.)
__host__ __device__ __forceinline__ int first_pitch(int m0) { return m0 | 1; }

// w^(k r), r = 1 .. R - 1, times the inputs: w^(k r) from the table for r <= 3
// and r = 4, 8, 12, the others as one product of two of these
template <int R, bool INV>
__device__ __forceinline__ void twiddle_inputs(float2 (&v)[R], const float2* __restrict__ tw, int kt) {
  auto get = [&](int r) {
    float2 w = __ldg(tw + kt * r);
    if (INV) w.y = -w.y;
    return w;
  };
  if constexpr (R <= 5) {
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = cmul(v[r], get(r));
  } else {
    float2 lo[4];
#pragma unroll
    for (int r = 1; r < 4; ++r) {
      lo[r] = get(r);
      v[r] = cmul(v[r], lo[r]);
    }
#pragma unroll
    for (int q = 4; q < R; q += 4) {
      const float2 hi = get(q);
      v[q] = cmul(v[q], hi);
#pragma unroll
      for (int r = 1; r < 4; ++r)
        if (q + r < R) v[q + r] = cmul(v[q + r], cmul(hi, lo[r]));
    }
  }
}

// One stage of radix R over the block's lines, in two halves around the
// barrier that ends the reads of the shared copy.  split(b, m, magic_m, &c,
// &j): line c and butterfly j of butterfly number b; load(c, i): element i of
// line c of the global input; store(q, c, i, value): its output element.  A
// thread takes butterflies threadIdx.x, + blockDim.x, ...; v holds their
// inputs one after another.  G > 0: loads or stores that carry the transfer
// function go in groups of that many, so that the FP64 phases of all of them
// are not live at once.  The shared forms get the pointer of line c's element
// 0 from at(c) and the elements' pitch (1, or the columns of a block).
template <int R, int E, int G, typename Split, typename Load>
__device__ __forceinline__ void stage_load_global(const LStage& s, int lines, Split split, Load load, float2 (&v)[E]) {
#pragma unroll
  for (int nb = 0; nb < butterflies(R, E); ++nb) {
    const int b = (int)threadIdx.x + nb * (int)blockDim.x;
    if (b < s.m * lines) {
      int c, j;
      split(b, s.m, s.magic_m, &c, &j);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        v[nb * R + r] = load(c, j + r * s.m);
        if (G > 0 && r % (G > 0 ? G : 1) == G - 1) sched_fence();
      }
    }
  }
}

// SECOND: the input lies as the first stage (radix r0, pitch p0) stored it
template <int R, int E, typename Split, typename At>
__device__ __forceinline__ void stage_load_shared(const LStage& s, int lines, bool second, int p0, Split split, At at,
                                                  int logp, float2 (&v)[E]) {
#pragma unroll
  for (int nb = 0; nb < butterflies(R, E); ++nb) {
    const int b = (int)threadIdx.x + nb * (int)blockDim.x;
    if (b < s.m * lines) {
      int c, j, base, step;
      split(b, s.m, s.magic_m, &c, &j);
      if (second) {  // ns = r0: j = q r0 + k
        const int q = (int)__umulhi((unsigned)j, s.magic_ns);
        base = (j - q * s.ns) * p0 + q;
        step = s.m_over_ns;
      } else {
        base = j;
        step = s.m;
      }
      const float2* src = at(c) + ((size_t)(unsigned)base << logp);
      step <<= logp;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        v[nb * R + r] = *src;
        src += step;
      }
    }
  }
}

// twiddles and butterflies in place: v[nb R + r] becomes output r
template <int R, int E, bool INV, bool FIRST, typename Split>
__device__ __forceinline__ void butterfly(const LStage& s, const float2* __restrict__ tw, int j, float2 (&a)[R], int* k) {
  *k = 0;
  if (!FIRST) {
    *k = j - (int)__umulhi((unsigned)j, s.magic_ns) * s.ns;
    twiddle_inputs<R, INV>(a, tw, *k * s.tstep);
  }
  reg_fft<R, INV>(a);
}

template <int R, int E, bool INV, bool FIRST, typename Split, typename At>
__device__ __forceinline__ void stage_store_shared(const LStage& s, int lines, int p0, const float2* __restrict__ tw,
                                                   Split split, At at, int logp, float2 (&v)[E]) {
#pragma unroll
  for (int nb = 0; nb < butterflies(R, E); ++nb) {
    const int b = (int)threadIdx.x + nb * (int)blockDim.x;
    if (b < s.m * lines) {
      int c, j, k;
      split(b, s.m, s.magic_m, &c, &j);
      float2 a[R];
#pragma unroll
      for (int r = 0; r < R; ++r) a[r] = v[nb * R + r];
      butterfly<R, E, INV, FIRST, Split>(s, tw, j, a, &k);
      float2* dst = at(c) + ((size_t)(unsigned)(FIRST ? j : (j - k) * R + k) << logp);
      const int step = (FIRST ? p0 : s.ns) << logp;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        *dst = a[r];
        dst += step;
      }
    }
  }
}

// the last stage: ns = m, so k = j and output r of butterfly j is element j + r m
template <int R, int E, int G, bool INV, typename Split, typename Store>
__device__ __forceinline__ void stage_store_global(const LStage& s, int lines, const float2* __restrict__ tw,
                                                   Split split, Store store, float2 (&v)[E]) {
#pragma unroll
  for (int nb = 0; nb < butterflies(R, E); ++nb) {
    const int b = (int)threadIdx.x + nb * (int)blockDim.x;
    if (b < s.m * lines) {
      int c, j;
      split(b, s.m, s.magic_m, &c, &j);
      float2 a[R];
#pragma unroll
      for (int r = 0; r < R; ++r) a[r] = v[nb * R + r];
      twiddle_inputs<R, INV>(a, tw, j);  // tstep = 1
      reg_fft<R, INV>(a);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        store(nb * R + r, c, j + r * s.m, a[r]);
        if (G > 0 && r % (G > 0 ? G : 1) == G - 1) sched_fence();
      }
    }
  }
}

#define RIHVR_EACH_RADIX(X) X(16) X(15) X(12) X(10) X(9) X(8) X(7) X(6) X(5) X(4) X(3) X(2)

// one of the functions above for the stage's radix.  A barrier inside the
// cases would make the compiler merge them around it (and spill up to 4 KB a
// thread): the barriers stand between these switches.
#define RIHVR_BY_RADIX(CALL)      \
  switch (s.r) {                  \
    RIHVR_EACH_RADIX(CALL)        \
    default: break;               \
  }

// all stages: src(c, i) the global input, dst(q, c, i, value) the global
// output, at(c) line c's place in the shared copy, its elements 2^logp apart
template <int E, bool INV, int LG = 0, int SG = 0, typename Split, typename Src, typename Dst, typename At>
__device__ __forceinline__ void line_fft(const LPlan& p, int lines, const float2* __restrict__ tw, Split split,
                                         Src src, Dst dst, At at, int logp) {
  float2 v[E];
  const int p0 = first_pitch(p.s[0].m);
  {
    const LStage& s = p.s[0];
#define RIHVR_CALL(RR) case RR: stage_load_global<RR, E, LG>(s, lines, split, src, v); break;
    RIHVR_BY_RADIX(RIHVR_CALL)
#undef RIHVR_CALL
    __syncthreads();
#define RIHVR_CALL(RR) case RR: stage_store_shared<RR, E, INV, true>(s, lines, p0, tw, split, at, logp, v); break;
    RIHVR_BY_RADIX(RIHVR_CALL)
#undef RIHVR_CALL
    __syncthreads();
  }
#pragma unroll 1
  for (int i = 1; i < p.nst; ++i) {
    const LStage& s = p.s[i];
#define RIHVR_CALL(RR) case RR: stage_load_shared<RR, E>(s, lines, i == 1, p0, split, at, logp, v); break;
    RIHVR_BY_RADIX(RIHVR_CALL)
#undef RIHVR_CALL
    if (i + 1 == p.nst) break;
    __syncthreads();
#define RIHVR_CALL(RR) case RR: stage_store_shared<RR, E, INV, false>(s, lines, p0, tw, split, at, logp, v); break;
    RIHVR_BY_RADIX(RIHVR_CALL)
#undef RIHVR_CALL
    __syncthreads();
  }
  const LStage& s = p.s[p.nst - 1];
#define RIHVR_CALL(RR) case RR: stage_store_global<RR, E, SG, INV>(s, lines, tw, split, dst, v); break;
  RIHVR_BY_RADIX(RIHVR_CALL)
#undef RIHVR_CALL
}

// ---------------------------------------------------------------------------
// rows: 2^logc contiguous lines a block, consecutive lanes on consecutive
// butterflies of a line
// ---------------------------------------------------------------------------
template <int E, bool INV, int IN>
__global__ void __launch_bounds__(kRowThreadsMax, 2)
    k_line_rows(const __grid_constant__ LPlan p, const float2* __restrict__ tw, const void* __restrict__ in,
                float2* __restrict__ out, long long nlines, float scale, int logc, int ls) {
  extern __shared__ __align__(128) float2 gbuf[];
  const long long l0 = (long long)blockIdx.x << logc;
  const int lines = (int)min(1LL << logc, nlines - l0);
  const size_t base = (size_t)l0 * p.n;
  const int n = p.n;
  line_fft<E, INV>(
      p, lines, tw,
      [](int b, int m, unsigned mg, int* c, int* j) {
        *c = (int)__umulhi((unsigned)b, mg);
        *j = b - *c * m;
      },
      [=](int c, int i) { return load_as<IN>(in, base + (size_t)(c * n + i)); },
      [=](int, int c, int i, float2 v) { out[base + (size_t)(c * n + i)] = cscale(v, scale); },
      [=](int c) { return gbuf + c * ls; }, 0);
}

// ---------------------------------------------------------------------------
// columns: 2^logc adjacent columns a block (column fastest over the lanes)
// ---------------------------------------------------------------------------
struct ColSplit {
  int logc;
  __device__ __forceinline__ void operator()(int b, int, unsigned, int* c, int* j) const {
    *c = b & ((1 << logc) - 1);
    *j = b >> logc;
  }
};
struct ColAt {
  float2* sm;
  __device__ __forceinline__ float2* operator()(int c) const { return sm + c; }
};

// adjoint: U_z(:, x) = IDFT_y(conj(H'_z(:, x)) Rs(:, x)), planes [zb, ze) of the block
template <int E>
__global__ void __launch_bounds__(kColThreadsMax, 1)
    k_line_adj_col(const __grid_constant__ LPlan p, const float2* __restrict__ tw, const float2* __restrict__ Rs,
                   const double* __restrict__ cturn, const double* __restrict__ zlist, float2* __restrict__ U, int W,
                   int z0, int z1, int zpb, int logc) {
  extern __shared__ __align__(128) float2 gbuf[];
  const int x0 = blockIdx.x << logc;
  const int lines = 1 << logc;
  const int zb = z0 + blockIdx.y * zpb, ze = min(zb + zpb, z1);
  const size_t HW = (size_t)p.n * W;
#pragma unroll 1
  for (int z = zb; z < ze; ++z) {
    const double zz = zlist[z];
    float2* Uz = U + (size_t)z * HW;
    line_fft<E, true, 4, 0>(
        p, lines, tw, ColSplit{logc},
        [=](int c, int y) {
          if (x0 + c >= W) return make_float2(0.f, 0.f);
          const unsigned i = (unsigned)(y * W + x0 + c);
          return cmul(__ldg(Rs + i), transfer(zz, __ldg(cturn + i), true));
        },
        [=](int, int c, int y, float2 v) {
          if (x0 + c < W) Uz[(unsigned)(y * W + x0 + c)] = v;
        },
        ColAt{gbuf}, logc);
  }
}

// forward with the z-sum: Spart[chunk](:, x) = sum_z H'_z(:, x) DFT_y(T_z(:, x)).
// The sums lie in shared memory after the exchange buffer; the last stage's
// outputs are the same elements of the same thread for every plane, so no
// barrier is involved.
template <int E>
__global__ void __launch_bounds__(kColThreadsMax, 1)
    k_line_fwd_col(const __grid_constant__ LPlan p, const float2* __restrict__ tw, const float2* __restrict__ T,
                   const double* __restrict__ cturn, const double* __restrict__ zlist, float2* __restrict__ Spart,
                   int W, int z0, int z1, int zpb, int logc, int places) {
  extern __shared__ __align__(128) float2 gbuf[];
  const int x0 = blockIdx.x << logc;
  const int lines = 1 << logc;
  const int zb = z0 + blockIdx.y * zpb, ze = min(zb + zpb, z1);
  const size_t HW = (size_t)p.n * W;
  float2* const acc = gbuf + (places << logc);
  for (int e = threadIdx.x; e < p.n << logc; e += blockDim.x) acc[e] = make_float2(0.f, 0.f);
  __syncthreads();
#pragma unroll 1
  for (int z = zb; z < ze; ++z) {
    const double zz = zlist[z];
    const float2* Tz = T + (size_t)z * HW;
    line_fft<E, false, 0, 4>(
        p, lines, tw, ColSplit{logc},
        [=](int c, int y) {
          return x0 + c < W ? __ldg(Tz + (unsigned)(y * W + x0 + c)) : make_float2(0.f, 0.f);
        },
        [=](int, int c, int y, float2 v) {
          if (x0 + c >= W) return;
          const float2 h = transfer(zz, __ldg(cturn + (unsigned)(y * W + x0 + c)), false);
          float2 a = acc[(y << logc) + c];
          a.x = fmaf(v.x, h.x, fmaf(-v.y, h.y, a.x));
          a.y = fmaf(v.x, h.y, fmaf(v.y, h.x, a.y));
          acc[(y << logc) + c] = a;
        },
        ColAt{gbuf}, logc);
  }
  __syncthreads();
  float2* Sp = Spart + (size_t)blockIdx.y * HW;
  for (int e = threadIdx.x; e < p.n << logc; e += blockDim.x) {
    const int c = e & (lines - 1), y = e >> logc;
    if (x0 + c < W) Sp[(unsigned)(y * W + x0 + c)] = acc[e];
  }
}

template <int E, bool INV>
__global__ void __launch_bounds__(kColThreadsMax, 1)
    k_line_plane_col(const __grid_constant__ LPlan p, const float2* __restrict__ tw, const float2* __restrict__ in,
                     float2* __restrict__ out, int W, float scale, int logc) {
  extern __shared__ __align__(128) float2 gbuf[];
  const int x0 = blockIdx.x << logc;
  line_fft<E, INV>(
      p, 1 << logc, tw, ColSplit{logc},
      [=](int c, int y) { return x0 + c < W ? in[(unsigned)(y * W + x0 + c)] : make_float2(0.f, 0.f); },
      [=](int, int c, int y, float2 v) {
        if (x0 + c < W) out[(unsigned)(y * W + x0 + c)] = cscale(v, scale);
      },
      ColAt{gbuf}, logc);
}

// the kernels of one number of elements a thread
struct LineKernels {
  using Rows = void (*)(LPlan, const float2*, const void*, float2*, long long, float, int, int);
  using AdjCol = void (*)(LPlan, const float2*, const float2*, const double*, const double*, float2*, int, int, int,
                          int, int);
  using FwdCol = void (*)(LPlan, const float2*, const float2*, const double*, const double*, float2*, int, int, int,
                          int, int, int);
  using PlaneCol = void (*)(LPlan, const float2*, const float2*, float2*, int, float, int);
  int elems;
  Rows inv_rows, rows_c32, rows_r32, rows_bf16, rows_f16;  // inverse of complex values; forward by input
  AdjCol adj_col;
  FwdCol fwd_col;
  PlaneCol plane_col, inv_plane_col;
};
template <int E>
LineKernels make_kernels() {
  return {E,
          k_line_rows<E, true, ELEM_C32>,
          k_line_rows<E, false, ELEM_C32>,
          k_line_rows<E, false, ELEM_R32>,
          k_line_rows<E, false, ELEM_STORE_BF16>,
          k_line_rows<E, false, ELEM_STORE_F16>,
          k_line_adj_col<E>,
          k_line_fwd_col<E>,
          k_line_plane_col<E, false>,
          k_line_plane_col<E, true>};
}
const LineKernels& long_kernels();  // kElemsLong, rihvr_lines_long.cu

}  // namespace lines
}  // namespace rihvr
