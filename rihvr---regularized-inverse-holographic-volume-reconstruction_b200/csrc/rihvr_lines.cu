// Line FFTs of plane sides without a register-resident four-step split (any
// even length from 16 to 4096 whose prime factors are 2, 3, 5 and 7, such as
// 480, 1080, 1280, 1536 or 2048).  The reference takes such sizes through
// cuFFT (sparse_compressive_holo.cu:98); W and H are multiples of 16 there
// (:126, 1948).
//
// A line of n = R_0 R_1 ... R_{S-1} is a self-sorting Stockham sequence of S
// butterfly stages with the largest radices that fit registers (up to 16): two
// stages to n = 256, three to 4096 for most lengths.  The first stage loads
// from global memory, the last one stores to it, and the stages exchange
// through ONE shared-memory copy of the block's lines: a thread reads the
// inputs of all its butterflies into registers (up to E elements) before a
// barrier and writes the outputs after it.
//
// What bounds it: instruction issue (butterflies, twiddles and index arithmetic;
// barriers and shared-memory latency keep issue near 40 %).  Radix-4/2/3/5/7
// stages between two shared-memory buffers, with an index division and a table
// load for every twiddle, took five stages at n = 1280: 883 us for a row pass of
// 1280 x 1024 x 64 on a B200, 407 us here (200 us at the memory's rate).
#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <utility>

#include "rihvr_device.cuh"
#include "rihvr_kernels.cuh"
#include "rihvr_launch.cuh"
#include "rihvr_lines.cuh"

namespace rihvr {

namespace {

constexpr int kMaxSide = 4096;
constexpr int kMaxStages = 6;
constexpr int kElems = 16;             // elements a thread holds at a time
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

constexpr int kRadices[] = {16, 15, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2};

// elements a thread holds of radix-r butterflies
constexpr int butterflies(int r, int e) { return e / r > 0 ? e / r : 1; }

// The shortest sequence of radices (at least two), the most even one among
// those (least sum), in falling order.
void search(int n, int most, int* cur, int depth, int* best, int* best_n, int* best_sum, int sum) {
  if (n == 1) {
    if (depth >= 2 && (depth < *best_n || (depth == *best_n && sum < *best_sum))) {
      *best_n = depth;
      *best_sum = sum;
      std::copy(cur, cur + depth, best);
    }
    return;
  }
  if (depth == kMaxStages || depth >= *best_n) return;
  for (int r : kRadices) {
    if (r > most || n % r != 0) continue;
    cur[depth] = r;
    search(n / r, r, cur, depth + 1, best, best_n, best_sum, sum + r);
  }
}

unsigned magic(int d) { return d == 1 ? 0u : (unsigned)((0x100000000ull + d - 1) / d); }

bool plan_make(int n, LPlan* p) {
  if (n < 4 || n > kMaxSide) return false;
  int cur[kMaxStages], best[kMaxStages], best_n = kMaxStages + 1, best_sum = 0;
  search(n, 16, cur, 0, best, &best_n, &best_sum, 0);
  if (best_n > kMaxStages) return false;
  p->n = n;
  p->nst = best_n;
  int ns = 1;
  for (int i = 0; i < best_n; ++i) {
    LStage& s = p->s[i];
    s.r = best[i];
    s.m = n / s.r;
    s.ns = ns;
    s.tstep = n / (ns * s.r);
    s.m_over_ns = s.m / ns;
    s.magic_m = magic(s.m);
    s.magic_ns = magic(ns);
    ns *= s.r;
  }
  return true;
}

// threads a block of `lines` lines needs so that every stage's butterflies fit e elements a thread
int plan_threads(const LPlan& p, int lines, int e) {
  int t = 32;
  for (int i = 0; i < p.nst; ++i) {
    const int b = p.s[i].m * lines, nb = butterflies(p.s[i].r, e);
    t = std::max(t, (b + nb - 1) / nb);
  }
  return (t + 31) / 32 * 32;
}

// places a line takes in the shared copy
int line_places(const LPlan& p) { return std::max(p.n, p.s[0].r * (p.s[0].m | 1)); }

int ilog2(int c) {
  int l = 0;
  while ((1 << l) < c) ++l;
  return l;
}

// rows per block: a power of two, at most kRowElems elements and the thread limit
int row_lines(const LPlan& p) {
  int c = 1;
  while (2 * c * p.n <= kRowElems && 2 * c <= kRowLinesMax && plan_threads(p, 2 * c, kElems) <= kRowThreadsMax) c *= 2;
  return c;
}

// columns per block: a power of two up to 16 (128-byte row segments), about
// 4600 elements where that leaves at least 4 columns (32-byte sectors)
int col_lines(const LPlan& p) {
  int c = 2;
  while (2 * c <= kColsMax && (2 * c <= 4 || 2 * c * p.n <= 4608) &&
         plan_threads(p, 2 * c, kElems) <= kColThreadsMax)
    c *= 2;
  return c;
}

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

// exp(-2 pi i k / n)
__global__ void k_line_twiddles(int n, float2* __restrict__ tw) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) {
    double s, c;
    sincospi(-2.0 * (double)k / (double)n, &s, &c);
    tw[k] = make_float2((float)c, (float)s);
  }
}

// exp(-2 pi i k / n), k < n: one table per (device, n), built once and kept
// for the life of the process (at most 32 KB each)
const float2* line_table(int n, cudaStream_t st, cudaError_t* err) {
  static std::mutex mu;
  static std::map<std::pair<int, int>, float2*> tables;
  int dev = 0;
  *err = cudaGetDevice(&dev);
  if (*err != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  auto it = tables.find({dev, n});
  if (it != tables.end()) return it->second;
  float2* t = nullptr;
  *err = cudaMalloc(&t, sizeof(float2) * (size_t)n);
  if (*err != cudaSuccess) return nullptr;
  k_line_twiddles<<<(n + 255) / 256, 256, 0, st>>>(n, t);
  *err = cudaStreamSynchronize(st);
  if (*err != cudaSuccess) {
    cudaFree(t);
    return nullptr;
  }
  tables[{dev, n}] = t;
  return t;
}

// the plan of a length, searched once per process
bool plan_of(int n, LPlan* p) {
  static std::mutex mu;
  static std::map<int, LPlan> plans;
  std::lock_guard<std::mutex> lock(mu);
  auto it = plans.find(n);
  if (it == plans.end()) {
    LPlan q;
    std::memset(&q, 0, sizeof(q));
    if (!plan_make(n, &q)) return false;
    it = plans.emplace(n, q).first;
  }
  *p = it->second;
  return true;
}

// ---------------------------------------------------------------------------
// rows: 2^logc contiguous lines a block, consecutive lanes on consecutive
// butterflies of a line
// ---------------------------------------------------------------------------
template <bool INV, int IN>
__global__ void __launch_bounds__(kRowThreadsMax, 2)
    k_line_rows(const __grid_constant__ LPlan p, const float2* __restrict__ tw, const void* __restrict__ in,
                float2* __restrict__ out, long long nlines, float scale, int logc, int ls) {
  extern __shared__ __align__(128) float2 gbuf[];
  const long long l0 = (long long)blockIdx.x << logc;
  const int lines = (int)min(1LL << logc, nlines - l0);
  const size_t base = (size_t)l0 * p.n;
  const int n = p.n;
  line_fft<kElems, INV>(
      p, lines, tw,
      [](int b, int m, unsigned mg, int* c, int* j) {
        *c = (int)__umulhi((unsigned)b, mg);
        *j = b - *c * m;
      },
      [=](int c, int i) { return load_as<IN>(in, base + (size_t)(c * n + i)); },
      [=](int, int c, int i, float2 v) { out[base + (size_t)(c * n + i)] = cscale(v, scale); },
      [=](int c) { return gbuf + c * ls; }, 0);
}

template <bool INV, int IN>
cudaError_t rows_launch(const LPlan& p, const float2* tw, const void* in, float2* out, long long nlines, float scale,
                        cudaStream_t st) {
  const int C = row_lines(p);
  const long long blocks = (nlines + C - 1) / C;
  if (blocks <= 0) return cudaSuccess;
  // an odd line pitch keeps lines apart in the banks
  const int ls = line_places(p) | 1;
  const size_t smem = sizeof(float2) * (size_t)C * ls;
  cudaError_t e = allow_smem(k_line_rows<INV, IN>, smem);
  if (e != cudaSuccess) return e;
  k_line_rows<INV, IN>
      <<<(unsigned)blocks, plan_threads(p, C, kElems), smem, st>>>(p, tw, in, out, nlines, scale, ilog2(C), ls);
  return cudaGetLastError();
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
    line_fft<kElems, true, 4, 0>(
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
    line_fft<kElems, false, 0, 4>(
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

template <bool INV>
__global__ void __launch_bounds__(kColThreadsMax, 1)
    k_line_plane_col(const __grid_constant__ LPlan p, const float2* __restrict__ tw, const float2* __restrict__ in,
                     float2* __restrict__ out, int W, float scale, int logc) {
  extern __shared__ __align__(128) float2 gbuf[];
  const int x0 = blockIdx.x << logc;
  line_fft<kElems, INV>(
      p, 1 << logc, tw, ColSplit{logc},
      [=](int c, int y) { return x0 + c < W ? in[(unsigned)(y * W + x0 + c)] : make_float2(0.f, 0.f); },
      [=](int, int c, int y, float2 v) {
        if (x0 + c < W) out[(unsigned)(y * W + x0 + c)] = cscale(v, scale);
      },
      ColAt{gbuf}, logc);
}

// plan, table, columns a block, threads and shared memory of a column launch
struct ColLaunch {
  LPlan p;
  const float2* tw = nullptr;
  int C = 0, logc = 0, strips = 0, threads = 0;
  size_t smem = 0;
};
cudaError_t col_launch(int W, int H, cudaStream_t st, ColLaunch* L) {
  if (!plan_of(H, &L->p)) return cudaErrorInvalidValue;
  cudaError_t e;
  L->tw = line_table(H, st, &e);
  if (!L->tw) return e;
  L->C = col_lines(L->p);
  L->logc = ilog2(L->C);
  L->strips = (W + L->C - 1) / L->C;
  L->threads = plan_threads(L->p, L->C, kElems);
  L->smem = sizeof(float2) * (size_t)line_places(L->p) * L->C;
  return cudaSuccess;
}

}  // namespace

bool generic_size_supported(int n) {
  if (n < 2 || n > kMaxSide) return false;
  for (int r : {2, 3, 5, 7})
    while (n % r == 0) n /= r;
  return n == 1;
}

int line_fwd_col_chunks(int W, int H, int Nz) {
  LPlan p;
  if (!plan_of(H, &p)) return 1;
  const int C = col_lines(p);
  const int strips = (W + C - 1) / C;
  int chunks = (4 * num_sms() + strips - 1) / strips;
  if (chunks > 16) chunks = 16;
  if (chunks > Nz) chunks = Nz;
  if (chunks < 1) chunks = 1;
  return chunks;
}

cudaError_t launch_line_rows(int inverse, int in_kind, const void* in, int out_kind, void* out, int W,
                             long long nlines, float scale, cudaStream_t st) {
  if (out_kind != ELEM_C32) return cudaErrorInvalidValue;
  LPlan p;
  if (!plan_of(W, &p)) return cudaErrorInvalidValue;
  cudaError_t e;
  const float2* tw = line_table(W, st, &e);
  if (!tw) return e;
  float2* o = static_cast<float2*>(out);
  if (inverse) {
    if (in_kind != ELEM_C32 && in_kind != ELEM_STORE_F32) return cudaErrorInvalidValue;
    return rows_launch<true, ELEM_C32>(p, tw, in, o, nlines, scale, st);
  }
  switch (in_kind) {
    case ELEM_C32:
    case ELEM_STORE_F32: return rows_launch<false, ELEM_C32>(p, tw, in, o, nlines, scale, st);
    case ELEM_R32: return rows_launch<false, ELEM_R32>(p, tw, in, o, nlines, scale, st);
    case ELEM_STORE_BF16: return rows_launch<false, ELEM_STORE_BF16>(p, tw, in, o, nlines, scale, st);
    case ELEM_STORE_F16: return rows_launch<false, ELEM_STORE_F16>(p, tw, in, o, nlines, scale, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_line_adj_col(const float2* Rs, const double* cturn, const double* zlist, float2* U, int W, int H,
                                int z0, int z1, cudaStream_t st, int chunks_hint) {
  const int nz = z1 - z0;
  if (nz <= 0) return cudaSuccess;
  ColLaunch L;
  cudaError_t e = col_launch(W, H, st, &L);
  if (e != cudaSuccess) return e;
  int chunks = chunks_hint > 0 ? chunks_hint : (8 * num_sms() + L.strips - 1) / L.strips;
  if (chunks > nz) chunks = nz;
  if (chunks < 1) chunks = 1;
  const int zpb = (nz + chunks - 1) / chunks;
  chunks = (nz + zpb - 1) / zpb;
  e = allow_smem(k_line_adj_col, L.smem);
  if (e != cudaSuccess) return e;
  k_line_adj_col<<<dim3(L.strips, chunks), L.threads, L.smem, st>>>(L.p, L.tw, Rs, cturn, zlist, U, W, z0, z1, zpb,
                                                                    L.logc);
  return cudaGetLastError();
}

cudaError_t launch_line_fwd_col(const float2* T, const double* cturn, const double* zlist, float2* Spart, int W,
                                int H, int z0, int z1, int nchunks, cudaStream_t st) {
  const int nz = z1 - z0;
  if (nz <= 0) return cudaSuccess;
  ColLaunch L;
  cudaError_t e = col_launch(W, H, st, &L);
  if (e != cudaSuccess) return e;
  const int zpb = (nz + nchunks - 1) / nchunks;
  const int chunks = (nz + zpb - 1) / zpb;
  if (chunks < nchunks) {  // unused chunk slots must read as zero
    e = cudaMemsetAsync(Spart + (size_t)chunks * H * W, 0, sizeof(float2) * (size_t)(nchunks - chunks) * H * W, st);
    if (e != cudaSuccess) return e;
  }
  const size_t smem = L.smem + sizeof(float2) * (size_t)H * L.C;  // exchange buffer and sums
  e = allow_smem(k_line_fwd_col, smem);
  if (e != cudaSuccess) return e;
  k_line_fwd_col<<<dim3(L.strips, chunks), L.threads, smem, st>>>(L.p, L.tw, T, cturn, zlist, Spart, W, z0, z1, zpb,
                                                                  L.logc, line_places(L.p));
  return cudaGetLastError();
}

cudaError_t launch_line_plane_col(int inverse, const float2* in, float2* out, int W, int H, float scale,
                                  cudaStream_t st) {
  ColLaunch L;
  cudaError_t e = col_launch(W, H, st, &L);
  if (e != cudaSuccess) return e;
  if (inverse) {
    e = allow_smem(k_line_plane_col<true>, L.smem);
    if (e != cudaSuccess) return e;
    k_line_plane_col<true><<<L.strips, L.threads, L.smem, st>>>(L.p, L.tw, in, out, W, scale, L.logc);
  } else {
    e = allow_smem(k_line_plane_col<false>, L.smem);
    if (e != cudaSuccess) return e;
    k_line_plane_col<false><<<L.strips, L.threads, L.smem, st>>>(L.p, L.tw, in, out, W, scale, L.logc);
  }
  return cudaGetLastError();
}

}  // namespace rihvr
