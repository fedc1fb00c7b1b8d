// Register-resident line FFT passes, as templates over the plane side: the row
// pass, the column passes of the adjoint and forward operators with the
// transfer function and the sum over z, and the plane passes.  The sides are
// compiled in groups (rihvr_fast_*.cu); rihvr_kernels.cu dispatches to them.
#pragma once
#include <cuda.h>  // CUtensorMap and its enums; the encoder is resolved at run time

#include <cstring>

#include "rihvr_device.cuh"
#include "rihvr_kernels.cuh"
#include "rihvr_launch.cuh"

namespace rihvr {

// ---------------------------------------------------------------------------
// line configurations: N = N1 * N2, N1 threads per line, N2 elements each.
// After the exchange a thread holds M stage-B rows of N1 elements (VS values).
// Where N1 divides N2 every thread holds N2 / N1 rows; otherwise (side 640 =
// 20 x 32) the N2 rows are dealt round-robin and a thread's last row exists
// only when t + N1 (M - 1) < N2 (EXACT false): the missing rows are computed
// on zeros and never stored.
// ---------------------------------------------------------------------------
template <int N>
struct LineCfg;
#define RIHVR_LINE(NN, NN1)                                                              \
  template <>                                                                            \
  struct LineCfg<NN> {                                                                   \
    static constexpr int N = NN, N1 = NN1, N2 = NN / NN1, M = (NN / NN1) / NN1;          \
    static constexpr int LD = NN1 + 1, VS = N2;                                          \
    static constexpr bool EXACT = true;                                                  \
    static_assert((NN / NN1) % NN1 == 0, "N1 must divide N2");                           \
  };
RIHVR_LINE(32, 4)
RIHVR_LINE(48, 4)
RIHVR_LINE(64, 8)
RIHVR_LINE(128, 8)
RIHVR_LINE(256, 16)
RIHVR_LINE(384, 8)
RIHVR_LINE(512, 16)
RIHVR_LINE(768, 16)
RIHVR_LINE(1024, 32)
RIHVR_LINE(2304, 48)  // the 2048 x 2048 hologram padded by 128 on each side
#undef RIHVR_LINE
template <>
struct LineCfg<640> {  // 20 threads a line, 32 elements each; 12 of them take a second stage-B row
  static constexpr int N = 640, N1 = 20, N2 = 32, M = 2;
  static constexpr int LD = N1 + 1, VS = M * N1;
  static constexpr bool EXACT = false;
};

// the first K values of a register array, as an array of K
template <int K, int L>
__device__ __forceinline__ float2 (&head(float2 (&a)[L]))[K] {
  static_assert(K <= L, "prefix longer than the array");
  return *reinterpret_cast<float2(*)[K]>(&a[0]);
}

// does stage-B row j of thread t exist (always, for the exact splits)
template <int N>
__device__ __forceinline__ bool row_ok(int t, int j) {
  using C = LineCfg<N>;
  if constexpr (C::EXACT) return true;
  else return t + C::N1 * j < C::N2;
}

#define RIHVR_FOR_EACH_SIZE(X) X(32) X(48) X(64) X(128) X(256) X(384) X(512) X(640) X(768) X(1024) X(2304)

template <int N1, int VS, bool INV>
__device__ __forceinline__ void stage_b_dft(float2 (&w)[VS]) {
  constexpr int M = VS / N1;
#pragma unroll
  for (int j = 0; j < M; ++j) {
    float2 s[N1];
#pragma unroll
    for (int k = 0; k < N1; ++k) s[k] = w[j * N1 + k];
    reg_fft<N1, INV>(s);
#pragma unroll
    for (int k = 0; k < N1; ++k) w[j * N1 + k] = s[k];
  }
}

// ---------------------------------------------------------------------------
// Row pass: one line per N1-thread group, lines contiguous in memory.
// ---------------------------------------------------------------------------
constexpr int kRowThreads = 256;

template <int N>
struct RowLayout {
  using C = LineCfg<N>;
  static constexpr int LPB = kRowThreads / C::N1;
  // lines of 48 threads straddle warps: the block then holds whole lines only
  // and exchanges through a block barrier instead of a warp one
  static constexpr bool WARP_LINES = (32 % C::N1) == 0;
  static constexpr int THREADS = LPB * C::N1;
  static constexpr int base_ls = C::N2 * C::LD;
  // pad the per-line stride so that lines sharing a half-warp hit different banks
  static constexpr int LS = (C::N1 >= 16) ? base_ls : base_ls + (((C::N1 % 16) - (base_ls % 16) + 16) % 16);
  static constexpr int SMEM = LPB * LS;  // float2 elements
  static constexpr size_t SMEM_BYTES = sizeof(float2) * SMEM;
};

// The input element kind is a template parameter: with it known at compile
// time the N2 loads of a thread issue back to back (a run-time kind switch
// around each load serialises them).  Output is complex FP32.
template <int N, bool INV, int IN>
__global__ void __launch_bounds__(kRowThreads) k_rows(const void* __restrict__ in, float2* __restrict__ out,
                                                     long long nlines, float scale) {
  using C = LineCfg<N>;
  using Lay = RowLayout<N>;
  constexpr int N1 = C::N1, N2 = C::N2, M = C::M, LD = C::LD;
  static_assert(Lay::WARP_LINES || Lay::THREADS <= kRowThreads, "whole lines per block");
  extern __shared__ __align__(128) float2 sm[];
  const int li = threadIdx.x / N1, t = threadIdx.x % N1;
  long long L = (long long)blockIdx.x * Lay::LPB + li;
  const bool active = L < nlines;
  if (!active) L = nlines - 1;
  const size_t base = (size_t)L * N;
  float2 v[C::VS];
#pragma unroll
  for (int n2 = 0; n2 < N2; ++n2) v[n2] = load_as<IN>(in, base + t + N1 * n2);
  reg_fft<N2, INV>(head<N2>(v));
  line_twiddle<N, N2, INV>(head<N2>(v), t);
  float2* sl = sm + li * Lay::LS;
#pragma unroll
  for (int k2 = 0; k2 < N2; ++k2) sl[k2 * LD + t] = v[k2];
  if constexpr (Lay::WARP_LINES) {
    __syncwarp();
  } else {
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < M; ++j) {
    const bool ok = row_ok<N>(t, j);
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) v[j * N1 + n1] = ok ? sl[(t + N1 * j) * LD + n1] : make_float2(0.f, 0.f);
  }
  stage_b_dft<N1, C::VS, INV>(v);
  if (active) {
#pragma unroll
    for (int j = 0; j < M; ++j)
      if (row_ok<N>(t, j))
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) out[base + t + N1 * j + N2 * k1] = cscale(v[j * N1 + k1], scale);
  }
}

template <int N, bool INV, int IN>
static cudaError_t rows_launch(const void* in, float2* out, long long nlines, float scale, cudaStream_t st) {
  using Lay = RowLayout<N>;
  const long long blocks = (nlines + Lay::LPB - 1) / Lay::LPB;
  if (blocks <= 0) return cudaSuccess;
  cudaError_t e = allow_smem(k_rows<N, INV, IN>, Lay::SMEM_BYTES);
  if (e != cudaSuccess) return e;
  k_rows<N, INV, IN><<<(unsigned)blocks, Lay::THREADS, Lay::SMEM_BYTES, st>>>(in, out, nlines, scale);
  return cudaGetLastError();
}

template <int N>
cudaError_t rows_n(int inverse, int in_kind, const void* in, int out_kind, void* out, long long nlines,
                          float scale, cudaStream_t st) {
  if (out_kind != ELEM_C32) return cudaErrorInvalidValue;
  float2* o = static_cast<float2*>(out);
  if (inverse) {
    if (in_kind != ELEM_C32 && in_kind != ELEM_STORE_F32) return cudaErrorInvalidValue;
    return rows_launch<N, true, ELEM_C32>(in, o, nlines, scale, st);
  }
  switch (in_kind) {
    case ELEM_C32:
    case ELEM_STORE_F32: return rows_launch<N, false, ELEM_C32>(in, o, nlines, scale, st);
    case ELEM_R32: return rows_launch<N, false, ELEM_R32>(in, o, nlines, scale, st);
    case ELEM_STORE_BF16: return rows_launch<N, false, ELEM_STORE_BF16>(in, o, nlines, scale, st);
    case ELEM_STORE_F16: return rows_launch<N, false, ELEM_STORE_F16>(in, o, nlines, scale, st);
    default: return cudaErrorInvalidValue;
  }
}

// ---------------------------------------------------------------------------
// Column passes: CC columns per block, N1 threads per column (lanes: column
// fastest so each warp-wide access covers CC*8 contiguous bytes of a row).
// Shared layout [k2][n1][c] with n1 padded to LD.
// ---------------------------------------------------------------------------
template <int N>
struct ColLayout {
  using C = LineCfg<N>;
  // columns per block.  Sides 256, 512 and 1024 take 128-thread blocks: two
  // or more blocks share an SM, so one block's barriers no longer idle the
  // whole SM (measured 10-17 % faster column passes than 256-thread blocks).
  // Sides 384 and 768 measured no gain or a loss and keep 256 threads.
  // Side 2304 (48 threads a column, 48 elements a thread) takes 4 columns:
  // 192 threads, so that the forward pass's 255 registers a thread fit.
  // Side 640 (20 threads a column) takes 8 columns: 160 threads.
  static constexpr int CC = (N == 256 || N == 512 || N == 1024) ? 128 / C::N1
                            : N == 2304                        ? 4
                            : N == 640                         ? 8
                                                               : (C::N1 >= 32 ? 8 : (C::N1 >= 16 ? 16 : 32));
  static constexpr int THREADS = CC * C::N1;
  static constexpr int SMEM_ELEMS = C::N2 * C::LD * CC;
  static constexpr size_t SMEM_BYTES = sizeof(float2) * SMEM_ELEMS;
  // one plane's column strip (N rows x CC columns) of complex values
  static constexpr size_t STRIP_ELEMS = (size_t)N * CC;
  // staging strips in shared memory next to the exchange buffer: two for the
  // forward pass (double-buffered prefetch), one complex + one FP64 strip for
  // the adjoint (spectrum and phase table, constant over z)
  // (only where two blocks still fit on an SM: side 2304 would take 222 KB)
  static constexpr bool STAGE = (N % CC == 0) && (SMEM_BYTES + 2 * sizeof(float2) * STRIP_ELEMS <= 113 * 1024);
  static constexpr size_t STAGE_BYTES = SMEM_BYTES + (STAGE ? 2 * sizeof(float2) * STRIP_ELEMS : 0);
};

// Copy the CC-column strip starting at column x0 of a plane of N rows of W
// elements into a dense [row][CC] shared buffer (16-byte pieces, two elements
// each, spread over the block).  Columns past the row's end are left as they
// are: W is even, so a piece lies inside the row or outside it.
template <int N, typename T>
__device__ __forceinline__ void strip_async(T* dst, const T* plane, int x0, int W) {
  static_assert(sizeof(T) == 8, "two elements a piece");
  using Lay = ColLayout<N>;
  constexpr int CC = Lay::CC;
  constexpr int PER_ROW = CC * (int)sizeof(T) / 16;  // 16-byte pieces per strip row
  constexpr int PIECES = N * PER_ROW;
  const char* src = reinterpret_cast<const char*>(plane + x0);
  char* d = reinterpret_cast<char*>(dst);
  for (int k = threadIdx.x; k < PIECES; k += Lay::THREADS) {
    const int row = k / PER_ROW, piece = k - row * PER_ROW;
    if (x0 + 2 * piece < W)
      cp_async16(d + ((size_t)row * CC * sizeof(T) + piece * 16), src + ((size_t)row * W * sizeof(T) + piece * 16));
  }
}

// Phase-table reads are issued in groups separated by a compiler scheduling
// fence so that the FP64 table values of a whole line are not all live at once.
constexpr int kPhaseGroup = 8;
// Hide a pointer's loop invariance from the compiler: the z loops re-read the
// phase table (and the residual spectrum) from L1/L2 every plane instead of
// pinning a whole line of them in registers.
template <typename T>
__device__ __forceinline__ const T* launder(const T* p) {
  asm volatile("mov.b64 %0, %0;" : "+l"(p));
  return p;
}
// Same for the twiddle index: recomputing a line's inter-stage twiddles every
// plane costs two sincospi and ~N2 complex products, far less than keeping
// N2 complex twiddles live across the z loop.
__device__ __forceinline__ int launder_i(int v) {
  asm volatile("mov.b32 %0, %0;" : "+r"(v));
  return v;
}

// Tensor-memory-accelerator (TMA) store of a dense shared-memory tile
// [rows][CC] of 8-byte elements to a 3-D (x, row, plane) tensor.  Stores only,
// no multicast.  The coordinates are non-negative and x * 8 bytes is a
// multiple of 16.
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, const void* smem, int x, int y, int z) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<unsigned long long>(map)),
               "r"(s), "r"(x), "r"(y), "r"(z)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// the source tiles of every committed store have been read
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// every committed store has completed
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// order this thread's shared-memory writes before later async-proxy reads
__device__ __forceinline__ void fence_smem_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// rows per TMA box: the largest divisor of N not above 256 (the box limit)
template <int N>
constexpr int tma_rows() {
  int r = 1;
  for (int d = 1; d <= 256 && d <= N; ++d)
    if (N % d == 0) r = d;
  return r;
}

// Exchange + stage B shared by all column kernels.  On entry v holds the
// twiddled stage-A output of this thread; on exit the stage-B output.
template <int N, bool INV>
__device__ __forceinline__ void col_exchange(float2 (&v)[LineCfg<N>::VS], float2* sm, int c, int t) {
  using C = LineCfg<N>;
  using Lay = ColLayout<N>;
  constexpr int N1 = C::N1, N2 = C::N2, M = C::M, LD = C::LD, CC = Lay::CC;
  __syncthreads();  // previous users of sm are done
#pragma unroll
  for (int k2 = 0; k2 < N2; ++k2) sm[(k2 * LD + t) * CC + c] = v[k2];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < M; ++j) {
    const bool ok = row_ok<N>(t, j);
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1)
      v[j * N1 + n1] = ok ? sm[((t + N1 * j) * LD + n1) * CC + c] : make_float2(0.f, 0.f);
  }
  stage_b_dft<N1, C::VS, INV>(v);
}

// The column passes walk many planes with the same thread-to-row assignment,
// so a thread's inter-stage twiddles are the same for every plane.  For lines
// of up to 32 elements a thread they are computed once and kept in registers
// (one complex product an element per plane instead of two plus the anchor
// products); shared memory limits the column passes to 8 warps per SM, which
// leaves the registers free.  Longer lines regenerate them every plane.
template <int N>
constexpr bool kHoistTw = LineCfg<N>::N2 <= 32 && LineCfg<N>::EXACT;

template <int N, int N2, bool INV>
__device__ __forceinline__ void apply_twiddles(float2 (&v)[N2], const float2 (&tw)[kHoistTw<N> ? N2 : 1], int t) {
  if constexpr (kHoistTw<N>) {
#pragma unroll
    for (int k = 1; k < N2; ++k) v[k] = cmul(v[k], tw[k]);
  } else {
    line_twiddle<N, N2, INV>(v, launder_i(t));
  }
}

// acc += v h: four fused multiply-adds where the twiddles are hoisted (lines
// of up to 32 elements a thread); the longer lines keep the product-then-add
// form, whose shorter live ranges keep them within the register file
template <int N>
__device__ __forceinline__ void cmac(float2& acc, float2 v, float2 h) {
  if constexpr (kHoistTw<N>) {
    acc.x = fmaf(v.x, h.x, fmaf(-v.y, h.y, acc.x));
    acc.y = fmaf(v.x, h.y, fmaf(v.y, h.x, acc.y));
  } else {
    acc = cadd(acc, cmul(v, h));
  }
}

// Adjoint column pass: U_z(:, x) = IDFT_y( conj(H'_z(:, x)) * Rs(:, x) ), z in [zb, ze).
// Planes of N rows of any even length W (the row pitch); SQ: W = N, which
// makes every element offset below a compile-time constant (a run-time pitch
// cost the square column passes 3 to 10 %).  Rs already carries 1/(W H).
// The spectrum and phase-table strips are the same for every plane: they are
// staged in shared memory once per block when they fit.
template <int N, bool TMA, bool SQ>
__global__ void __launch_bounds__(ColLayout<N>::THREADS) k_adj_col(const float2* __restrict__ Rs,
                                                                   const double* __restrict__ cturn,
                                                                   const double* __restrict__ zlist,
                                                                   float2* __restrict__ U, int z0, int z1,
                                                                   int zpb, int Wr,
                                                                   const __grid_constant__ CUtensorMap umap) {
  const int W = SQ ? N : Wr;
  using C = LineCfg<N>;
  using Lay = ColLayout<N>;
  constexpr int N1 = C::N1, N2 = C::N2, M = C::M, CC = Lay::CC;
  extern __shared__ __align__(128) float2 sm[];  // TMA sources need 128-byte alignment
  const int c = threadIdx.x % CC, t = threadIdx.x / CC;
  const int xr = blockIdx.x * CC + c;
  const bool col_ok = xr < W;
  const int x = col_ok ? xr : W - 1;
  const int zb = z0 + blockIdx.y * zpb, ze = min(zb + zpb, z1);
  const size_t HW = (size_t)N * W;
  float2* s_rs = sm + Lay::SMEM_ELEMS;
  double* s_ct = reinterpret_cast<double*>(s_rs + Lay::STRIP_ELEMS);
  if constexpr (Lay::STAGE) {
    strip_async<N>(s_rs, Rs, blockIdx.x * CC, W);
    strip_async<N>(s_ct, cturn, blockIdx.x * CC, W);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
  }
  const float2* rs = Rs + (size_t)t * W + x;
  const double* ct = cturn + (size_t)t * W + x;
  float2 tw[kHoistTw<N> ? N2 : 1];
  if constexpr (kHoistTw<N>) line_twiddles<N, N2, true>(tw, t);
  double znext = zb < ze ? zlist[zb] : 0.0;
#pragma unroll 1
  for (int z = zb; z < ze; ++z) {
    const double zz = znext;
    if (z + 1 < ze) znext = zlist[z + 1];  // in flight during this plane
    float2 v[C::VS];
    if constexpr (Lay::STAGE) {
#pragma unroll
      for (int n2 = 0; n2 < N2; ++n2) {
        const int i = (t + N1 * n2) * CC + c;
        v[n2] = cmul(s_rs[i], transfer(zz, s_ct[i], true));
      }
    } else {
      const float2* rsz = launder(rs);
      const double* ctz = launder(ct);
#pragma unroll
      for (int g = 0; g < N2; g += kPhaseGroup) {
#pragma unroll
        for (int q = 0; q < kPhaseGroup; ++q) {
          const int n2 = g + q;
          v[n2] = cmul(__ldg(rsz + (size_t)n2 * N1 * W), transfer(zz, __ldg(ctz + (size_t)n2 * N1 * W), true));
        }
        sched_fence();
      }
    }
    reg_fft<N2, true>(head<N2>(v));
    apply_twiddles<N, N2, true>(head<N2>(v), tw, t);
    // the exchange buffer also holds the previous plane's output tile: its
    // store must have read it (the exchange starts with a barrier)
    if (TMA && threadIdx.x == 0) bulk_wait_read_all();
    col_exchange<N, true>(v, sm, c, t);
    if constexpr (TMA) {
      // plane z's [N][CC] column strip goes out through the TMA from the
      // exchange buffer, as a few bulk stores instead of N2 8-byte stores a thread
      __syncthreads();  // every thread is done reading the exchange
#pragma unroll
      for (int j = 0; j < M; ++j)
        if (row_ok<N>(t, j))
#pragma unroll
          for (int k1 = 0; k1 < N1; ++k1) sm[(N1 * j + N2 * k1 + t) * CC + c] = v[j * N1 + k1];
      fence_smem_async();
      __syncthreads();
      if (threadIdx.x == 0) {
        constexpr int R = tma_rows<N>();
#pragma unroll 1
        for (int b = 0; b < N; b += R) tma_store_3d(&umap, sm + b * CC, blockIdx.x * CC, b, z);
        bulk_commit();
      }
    } else if (col_ok) {
      float2* Uz = U + (size_t)z * HW + (size_t)t * W + x;
#pragma unroll
      for (int j = 0; j < M; ++j)
        if (row_ok<N>(t, j))
#pragma unroll
          for (int k1 = 0; k1 < N1; ++k1) Uz[(size_t)(N1 * j + N2 * k1) * W] = v[j * N1 + k1];
    }
  }
  if (TMA && threadIdx.x == 0) bulk_wait_all();
}

// Inter-stage twiddles as a per-block table in shared memory, for column
// kernels that run three blocks an SM: w^(t k) for the N1 thread rows t and
// the N2 elements k of a line, the same values (same FP32 expression) that
// line_twiddles keeps in registers, so results are bit-identical to the
// register-resident form while 2 N2 registers a thread are freed.  Rows are
// padded to an even length (16-byte aligned pairs) that spreads the 8 rows a
// warp reads over all 32 banks.
template <int N>
struct TwTable {
  using C = LineCfg<N>;
  static constexpr int LDT = C::N2 + 2;  // float2 per row
  static constexpr int ELEMS = C::N1 * LDT;
  static constexpr size_t BYTES = sizeof(float2) * ELEMS;
};

// Blocks an SM the table-twiddle column kernels are compiled for: three for
// lines of up to 32 elements a thread; one for 48 (sides 384, 768 and 2304),
// whose lines alone take most of the register file.
template <int N>
constexpr int col3_minb() {
  return LineCfg<N>::N2 <= 32 ? 3 : 1;
}

template <int N, bool INV>
__device__ __forceinline__ void tw_table_build(float2* tab) {
  using C = LineCfg<N>;
  constexpr int N2 = C::N2, LDT = TwTable<N>::LDT;
  const float sgn = INV ? 2.0f : -2.0f;
  for (int i = threadIdx.x; i < C::N1 * N2; i += ColLayout<N>::THREADS) {
    const int t = i / N2, k = i - t * N2;
    float s, c;
    sincospif(sgn * (float)((t * k) % N) / (float)N, &s, &c);
    tab[t * LDT + k] = make_float2(c, s);
  }
}

// v[k] *= w^(t k), k >= 1, from the table (pairs of twiddles per 16-byte load)
template <int N>
__device__ __forceinline__ void tw_table_apply(float2 (&v)[LineCfg<N>::N2], const float2* tab, int t) {
  constexpr int N2 = LineCfg<N>::N2;
  static_assert(N2 % 2 == 0, "twiddle pairs");
  const float4* row = reinterpret_cast<const float4*>(tab + t * TwTable<N>::LDT);
#pragma unroll
  for (int k = 0; k < N2; k += 2) {
    const float4 q = row[k / 2];
    if (k > 0) v[k] = cmul(v[k], make_float2(q.x, q.y));
    v[k + 1] = cmul(v[k + 1], make_float2(q.z, q.w));
  }
}

// Transfer function H'_z = exp(i 2 pi u), u = frac(z * cturn), with the
// accurate sincospi: used where a value seeds many planes (the recurrence
// below), so its error is not multiplied by the plane count.
__device__ __forceinline__ float2 transfer_accurate(double z, double cturn, bool conj_) {
  double u = z * cturn;
  u -= rint(u);
  float s, c;
  sincospif(2.0f * (float)u, &s, &c);
  return make_float2(c, conj_ ? -s : s);
}

// What Horner's sum over planes 0 .. n with the rotation d (D = H'_dz in FP32) is
// multiplied by: H'_z of its first plane, turned by what d^(n/2) has drifted from
// D^(n/2), so that term k carries the drift of |k - n/2| steps instead of k.  `drift`
// holds D / d - 1 (HornerTable); left out where a chunk has too few planes to drift by
// an ulp.  512 x 512 x 100, 17 planes a chunk: 4.1e-7 from the exact sum with d from a
// phase rounded to FP32 and no drift, 3.2e-7 so; the volume of a solve at 1024 x 1024 x
// 1000, 200 planes a chunk: 1.6e-6 and 4.3e-7.
constexpr int kHornerDrift = 8;
template <bool DRIFT>
__device__ __forceinline__ float2 horner_anchor(double z, double cturn, const __half2* drift, int n) {
  const float2 h = transfer_accurate(z, cturn, false);
  if (!DRIFT) return h;
  const float2 e = __half22float2(__ldg(drift));
  return cadd(h, cmul(h, cscale(e, 0.5f * (float)n / kHornerDriftScale)));
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Planes between exact re-anchorings of the adjoint recurrence.  FP32
// rotations drift by about one rounding a step; 16 steps keep that near 1e-6.
constexpr int kAdjAnchor = 16;

// Adjoint column pass for evenly spaced planes (z_{k+1} - z_k = dz for all k):
// Y_z = conj(H'_z) Rs advances from plane to plane by the rotation
// D = conj(H'_dz), one complex product an element, instead of an FP64 phase
// reduction and a sincos.  Y lives in registers and D in shared memory, which
// replaces both staged strips of k_adj_col (spectrum and phase table): 66 KB
// a block at side 1024 instead of 98 KB, so three blocks share an SM.  Every
// kAdjAnchor planes Y is recomputed exactly from Rs and the FP64 phase table.
// Lines of up to 32 elements a thread only (the inter-stage twiddles are
// regenerated each plane to leave registers for Y).
//
// TWM selects the inter-stage twiddles: 1 keeps them in registers as k_adj_col
// does (fewest instructions a plane, two blocks an SM); 0 regenerates them
// each plane (three blocks fit, twice the instructions); 2 reads them from a
// per-block shared table (one 16-byte load per two elements, three blocks an
// SM).  The autotuner picks one of these or the direct evaluation.
template <int N, bool TMA, int TWM, bool SQ>
__global__ void __launch_bounds__(ColLayout<N>::THREADS, TWM == 1 ? 2 : col3_minb<N>())
    k_adj_col_rec(const float2* __restrict__ Rs, const double* __restrict__ cturn, const double* __restrict__ zlist,
                  double dz, float2* __restrict__ U, int z0, int z1, int zpb, int Wr,
                  const __grid_constant__ CUtensorMap umap) {
  const int W = SQ ? N : Wr;
  constexpr bool HOIST = TWM == 1;
  using C = LineCfg<N>;
  using Lay = ColLayout<N>;
  constexpr int N1 = C::N1, N2 = C::N2, M = C::M, CC = Lay::CC;
  static_assert(N2 <= (TWM == 2 ? 48 : 32), "the recurrence keeps a line's elements in registers");
  extern __shared__ __align__(128) float2 sm[];
  const int c = threadIdx.x % CC, t = threadIdx.x / CC;
  const int xr = blockIdx.x * CC + c;
  const bool col_ok = xr < W;
  const int x = col_ok ? xr : W - 1;
  const int zb = z0 + blockIdx.y * zpb, ze = min(zb + zpb, z1);
  if (zb >= ze) return;
  float2* s_d = sm + Lay::SMEM_ELEMS;  // this thread's rotations, [row][CC] (thread-private slots)
  float2* s_tw = s_d + Lay::STRIP_ELEMS;  // twiddle table (TWM 2)
  const float2* rs = Rs + (size_t)t * W + x;
  const double* ct = cturn + (size_t)t * W + x;
  float2 tw[HOIST ? N2 : 1];
  if constexpr (HOIST) line_twiddles<N, N2, true>(tw, t);
  if constexpr (TWM == 2) {
    tw_table_build<N, true>(s_tw);
    __syncthreads();
  }
  float2 y[N2];
#pragma unroll
  for (int n2 = 0; n2 < N2; ++n2) {
    const double cn = __ldg(ct + (size_t)n2 * N1 * W);
    s_d[(t + N1 * n2) * CC + c] = transfer_accurate(dz, cn, true);
    y[n2] = cmul(__ldg(rs + (size_t)n2 * N1 * W), transfer_accurate(zlist[zb], cn, true));
  }
#pragma unroll 1
  for (int z = zb; z < ze; ++z) {
    if (z > zb) {
      if ((z - zb) % kAdjAnchor == 0) {
        const double zz = zlist[z];
        const float2* rsz = launder(rs);
        const double* ctz = launder(ct);
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2)
          y[n2] = cmul(__ldg(rsz + (size_t)n2 * N1 * W), transfer_accurate(zz, __ldg(ctz + (size_t)n2 * N1 * W), true));
      } else {
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) y[n2] = cmul(y[n2], s_d[(t + N1 * n2) * CC + c]);
      }
    }
    float2 v[N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2) v[n2] = y[n2];
    reg_fft<N2, true>(v);
    if constexpr (HOIST) {
#pragma unroll
      for (int k = 1; k < N2; ++k) v[k] = cmul(v[k], tw[k]);
    } else if constexpr (TWM == 2) {
      tw_table_apply<N>(v, s_tw, t);
    } else {
      line_twiddle<N, N2, true>(v, launder_i(t));
    }
    if (TMA && threadIdx.x == 0) bulk_wait_read_all();
    col_exchange<N, true>(v, sm, c, t);
    if constexpr (TMA) {
      __syncthreads();
#pragma unroll
      for (int j = 0; j < M; ++j)
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) sm[(N1 * j + N2 * k1 + t) * CC + c] = v[j * N1 + k1];
      fence_smem_async();
      __syncthreads();
      if (threadIdx.x == 0) {
        constexpr int R = tma_rows<N>();
#pragma unroll 1
        for (int b = 0; b < N; b += R) tma_store_3d(&umap, sm + b * CC, blockIdx.x * CC, b, z);
        bulk_commit();
      }
    } else if (col_ok) {
      float2* Uz = U + (size_t)z * ((size_t)N * W) + (size_t)t * W + x;
#pragma unroll
      for (int j = 0; j < M; ++j)
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) Uz[(size_t)(N1 * j + N2 * k1) * W] = v[j * N1 + k1];
    }
  }
  if (TMA && threadIdx.x == 0) bulk_wait_all();
}

// Forward column pass with the z-sum: Spart[chunk](:, x) = sum_z H'_z(:, x) DFT_y(T_z(:, x)).
// When they fit next to the exchange buffer, the block's strip of the phase
// table (constant over z) and one strip of T are staged in shared memory:
// plane z+1's strip is fetched asynchronously once the exchange of plane z has
// consumed the buffer, and overlaps the transfer-function multiply and sum.
template <int N, bool SQ>
__global__ void __launch_bounds__(ColLayout<N>::THREADS) k_fwd_col(const float2* __restrict__ T,
                                                                   const double* __restrict__ cturn,
                                                                   const double* __restrict__ zlist,
                                                                   float2* __restrict__ Spart, int z0, int z1,
                                                                   int zpb, int Wr) {
  const int W = SQ ? N : Wr;
  using C = LineCfg<N>;
  using Lay = ColLayout<N>;
  constexpr int N1 = C::N1, N2 = C::N2, M = C::M, CC = Lay::CC;
  extern __shared__ __align__(128) float2 sm[];
  const int c = threadIdx.x % CC, t = threadIdx.x / CC;
  const int xr = blockIdx.x * CC + c;
  const bool col_ok = xr < W;
  const int x = col_ok ? xr : W - 1;
  const int zb = z0 + blockIdx.y * zpb, ze = min(zb + zpb, z1);
  const size_t HW = (size_t)N * W;
  const double* ct = cturn + (size_t)t * W + x;
  float2* const s_t = sm + Lay::SMEM_ELEMS;                                  // one strip of T
  const double* const s_ct = reinterpret_cast<const double*>(s_t + Lay::STRIP_ELEMS);  // phase-table strip
  if constexpr (Lay::STAGE) {
    strip_async<N>(const_cast<double*>(s_ct), cturn, blockIdx.x * CC, W);
    if (zb < ze) strip_async<N>(s_t, T + (size_t)zb * HW, blockIdx.x * CC, W);
    cp_async_commit();
  }
  float2 acc[C::VS];
#pragma unroll
  for (int i = 0; i < C::VS; ++i) acc[i] = make_float2(0.f, 0.f);
  float2 tw[kHoistTw<N> ? N2 : 1];
  if constexpr (kHoistTw<N>) line_twiddles<N, N2, false>(tw, t);
  double znext = zb < ze ? zlist[zb] : 0.0;
#pragma unroll 1
  for (int z = zb; z < ze; ++z) {
    const double zz = znext;
    if (z + 1 < ze) znext = zlist[z + 1];  // in flight during this plane
    float2 v[C::VS];
    if constexpr (Lay::STAGE) {
      cp_async_wait<0>();
      __syncthreads();
#pragma unroll
      for (int n2 = 0; n2 < N2; ++n2) v[n2] = s_t[(t + N1 * n2) * CC + c];
    } else {
      const float2* Tz = T + (size_t)z * HW + (size_t)t * W + x;
#pragma unroll
      for (int n2 = 0; n2 < N2; ++n2) v[n2] = Tz[(size_t)n2 * N1 * W];
    }
    reg_fft<N2, false>(head<N2>(v));
    apply_twiddles<N, N2, false>(head<N2>(v), tw, t);
    // the exchange's first barrier also orders every thread's reads of s_t
    // before the refill below
    col_exchange<N, false>(v, sm, c, t);
    if constexpr (Lay::STAGE) {
      if (z + 1 < ze) strip_async<N>(s_t, T + (size_t)(z + 1) * HW, blockIdx.x * CC, W);
      cp_async_commit();
#pragma unroll
      for (int j = 0; j < M; ++j)
        if (row_ok<N>(t, j))
#pragma unroll
          for (int k1 = 0; k1 < N1; ++k1) {
            const float2 h = transfer(zz, s_ct[(N1 * j + N2 * k1 + t) * CC + c], false);
            cmac<N>(acc[j * N1 + k1], v[j * N1 + k1], h);
          }
    } else {
      const double* ctz = launder(ct);
#pragma unroll
      for (int g = 0; g < C::VS; g += kPhaseGroup) {
#pragma unroll
        for (int q = 0; q < kPhaseGroup; ++q) {
          const int j = (g + q) / N1, k1 = (g + q) % N1;
          if (row_ok<N>(t, j)) {
            const float2 h = transfer(zz, __ldg(ctz + (size_t)(N1 * j + N2 * k1) * W), false);
            cmac<N>(acc[j * N1 + k1], v[j * N1 + k1], h);
          }
        }
        sched_fence();
      }
    }
  }
  if constexpr (Lay::STAGE) cp_async_wait<0>();
  if (col_ok) {
    float2* Sp = Spart + (size_t)blockIdx.y * HW + (size_t)t * W + x;
#pragma unroll
    for (int j = 0; j < M; ++j)
      if (row_ok<N>(t, j))
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) Sp[(size_t)(N1 * j + N2 * k1) * W] = acc[j * N1 + k1];
  }
}

// Forward column pass for evenly spaced planes, by Horner's scheme: with
// H'_z = H'_{zb} D^(z - zb) and D = H'_dz,
//   sum_{z in [zb, ze)} H'_z V_z = H'_{zb} (((V_{ze-1} D + V_{ze-2}) D + ...) D + V_{zb}),
// so each plane costs one complex multiply-add by D (held in shared memory in
// place of the FP64 phase-table strip) instead of an FP64 phase reduction, a
// sincos and a multiply-add; H'_{zb} is applied once, exactly, at the end.  The
// planes go in descending order.  D^k carries the rounding of D k times (about
// k x 2e-8 in phase); horner_anchor halves it.
template <int N>
__global__ void __launch_bounds__(ColLayout<N>::THREADS) k_fwd_col_horner(const float2* __restrict__ T,
                                                                          const double* __restrict__ cturn,
                                                                          const double* __restrict__ zlist,
                                                                          const HornerTable table,
                                                                          float2* __restrict__ Spart, int z0, int z1,
                                                                          int zpb) {
  constexpr int W = N;  // square planes
  using C = LineCfg<N>;
  using Lay = ColLayout<N>;
  constexpr int N1 = C::N1, N2 = C::N2, M = C::M, CC = Lay::CC;
  static_assert(Lay::STAGE && C::EXACT, "staged sides only");
  extern __shared__ __align__(128) float2 sm[];
  const int c = threadIdx.x % CC, t = threadIdx.x / CC;
  const int xr = blockIdx.x * CC + c;
  const bool col_ok = xr < W;
  const int x = col_ok ? xr : W - 1;
  const int zb = z0 + blockIdx.y * zpb, ze = min(zb + zpb, z1);
  const size_t HW = (size_t)N * W;
  const double* ct = cturn + (size_t)t * W + x;
  const float2* rot = table.d + (size_t)t * W + x;
  float2* const s_t = sm + Lay::SMEM_ELEMS;       // one strip of T
  float2* const s_d = s_t + Lay::STRIP_ELEMS;     // this thread's rotations D, stage-B layout
  if (zb < ze) strip_async<N>(s_t, T + (size_t)(ze - 1) * HW, blockIdx.x * CC, W);
  cp_async_commit();
#pragma unroll
  for (int j = 0; j < M; ++j)
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1)
      s_d[(N1 * j + N2 * k1 + t) * CC + c] = __ldg(rot + (size_t)(N1 * j + N2 * k1) * W);
  float2 acc[N2];
#pragma unroll
  for (int i = 0; i < N2; ++i) acc[i] = make_float2(0.f, 0.f);
  float2 tw[kHoistTw<N> ? N2 : 1];
  if constexpr (kHoistTw<N>) line_twiddles<N, N2, false>(tw, t);
#pragma unroll 1
  for (int z = ze - 1; z >= zb; --z) {
    cp_async_wait<0>();
    __syncthreads();
    float2 v[N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2) v[n2] = s_t[(t + N1 * n2) * CC + c];
    reg_fft<N2, false>(v);
    apply_twiddles<N, N2, false>(v, tw, t);
    // the exchange's first barrier orders every thread's reads of s_t before the refill
    col_exchange<N, false>(v, sm, c, t);
    if (z - 1 >= zb) strip_async<N>(s_t, T + (size_t)(z - 1) * HW, blockIdx.x * CC, W);
    cp_async_commit();
#pragma unroll
    for (int j = 0; j < M; ++j)
#pragma unroll
      for (int k1 = 0; k1 < N1; ++k1) {
        const float2 d = s_d[(N1 * j + N2 * k1 + t) * CC + c];
        float2& a = acc[j * N1 + k1];
        const float2 u = v[j * N1 + k1];
        const float ax = a.x;
        a.x = fmaf(ax, d.x, fmaf(-a.y, d.y, u.x));
        a.y = fmaf(ax, d.y, fmaf(a.y, d.x, u.y));
      }
  }
  cp_async_wait<0>();
  if (col_ok && zb < ze) {
    const double zz = zlist[zb];
    const int We = W;
    float2* Sp = Spart + (size_t)blockIdx.y * HW + (size_t)t * W + x;
    const __half2* dr = table.drift + (size_t)t * W + x;
    const auto finish = [&](auto with) {  // one test for the chunk: the loads of all elements can be in flight
#pragma unroll
      for (int j = 0; j < M; ++j)
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) {
          const size_t o = (size_t)(N1 * j + N2 * k1) * We;
          Sp[o] = cmul(acc[j * N1 + k1], horner_anchor<decltype(with)::value>(zz, __ldg(ct + o), dr + o, ze - 1 - zb));
        }
    };
    if (ze - 1 - zb < kHornerDrift) finish(std::false_type{});
    else finish(std::true_type{});
  } else if (col_ok) {
    float2* Sp = Spart + (size_t)blockIdx.y * HW + (size_t)t * W + x;
#pragma unroll
    for (int j = 0; j < M; ++j)
#pragma unroll
      for (int k1 = 0; k1 < N1; ++k1) Sp[(size_t)(N1 * j + N2 * k1) * W] = make_float2(0.f, 0.f);
  }
}

// The same Horner sum with three blocks an SM instead of two.  Shared memory
// per block drops from three column strips to two plus the twiddle table: T
// lands in the exchange buffer itself, and plane z-1's strip is requested as
// soon as every thread has read plane z's exchange, so its load overlaps the
// second DFT stage and the multiply-add (and the other blocks' work).  The
// inter-stage twiddles come from the per-block table, which frees the
// registers the third block needs.  Same arithmetic, same bits as
// k_fwd_col_horner.
template <int N>
constexpr size_t horner1_smem() {
  using Lay = ColLayout<N>;
  constexpr size_t buf = Lay::SMEM_ELEMS > Lay::STRIP_ELEMS ? (size_t)Lay::SMEM_ELEMS : Lay::STRIP_ELEMS;
  return sizeof(float2) * (buf + Lay::STRIP_ELEMS) + TwTable<N>::BYTES + 16;  // + the mbarrier
}

// Sides that have the table-twiddle forms (k_fwd_col_horner1, and
// k_adj_col_rec with TWM 2): whole lines a thread (N1 | N2), column blocks
// that tile the row, up to 48 elements a thread, and the exchange buffer,
// the rotation strip and the table within the 227 KB a block may take.
template <int N>
constexpr bool kTableCols = LineCfg<N>::EXACT && (N % ColLayout<N>::CC == 0) && LineCfg<N>::N2 <= 48 &&
                            LineCfg<N>::N2 % 2 == 0 && horner1_smem<N>() <= 227 * 1024;

// Where the TMA-fed column passes count bounded waits that ran out
// (col_wait_timeouts): device memory of the current device.  None is expected:
// a wait covers one strip copy.
unsigned* col_timeout_counter();
constexpr unsigned kColMaxSpins = 1u << 26;

__device__ __forceinline__ void col_mbar_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(bar),
               "r"(bytes)
               : "memory");
}

// wait for phase `parity` of the mbarrier, at most kColMaxSpins tries; false when the bound ran out
__device__ __forceinline__ bool col_mbar_wait(unsigned bar, unsigned parity) {
  for (unsigned i = 0; i < kColMaxSpins; ++i) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// TMA load of a [rows][CC] box of 8-byte elements (x, row, plane) into shared
// memory, completing on the mbarrier.  No multicast; x * 8 bytes is a multiple
// of 16 and every coordinate lies inside the tensor.
__device__ __forceinline__ void tma_load_3d(void* smem, const CUtensorMap* map, int x, int y, int z, unsigned bar) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(d),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}

// With TMA, one thread loads each plane's strip as tma_rows<N>-row boxes that
// complete on an mbarrier, instead of every thread issuing 16-byte cp.async
// pieces.  Every wait on the mbarrier is bounded: when one runs out, the block
// counts it at `timeouts` (read back by col_wait_timeouts), gives the
// copy in flight one more bounded wait and leaves without writing its sums.
template <int N, bool TMA, bool SQ>
__global__ void __launch_bounds__(ColLayout<N>::THREADS, col3_minb<N>())
    k_fwd_col_horner1(const float2* __restrict__ T, const double* __restrict__ cturn,
                      const double* __restrict__ zlist, const HornerTable table,
                      float2* __restrict__ Spart, int z0, int z1, int zpb, int Wr,
                      const __grid_constant__ CUtensorMap tmap, unsigned* timeouts) {
  const int W = SQ ? N : Wr;
  using C = LineCfg<N>;
  using Lay = ColLayout<N>;
  constexpr int N1 = C::N1, N2 = C::N2, M = C::M, LD = C::LD, CC = Lay::CC;
  static_assert(C::EXACT && N % CC == 0 && N2 <= 48, "sides of up to 48 elements a thread");
  constexpr size_t BUF = Lay::SMEM_ELEMS > Lay::STRIP_ELEMS ? (size_t)Lay::SMEM_ELEMS : Lay::STRIP_ELEMS;
  extern __shared__ __align__(128) float2 sm[];
  const int c = threadIdx.x % CC, t = threadIdx.x / CC;
  const int xr = blockIdx.x * CC + c;
  const bool col_ok = xr < W;
  const int x = col_ok ? xr : W - 1;
  const int zb = z0 + blockIdx.y * zpb, ze = min(zb + zpb, z1);
  const size_t HW = (size_t)N * W;
  const double* ct = cturn + (size_t)t * W + x;
  const float2* rot = table.d + (size_t)t * W + x;
  float2* const s_d = sm + BUF;                  // this thread's rotations D, stage-B layout
  float2* const s_tw = s_d + Lay::STRIP_ELEMS;   // twiddle table
  uint64_t* const bar = reinterpret_cast<uint64_t*>(s_tw + TwTable<N>::ELEMS);
  const unsigned sbar = (unsigned)__cvta_generic_to_shared(bar);
  unsigned phase = 0;
  constexpr int R = tma_rows<N>();
  constexpr unsigned kStripBytes = (unsigned)(sizeof(float2) * Lay::STRIP_ELEMS);
  // plane z's strip into the buffer: by TMA (thread 0) or cp.async (all threads)
  auto request = [&](int z) {
    if constexpr (TMA) {
      if (threadIdx.x == 0) {
        fence_smem_async();  // the block's reads of the buffer come before the copy's writes
        col_mbar_expect_tx(sbar, kStripBytes);
#pragma unroll 1
        for (int b = 0; b < N; b += R) tma_load_3d(sm + b * CC, &tmap, blockIdx.x * CC, b, z, sbar);
      }
    } else {
      strip_async<N>(sm, T + (size_t)z * HW, blockIdx.x * CC, W);
      cp_async_commit();
    }
  };
  if constexpr (TMA) {
    if (threadIdx.x == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sbar) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
  }
  if (zb < ze) request(ze - 1);
  tw_table_build<N, false>(s_tw);
#pragma unroll
  for (int j = 0; j < M; ++j)
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1)
      s_d[(N1 * j + N2 * k1 + t) * CC + c] = __ldg(rot + (size_t)(N1 * j + N2 * k1) * W);
  {  // the phases are next read at the end, by all blocks of a wave at once
    const int Wp = SQ ? N : launder_i(Wr);
#pragma unroll
    for (int i = 0; i < N; i += N1) prefetch_l2(ct + (size_t)i * Wp);
  }
  float2 acc[N2];
#pragma unroll
  for (int i = 0; i < N2; ++i) acc[i] = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int z = ze - 1; z >= zb; --z) {
    if constexpr (TMA) {
      const bool ok = col_mbar_wait(sbar, phase);
      if (__syncthreads_or(!ok)) {  // a wait ran out: count it, let the copy land, leave
        if (threadIdx.x == 0) {
          atomicAdd(timeouts, 1u);
          col_mbar_wait(sbar, phase);
        }
        return;
      }
      phase ^= 1u;
    } else {
      cp_async_wait<0>();
      __syncthreads();  // plane z's strip (and, the first time, the table) is visible
    }
    float2 v[N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2) v[n2] = sm[(t + N1 * n2) * CC + c];
    reg_fft<N2, false>(v);
    tw_table_apply<N>(v, s_tw, t);
    __syncthreads();  // every thread has read the strip: the buffer becomes the exchange
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) sm[(k2 * LD + t) * CC + c] = v[k2];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < M; ++j)
#pragma unroll
      for (int n1 = 0; n1 < N1; ++n1) v[j * N1 + n1] = sm[((t + N1 * j) * LD + n1) * CC + c];
    __syncthreads();  // every thread has read the exchange: refill with plane z-1
    if (z - 1 >= zb) request(z - 1);
    stage_b_dft<N1, C::VS, false>(v);
#pragma unroll
    for (int j = 0; j < M; ++j)
#pragma unroll
      for (int k1 = 0; k1 < N1; ++k1) {
        const float2 d = s_d[(N1 * j + N2 * k1 + t) * CC + c];
        float2& a = acc[j * N1 + k1];
        const float2 u = v[j * N1 + k1];
        const float ax = a.x;
        a.x = fmaf(ax, d.x, fmaf(-a.y, d.y, u.x));
        a.y = fmaf(ax, d.y, fmaf(a.y, d.x, u.y));
      }
  }
  if constexpr (!TMA) cp_async_wait<0>();
  if (col_ok && zb < ze) {
    const double zz = zlist[zb];
    const int We = SQ ? N : launder_i(Wr);  // own row offsets: kept from the start, they would take the sums' registers
    float2* Sp = Spart + (size_t)blockIdx.y * HW + (size_t)t * W + x;
    const __half2* dr = table.drift + (size_t)t * W + x;
    const auto finish = [&](auto with) {  // one test for the chunk: the loads of all elements can be in flight
#pragma unroll
      for (int j = 0; j < M; ++j)
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) {
          const size_t o = (size_t)(N1 * j + N2 * k1) * We;
          Sp[o] = cmul(acc[j * N1 + k1], horner_anchor<decltype(with)::value>(zz, __ldg(ct + o), dr + o, ze - 1 - zb));
        }
    };
    if (ze - 1 - zb < kHornerDrift) finish(std::false_type{});
    else finish(std::true_type{});
  } else if (col_ok) {
    float2* Sp = Spart + (size_t)blockIdx.y * HW + (size_t)t * W + x;
#pragma unroll
    for (int j = 0; j < M; ++j)
#pragma unroll
      for (int k1 = 0; k1 < N1; ++k1) Sp[(size_t)(N1 * j + N2 * k1) * W] = make_float2(0.f, 0.f);
  }
}

// Plain column DFT of one plane.
template <int N, bool INV, bool SQ>
__global__ void __launch_bounds__(ColLayout<N>::THREADS) k_plane_col(const float2* __restrict__ in,
                                                                     float2* __restrict__ out, int Wr, float scale) {
  const int W = SQ ? N : Wr;
  using C = LineCfg<N>;
  using Lay = ColLayout<N>;
  constexpr int N1 = C::N1, N2 = C::N2, M = C::M, CC = Lay::CC;
  extern __shared__ __align__(128) float2 sm[];
  const int c = threadIdx.x % CC, t = threadIdx.x / CC;
  const int xr = blockIdx.x * CC + c;
  const bool col_ok = xr < W;
  const int x = col_ok ? xr : W - 1;
  const float2* src = in + (size_t)t * W + x;
  float2 v[C::VS];
#pragma unroll
  for (int n2 = 0; n2 < N2; ++n2) v[n2] = src[(size_t)n2 * N1 * W];
  reg_fft<N2, INV>(head<N2>(v));
  line_twiddle<N, N2, INV>(head<N2>(v), t);
  col_exchange<N, INV>(v, sm, c, t);
  if (col_ok) {
    float2* dst = out + (size_t)t * W + x;
#pragma unroll
    for (int j = 0; j < M; ++j)
      if (row_ok<N>(t, j))
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) dst[(size_t)(N1 * j + N2 * k1) * W] = cscale(v[j * N1 + k1], scale);
  }
}

template <int N>
static int col_strips(int W) {
  return (W + ColLayout<N>::CC - 1) / ColLayout<N>::CC;
}

// cuTensorMapEncodeTiled, resolved once through the runtime (no link-time
// dependence on the driver library); null when unavailable
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline EncodeTiledFn encode_tiled() {
  static const EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

// 3-D map (column, row, plane) of nz planes of h rows of w 8-byte elements
// with a box of cc columns x rows rows x 1 plane; rows must be whole 16-byte
// pieces and at least a box wide (columns of a box past the row's end are
// zero-filled on a load and dropped on a store)
inline bool plane_stack_map(CUtensorMap* m, void* base, int w, int h, int nz, int cc, int rows) {
  const EncodeTiledFn enc = encode_tiled();
  if (!enc || (reinterpret_cast<uintptr_t>(base) & 15) != 0 || (w & 1) || w < cc) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)nz};
  const cuuint64_t strides[2] = {(cuuint64_t)w * 8, (cuuint64_t)w * h * 8};
  const cuuint32_t box[3] = {(cuuint32_t)cc, (cuuint32_t)rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_INT64, 3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

template <int N>
cudaError_t adj_col_n(const float2* Rs, const double* cturn, const double* zlist, float2* U, int W,
                             int z0, int z1, cudaStream_t st, int chunks_hint, double dz_uniform, int rec_mode) {
  using Lay = ColLayout<N>;
  const int nz = z1 - z0;
  if (nz <= 0) return cudaSuccess;
  const int strips = col_strips<N>(W);
  // the recurrence variants: evenly spaced planes, lines of <= 32 elements a
  // thread; `rec_mode` 1 regenerates the twiddles each plane, 2 keeps them;
  // 3 reads them from a shared table (lines of up to 48 elements)
  constexpr bool kRecOk = kHoistTw<N> && (N % Lay::CC == 0);
  const bool rec = dz_uniform != 0.0 && ((kRecOk && rec_mode != 0) || (kTableCols<N> && rec_mode == 3));
  const int target = (rec && rec_mode != 2 ? 12 : 8) * num_sms();
  int chunks = chunks_hint > 0 ? chunks_hint : (target + strips - 1) / strips;
  if (chunks > nz) chunks = nz;
  if (chunks < 1) chunks = 1;
  const int zpb = (nz + chunks - 1) / chunks;
  chunks = (nz + zpb - 1) / zpb;
  CUtensorMap umap;
  std::memset(&umap, 0, sizeof(umap));
  const bool tma = plane_stack_map(&umap, U, W, N, z1, Lay::CC, tma_rows<N>());
  cudaError_t e;
  const bool sq = W == N;
  // rectangular planes: the recurrence in its TMA form only, twiddles kept or from the table
  if constexpr (kRecOk || kTableCols<N>) {
    if (rec && (sq || tma)) {
      // the twiddle table follows the rotation strip (rec_mode 3)
      const size_t smem =
          Lay::SMEM_BYTES + sizeof(float2) * Lay::STRIP_ELEMS + (rec_mode == 3 ? TwTable<N>::BYTES : 0);
      auto go = [&](auto kern) -> cudaError_t {
        cudaError_t e2 = allow_smem(kern, smem);
        if (e2 != cudaSuccess) return e2;
        kern<<<dim3(strips, chunks), Lay::THREADS, smem, st>>>(Rs, cturn, zlist, dz_uniform, U, z0, z1, zpb, W, umap);
        return cudaGetLastError();
      };
      if constexpr (kTableCols<N>) {
        if (rec_mode == 3)
          return !sq ? go(k_adj_col_rec<N, true, 2, false>)
                     : tma ? go(k_adj_col_rec<N, true, 2, true>) : go(k_adj_col_rec<N, false, 2, true>);
      }
      if constexpr (kRecOk) {
        if (!sq) return go(k_adj_col_rec<N, true, 1, false>);
        if (rec_mode == 2) return tma ? go(k_adj_col_rec<N, true, 1, true>) : go(k_adj_col_rec<N, false, 1, true>);
        return tma ? go(k_adj_col_rec<N, true, 0, true>) : go(k_adj_col_rec<N, false, 0, true>);
      }
    }
  }
  auto direct = [&](auto kern) -> cudaError_t {
    e = allow_smem(kern, Lay::STAGE_BYTES);
    if (e != cudaSuccess) return e;
    kern<<<dim3(strips, chunks), Lay::THREADS, Lay::STAGE_BYTES, st>>>(Rs, cturn, zlist, U, z0, z1, zpb, W, umap);
    return cudaGetLastError();
  };
  if (sq) return tma ? direct(k_adj_col<N, true, true>) : direct(k_adj_col<N, false, true>);
  return tma ? direct(k_adj_col<N, true, false>) : direct(k_adj_col<N, false, false>);
}

template <int N>
cudaError_t fwd_col_n(const float2* T, const double* cturn, const double* zlist, float2* Spart, int W,
                             int z0, int z1, int nchunks, cudaStream_t st, int horner_mode,
                             const HornerTable& table) {
  using Lay = ColLayout<N>;
  const int nz = z1 - z0;
  if (nz <= 0) return cudaSuccess;
  const int strips = col_strips<N>(W);
  const int zpb = (nz + nchunks - 1) / nchunks;
  const int chunks = (nz + zpb - 1) / zpb;
  const bool horner = horner_mode != 0 && table.d;
  cudaError_t e;
  if (chunks < nchunks) {  // unused chunk slots must read as zero
    e = cudaMemsetAsync(Spart + (size_t)chunks * N * W, 0, sizeof(float2) * (size_t)(nchunks - chunks) * N * W, st);
    if (e != cudaSuccess) return e;
  }
  if constexpr (kTableCols<N>) {
    if (horner && (horner_mode == 2 || horner_mode == 3)) {
      constexpr size_t smem = horner1_smem<N>();
      CUtensorMap tmap;
      std::memset(&tmap, 0, sizeof(tmap));
      // mode 3: TMA strip loads where the map can be made
      const bool tma =
          horner_mode == 3 && plane_stack_map(&tmap, const_cast<float2*>(T), W, N, z1, Lay::CC, tma_rows<N>());
      auto go = [&](auto kern) -> cudaError_t {
        cudaError_t e2 = allow_smem(kern, smem);
        if (e2 != cudaSuccess) return e2;
        unsigned* const timeouts = col_timeout_counter();
        if (!timeouts) return cudaErrorUnknown;
        kern<<<dim3(strips, chunks), Lay::THREADS, smem, st>>>(T, cturn, zlist, table, Spart, z0, z1, zpb, W, tmap,
                                                               timeouts);
        return cudaGetLastError();
      };
      if (W == N) return tma ? go(k_fwd_col_horner1<N, true, true>) : go(k_fwd_col_horner1<N, false, true>);
      if (tma) return go(k_fwd_col_horner1<N, true, false>);
    }
  }
  if constexpr (Lay::STAGE && LineCfg<N>::EXACT) {
    if (horner && W == N) {
      e = allow_smem(k_fwd_col_horner<N>, Lay::STAGE_BYTES);
      if (e != cudaSuccess) return e;
      k_fwd_col_horner<N><<<dim3(strips, chunks), Lay::THREADS, Lay::STAGE_BYTES, st>>>(T, cturn, zlist, table,
                                                                                         Spart, z0, z1, zpb);
      return cudaGetLastError();
    }
  }
  auto direct = [&](auto kern) -> cudaError_t {
    e = allow_smem(kern, Lay::STAGE_BYTES);
    if (e != cudaSuccess) return e;
    kern<<<dim3(strips, chunks), Lay::THREADS, Lay::STAGE_BYTES, st>>>(T, cturn, zlist, Spart, z0, z1, zpb, W);
    return cudaGetLastError();
  };
  return W == N ? direct(k_fwd_col<N, true>) : direct(k_fwd_col<N, false>);
}

template <int N>
cudaError_t plane_col_n(int inverse, const float2* in, float2* out, int W, float scale, cudaStream_t st) {
  using Lay = ColLayout<N>;
  const int strips = col_strips<N>(W);
  auto go = [&](auto kern) -> cudaError_t {
    cudaError_t e = allow_smem(kern, Lay::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    kern<<<strips, Lay::THREADS, Lay::SMEM_BYTES, st>>>(in, out, W, scale);
    return cudaGetLastError();
  };
  if (W == N) return inverse ? go(k_plane_col<N, true, true>) : go(k_plane_col<N, false, true>);
  return inverse ? go(k_plane_col<N, true, false>) : go(k_plane_col<N, false, false>);
}


// the functions a side is reached through
#define RIHVR_FAST_SIDE(LINKAGE, NN)                                                                                \
  LINKAGE template cudaError_t rows_n<NN>(int, int, const void*, int, void*, long long, float, cudaStream_t);       \
  LINKAGE template cudaError_t adj_col_n<NN>(const float2*, const double*, const double*, float2*, int, int, int,   \
                                             cudaStream_t, int, double, int);                                      \
  LINKAGE template cudaError_t fwd_col_n<NN>(const float2*, const double*, const double*, float2*, int, int, int,   \
                                             int, cudaStream_t, int, const HornerTable&);                          \
  LINKAGE template cudaError_t plane_col_n<NN>(int, const float2*, float2*, int, float, cudaStream_t);

}  // namespace rihvr
