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
#include "rihvr_line_fft.cuh"
#include "rihvr_lines.cuh"

namespace rihvr {

using namespace lines;

namespace {

constexpr int kRadices[] = {16, 15, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2};

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

// kernels for a block of at least `lines` lines and at most `most` threads
const LineKernels& kernels_for(const LPlan& p, int lines, int most) {
  static const LineKernels k = make_kernels<kElems>();
  return plan_threads(p, lines, kElems) <= most ? k : long_kernels();
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

cudaError_t rows_launch(LineKernels::Rows LineKernels::* which, const LPlan& p, const float2* tw, const void* in,
                        float2* out, long long nlines, float scale, cudaStream_t st) {
  const int C = row_lines(p);
  const long long blocks = (nlines + C - 1) / C;
  if (blocks <= 0) return cudaSuccess;
  // an odd line pitch keeps lines apart in the banks
  const int ls = line_places(p) | 1;
  const size_t smem = sizeof(float2) * (size_t)C * ls;
  const LineKernels& k = kernels_for(p, 1, kRowThreadsMax);
  const LineKernels::Rows kern = k.*which;
  cudaError_t e = allow_smem(kern, smem);
  if (e != cudaSuccess) return e;
  kern<<<(unsigned)blocks, plan_threads(p, C, k.elems), smem, st>>>(p, tw, in, out, nlines, scale, ilog2(C), ls);
  return cudaGetLastError();
}

// plan, table, columns a block, threads and shared memory of a column launch
struct ColLaunch {
  LPlan p;
  const float2* tw = nullptr;
  const LineKernels* k = nullptr;
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
  L->k = &kernels_for(L->p, 2, kColThreadsMax);
  L->threads = plan_threads(L->p, L->C, L->k->elems);
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
    return rows_launch(&LineKernels::inv_rows, p, tw, in, o, nlines, scale, st);
  }
  switch (in_kind) {
    case ELEM_C32:
    case ELEM_STORE_F32: return rows_launch(&LineKernels::rows_c32, p, tw, in, o, nlines, scale, st);
    case ELEM_R32: return rows_launch(&LineKernels::rows_r32, p, tw, in, o, nlines, scale, st);
    case ELEM_STORE_BF16: return rows_launch(&LineKernels::rows_bf16, p, tw, in, o, nlines, scale, st);
    case ELEM_STORE_F16: return rows_launch(&LineKernels::rows_f16, p, tw, in, o, nlines, scale, st);
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
  const auto kern = L.k->adj_col;
  e = allow_smem(kern, L.smem);
  if (e != cudaSuccess) return e;
  kern<<<dim3(L.strips, chunks), L.threads, L.smem, st>>>(L.p, L.tw, Rs, cturn, zlist, U, W, z0, z1, zpb, L.logc);
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
  const auto kern = L.k->fwd_col;
  e = allow_smem(kern, smem);
  if (e != cudaSuccess) return e;
  kern<<<dim3(L.strips, chunks), L.threads, smem, st>>>(L.p, L.tw, T, cturn, zlist, Spart, W, z0, z1, zpb, L.logc,
                                                        line_places(L.p));
  return cudaGetLastError();
}

cudaError_t launch_line_plane_col(int inverse, const float2* in, float2* out, int W, int H, float scale,
                                  cudaStream_t st) {
  ColLaunch L;
  cudaError_t e = col_launch(W, H, st, &L);
  if (e != cudaSuccess) return e;
  const auto kern = inverse ? L.k->inv_plane_col : L.k->plane_col;
  e = allow_smem(kern, L.smem);
  if (e != cudaSuccess) return e;
  kern<<<L.strips, L.threads, L.smem, st>>>(L.p, L.tw, in, out, W, scale, L.logc);
  return cudaGetLastError();
}

}  // namespace rihvr
