// Line FFT passes of plane sides without a register-resident split
// (rihvr_lines.cu), behind the dispatchers of rihvr_kernels.cu.
#pragma once
#include <cuda_runtime.h>

namespace rihvr {

int line_fwd_col_chunks(int W, int H, int Nz);
cudaError_t launch_line_rows(int inverse, int in_kind, const void* in, int out_kind, void* out, int W,
                             long long nlines, float scale, cudaStream_t st);
cudaError_t launch_line_adj_col(const float2* Rs, const double* cturn, const double* zlist, float2* U, int W, int H,
                                int z0, int z1, cudaStream_t st, int chunks_hint);
cudaError_t launch_line_fwd_col(const float2* T, const double* cturn, const double* zlist, float2* Spart, int W,
                                int H, int z0, int z1, int nchunks, cudaStream_t st);
cudaError_t launch_line_plane_col(int inverse, const float2* in, float2* out, int W, int H, float scale,
                                  cudaStream_t st);

}  // namespace rihvr
