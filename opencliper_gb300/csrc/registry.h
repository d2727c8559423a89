// Per-transform-length kernel table.  Each supported length L (see
// fft_size_ok) has one entry with host launchers for the templated kernels.
#pragma once

#include <cuda_runtime.h>
#include "types.h"

namespace gbn {

struct SizeKernels {
  int L;
  // The fused kernels take a device table of instances (all with H = L for the
  // column passes, W = L for the row pass) and the launch's BatchMap.
  // forward column pass (k_fwd_cols<L>), grid (W/8, coil groups, total frames)
  void (*fwd_cols)(const FusedArgs* tab, const BatchMap& bm, int it, int coils_per_block, dim3 grid, cudaStream_t s);
  // row pass (k_rows<L, resid>), 1-D persistent grid
  void (*rows)(const FusedArgs* tab, const BatchMap& bm, int it, bool resid, int grid, cudaStream_t s);
  // adjoint column pass (k_inv_cols<L, update>), grid (W/8, 2, total frames) in clusters of 2
  void (*inv_cols)(const FusedArgs* tab, const BatchMap& bm, int it, bool update, dim3 grid, cudaStream_t s);
  // dense FFT passes: rows (k_fft_rows_dense; mask [F][H][W] or nullptr, rows of C
  // coils), columns of images (k_fft_cols_dense), of S_c x_f (k_enc_cols), and
  // backward columns combined over the coils (k_adj_cols; S, or nullptr for the root
  // sum of squares) in clusters of cs CTAs
  void (*fft_rows)(const float2* in, float2* out, int nrows, int inv, float scale, const float2* tw,
                   const uint8_t* mask, int C, int H, int grid, bool first, cudaStream_t s);
  // fft_cols, adj_cols: after fft_rows, which releases them; fft_rows not first: after enc_cols
  void (*fft_cols)(const float2* in, float2* out, int W, int nimg, int inv, float scale, const float2* tw, int nsm,
                   cudaStream_t s);
  void (*enc_cols)(const float2* x, const float2* S, float2* out, int W, int C, int F, const float2* tw,
                   cudaStream_t s);
  void (*adj_cols)(const float2* T, const float2* S, float2* x, int W, int C, int F, float scale, const float2* tw,
                   int cs, cudaStream_t s);
  // row-local inner iteration: k_iter_pair<L, motion> where pair_cols, else
  // k_iter_cols<L, motion> on grid (W/8, 2, total frames) in clusters of 2; nullptr
  // for lengths that run only the three-pass iteration
  void (*iter_cols)(const FusedArgs* tab, const BatchMap& bm, int it, bool motion, dim3 grid, cudaStream_t s);
  // the sums and scalar step of iteration it - 1 alone (column-pair form)
  void (*iter_finish)(const FusedArgs* tab, const BatchMap& bm, int it, dim3 grid, cudaStream_t s);
  int pair_cols;     // columns per tile of the column-pair form of iter_cols; 0: iter_cols works on natural buffers
  int adj_per_sm[2];  // CTAs of adj_cols that share an SM: with S, and without
  int rows_per_cta;  // rows processed per CTA step by the row kernels
  int (*rows_occupancy)(bool resid);  // resident row-kernel CTAs per SM
};

// Returns the table entry for length L or nullptr when L is unsupported.
const SizeKernels* find_size(int L);

// Lengths with an entry, ascending.
int supported_sizes(int* out, int cap);

}  // namespace gbn
