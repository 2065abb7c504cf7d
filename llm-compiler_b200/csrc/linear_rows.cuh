// Projections of a few rows (linear_rows.cu): which calls it takes, and a call.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

struct FewRowsCall {
  const void* input;
  const void* weight;
  const void* bias;
  const void* residual;
  void* output;
  int64_t m, k, n, input_row_stride;
  int epilogue;
  int splits = 1;                // K slices, each summed in one chain and added in slice order
  float* sums = nullptr;         // [splits, m, n]: the slices' fp32 sums instead of `output`, no epilogue
  float* row_squares = nullptr;  // [splits, m], with `sums`: sum(x_r^2) over each slice
  // With a residual: sum(y_r^2) in the slices [(tile, K slice), m] that the cluster form of linear_tcgen05.cu leaves
  float* squares_out = nullptr;
  int tile_columns = 0;
  // Folded RMSNorm: row r scaled by rsqrt(mean(x_r^2) + norm_eps) in front of the bias, the mean from such slices
  const float* norm_squares = nullptr;
  int norm_slices = 0;
  double norm_eps = 0.0;
};

// Runs a 16-bit projection of up to 8 rows whose rows allow 16-byte loads; false: not one of its sizes.
bool takes_few_rows(const FewRowsCall& call);
int linear_few_rows(const FewRowsCall& call, int dtype, cudaStream_t stream);

}  // namespace b200
