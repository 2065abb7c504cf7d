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
  float* sums = nullptr;         // [m, n]: the fp32 products instead of `output`, no epilogue
  float* row_squares = nullptr;  // [m], with `sums`: sum(x_r^2)
  int64_t m, k, n, input_row_stride;
  int epilogue;
  bool fold_norm = false;        // scale row r by rsqrt(mean(x_r^2) + norm_eps) in front of the bias
  double norm_eps = 0.0;
};

// Whether a 16-bit projection of this many rows runs in linear_few_rows. Its operands' rows allow 16-byte loads.
bool takes_few_rows(int64_t m);
int linear_few_rows(const FewRowsCall& call, int dtype, cudaStream_t stream);

}  // namespace b200
