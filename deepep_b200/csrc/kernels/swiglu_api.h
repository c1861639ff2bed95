// SwiGLU forward and backward, and the product of rows with their routing weights (the training layer).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace dep {

struct SwigluParams {
  const __nv_bfloat16* gu;     // [rows][2 * inter]: gate columns, then up columns
  __nv_bfloat16* h;            // forward: [rows][inter] = silu(gate) * up
  const __nv_bfloat16* dh;     // backward: [rows][inter] gradient of h
  __nv_bfloat16* dgu;          // backward: [rows][2 * inter]
  long long rows;
  int inter, pad;              // inter: a multiple of 8
};
// out = a * w per row, and in the same pass prod = a * b (backward: a is the gradient, b the rows, prod the terms of the weight's
// gradient).  The weight is rounded to bf16 first, every product once.
struct RowScaleParams {
  const __nv_bfloat16* a;      // [rows][width]
  const float* w;              // [rows]
  __nv_bfloat16* out;          // [rows][width], or null
  const __nv_bfloat16* b;      // [rows][width], or null
  __nv_bfloat16* prod;         // [rows][width] when b is given
  long long rows;
  int width, pad;              // width: a multiple of 8
};
cudaError_t launch_row_scale(const RowScaleParams& p, int blocks, cudaStream_t stream);
cudaError_t launch_swiglu(const SwigluParams& p, bool backward, int blocks, cudaStream_t stream);

}  // namespace dep
