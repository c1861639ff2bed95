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
// Backward of a combine with weighed rows: the gradient g of a token's sum goes to the rows of its slots, dy[row] = g * w[row], and
// dw[row] = sum(g * y[row]).  The weight is rounded to bf16 first, every product once; the sum is taken in fp32 and rounded to bf16.
struct ReturnGradParams {
  const __nv_bfloat16* g;      // [tokens][width]
  const __nv_bfloat16* y;      // [rows][width]
  const float* w;              // [rows]
  const int* slot_row;         // [tokens][topk] row of every slot, -1 for none
  __nv_bfloat16* dy;           // [rows][width], or null
  float* dw;                   // [rows], or null
  long long rows;
  int tokens, topk, width, pad;
};
cudaError_t launch_return_grad(const ReturnGradParams& p, cudaStream_t stream);
cudaError_t launch_row_scale(const RowScaleParams& p, int blocks, cudaStream_t stream);
cudaError_t launch_swiglu(const SwigluParams& p, bool backward, cudaStream_t stream);

}  // namespace dep
