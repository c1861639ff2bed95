// SwiGLU with a per-row factor, forward and backward (the expert activation of the training layer).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace dep {

struct SwigluParams {
  const __nv_bfloat16* gu;     // [rows][2 * inter]: gate columns, then up columns
  const float* w;              // [rows] factor of every row, or null (one)
  __nv_bfloat16* h;            // forward: [rows][inter] = silu(gate) * up * w
  const __nv_bfloat16* dh;     // backward: [rows][inter] gradient of h
  __nv_bfloat16* dgu;          // backward: [rows][2 * inter]
  float* dw;                   // backward: [rows] gradient of w, or null
  long long rows;
  int inter, pad;              // inter: a multiple of 8
};
cudaError_t launch_swiglu(const SwigluParams& p, bool backward, int blocks, cudaStream_t stream);

}  // namespace dep
