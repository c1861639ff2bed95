// SwiGLU forward and backward (the expert activation of the training layer).
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
cudaError_t launch_swiglu(const SwigluParams& p, bool backward, int blocks, cudaStream_t stream);

}  // namespace dep
