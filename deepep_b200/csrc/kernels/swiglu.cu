// silu(gate) * up over rows of [gate | up], and its backward pass (see swiglu_api.h).
//
// The results are those of the separate bf16 operations, bit for bit: every intermediate that they would store (silu(gate),
// dh * up) is rounded to bf16 here too.  silu(gate) is the gate times the reciprocal of 1 + exp(-gate), in the forward pass with the
// fast exponential: a gate is one of 65536 values, and for every one of them the rounded product is that of the accurate exponential
// and division (the tests go through all of them).  The backward pass needs the sigmoid in fp32 and takes the accurate exponential.
//
// One 16-byte piece of every operand per thread, in as many blocks as that takes: forward reads 4 and writes 2 bytes per value,
// backward reads 6 and writes 4.  Arithmetic and memory bound it about alike.  49152 rows of 1536: forward 85 us (5.3 TB/s), backward
// 128 us (5.9 TB/s); with a division in either 99 and 146 us, and as warps that loop over rows 97 and 163 us.  As library passes over
// the two strided halves (silu, product, their gradients and a concatenation): 382 and 575 us.
#include "swiglu_api.h"

namespace dep {

constexpr int kSwigluThreads = 256;

struct Vec8 { float v[8]; };
__device__ __forceinline__ Vec8 unpack8(const int4& q) {
  Vec8 r;
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) { r.v[2 * i] = __low2float(h[i]); r.v[2 * i + 1] = __high2float(h[i]); }
  return r;
}
__device__ __forceinline__ int4 pack8(const Vec8& r) {
  int4 q;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(r.v[2 * i], r.v[2 * i + 1]);
  return q;
}
__device__ __forceinline__ float as_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

template <bool kBackward>
__global__ void __launch_bounds__(kSwigluThreads) swiglu_kernel(const __grid_constant__ SwigluParams p) {
  const int units = p.inter / 8;
  const long long i = (long long)blockIdx.x * kSwigluThreads + threadIdx.x, row = i / units;
  if (row >= p.rows) return;
  const int u = (int)(i - row * units);
  const int4* gate = reinterpret_cast<const int4*>(p.gu) + row * 2 * units;
  const int4 g4 = __ldg(gate + u), u4 = __ldg(gate + units + u);
  int4 d4;
  if (kBackward) d4 = __ldg(reinterpret_cast<const int4*>(p.dh) + i);
  const Vec8 g = unpack8(g4), up = unpack8(u4);
  if (!kBackward) {
    Vec8 h;
#pragma unroll
    for (int e = 0; e < 8; ++e) h.v[e] = as_bf16(g.v[e] * __frcp_rn(1.f + __expf(-g.v[e]))) * up.v[e];
    reinterpret_cast<int4*>(p.h)[i] = pack8(h);
  } else {
    const Vec8 d = unpack8(d4);
    Vec8 dg, du;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float s = __frcp_rn(1.f + expf(-g.v[e]));
      du.v[e] = d.v[e] * as_bf16(g.v[e] * s);
      dg.v[e] = as_bf16(d.v[e] * up.v[e]) * s * (1.f + g.v[e] * (1.f - s));
    }
    int4* out = reinterpret_cast<int4*>(p.dgu) + row * 2 * units;
    out[u] = pack8(dg);
    out[units + u] = pack8(du);
  }
}

// Bound by memory.  49152 rows of 4096: 129 us one product, 257 us both (6.2 TB/s); as a library product with a broadcast factor
// 449 us each way, and 173 us for the terms of the weight's gradient.
__global__ void __launch_bounds__(kSwigluThreads) row_scale_kernel(const __grid_constant__ RowScaleParams p) {
  const int lane = threadIdx.x & 31, units = p.width / 8;
  const long long warps = (long long)gridDim.x * (kSwigluThreads / 32);
  for (long long row = (long long)blockIdx.x * (kSwigluThreads / 32) + (threadIdx.x >> 5); row < p.rows; row += warps) {
    const int4* a = reinterpret_cast<const int4*>(p.a) + row * units;
    const int4* b = reinterpret_cast<const int4*>(p.b) + row * units;
    const float w = as_bf16(__ldg(p.w + row));
    constexpr int U = 4;                       // 16-byte pieces of every operand in flight per lane
    for (int u0 = lane; u0 < units; u0 += 32 * U) {
      int4 a4[U], b4[U];
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const int u = u0 + i * 32;
        if (u < units) {
          a4[i] = __ldg(a + u);
          if (p.b) b4[i] = __ldg(b + u);
        }
      }
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const int u = u0 + i * 32;
        if (u >= units) break;
        const Vec8 x = unpack8(a4[i]);
        Vec8 r;
        if (p.out) {
#pragma unroll
          for (int e = 0; e < 8; ++e) r.v[e] = x.v[e] * w;
          reinterpret_cast<int4*>(p.out)[row * units + u] = pack8(r);
        }
        if (p.b) {
          const Vec8 y = unpack8(b4[i]);
#pragma unroll
          for (int e = 0; e < 8; ++e) r.v[e] = x.v[e] * y.v[e];
          reinterpret_cast<int4*>(p.prod)[row * units + u] = pack8(r);
        }
      }
    }
  }
}

// One block per token: the token's gradient is read once and stays in registers, kReturnRows of its rows are in flight at a time.
// Bound by memory (rows read once, their gradients written once).  49152 rows of 4096, six per token: 140 us in a training step; as a
// dispatch of the gradient, a product with two outputs and a sum 480 us there.
constexpr int kReturnRows = 3;
constexpr int kReturnThreads = 256;

template <int G>      // 16-byte pieces per thread
__global__ void __launch_bounds__(kReturnThreads) return_grad_kernel(const __grid_constant__ ReturnGradParams p) {
  __shared__ float s_dw[kReturnThreads / 32][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, threads = blockDim.x, units = p.width / 8, t = blockIdx.x;
  const int4* gsrc = reinterpret_cast<const int4*>(p.g) + (size_t)t * units;
  int4 g[G];
#pragma unroll
  for (int i = 0; i < G; ++i) {
    const int u = tid + i * threads;
    g[i] = u < units ? __ldg(gsrc + u) : make_int4(0, 0, 0, 0);
  }
  int row = lane < p.topk ? __ldg(p.slot_row + (size_t)t * p.topk + lane) : -1;
  if (row >= p.rows) row = -1;
  const float w = row >= 0 ? as_bf16(__ldg(p.w + row)) : 0.f;
  for (unsigned m = __ballot_sync(0xffffffffu, row >= 0); m;) {
    int4 y[kReturnRows][G];
    int at[kReturnRows], slot[kReturnRows];
    const int n = min(__popc(m), kReturnRows);
#pragma unroll
    for (int q = 0; q < kReturnRows; ++q) {
      if (q < n) {
        slot[q] = __ffs(m) - 1;
        m &= m - 1;
        at[q] = __shfl_sync(0xffffffffu, row, slot[q]);
        if (p.dw) {
#pragma unroll
          for (int i = 0; i < G; ++i) {
            const int u = tid + i * threads;
            y[q][i] = u < units ? __ldg(reinterpret_cast<const int4*>(p.y) + (size_t)at[q] * units + u) : make_int4(0, 0, 0, 0);
          }
        }
      }
    }
#pragma unroll
    for (int q = 0; q < kReturnRows; ++q) {
      if (q < n) {
        const float wq = __shfl_sync(0xffffffffu, w, slot[q]);
        float dot = 0.f;
#pragma unroll
        for (int i = 0; i < G; ++i) {
          const int u = tid + i * threads;
          const Vec8 gv = unpack8(g[i]);
          if (p.dw) {
            const Vec8 yv = unpack8(y[q][i]);
#pragma unroll
            for (int e = 0; e < 8; ++e) dot += as_bf16(gv.v[e] * yv.v[e]);
          }
          if (p.dy && u < units) {
            Vec8 r;
#pragma unroll
            for (int e = 0; e < 8; ++e) r.v[e] = gv.v[e] * wq;
            reinterpret_cast<int4*>(p.dy)[(size_t)at[q] * units + u] = pack8(r);
          }
        }
        if (p.dw) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
          if (lane == 0) s_dw[warp][slot[q]] = dot;
        }
      }
    }
  }
  if (!p.dw) return;
  __syncthreads();
  if (warp == 0 && row >= 0) {
    float sum = 0.f;
    for (int i = 0; i < threads / 32; ++i) sum += s_dw[i][lane];
    p.dw[row] = as_bf16(sum);
  }
}

cudaError_t launch_return_grad(const ReturnGradParams& p, cudaStream_t stream) {
  if (p.tokens == 0 || p.rows == 0) return cudaSuccess;
  const int units = p.width / 8, threads = units >= kReturnThreads ? kReturnThreads : (units + 31) / 32 * 32;
  const int pieces = (units + threads - 1) / threads;
  if (pieces <= 1) return_grad_kernel<1><<<p.tokens, threads, 0, stream>>>(p);
  else if (pieces <= 2) return_grad_kernel<2><<<p.tokens, threads, 0, stream>>>(p);
  else if (pieces <= 4) return_grad_kernel<4><<<p.tokens, threads, 0, stream>>>(p);
  else return cudaErrorInvalidValue;       // (the dispatch takes rows of at most 8192 values)
  return cudaGetLastError();
}

cudaError_t launch_row_scale(const RowScaleParams& p, int blocks, cudaStream_t stream) {
  if (p.rows == 0) return cudaSuccess;
  row_scale_kernel<<<blocks, kSwigluThreads, 0, stream>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_swiglu(const SwigluParams& p, bool backward, cudaStream_t stream) {
  if (p.rows == 0) return cudaSuccess;
  const unsigned grid = (unsigned)((p.rows * (p.inter / 8) + kSwigluThreads - 1) / kSwigluThreads);
  if (backward) swiglu_kernel<true><<<grid, kSwigluThreads, 0, stream>>>(p);
  else swiglu_kernel<false><<<grid, kSwigluThreads, 0, stream>>>(p);
  return cudaGetLastError();
}

}  // namespace dep
