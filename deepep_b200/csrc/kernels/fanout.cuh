// Warp-wide copies of one row, or a piece of it, to several destinations, and the rows of an aligned layout that no token fills.
// Used by the high-throughput dispatch and the V1 expand operator.
#pragma once
#include "common.cuh"

namespace dep {

constexpr int kCopyUnroll = 7;    // 16-byte pieces per lane and pass: 3.5 KB in flight per warp

__device__ __forceinline__ unsigned long long shfl_u64(unsigned long long v, int src) {
  return __shfl_sync(0xffffffffu, v, src);
}

// Copies `units` 16-byte pieces from `src` to every destination in `mask`: lane l of the mask holds its
// destination in `dst`.  All loads of a pass are issued before the first store.
template <bool kPeerWritten, int U = kCopyUnroll>
__device__ __forceinline__ void warp_fanout(const int4* src, int units, unsigned long long dst, unsigned mask, int lane) {
  for (int u0 = 0; u0 < units; u0 += 32 * U) {
    int4 v[U];
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const int u = u0 + i * 32 + lane;
      if (u < units) v[i] = kPeerWritten ? __ldcg(src + u) : __ldg(src + u);
    }
    for (unsigned m = mask; m; m &= m - 1) {
      int4* d = reinterpret_cast<int4*>(shfl_u64(dst, __ffs(m) - 1));
#pragma unroll
      for (int i = 0; i < U; ++i) {
        const int u = u0 + i * 32 + lane;
        if (u < units) d[u] = v[i];
      }
    }
  }
}

// The same for a short run of floats (the scales of an fp8 row).
template <bool kPeerWritten>
__device__ __forceinline__ void warp_fanout_f32(const float* src, int n, unsigned long long dst, unsigned mask, int lane) {
  for (int b0 = 0; b0 < n; b0 += 32) {   // the trip count is the same for every lane: all of them take part in the shuffles
    const int b = b0 + lane;
    float v = 0.f;
    if (b < n) v = kPeerWritten ? __ldcg(src + b) : __ldg(src + b);
    for (unsigned m = mask; m; m &= m - 1) {
      float* d = reinterpret_cast<float*>(shfl_u64(dst, __ffs(m) - 1));
      if (b < n) d[b] = v;
    }
  }
}

// Calls f(row) for the rows between the end of every expert's rows (offsets[e] + counts[e]) and the next expert's first, and for
// those from offsets[experts] up to `total`.  Warp `gw` of `warps`; the warps are dealt out to the experts in turn.
template <class F>
__device__ __forceinline__ void for_padding_rows(const int* offsets, const int* counts, int experts, int total, int gw, int warps, F f) {
  const int per = max(1, warps / experts);            // warps per expert
  for (int i = gw; i < experts * per; i += warps) {
    const int e = i % experts, end = min(offsets[e + 1], total);
    for (int row = offsets[e] + counts[e] + i / experts; row < end; row += per) f(row);
  }
  for (int row = offsets[experts] + gw; row < total; row += warps) f(row);
}

__device__ __forceinline__ void zero_row(uint8_t* row, int row_bytes, float* sf, int nsf, int lane) {
  for (int u = lane; u < row_bytes / 16; u += 32) reinterpret_cast<int4*>(row)[u] = make_int4(0, 0, 0, 0);
  for (int b = lane; b < nsf; b += 32) sf[b] = 0.f;
}

}  // namespace dep
