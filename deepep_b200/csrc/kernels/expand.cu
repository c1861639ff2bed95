// ep_expand / ep_aggregate: the V1 interface's local layout operators (see expand_api.h).
//
// expand: rows of the rank-deduplicated layout carry up to K local expert ids; every (row, slot) gets its own row
// in the expert-major output, ordered inside an expert by (row, slot).  Ranking is deterministic: bit masks per expert, ranks from
// popcounts.  A plan kernel (none with a saved mapping) is followed by a kernel of copies, in which every warp moves one piece of a
// row; rows between an expert's real count and its capacity are zeroed.
// aggregate: out[r] = sum over the slots of row r of (w *) x[mapping[r][k]], fp32 in slot order, one piece of a row per warp.
//
// The copies are bound by the bytes that they write or read, and blocks that the hardware deals out as they finish move them faster
// than persistent ones (2048 rows of 4096 bf16, top-6 of 64: expand 51 us as one cooperative kernel of 296 blocks with grid barriers
// between its passes, 6 us of plan and 18 of copies here; aggregate 47 us in 296 blocks that hold sixteen rows at a time, 25 here).
#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "expand_api.h"
#include "fanout.cuh"
#include "local_tile.cuh"

namespace cg = cooperative_groups;

namespace dep {

constexpr int kExpandThreads = 256;

// The host polls this word, which is in its memory, while the copies of the rows are queued behind the plan.
__device__ __forceinline__ void report(int* flag, int value) { *reinterpret_cast<volatile int*>(flag) = value; }

// The plan, by one cluster that keeps the table in shared memory.
__global__ void __launch_bounds__(kTileThreads) ep_expand_plan_kernel(const __grid_constant__ ExpandParams p) {
  cg::cluster_group cluster = cg::this_cluster();
  const int c = blockIdx.x % kTileCtas, share = blockIdx.x / kTileCtas, shares = gridDim.x / kTileCtas, tid = threadIdx.x;
  const int R = p.R, K = p.K, L = p.L, per = LocalTile::tokens(R), stride = LocalTile::stride(per);
  const int t0 = min(R, c * per), live = min(per, R - t0);
  extern __shared__ __align__(16) unsigned char smem[];
  const LocalTile s(smem, per, L);
  __shared__ int s_warp[kTileThreads / 32], s_hits[2];
  s.count(p.topk_idx + (size_t)t0 * K, live * K, per, K, L);
  cluster.sync();
  int before, tot;
  s.gather(cluster, c, L, s_hits, before, tot);
  const int cap = tid < L ? p.caps[tid] : 0, first = tile_prefix(cap, s_warp);
  if (tid < L) { s.off[tid + 1] = first + cap; s.base[tid] = first + before; }
  const int over = __syncthreads_or(tid < L && tot > cap);
  if (blockIdx.x == 0) {
    if (tid < L) { p.expert_offsets[tid] = first; p.actual_counts[tid] = tot; }
    if (tid == 0) {
      p.expert_offsets[L] = s.off[L];
      report(p.error_flag, over != 0);
    }
  }
  const int rows = (live + shares - 1) / shares, begin = min(live, share * rows), end = min(live, begin + rows);
  for (int i = begin * K + tid; i < end * K; i += kTileThreads) {
    const int r = i / K, k = i - r * K, e = s.id[i];
    int dst = -1;
    if ((s.valid[r] >> k) & 1u) {
      dst = s.base[e] + LocalTile::below(s.mask + e * stride, r);
      if (dst >= s.off[e + 1]) dst = -1;
    }
    p.mapping[(size_t)t0 * K + i] = dst;
  }
  cluster.sync();           // nobody reads another CTA's counts any more
}

// The plan of tables that do not fit a cluster's shared memory: three passes over tiles of 64 rows with grid barriers between them.
__global__ void __launch_bounds__(kExpandThreads) ep_expand_plan_grid_kernel(const __grid_constant__ ExpandParams p) {
  cg::grid_group grid = cg::this_grid();
  const int tiles = (p.R + kExpandTile - 1) / kExpandTile, L = p.L, K = p.K;
  __shared__ unsigned s_mask[kMaxExperts][2];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    int run = 0;
    for (int e = 0; e < L; ++e) { p.expert_offsets[e] = run; run += p.caps[e]; }
    p.expert_offsets[L] = run;
  }
  // ---- pass 1: rows per (tile, expert)
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    for (int i = threadIdx.x; i < L * 2; i += kExpandThreads) (&s_mask[0][0])[i] = 0u;
    __syncthreads();
    for (int i = threadIdx.x; i < kExpandTile * K; i += kExpandThreads) {
      const int r = tile * kExpandTile + i / K;
      if (r >= p.R) continue;
      const long long e = p.topk_idx[(size_t)r * K + i % K];
      if (e >= 0 && e < L) atomicOr(&s_mask[e][(i / K) >> 5], 1u << ((i / K) & 31));
    }
    __syncthreads();
    for (int e = threadIdx.x; e < L; e += kExpandThreads) p.tile_counts[(size_t)tile * L + e] = __popc(s_mask[e][0]) + __popc(s_mask[e][1]);
    __syncthreads();
  }
  __threadfence();
  grid.sync();
  // ---- pass 2: exclusive scan over the tiles, one thread per expert of the first block
  if (blockIdx.x == 0) {
    int over = 0;
    for (int e = threadIdx.x; e < L; e += kExpandThreads) {
      int run = 0;
      for (int t = 0; t < tiles; ++t) { const int c = p.tile_counts[(size_t)t * L + e]; p.tile_counts[(size_t)t * L + e] = run; run += c; }
      p.actual_counts[e] = run;
      over |= run > p.caps[e];
    }
    over = __syncthreads_or(over);
    if (threadIdx.x == 0) report(p.error_flag, over != 0);
  }
  __threadfence();
  grid.sync();
  // ---- pass 3: the mapping
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    for (int i = threadIdx.x; i < L * 2; i += kExpandThreads) (&s_mask[0][0])[i] = 0u;
    __syncthreads();
    for (int i = threadIdx.x; i < kExpandTile * K; i += kExpandThreads) {
      const int r = tile * kExpandTile + i / K;
      if (r >= p.R) continue;
      const long long e = p.topk_idx[(size_t)r * K + i % K];
      if (e >= 0 && e < L) atomicOr(&s_mask[e][(i / K) >> 5], 1u << ((i / K) & 31));
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kExpandTile * K; i += kExpandThreads) {
      const int rt = i / K, r = tile * kExpandTile + rt;
      if (r >= p.R) continue;
      const long long e = p.topk_idx[(size_t)r * K + i % K];
      int dst = -1;
      if (e >= 0 && e < L) {
        bool first = true;                 // a repeated id inside a row keeps its first slot only
        for (int k = 0; k < i % K; ++k) first = first && p.topk_idx[(size_t)r * K + k] != e;
        if (first) {
          const int below = rt < 32 ? __popc(s_mask[e][0] & ((1u << rt) - 1u)) : __popc(s_mask[e][0]) + __popc(s_mask[e][1] & ((1u << (rt - 32)) - 1u));
          const int pos = p.tile_counts[(size_t)tile * L + e] + below;
          if (pos < p.expert_offsets[e + 1] - p.expert_offsets[e]) dst = p.expert_offsets[e] + pos;
        }
      }
      p.mapping[(size_t)r * K + i % K] = dst;
    }
    __syncthreads();
  }
}

// One piece of a row per warp, to all the row's destinations; the first p.pad_blocks blocks zero the padding rows.
constexpr int kExpandUnroll = 4;       // 16-byte pieces per lane and item

__global__ void __launch_bounds__(kExpandThreads) ep_expand_copy_kernel(const __grid_constant__ ExpandParams p) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = kExpandThreads / 32, units = p.row_bytes / 16;
  if ((int)blockIdx.x < p.pad_blocks) {
    for_padding_rows(p.expert_offsets, p.actual_counts, p.L, p.N, warp * p.pad_blocks + blockIdx.x, p.pad_blocks * nwarps, [&](int row) {
      zero_row(p.out + (size_t)row * p.row_bytes, p.row_bytes, p.out_sf + (size_t)row * p.num_sf, p.num_sf, lane);
      if (p.out_w && lane == 0) p.out_w[row] = 0.f;
    });
    return;
  }
  const int item = ((int)blockIdx.x - p.pad_blocks) * nwarps + warp, r = item / p.pieces, piece = item - r * p.pieces;
  if (r >= p.R) return;
  const int per_piece = ((units + p.pieces - 1) / p.pieces + 31) / 32 * 32, u_begin = min(units, piece * per_piece);
  int row = lane < p.K ? __ldg(p.mapping + (size_t)r * p.K + lane) : -1;
  if (row >= p.N) row = -1;
  const unsigned mask = __ballot_sync(0xffffffffu, row >= 0);
  if (mask == 0) return;
  if (piece == 0) {
    if (p.out_w && row >= 0) p.out_w[row] = p.topk_w ? __ldg(p.topk_w + (size_t)r * p.K + lane) : 0.f;
    if (p.num_sf > 0)
      warp_fanout_f32<false>(p.x_sf + (size_t)r * p.num_sf, p.num_sf, reinterpret_cast<unsigned long long>(p.out_sf + (long long)row * p.num_sf),
                             mask, lane);
  }
  warp_fanout<false, kExpandUnroll>(reinterpret_cast<const int4*>(p.x + (size_t)r * p.row_bytes) + u_begin, min(units - u_begin, per_piece),
                                    reinterpret_cast<unsigned long long>(p.out + (long long)row * p.row_bytes) + (size_t)u_begin * 16, mask, lane);
}

long long expand_scratch(int R, int L, int K) {
  return LocalTile::bytes(LocalTile::tokens(R), L, K) <= kTileSmemLimit ? 0 : (long long)(R + kExpandTile - 1) / kExpandTile * L;
}

cudaError_t launch_expand(const ExpandParams& params, int blocks, cudaStream_t stream) {
  ExpandParams p = params;
  if (!p.cached) {
    constexpr int kSlots = kTileCtas * kTileThreads;
    cudaError_t e;
    if (expand_scratch(p.R, p.L, p.K) == 0) {
      const size_t smem = LocalTile::bytes(LocalTile::tokens(p.R), p.L, p.K);
      e = launch_tiles((const void*)ep_expand_plan_kernel, &p, std::max(1, std::min(4, (p.R * p.K + kSlots - 1) / kSlots)), smem, stream);
    } else {
      void* args[] = {&p};
      e = cudaLaunchCooperativeKernel((const void*)ep_expand_plan_grid_kernel, dim3(blocks), dim3(kExpandThreads), args, 0, stream);
    }
    if (e != cudaSuccess) return e;
  }
  const int units = p.row_bytes / 16, warps = kExpandThreads / 32;
  p.pieces = (units + 32 * kExpandUnroll - 1) / (32 * kExpandUnroll);
  p.pad_blocks = std::min(148, (p.N + warps - 1) / warps);
  const long long grid = p.pad_blocks + ((long long)p.R * p.pieces + warps - 1) / warps;
  if (grid == 0) return cudaSuccess;
  ep_expand_copy_kernel<<<(unsigned)grid, kExpandThreads, 0, stream>>>(p);
  return cudaGetLastError();
}

template <class T2> __device__ __forceinline__ float2 to_float2(uint32_t v);
template <> __device__ __forceinline__ float2 to_float2<__nv_bfloat162>(uint32_t v) { return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&v)); }
template <> __device__ __forceinline__ float2 to_float2<__half2>(uint32_t v) { return __half22float2(*reinterpret_cast<__half2*>(&v)); }
template <class T2> __device__ __forceinline__ uint32_t from_float2(float a, float b);
template <> __device__ __forceinline__ uint32_t from_float2<__nv_bfloat162>(float a, float b) { __nv_bfloat162 h = __floats2bfloat162_rn(a, b); return *reinterpret_cast<uint32_t*>(&h); }
template <> __device__ __forceinline__ uint32_t from_float2<__half2>(float a, float b) { __half2 h = __floats2half2_rn(a, b); return *reinterpret_cast<uint32_t*>(&h); }

constexpr int kAggregateRows = 3;      // rows in flight per lane; few registers, so that an SM holds all its warps

template <class T2>
__global__ void __launch_bounds__(kExpandThreads) ep_aggregate_kernel(const __grid_constant__ AggregateParams p) {
  const int lane = threadIdx.x & 31, units = p.H / 8, pieces = (units + 31) / 32;
  const long long item = (long long)blockIdx.x * (kExpandThreads / 32) + (threadIdx.x >> 5);
  const int r = (int)(item / pieces), u = (int)(item - (long long)r * pieces) * 32 + lane;
  if (r >= p.R) return;
  int row = lane < p.K ? __ldg(p.mapping + (size_t)r * p.K + lane) : -1;
  if (row >= p.N) row = -1;
  const unsigned mask = __ballot_sync(0xffffffffu, row >= 0);
  if (p.out_values && u == lane && lane < p.K) p.out_values[(size_t)r * p.K + lane] = row >= 0 && p.values ? __ldg(p.values + row) : 0.f;
  const float w = row >= 0 && p.row_w ? __ldg(p.row_w + row) : 1.f;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (unsigned m = mask; m;) {
    int4 v[kAggregateRows];
    float wq[kAggregateRows];
    const int n = __popc(m);
#pragma unroll
    for (int q = 0; q < kAggregateRows; ++q) {
      if (q < n) {
        const int k = __ffs(m) - 1;
        m &= m - 1;
        const int4* src = reinterpret_cast<const int4*>(p.x + (size_t)__shfl_sync(0xffffffffu, row, k) * p.H * 2);
        wq[q] = __shfl_sync(0xffffffffu, w, k);
        if (u < units) v[q] = __ldg(src + u);
      }
    }
#pragma unroll
    for (int q = 0; q < kAggregateRows; ++q) {
      if (q < n && u < units) {
        const uint32_t* h = reinterpret_cast<const uint32_t*>(&v[q]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {        // product and sum rounded separately (slot order)
          const float2 f = to_float2<T2>(h[j]);
          acc[2 * j] = __fadd_rn(acc[2 * j], __fmul_rn(wq[q], f.x));
          acc[2 * j + 1] = __fadd_rn(acc[2 * j + 1], __fmul_rn(wq[q], f.y));
        }
      }
    }
  }
  if (u < units)
    reinterpret_cast<int4*>(p.out + (size_t)r * p.H * 2)[u] =
        make_int4((int)from_float2<T2>(acc[0], acc[1]), (int)from_float2<T2>(acc[2], acc[3]), (int)from_float2<T2>(acc[4], acc[5]),
                  (int)from_float2<T2>(acc[6], acc[7]));
}

cudaError_t launch_aggregate(const AggregateParams& p, cudaStream_t stream) {
  const long long items = (long long)p.R * ((p.H / 8 + 31) / 32), per = kExpandThreads / 32;
  const unsigned grid = (unsigned)((items + per - 1) / per);
  if (p.is_half) ep_aggregate_kernel<__half2><<<grid, kExpandThreads, 0, stream>>>(p);
  else ep_aggregate_kernel<__nv_bfloat162><<<grid, kExpandThreads, 0, stream>>>(p);
  return cudaGetLastError();
}

}  // namespace dep
