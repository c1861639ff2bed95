// ep_layout: the routing summary of upstream DeepEP's V1 `get_dispatch_layout`.
//
// From topk_idx [T, K] (int64, < 0 or >= E marks an empty slot): tokens per destination rank, tokens per expert,
// and is_token_in_rank [T, P].  One thread per token; every block counts in shared memory.  Integer sums: the result does not depend on
// the order of arrival.  A short table is counted by one cluster, whose CTAs add their counts up through distributed shared memory, in
// a single launch.  A long one wants the shared-memory atomics of more than 16 SMs, and more experts cost a cluster's sums more: a grid
// adds its counts to outputs that a kernel of one block clears (1 us; two fills take 2 us each).
// us in a graph and, in brackets, of an eager call until the device is idle, cluster / clear and grid: 1 token, top-2 of 8, 3.4 / 3.7
// (26 / 32); 2048 tokens, top-6 of 64, 4.3 / 4.5, top-8 of 256 5.1 / 5.0 (19.0 / 20.2), top-16 of 1024 8.0 / 6.8 (21.7 / 22.0); 4096, top-8
// of 256, 5.5 / 4.9 (19.4 / 20.2), 16384 7.1 / 4.9 (21.0 / 20.1), 60000 14.1 / 6.7; 16384, top-16 of 1024, 15.3 / 7.1.
// Counterpart of the reference's dispatch_layout_kernel (csrc/direct/kernels/dispatch/dispatch_layout.cpp:35),
// which builds the same three outputs from per-core partial counts.
#include <algorithm>

#include "api.h"
#include "local_tile.cuh"

namespace cg = cooperative_groups;

namespace dep {

constexpr int kLayoutThreads = 256;                                   // of a block of the grid
constexpr int kLayoutClusterTokens = 2048, kLayoutClusterExperts = 512;

struct LayoutParams {
  const long long* topk_idx;
  int T, K, E, P;
  int* tokens_per_rank;        // [P]
  int* tokens_per_expert;      // [E]
  bool* is_token_in_rank;      // [T][P]
};

struct LayoutCounts { int expert[kMaxExperts], rank[kMaxRanks]; };    // of a block, in shared memory

// Tokens first, first + stride, ... of this thread, into counts that the block clears first.
__device__ __forceinline__ void count_tokens(const LayoutParams& p, LayoutCounts& s, int first, int stride) {
  for (int e = threadIdx.x; e < p.E; e += (int)blockDim.x) s.expert[e] = 0;
  if (threadIdx.x < kMaxRanks) s.rank[threadIdx.x] = 0;
  __syncthreads();
  const int Lx = p.E / p.P;
  for (int t = first; t < p.T; t += stride) {
    unsigned rank_mask = 0;
    for (int k = 0; k < p.K; ++k) {
      const long long e = __ldg(p.topk_idx + (size_t)t * p.K + k);
      if (e < 0 || e >= p.E) continue;
      atomicAdd(&s.expert[(int)e], 1);              // per-expert counts include every valid slot, as upstream counts them
      rank_mask |= 1u << ((int)e / Lx);
    }
    for (int r = 0; r < p.P; ++r) {
      const bool in = (rank_mask >> r) & 1u;
      p.is_token_in_rank[(size_t)t * p.P + r] = in;
      if (in) atomicAdd(&s.rank[r], 1);
    }
  }
}

__global__ void __launch_bounds__(kTileThreads) ep_layout_cluster_kernel(const __grid_constant__ LayoutParams p) {
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ LayoutCounts s;
  const int tid = threadIdx.x, c = blockIdx.x;
  count_tokens(p, s, ((tid >> 5) * kTileCtas + c) * 32 + (tid & 31), kTileCtas * kTileThreads);      // the CTAs take warps of tokens in turn
  cluster.sync();
  auto sum = [&](int* mine, int i) {
    int v = 0;
#pragma unroll
    for (int r = 0; r < kTileCtas; ++r) v += cluster.map_shared_rank(mine, r)[i];
    return v;
  };
  for (int e = c + tid * kTileCtas; e < p.E; e += kTileCtas * kTileThreads) p.tokens_per_expert[e] = sum(s.expert, e);
  if (c == 0 && tid < p.P) p.tokens_per_rank[tid] = sum(s.rank, tid);
  cluster.sync();                                   // nobody reads another CTA's counts any more
}

__global__ void __launch_bounds__(kMaxExperts) ep_layout_clear_kernel(const __grid_constant__ LayoutParams p) {
  if ((int)threadIdx.x < p.E) p.tokens_per_expert[threadIdx.x] = 0;
  if ((int)threadIdx.x < p.P) p.tokens_per_rank[threadIdx.x] = 0;
}

__global__ void __launch_bounds__(kLayoutThreads) ep_layout_kernel(const __grid_constant__ LayoutParams p) {
  __shared__ LayoutCounts s;
  count_tokens(p, s, blockIdx.x * kLayoutThreads + threadIdx.x, gridDim.x * kLayoutThreads);
  __syncthreads();
  for (int e = threadIdx.x; e < p.E; e += kLayoutThreads)
    if (s.expert[e]) atomicAdd(&p.tokens_per_expert[e], s.expert[e]);
  if ((int)threadIdx.x < p.P && s.rank[threadIdx.x]) atomicAdd(&p.tokens_per_rank[threadIdx.x], s.rank[threadIdx.x]);
}

// All outputs are fully written.
cudaError_t launch_layout(const long long* topk_idx, int T, int K, int E, int P, int* tokens_per_rank, int* tokens_per_expert,
                          bool* is_token_in_rank, cudaStream_t stream) {
  if (T < 0 || K < 1 || K > kMaxTopk || E < P || E > kMaxExperts || E % P || P < 1 || P > kMaxRanks) return cudaErrorInvalidValue;
  const LayoutParams p = {topk_idx, T, K, E, P, tokens_per_rank, tokens_per_expert, is_token_in_rank};
  if (T <= kLayoutClusterTokens && E <= kLayoutClusterExperts) return launch_tiles((const void*)ep_layout_cluster_kernel, &p, 1, 0, stream);
  ep_layout_clear_kernel<<<1, std::max(E, P), 0, stream>>>(p);
  if (T > 0)
    ep_layout_kernel<<<std::min(148, (T + kLayoutThreads - 1) / kLayoutThreads), kLayoutThreads, 0, stream>>>(p);
  return cudaGetLastError();
}

}  // namespace dep
