// ep_layout: the routing summary of upstream DeepEP's V1 `get_dispatch_layout`.
//
// From topk_idx [T, K] (int64, < 0 or >= E marks an empty slot): tokens per destination rank, tokens per expert,
// and is_token_in_rank [T, P].  One thread per token; the CTAs of one cluster count in shared memory and add their counts up through
// distributed shared memory, so that nothing has to be cleared before the launch (the kernel takes 3 us either way; two fills of 1 us
// and their launches are gone).
// Counterpart of the reference's dispatch_layout_kernel (csrc/direct/kernels/dispatch/dispatch_layout.cpp:35),
// which builds the same three outputs from per-core partial counts.
#include "api.h"
#include "local_tile.cuh"

namespace cg = cooperative_groups;

namespace dep {

struct LayoutParams {
  const long long* topk_idx;
  int T, K, E, P;
  int* tokens_per_rank;        // [P]
  int* tokens_per_expert;      // [E]
  bool* is_token_in_rank;      // [T][P]
};

__global__ void __launch_bounds__(kTileThreads) ep_layout_kernel(const __grid_constant__ LayoutParams p) {
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ int s_expert[kMaxExperts];
  __shared__ int s_rank[kMaxRanks];
  const int tid = threadIdx.x, c = blockIdx.x, Lx = p.E / p.P;
  for (int e = tid; e < p.E; e += kTileThreads) s_expert[e] = 0;
  if (tid < kMaxRanks) s_rank[tid] = 0;
  __syncthreads();
  for (int t = c * kTileThreads + tid; t < p.T; t += kTileCtas * kTileThreads) {
    unsigned rank_mask = 0;
    for (int k = 0; k < p.K; ++k) {
      const long long e = __ldg(p.topk_idx + (size_t)t * p.K + k);
      if (e < 0 || e >= p.E) continue;
      atomicAdd(&s_expert[(int)e], 1);              // per-expert counts include every valid slot, as upstream counts them
      rank_mask |= 1u << ((int)e / Lx);
    }
    for (int r = 0; r < p.P; ++r) {
      const bool in = (rank_mask >> r) & 1u;
      p.is_token_in_rank[(size_t)t * p.P + r] = in;
      if (in) atomicAdd(&s_rank[r], 1);
    }
  }
  cluster.sync();
  auto sum = [&](int* mine, int i) {
    int v = 0;
#pragma unroll
    for (int r = 0; r < kTileCtas; ++r) v += cluster.map_shared_rank(mine, r)[i];
    return v;
  };
  for (int e = c + tid * kTileCtas; e < p.E; e += kTileCtas * kTileThreads) p.tokens_per_expert[e] = sum(s_expert, e);
  if (c == 0 && tid < p.P) p.tokens_per_rank[tid] = sum(s_rank, tid);
  cluster.sync();                                   // nobody reads another CTA's counts any more
}

// All outputs are fully written.
cudaError_t launch_layout(const long long* topk_idx, int T, int K, int E, int P, int* tokens_per_rank, int* tokens_per_expert,
                          bool* is_token_in_rank, cudaStream_t stream) {
  if (T < 0 || K < 1 || K > kMaxTopk || E < P || E > kMaxExperts || E % P || P < 1 || P > kMaxRanks) return cudaErrorInvalidValue;
  const LayoutParams p = {topk_idx, T, K, E, P, tokens_per_rank, tokens_per_expert, is_token_in_rank};
  return launch_tiles((const void*)ep_layout_kernel, &p, 1, 0, stream);
}

}  // namespace dep
