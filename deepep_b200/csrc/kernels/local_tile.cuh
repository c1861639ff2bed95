// Counts and ranks of a routing table [T][K] by one cluster of CTAs: every CTA owns a range of tokens (whole 64-token tiles), keeps
// its ids and one bit per (expert, token) in shared memory, and learns the others' counts through distributed shared memory.  Used
// by the routing pass of a single rank and by the V1 expand operator.
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"

namespace dep {

constexpr int kTileThreads = 1024;
constexpr int kTileCtas = 16;              // largest cluster of this device class
constexpr unsigned kRepeated = 1u << 31;   // in LocalTile::valid: two slots of the token name one expert
constexpr size_t kTileSmemLimit = 200 << 10;

// Shared memory of a CTA that owns `per` tokens.
struct LocalTile {
  unsigned* mask;      // [E][stride]: tokens of the expert, `stride` odd so that a column of it meets all banks
  unsigned* hit;       // [per / 32]: tokens with at least one slot that counts
  int* cnt;            // [E + 1]: tokens per expert of this CTA, then tokens with a hit (read by the other CTAs)
  int* tot;            // [E] rows of the expert
  int* off;            // [E + 1] first row of the expert
  int* base;           // [E] first row of this CTA's tokens
  unsigned* valid;     // [per] bit k: slot k counts (its id is in range and no earlier slot of the token has the same)
  short* id;           // [per][K], -1: no expert
  __host__ __device__ static int tokens(int T) {          // per CTA: whole tiles
    const int tiles = (T + kChunkTokens - 1) / kChunkTokens;
    return (tiles > kTileCtas ? (tiles + kTileCtas - 1) / kTileCtas : 1) * kChunkTokens;
  }
  __host__ __device__ static int stride(int per) { return per / 32 | 1; }
  __host__ __device__ static size_t bytes(int per, int E, int K) {
    return 4 * ((size_t)E * stride(per) + per / 32 + 4 * E + 2 + per) + 2 * (size_t)per * K;
  }
#ifdef __CUDACC__
  __device__ LocalTile(void* smem, int per, int E) {
    mask = reinterpret_cast<unsigned*>(smem);
    hit = mask + (size_t)E * stride(per);
    cnt = reinterpret_cast<int*>(hit + per / 32);
    tot = cnt + E + 1; off = tot + E; base = off + E + 1;
    valid = reinterpret_cast<unsigned*>(base + E);
    id = reinterpret_cast<short*>(valid + per);
  }

  // Bits of m below bit t.
  static __device__ __forceinline__ int below(const unsigned* m, int t) {
    int n = 0;
    for (int w = 0; w < t >> 5; ++w) n += __popc(m[w]);
    return n + ((t & 31) ? __popc(m[t >> 5] & ((1u << (t & 31)) - 1u)) : 0);
  }

  // Ids, masks, valid slots and counts of the `n` slots at `table`.  The caller's cluster barrier follows.
  __device__ void count(const long long* table, int n, int per, int K, int E) const {
    const int tid = threadIdx.x, words = per / 32, st = stride(per);
    for (int i0 = tid; i0 < n; i0 += kTileThreads * 4) {
      long long v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = i0 + j * kTileThreads < n ? __ldg(table + i0 + j * kTileThreads) : -1;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (i0 + j * kTileThreads < n) id[i0 + j * kTileThreads] = (short)((v[j] < 0 || v[j] >= E) ? -1 : (int)v[j]);
    }
    for (int i = tid; i < E * st; i += kTileThreads) mask[i] = 0u;
    for (int i = tid; i < per; i += kTileThreads) valid[i] = 0u;
    __syncthreads();
    for (int i = tid; i < n; i += kTileThreads) {
      const int tl = i / K, k = i - tl * K, e = id[i];
      if (e < 0) continue;
      const unsigned bit = 1u << (tl & 31);
      const bool again = atomicOr(&mask[e * st + (tl >> 5)], bit) & bit;
      atomicOr(&valid[tl], 1u << k | (again ? kRepeated : 0u));
    }
    __syncthreads();
    for (int i = tid; i < per; i += kTileThreads) {                 // per is a multiple of 64: whole warps
      unsigned v = valid[i];
      if (v & kRepeated) {                                          // only the first of a token's slots with one expert counts
        v &= ~kRepeated;
        for (int k = 1; k < K; ++k)
          for (int j = 0; j < k; ++j)
            if (id[i * K + j] == id[i * K + k]) v &= ~(1u << k);
        valid[i] = v;
      }
      const unsigned word = __ballot_sync(0xffffffffu, v != 0u);
      if ((tid & 31) == 0) hit[i >> 5] = word;
    }
    for (int e = tid; e < E; e += kTileThreads) {
      int v = 0;
      for (int w = 0; w < words; ++w) v += __popc(mask[e * st + w]);
      cnt[e] = v;
    }
    __syncthreads();
    if (tid == 0) {
      int v = 0;
      for (int w = 0; w < words; ++w) v += __popc(hit[w]);
      cnt[E] = v;
    }
  }

  // Thread e < E: the tokens of expert e in the CTAs before CTA c, and in all.  hits: the same for tokens with a hit (valid after the
  // next block barrier).
  template <class Cluster>
  __device__ void gather(Cluster& cluster, int c, int E, int hits[2], int& before, int& tot) const {
    const int tid = threadIdx.x, lane = tid & 31;
    before = tot = 0;
    if (tid < E) {
      int v[kTileCtas];
#pragma unroll
      for (int r = 0; r < kTileCtas; ++r) v[r] = cluster.map_shared_rank(cnt, r)[tid];
#pragma unroll
      for (int r = 0; r < kTileCtas; ++r) {
        if (r < c) before += v[r];
        tot += v[r];
      }
    }
    if (tid >= kTileThreads - 32) {
      int v = lane < kTileCtas ? cluster.map_shared_rank(cnt, lane)[E] : 0, b = lane < c ? v : 0;
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) { b += __shfl_xor_sync(0xffffffffu, b, d); v += __shfl_xor_sync(0xffffffffu, v, d); }
      if (lane == 0) { hits[0] = b; hits[1] = v; }
    }
  }
#endif
};

#ifdef __CUDACC__
// Sum of `v` over the threads before this one of a block of kTileThreads; s_warp: one int per warp.
__device__ __forceinline__ int tile_prefix(int v, int* s_warp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += o;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  int warps = lane < warp ? s_warp[lane] : 0;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) warps += __shfl_xor_sync(0xffffffffu, warps, d);
  return warps + incl - v;
}
#endif

// Launches `clusters` clusters of kTileCtas CTAs of `fn`, whose only argument is *params.
inline cudaError_t launch_tiles(const void* fn, const void* params, int clusters, size_t smem, cudaStream_t stream) {
  // attributes belong to the current device, so they are set on every launch (a process may drive several GPUs)
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess && smem > 48 * 1024) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kTileCtas * clusters); cfg.blockDim = dim3(kTileThreads); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = kTileCtas; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  void* args[] = {const_cast<void*>(params)};
  return cudaLaunchKernelExC(&cfg, fn, args);
}

}  // namespace dep
