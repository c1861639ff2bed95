// Stand-alone launches of the MegaMoE routing/pull and finishing phases (see mega_route.cuh), the copy of a call's inputs, and the
// final reduction of a single rank.
#include "mega_route.cuh"

namespace dep {

constexpr int kRouteThreads = 256;

long long mega_input_bytes(int M, int H, int K) { return mega_input_layout(M, H, K).total; }
void mega_input_offsets(int M, int H, int K, long long* out) {
  MegaInput l = mega_input_layout(M, H, K);
  out[0] = l.hdr; out[1] = l.x; out[2] = l.x_sf; out[3] = l.idx; out[4] = l.w; out[5] = l.total;
}

// Bound by its launch for decode batches (4096 tokens of 7168: 60 MB); as separate copies and conversions it was five launches.
__global__ void __launch_bounds__(kRouteThreads) mega_load_kernel(const __grid_constant__ MegaLoadArgs a) {
  const long long i = (long long)blockIdx.x * kRouteThreads + threadIdx.x, n = (long long)a.T * a.H, slots = (long long)a.T * a.K;
  if (a.x && i < n / 16) a.x_to[i] = __ldg(a.x + i);
  if (a.x && i < n / 256) a.sf_to[i] = __ldg(a.sf + i);
  if (i < slots) {
    a.idx_to[i] = a.idx64 ? (int)__ldg(reinterpret_cast<const long long*>(a.idx) + i) : __ldg(reinterpret_cast<const int*>(a.idx) + i);
    a.w_to[i] = __ldg(a.w + i);
  }
}

cudaError_t launch_mega_load(const MegaLoadArgs& a, cudaStream_t stream) {
  const long long n = a.x ? (long long)a.T * a.H / 16 : 0, slots = (long long)a.T * a.K, threads = n > slots ? n : slots;
  if (threads == 0) return cudaSuccess;
  mega_load_kernel<<<(unsigned)((threads + kRouteThreads - 1) / kRouteThreads), kRouteThreads, 0, stream>>>(a);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(kRouteThreads) mega_route_kernel(const __grid_constant__ MegaRouteParams p) {
  cg::grid_group grid = cg::this_grid();
  route_phase(p.r[blockIdx.y], grid);
}

cudaError_t launch_mega_route(const MegaRouteParams& p, int nranks, int blocks, cudaStream_t stream) {
  dim3 grid(blocks, nranks), block(kRouteThreads);
  void* args[] = {const_cast<MegaRouteParams*>(&p)};
  return cudaLaunchCooperativeKernel((const void*)mega_route_kernel, grid, block, args, 0, stream);
}

__global__ void __launch_bounds__(kRouteThreads) mega_finish_kernel(const __grid_constant__ MegaFinishParams p) {
  finish_phase(p.r[blockIdx.y], true);
}

cudaError_t launch_mega_finish(const MegaFinishParams& p, int nranks, int blocks, cudaStream_t stream) {
  dim3 grid(blocks, nranks), block(kRouteThreads);
  void* args[] = {const_cast<MegaFinishParams*>(&p)};
  return cudaLaunchCooperativeKernel((const void*)mega_finish_kernel, grid, block, args, 0, stream);
}

// One span of 32 16-byte pieces of a token per warp, three slots in flight: the loads of 2048 threads an SM instead of the layer's
// 384, and a kernel's end instead of a grid barrier before it.  Inside the layer's kernel the barrier took 4.5 us and the reduction
// 5 to 10 (4096 tokens of 7168: 113).  32 experts, top-8, intermediate 2048, the layer in captured graphs, us inside / behind: 1 token
// 82.3 / 76.4, 8 149.7 / 144.8, 64 158.4 / 155.4, 128 173.0 / 166.8, 512 267 / 258.  This kernel by itself, 4096 tokens of 7168, 8 slots:
// 88 us, 6.0 TB/s (memory); with the 40 registers that the compiler takes unasked, 1536 threads an SM, 92.
constexpr int kReduceThreads = 256, kReduceSlots = 3;
__global__ void __launch_bounds__(kReduceThreads, 8) mega_reduce_kernel(const __grid_constant__ MegaFinishArgs a) {
  const int K = a.K, Kp = K + a.S, units = a.H / 8, spans = (units + 31) / 32, lane = threadIdx.x & 31;
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) ++control_of(a.ctx.ws[0])->epoch[kOpMega];
    if (a.stats)
      for (int l = threadIdx.x; l < a.E; l += kReduceThreads) a.stats[l] = (a.stats_set ? 0 : a.stats[l]) + __ldg(a.expert_rows + l);
  }
  if (a.ready && blockIdx.x == gridDim.x - 1) {
    for (int i = threadIdx.x; i < a.max_mtiles; i += kReduceThreads) a.ready[i] = a.pulled[i] = 0;
    if (threadIdx.x == 0 && a.tile_counter) *a.tile_counter = 0;
  }
  const int item = blockIdx.x * (kReduceThreads / 32) + (threadIdx.x >> 5), t = item / spans;
  if (t >= a.T) return;
  const int u = (item - t * spans) * 32 + lane;
  const MegaInput in = mega_input_layout(a.max_tokens, a.H, K);
  // lane k holds slot k: its weight and whether it counts (shared experts: every token, weight one)
  int e = -1;
  float weight = 1.f;
  if (lane < K) {
    e = __ldg(reinterpret_cast<const int*>(a.ctx.ws[0] + a.in_off + in.idx) + (size_t)t * K + lane);
    weight = __ldg(reinterpret_cast<const float*>(a.ctx.ws[0] + a.in_off + in.w) + (size_t)t * K + lane);
  }
  const int4* rows = reinterpret_cast<const int4*>(a.ctx.ws[0] + a.comb_off) + (size_t)t * Kp * units + min(u, units - 1);
  float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (unsigned m = __ballot_sync(0xffffffffu, lane < K ? e >= 0 && e < a.E : lane < Kp); m;) {
    int4 v[kReduceSlots];
    unsigned taken = m;
#pragma unroll
    for (int q = 0; q < kReduceSlots; ++q) {
      if (m) v[q] = __ldg(rows + (__ffs(m) - 1) * units);
      m &= m - 1;
    }
#pragma unroll
    for (int q = 0; q < kReduceSlots; ++q) {
      if (taken) {
        const float w = __shfl_sync(0xffffffffu, weight, __ffs(taken) - 1);
        taken &= taken - 1;
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v[q]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {   // product and sum rounded separately, as the CPU oracle does
          sum[2 * i] = __fadd_rn(sum[2 * i], __fmul_rn(w, __low2float(h[i])));
          sum[2 * i + 1] = __fadd_rn(sum[2 * i + 1], __fmul_rn(w, __high2float(h[i])));
        }
      }
    }
  }
  if (u >= units) return;
  int4 o;
  __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
  for (int i = 0; i < 4; ++i) oh[i] = __floats2bfloat162_rn(sum[2 * i], sum[2 * i + 1]);
  reinterpret_cast<int4*>(a.y)[(size_t)t * units + u] = o;
}

cudaError_t launch_mega_reduce(const MegaFinishArgs& a, cudaStream_t stream) {
  const long long warps = (long long)a.T * ((a.H / 8 + 31) / 32), blocks = (warps * 32 + kReduceThreads - 1) / kReduceThreads;
  mega_reduce_kernel<<<(unsigned)(blocks > 0 ? blocks : 1), kReduceThreads, 0, stream>>>(a);
  return cudaGetLastError();
}

}  // namespace dep
