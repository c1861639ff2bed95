// ep_dispatch_ll / ep_combine_ll: latency-oriented dispatch and combine for decode batches
// (at most 256 tokens per rank).
//
// One kernel per direction and no separate layout pass.  Dispatch: every rank pushes its tiny
// routing table ([T, K] expert ids and weights) to all peers (one block per peer, 16-byte stores)
// and, at the same time, pushes each token row once per destination GPU into a fixed staging slot
// there, as four column parts that different warps carry, each followed by its own release flag.
// A receiver derives the expert-major layout (sorted by local expert, source rank, source token,
// slot) from the gathered tables with bit masks and popcounts in shared memory, then polls the
// part flags and writes every output row.  Combine returns each expert row, again part by part, to
// a fixed (token, slot) slot at its source; the source waits per part and computes
// sum_k w_k * row_k in slot order in fp32.
//
// What stays on the rank takes neither detour: its tokens are routed from the caller's table, its rows go
// from the caller's tensor straight into the output rows (quantised on the way, cut into as many pieces as
// there are warps), and the combine reads the rows of its own experts where they lie, through the row of
// every (token, slot) that the dispatch leaves behind.  A single rank, where that is all there is, has kernels of
// its own (the *_local kernels).  What bounds all of them is the launch and the chain of dependent steps, not
// bytes: on one GPU a captured round (hidden 7168, 256 experts, top-8, fp8) took 34.8 us for one token while own
// rows went through flags and the staging area and one thread scanned the experts, 18.4 us in the kernels for
// several ranks, 9.6 us in those for one; 93 bf16 tokens of 4096 (64 experts, top-6) 41.3, 20.5 and 10.3 us.
//
// Re-entrancy: epochs live in device memory and select one of two banks, flags hold epochs and
// are never cleared, a bank is reused only after the peers acknowledged the call before last.
// Nothing depends on host state, so both kernels can be captured in a CUDA graph.
//
// Parity: csrc/kernels/dispatch/low_latency/dispatch_server_dedup_kernel.h:37-58 and
// csrc/kernels/combine/low_latency/combine_server_dedup_kernel.h:102-127 of the reference
// (count exchange, cumsum, flagged packets, ping-pong banks; weights applied at the source).
#include <cooperative_groups.h>

#include "ll_api.h"

namespace dep {

constexpr int kLLThreads = 512;
constexpr int kLLLocalThreads = 128; // combine of one rank
constexpr int kLLSendWarps = 8;      // dispatch: warps that push rows; the other warps of the block derive the layout meanwhile
constexpr int kLLMaxTokens = 256;
constexpr int kLLWords = kLLMaxTokens / 32;  // a token set as 32-bit masks

// A row travels as kLLParts column parts, each with its own flag, so that a row is spread over several warps on both
// sides.  Parts are whole groups of 128 values (the granularity of the fp8 scales): part p covers values [v0, v1).
struct LLPart { int v0, v1, b0, b1; };
__device__ __forceinline__ LLPart ll_part(int H, int p) {
  const int nblk = (H + 127) / 128, bpp = (nblk + kLLParts - 1) / kLLParts;
  LLPart r;
  r.b0 = min(nblk, p * bpp); r.b1 = min(nblk, (p + 1) * bpp);
  r.v0 = min(H, r.b0 * 128); r.v1 = min(H, r.b1 * 128);
  return r;
}

// Flags of finished parts are published together: lane i of the warp keeps the address of the i-th pending flag.
struct PendingFlags {
  unsigned long long* mine = nullptr;
  int count = 0;
  __device__ __forceinline__ void add(unsigned long long* flag, unsigned long long epoch, int lane) {
    if (count == 32) publish(epoch, lane);
    if (lane == count) mine = flag;
    ++count;
  }
  // every lane's stores are ordered before the flags by the warp barrier + release
  __device__ __forceinline__ void publish(unsigned long long epoch, int lane) {
    __syncwarp();
    if (lane < count) st_release_sys(mine, epoch);
    count = 0;
  }
};

__device__ __forceinline__ int below8(const unsigned* m, int t) {
  int n = 0;
  const int w = t >> 5;
  for (int i = 0; i < w; ++i) n += __popc(m[i]);
  return n + __popc(m[w] & ((1u << (t & 31)) - 1u));
}
__device__ __forceinline__ bool counts_ll(const int* row, int k, int E) {
  int e = row[k];
  if (e < 0 || e >= E) return false;
  for (int j = 0; j < k; ++j)
    if (row[j] == e) return false;
  return true;
}

// ------------------------------------------------------------------------------------------ dispatch
// One 16-byte piece (8 bf16 values) -> 8 e4m3 codes and the fp32 scale of its group of 128 values, which 16 consecutive
// lanes hold together (a step of a warp covers two groups).  Lanes past the end pass zeros.
__device__ __forceinline__ uint2 quant8(const int4& v, float& scale) {
  float f[8];
  const __nv_bfloat162* hh = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int q = 0; q < 4; ++q) { f[2 * q] = __low2float(hh[q]); f[2 * q + 1] = __high2float(hh[q]); }
  float amax = 0.f;
#pragma unroll
  for (int q = 0; q < 8; ++q) amax = fmaxf(amax, fabsf(f[q]));
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  amax = fmaxf(amax, 1e-4f);
  const float inv = __frcp_rn(amax) * 448.0f;   // torch evaluates `448 / amax` (scalar / tensor) as reciprocal, then multiply
  uint32_t q2[2] = {0u, 0u};
#pragma unroll
  for (int q = 0; q < 8; ++q)
    q2[q >> 2] |= (uint32_t)__nv_cvt_float_to_fp8(f[q] * inv, __NV_SATFINITE, __NV_E4M3) << (8 * (q & 3));
  scale = amax / 448.0f;
  return make_uint2(q2[0], q2[1]);
}

// Column range of piece `p` of `n` equal pieces of a row, in groups of 128 values (the last group may be short).
__device__ __forceinline__ LLPart ll_piece(int H, int p, int n) {
  const int nblk = (H + 127) / 128, bpp = (nblk + n - 1) / n;
  LLPart r;
  r.b0 = min(nblk, p * bpp); r.b1 = min(nblk, (p + 1) * bpp);
  r.v0 = min(H, r.b0 * 128); r.v1 = min(H, r.b1 * 128);
  return r;
}

constexpr int kOwnUnroll = 4;   // 16-byte pieces per lane of an own row that are read ahead of the layout

// One piece of token t of the caller's tensor, quantised on the way in mode 2, into the output rows of its slots: lane l of
// `live` holds an output row.  `ahead`: the piece's first loads, when they were issued earlier.
__device__ __forceinline__ void write_own_piece(const LLDispatchArgs& a, uint8_t* recv_x, int t, const LLPart& pr, int row, unsigned live,
                                                int H, int nsf, int row_bytes, int src_bytes, const int4* ahead, int lane) {
  const int4* src = reinterpret_cast<const int4*>(reinterpret_cast<const uint8_t*>(a.x) + (size_t)t * src_bytes);
  const int lo = (a.mode == 1 ? pr.v0 : pr.v0 * 2) / 16, hi = (a.mode == 1 ? pr.v1 : pr.v1 * 2) / 16;
  for (int u0 = lo; u0 < hi; u0 += 32 * kOwnUnroll) {
    int4 v[kOwnUnroll];
#pragma unroll
    for (int i = 0; i < kOwnUnroll; ++i) {
      const int u = u0 + i * 32 + lane;
      if (ahead && u0 == lo) v[i] = ahead[i];
      else v[i] = u < hi ? __ldg(src + u) : make_int4(0, 0, 0, 0);
    }
#pragma unroll
    for (int i = 0; i < kOwnUnroll; ++i) {
      const int u = u0 + i * 32 + lane;
      if (u0 + i * 32 >= hi) break;               // warp-uniform
      if (a.mode == 2) {
        float scale;
        const uint2 q = quant8(v[i], scale);
        for (unsigned m = live; m; m &= m - 1) {
          const size_t o = __shfl_sync(0xffffffffu, row, __ffs(m) - 1);
          if (u < hi) {
            *reinterpret_cast<uint2*>(recv_x + o * H + (size_t)u * 8) = q;
            if ((lane & 15) == 0) a.recv_sf[o * nsf + u / 16] = scale;
          }
        }
      } else {
        for (unsigned m = live; m; m &= m - 1) {
          const size_t o = __shfl_sync(0xffffffffu, row, __ffs(m) - 1);
          if (u < hi) reinterpret_cast<int4*>(recv_x + o * row_bytes)[u] = v[i];
        }
      }
    }
  }
  if (a.mode == 1)
    for (int b = pr.b0; b < pr.b1; b += 32) {
      const float sf = b + lane < pr.b1 ? __ldg(a.x_sf + (size_t)t * nsf + b + lane) : 0.f;
      for (unsigned m = live; m; m &= m - 1) {
        const size_t o = __shfl_sync(0xffffffffu, row, __ffs(m) - 1);
        if (b + lane < pr.b1) a.recv_sf[o * nsf + b + lane] = sf;
      }
    }
}

template <bool kProfile>
__global__ void __launch_bounds__(kLLThreads) ep_dispatch_ll_kernel(const __grid_constant__ LLDispatchParams p) {
  const LLDispatchArgs& a = p.r[blockIdx.y];
  const WsLayout& lay = p.lay;
  const RankCtx& ctx = a.ctx;
  const int P = ctx.world, me = ctx.rank, M = lay.max_tokens, K = lay.topk, H = lay.hidden, E = a.E, Lx = E / P;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = kLLThreads / 32;
  // consecutive work items go to different SMs, so a short list of items spreads over the whole GPU
  const int gw = warp * gridDim.x + blockIdx.x, total_warps = gridDim.x * nwarps;
  Control* ctl = control_of(ctx.ws[me]);
  const unsigned long long epoch = ctl->epoch[kOpLLDispatch] + 1;
  const LLLayout ll = make_ll_layout(P, M, K, H);
  const long long bank_off = lay.ll + (long long)(epoch & 1) * ll.bank_bytes;
  const bool fp8 = a.mode != 0;
  const int nsf = H / 128, row_bytes = fp8 ? H : H * 2, src_bytes = a.mode == 1 ? H : H * 2;

  __shared__ unsigned s_emask[kMaxExperts][kLLWords];   // [(source, local expert)] -> tokens
  __shared__ unsigned s_hit[kMaxRanks][kLLWords];       // tokens of source r that reach this rank
  __shared__ unsigned s_own[kMaxRanks][kLLWords];       // my tokens that reach rank d
  __shared__ int s_off[kMaxExperts];                    // first output row of (source, local expert)
  __shared__ int s_warp_rows[kLLThreads / 32];          // rows of the experts that each layout warp scans
  __shared__ int s_T[kMaxRanks];
  __shared__ int s_fail;                                // a wait of the layout warps ran out

  // profile instantiation only: phase stamps (nanoseconds since kernel start) of block 0 in Control::dbg[0..7]; the
  // first thread of the sending warps and the first thread of the layout warps stamp their own phases
  unsigned long long t_start = 0;
  if constexpr (kProfile) t_start = global_timer_ns();
  auto stamp = [&](int i, int who = 0) {
    if constexpr (kProfile)
      if (blockIdx.x == 0 && (int)threadIdx.x == who) ctl->dbg[i] = global_timer_ns() - t_start;
  };
  constexpr int kLayoutFirst = kLLSendWarps * 32, LT = kLLThreads - kLayoutFirst;   // the layout warps and their thread count
  const int lt = (int)threadIdx.x - kLayoutFirst;
  auto layout_sync = [&]() { asm volatile("bar.sync 1, %0;" ::"n"(LT) : "memory"); };
  if (threadIdx.x == 0) s_fail = 0;

  // ---- everything that needs no peer starts at once: this warp's first piece of an own row is read ahead, the masks are cleared
  const int nblk = (H + 127) / 128;
  const int pieces = max(1, min(nblk, total_warps / max(a.T, 1)));      // pieces of an own row
  int4 ahead[kOwnUnroll];
  LLPart own_pr = {0, 0, 0, 0};
  if (gw < a.T * pieces) {
    own_pr = ll_piece(H, gw % pieces, pieces);
    const int lo = (a.mode == 1 ? own_pr.v0 : own_pr.v0 * 2) / 16, hi = (a.mode == 1 ? own_pr.v1 : own_pr.v1 * 2) / 16;
    const int4* src = reinterpret_cast<const int4*>(reinterpret_cast<const uint8_t*>(a.x) + (size_t)(gw / pieces) * src_bytes);
#pragma unroll
    for (int i = 0; i < kOwnUnroll; ++i) {
      const int u = lo + i * 32 + lane;
      ahead[i] = u < hi ? __ldg(src + u) : make_int4(0, 0, 0, 0);
    }
  }
  for (int i = threadIdx.x; i < E * kLLWords; i += kLLThreads) (&s_emask[0][0])[i] = 0u;
  for (int i = threadIdx.x; i < kMaxRanks * kLLWords; i += kLLThreads) { (&s_own[0][0])[i] = 0u; (&s_hit[0][0])[i] = 0u; }
  // ---- bank reuse: the call before last must have been consumed by the peers (this rank's own calls are ordered)
  int ok = 1;
  if (threadIdx.x < P && threadIdx.x != me && epoch > 2)
    ok = wait_flag_ge(&ctl->ll_disp_ack[threadIdx.x], epoch - 2, ctx, kOpLLDispatch, 0, threadIdx.x);
  int alive = __syncthreads_and(ok);

  // ---- my own routing: which ranks does each token reach, and which experts of this rank
  for (int t = threadIdx.x; t < a.T; t += kLLThreads) {   // one thread per token: K independent loads, dedup in registers
    int row[kMaxTopk];
#pragma unroll
    for (int k = 0; k < kMaxTopk; ++k) {
      long long v = k < K ? a.topk_idx[(size_t)t * K + k] : -1;
      row[k] = (v < 0 || v >= E) ? -1 : (int)v;
    }
#pragma unroll
    for (int k = 0; k < kMaxTopk; ++k)
      if (k < K && counts_ll(row, k, E)) {
        const int d = row[k] / Lx;
        atomicOr(&s_own[d][t >> 5], 1u << (t & 31));
        if (d == me) atomicOr(&s_emask[me * Lx + (row[k] - me * Lx)][t >> 5], 1u << (t & 31));
      }
  }
  __syncthreads();

  stamp(0);
  if (alive) {
    // ---- routing table: block b writes it to peer (me + 1 + b) % P (16-byte stores when the table allows), so all peers are
    // served at once and the table leaves in a couple of microseconds; rows to their destinations (all warps)
    {
      const int n = a.T * K;
      const bool vec = ((M * K) & 3) == 0 && (reinterpret_cast<uintptr_t>(a.topk_idx) & 15) == 0 &&
                       (!a.topk_w || (reinterpret_cast<uintptr_t>(a.topk_w) & 15) == 0);
      for (int s = blockIdx.x + 1; s < P; s += gridDim.x) {
        const int d = (me + s) % P;
        uint8_t* base = ctx.ws[d] + bank_off;
        int* gi = reinterpret_cast<int*>(base + ll.gather_idx) + (size_t)me * M * K;
        float* gwt = reinterpret_cast<float*>(base + ll.gather_w) + (size_t)me * M * K;
        const int n4 = vec ? n / 4 : 0;
        for (int i = threadIdx.x; i < n4; i += kLLThreads) {
          const longlong2 lo = __ldg(reinterpret_cast<const longlong2*>(a.topk_idx) + 2 * i);
          const longlong2 hi = __ldg(reinterpret_cast<const longlong2*>(a.topk_idx) + 2 * i + 1);
          const long long v[4] = {lo.x, lo.y, hi.x, hi.y};
          int o[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) o[j] = (v[j] < 0 || v[j] >= E) ? -1 : (int)v[j];
          reinterpret_cast<int4*>(gi)[i] = make_int4(o[0], o[1], o[2], o[3]);
          reinterpret_cast<float4*>(gwt)[i] = a.topk_w ? __ldg(reinterpret_cast<const float4*>(a.topk_w) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        for (int j = n4 * 4 + threadIdx.x; j < n; j += kLLThreads) {
          const long long v = a.topk_idx[j];
          gi[j] = (v < 0 || v >= E) ? -1 : (int)v;
          gwt[j] = a.topk_w ? a.topk_w[j] : 0.f;
        }
        if (threadIdx.x == 0) reinterpret_cast<int*>(base + ll.gather_hdr)[me * 4] = a.T;
        __syncthreads();   // the block's stores are ordered before the flag by the block barrier + release
        if (threadIdx.x == 0) st_release_sys(reinterpret_cast<unsigned long long*>(base + ll.idx_flag) + me, epoch);
      }
    }
    stamp(6);
    uint8_t* mine = ctx.ws[me] + bank_off;
    const int* gidx = reinterpret_cast<const int*>(mine + ll.gather_idx);
    if (warp < kLLSendWarps) {
    // ================================================================ sending warps: every row part to its remote destinations
    PendingFlags pending;
    for (int item = warp * gridDim.x + blockIdx.x; item < a.T * (P - 1) * kLLParts; item += gridDim.x * kLLSendWarps) {
      const int part = item % kLLParts, td = item / kLLParts;
      const int t = td / (P - 1), d = (me + 1 + td % (P - 1)) % P;
      if (!((s_own[d][t >> 5] >> (t & 31)) & 1u)) continue;
      const LLPart pr = ll_part(H, part);
      if (pr.v0 >= pr.v1) continue;
      const int j = below8(s_own[d], t);
      uint8_t* base = ctx.ws[d] + bank_off;
      uint8_t* dst = base + ll.stage + ((size_t)me * M + j) * ll.msg_bytes;
      if (a.mode == 2) {  // bf16 -> e4m3 with one fp32 scale per 128 values, straight into the peer
        const int4* src = reinterpret_cast<const int4*>(reinterpret_cast<const uint8_t*>(a.x) + (size_t)t * H * 2);
        const int u_lo = pr.v0 / 8, u_hi = pr.v1 / 8, half = lane >> 4;
        constexpr int U = 8;
        for (int u0 = u_lo; u0 < u_hi; u0 += 32 * U) {
          int4 v[U];
#pragma unroll
          for (int i = 0; i < U; ++i) {
            const int u = u0 + i * 32 + lane;
            v[i] = u < u_hi ? __ldg(src + u) : make_int4(0, 0, 0, 0);
          }
#pragma unroll
          for (int i = 0; i < U; ++i) {
            const int u = u0 + i * 32 + lane;
            if (u0 + i * 32 >= u_hi) break;           // warp-uniform
            float scale;
            const uint2 q = quant8(v[i], scale);      // groups are whole, so a step is all-or-nothing per half warp
            if (u < u_hi) {
              *reinterpret_cast<uint2*>(dst + (size_t)u * 8) = q;
              if ((lane & 15) == 0) reinterpret_cast<float*>(dst + H)[(u0 + i * 32) / 16 + half] = scale;
            }
          }
        }
      } else {
        const int b_lo = fp8 ? pr.v0 : pr.v0 * 2, b_hi = fp8 ? pr.v1 : pr.v1 * 2;   // byte range of the part in the row
        warp_copy_row1(reinterpret_cast<int4*>(dst + b_lo),
                       reinterpret_cast<const int4*>(reinterpret_cast<const uint8_t*>(a.x) + (size_t)t * row_bytes + b_lo),
                       (b_hi - b_lo) / 16, lane);
        if (a.mode == 1)
          for (int q = pr.b0 + lane; q < pr.b1; q += 32) reinterpret_cast<float*>(dst + H)[q] = a.x_sf[(size_t)t * nsf + q];
      }
      stamp(7);
      pending.add(reinterpret_cast<unsigned long long*>(base + ll.row_flag) + ((size_t)me * M + j) * kLLParts + part, epoch, lane);
    }
    pending.publish(epoch, lane);
    stamp(1);
    } else {
    // ================================================================ layout warps: wait for the peers' routing tables, derive the layout
    int ok = 1;
    if (lt < P && lt != me)
      ok = wait_flag_ge(reinterpret_cast<unsigned long long*>(mine + ll.idx_flag) + lt, epoch, ctx, kOpLLDispatch, 1, lt);
    if (!ok) s_fail = 1;
    if (lt < kMaxRanks)
      s_T[lt] = lt == me ? a.T : (ok && lt < P) ? __ldcg(reinterpret_cast<const int*>(mine + ll.gather_hdr) + lt * 4) : 0;
    layout_sync();
    stamp(2, kLayoutFirst);
    if (!s_fail) {
    int maxT = 1;
    for (int r = 0; r < P; ++r) maxT = max(maxT, min(s_T[r], M));
    const int words = (maxT + 31) >> 5;               // mask words in use
    // one thread per (source, token) of the peers (this rank's masks are already set); the loads of four items are issued
    // before the first of them is used
    constexpr int kBatch = 4;
    for (int i0 = lt; i0 < P * maxT; i0 += LT * kBatch) {
      int row[kBatch][kMaxTopk];
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        const int i = i0 + b * LT, r = i / maxT, t = i - r * maxT;
        const bool live = i < P * maxT && t < s_T[r] && r != me;
#pragma unroll
        for (int k = 0; k < kMaxTopk; ++k) row[b][k] = (live && k < K) ? __ldcg(gidx + ((size_t)r * M + t) * K + k) : -1;
      }
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        const int i = i0 + b * LT, r = i / maxT, t = i - r * maxT;
        if (i >= P * maxT) break;
#pragma unroll
        for (int k = 0; k < kMaxTopk; ++k) {
          if (k < K && counts_ll(row[b], k, E) && row[b][k] / Lx == me) {
            atomicOr(&s_emask[r * Lx + (row[b][k] - me * Lx)][t >> 5], 1u << (t & 31));
            atomicOr(&s_hit[r][t >> 5], 1u << (t & 31));
          }
        }
      }
    }
    layout_sync();
    // rows per local expert and their exclusive prefix: every thread owns `per` consecutive experts, a warp scan and the
    // warps' totals give its first row (a serial scan by one thread took 6 us for 384 experts)
    const int per = (Lx + LT - 1) / LT, l0 = min(Lx, lt * per), l1 = min(Lx, l0 + per);
    auto rows_of = [&](int r, int l) {
      int n = 0;
      for (int w = 0; w < words; ++w) n += __popc(s_emask[r * Lx + l][w]);
      return n;
    };
    int tot = 0;
    for (int l = l0; l < l1; ++l)
      for (int r = 0; r < P; ++r) { const int n = rows_of(r, l); s_off[r * Lx + l] = n; tot += n; }
    int incl = tot;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += o;
    }
    if (lane == 31) s_warp_rows[warp] = incl;
    layout_sync();
    int run = incl - tot, all = 0;
    for (int w = kLLSendWarps; w < nwarps; ++w) {
      if (w < warp) run += s_warp_rows[w];
      all += s_warp_rows[w];
    }
    for (int l = l0; l < l1; ++l) {
      const int begin = run;
      for (int r = 0; r < P; ++r) { const int n = s_off[r * Lx + l]; s_off[r * Lx + l] = run; run += n; }
      if (blockIdx.x == 0) {
        a.expert_offsets[l] = begin;
        a.expert_counts[l] = run - begin;
        if (a.mailbox) a.mailbox[4 + l] = run - begin;
      }
    }
    if (blockIdx.x == 0) {
      if (a.mailbox) __threadfence_system();     // the last block of the launch publishes the call's number
      if (lt == 0) {
        a.expert_offsets[Lx] = all;
        *a.num_rows = all;
        if (a.mailbox) { a.mailbox[0] = all; __threadfence_system(); }
      }
    }
    }
    stamp(3, kLayoutFirst);
    }
    // ---- both halves of the block meet: the rows are on their way and the layout is known
    __syncthreads();
    alive = !s_fail;
  }
  if (!alive) {     // a wait ran out: the handle names no rows (a combine may be queued behind this launch already)
    for (int i = blockIdx.x * kLLThreads + threadIdx.x; i < a.T * K; i += gridDim.x * kLLThreads) a.local_row[i] = -1;
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.num_rows = 0;
  }
  if (alive) {
    uint8_t* mine = ctx.ws[me] + bank_off;
    const int* gidx = reinterpret_cast<const int*>(mine + ll.gather_idx);
    const float* gw_ = reinterpret_cast<const float*>(mine + ll.gather_w);
    uint8_t* recv_x = reinterpret_cast<uint8_t*>(a.recv_x);
    // lane k: the output row of slot k of token t of source r (-1: its expert lives elsewhere, or the slot is empty or repeated)
    auto out_row_of = [&](int r, int t, int e) {
      bool counts = e >= 0 && e < E && e / Lx == me;
      for (int z = 0; z < K; ++z) {
        const int ez = __shfl_sync(0xffffffffu, e, z);
        if (z < lane && ez == e) counts = false;
      }
      if (!counts) return -1;
      const int at = r * Lx + e - me * Lx, row = s_off[at] + below8(s_emask[at], t);
      return row < a.capacity ? row : -1;
    };

    // ---- rows of this rank's own tokens: from the caller's tensor straight into every output row
    for (int item = gw; item < a.T * pieces; item += total_warps) {
      const int piece = item % pieces, t = item / pieces;
      const LLPart pr = item == gw ? own_pr : ll_piece(H, piece, pieces);
      int e = -1;
      if (lane < K) {
        const long long v = a.topk_idx[(size_t)t * K + lane];
        e = (v < 0 || v >= E) ? -1 : (int)v;
      }
      const int row = out_row_of(me, t, e);
      if (piece == 0 && lane < K) {
        a.local_row[(size_t)t * K + lane] = row;
        if (row >= 0) {
          a.recv_row_src[row] = (me * M + t) * K + lane;
          a.recv_w[row] = a.topk_w ? a.topk_w[(size_t)t * K + lane] : 0.f;
        }
      }
      const unsigned live = __ballot_sync(0xffffffffu, row >= 0);
      if (live == 0 || pr.v0 >= pr.v1) continue;
      write_own_piece(a, recv_x, t, pr, row, live, H, nsf, row_bytes, src_bytes, item == gw ? ahead : nullptr, lane);
    }

    // ---- rows of the peers: poll the part flags and write the output rows
    int maxT = 1;
    for (int r = 0; r < P; ++r) if (r != me) maxT = max(maxT, min(s_T[r], M));
    const uint8_t* stage = mine + ll.stage;
    // a staged row is materialised part by part, by whichever warp draws the part
    for (int item = gw; item < (P - 1) * maxT * kLLParts; item += total_warps) {
      const int part = item % kLLParts, it = item / kLLParts;
      const int r = (me + 1 + it / maxT) % P, t = it % maxT;
      if (t >= s_T[r] || !((s_hit[r][t >> 5] >> (t & 31)) & 1u)) continue;
      const LLPart pr = ll_part(H, part);
      if (pr.v0 >= pr.v1) continue;
      const int j = below8(s_hit[r], t);
      const int e = lane < K ? __ldcg(gidx + ((size_t)r * M + t) * K + lane) : -1;   // issued before the flag wait
      int got = 1;
      if (lane == 0)
        got = wait_flag_ge(reinterpret_cast<unsigned long long*>(mine + ll.row_flag) + ((size_t)r * M + j) * kLLParts + part, epoch,
                           ctx, kOpLLDispatch, 2, r);
      if (!__shfl_sync(0xffffffffu, got, 0)) break;
      const int row = out_row_of(r, t, e);
      if (part == 0 && row >= 0) {
        a.recv_row_src[row] = (r * M + t) * K + lane;
        a.recv_w[row] = __ldcg(gw_ + ((size_t)r * M + t) * K + lane);
      }
      const unsigned live = __ballot_sync(0xffffffffu, row >= 0);
      const uint8_t* src = stage + ((size_t)r * M + j) * ll.msg_bytes;
      const int b_lo = fp8 ? pr.v0 : pr.v0 * 2, b_hi = fp8 ? pr.v1 : pr.v1 * 2, n = (b_hi - b_lo) / 16;
      for (int u0 = 0; u0 < n; u0 += 32 * 8) {
        int4 v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int u = u0 + i * 32 + lane;
          if (u < n) v[i] = __ldcg(reinterpret_cast<const int4*>(src + b_lo) + u);
        }
        for (unsigned m = live; m; m &= m - 1) {
          int4* d = reinterpret_cast<int4*>(recv_x + (size_t)__shfl_sync(0xffffffffu, row, __ffs(m) - 1) * row_bytes + b_lo);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int u = u0 + i * 32 + lane;
            if (u < n) d[u] = v[i];
          }
        }
      }
      if (fp8)
        for (int b = pr.b0; b < pr.b1; b += 32) {
          const float sf = b + lane < pr.b1 ? __ldcg(reinterpret_cast<const float*>(src + H) + b + lane) : 0.f;
          for (unsigned m = live; m; m &= m - 1) {
            const size_t o = __shfl_sync(0xffffffffu, row, __ffs(m) - 1);
            if (b + lane < pr.b1) a.recv_sf[o * nsf + b + lane] = sf;
          }
        }
    }
  }

  stamp(4);
  if (last_block_of_rank(ctl, kOpLLDispatch, gridDim.x)) {
    stamp(5);
    if (!ld_volatile_int(&ctl->abort) && threadIdx.x < P)
      st_release_sys(&control_of(ctx.ws[threadIdx.x])->ll_disp_ack[me], epoch);
    if (threadIdx.x == 0) {
      ctl->epoch[kOpLLDispatch] = epoch;
      // A host that waits for the counts goes on when the rows of the peers are in place too: a wait for them that ran out is in the
      // status by now (the blocks arrive behind their own waits), and the host looks there next.
      if (a.mailbox) {
        __threadfence_system();
        a.mailbox[3] = a.seq;
      }
    }
  }
}

// One rank: nothing is sent and nobody is waited for, so every block derives the layout from the caller's table by itself and
// writes its share of the rows.  What bounds it is the launch and the chain routes -> masks -> scan -> rows; the table's and the
// first row's loads are issued before anything else.  Because no block waits for another an ordinary launch will do: a captured
// dispatch of one fp8 token (hidden 7168, 256 experts, top-8) took 12.4 us as a cooperative launch of the kernel above, of which 6.9
// were spent inside, and takes 6.3 here (3.8 inside); 64 tokens 12.5 and 6.7 us, 128 tokens 14.7 and 8.7.
template <bool kProfile>
__global__ void __launch_bounds__(kLLThreads) ep_dispatch_ll_local_kernel(const __grid_constant__ LLDispatchParams p) {
  const LLDispatchArgs& a = p.r[0];
  const WsLayout& lay = p.lay;
  const int K = lay.topk, H = lay.hidden, E = a.E, T = a.T, n = T * K;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gw = warp * gridDim.x + blockIdx.x, total_warps = gridDim.x * (kLLThreads / 32);
  const bool fp8 = a.mode != 0;
  const int nsf = H / 128, row_bytes = fp8 ? H : H * 2, src_bytes = a.mode == 1 ? H : H * 2, words = (T + 31) >> 5;

  __shared__ unsigned s_emask[kMaxExperts * kLLWords];    // [expert][words]: its tokens
  __shared__ int s_off[kMaxExperts];                      // first output row of the expert
  __shared__ short s_id[kLLMaxTokens * kMaxTopk];         // the table; -1: no expert
  __shared__ int s_warp_rows[kLLThreads / 32];

  Control* ctl = control_of(a.ctx.ws[0]);
  unsigned long long t_start = 0;
  if constexpr (kProfile) t_start = global_timer_ns();
  auto stamp = [&](int i) {
    if constexpr (kProfile)
      if (blockIdx.x == 0 && threadIdx.x == 0) ctl->dbg[i] = global_timer_ns() - t_start;
  };

  // ---- the routes and this warp's first piece of a row (loops over the table stay rolled: a launch starts with a cold instruction
  // cache, and copies of a loop's body cost more than its iterations)
  constexpr int kIds = 4;
#pragma unroll 1
  for (int i0 = threadIdx.x; i0 < n; i0 += kLLThreads * kIds) {
    long long v[kIds];
#pragma unroll
    for (int j = 0; j < kIds; ++j) v[j] = i0 + j * kLLThreads < n ? __ldg(a.topk_idx + i0 + j * kLLThreads) : -1;
#pragma unroll
    for (int j = 0; j < kIds; ++j)
      if (i0 + j * kLLThreads < n) s_id[i0 + j * kLLThreads] = (short)((v[j] < 0 || v[j] >= E) ? -1 : (int)v[j]);
  }
  const int pieces = max(1, min((H + 127) / 128, total_warps / max(T, 1)));
  int4 ahead[kOwnUnroll];
  LLPart first_part = {0, 0, 0, 0};
  if (gw < T * pieces) {
    first_part = ll_piece(H, gw % pieces, pieces);
    const int lo = (a.mode == 1 ? first_part.v0 : first_part.v0 * 2) / 16, hi = (a.mode == 1 ? first_part.v1 : first_part.v1 * 2) / 16;
    const int4* src = reinterpret_cast<const int4*>(reinterpret_cast<const uint8_t*>(a.x) + (size_t)(gw / pieces) * src_bytes);
#pragma unroll
    for (int i = 0; i < kOwnUnroll; ++i) {
      const int u = lo + i * 32 + lane;
      ahead[i] = u < hi ? __ldg(src + u) : make_int4(0, 0, 0, 0);
    }
  }
#pragma unroll 1
  for (int i = threadIdx.x; i < E * words; i += kLLThreads) s_emask[i] = 0u;
  const bool head = gw < T * pieces && gw % pieces == 0;      // this warp starts with the first piece of a token: its weights too
  const float first_w = head && lane < K && a.topk_w ? __ldg(a.topk_w + (size_t)(gw / pieces) * K + lane) : 0.f;
  __syncthreads();
  stamp(0);

  // ---- tokens of every expert: a repeated id sets the same bit again
#pragma unroll 1
  for (int i = threadIdx.x; i < n; i += kLLThreads) {
    const int e = s_id[i], t = i / K;
    if (e >= 0) atomicOr(&s_emask[e * words + (t >> 5)], 1u << (t & 31));
  }
  __syncthreads();
  stamp(2);

  // ---- first row of every expert: two consecutive experts per thread, a warp scan and the warps' totals
  constexpr int kPer = kMaxExperts / kLLThreads;
  const int per = E > kLLThreads ? kPer : 1;
  int rows[kPer] = {}, tot = 0;
  for (int j = 0; j < per; ++j) {
    const int e = (int)threadIdx.x * per + j;
    if (e < E)
      for (int w = 0; w < words; ++w) rows[j] += __popc(s_emask[e * words + w]);
    tot += rows[j];
  }
  int incl = tot;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += o;
  }
  if (lane == 31) s_warp_rows[warp] = incl;
  __syncthreads();
  int run = incl - tot, all = 0;
#pragma unroll
  for (int w = 0; w < kLLThreads / 32; ++w) {
    const int r = s_warp_rows[w];
    if (w < warp) run += r;
    all += r;
  }
  for (int j = 0; j < per; ++j) {
    const int e = (int)threadIdx.x * per + j;
    if (e >= E) break;
    s_off[e] = run;
    if (blockIdx.x == 0) {
      a.expert_offsets[e] = run;
      a.expert_counts[e] = rows[j];
      if (a.mailbox) a.mailbox[4 + e] = rows[j];
    }
    run += rows[j];
  }
  __syncthreads();
  stamp(3);

  // ---- the rows, each piece from the caller's tensor into every output row of its token
  uint8_t* recv_x = reinterpret_cast<uint8_t*>(a.recv_x);
  for (int item = gw; item < T * pieces; item += total_warps) {
    const int piece = item % pieces, t = item / pieces;
    const LLPart pr = item == gw ? first_part : ll_piece(H, piece, pieces);
    const int e = lane < K ? s_id[t * K + lane] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, e);
    int row = -1;
    if (e >= 0 && (same & ((1u << lane) - 1u)) == 0) {
      row = s_off[e] + below8(s_emask + e * words, t);
      if (row >= a.capacity) row = -1;
    }
    if (piece == 0 && lane < K) {
      a.local_row[(size_t)t * K + lane] = row;
      if (row >= 0) {
        a.recv_row_src[row] = t * K + lane;
        a.recv_w[row] = item == gw ? first_w : a.topk_w ? __ldg(a.topk_w + (size_t)t * K + lane) : 0.f;
      }
    }
    const unsigned live = __ballot_sync(0xffffffffu, row >= 0);
    if (live == 0 || pr.v0 >= pr.v1) continue;
    write_own_piece(a, recv_x, t, pr, row, live, H, nsf, row_bytes, src_bytes, item == gw ? ahead : nullptr, lane);
  }
  stamp(4);

  // ---- the host's copy of the counts, and the epoch (nothing but this block reads it)
  if (blockIdx.x == 0) {
    if (a.mailbox) __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) {
      const unsigned long long epoch = ctl->epoch[kOpLLDispatch] + 1;
      a.expert_offsets[E] = all;
      *a.num_rows = all;
      if (a.mailbox) {
        a.mailbox[0] = all;
        __threadfence_system();
        a.mailbox[3] = a.seq;
      }
      ctl->ll_disp_ack[0] = epoch;
      ctl->epoch[kOpLLDispatch] = epoch;
    }
    stamp(5);
  }
}

cudaError_t launch_ll_dispatch(const LLDispatchParams& p, int nranks, int blocks, cudaStream_t stream) {
  if (p.lay.world == 1 && nranks == 1) {
    const LLDispatchArgs& a = p.r[0];
    // no more blocks than pieces of 128 values: every block derives the whole layout
    const int items = a.T * ((p.lay.hidden + 127) / 128), grid = max(1, min(blocks, items));
    if (p.profile) ep_dispatch_ll_local_kernel<true><<<grid, kLLThreads, 0, stream>>>(p);
    else ep_dispatch_ll_local_kernel<false><<<grid, kLLThreads, 0, stream>>>(p);
    return cudaGetLastError();
  }
  dim3 grid(blocks, nranks), block(kLLThreads);
  void* args[] = {const_cast<LLDispatchParams*>(&p)};
  const void* fn = p.profile ? (const void*)ep_dispatch_ll_kernel<true> : (const void*)ep_dispatch_ll_kernel<false>;
  return cudaLaunchCooperativeKernel(fn, grid, block, args, 0, stream);
}

// ------------------------------------------------------------------------------------------ combine
template <bool kProfile>
__global__ void __launch_bounds__(kLLThreads) ep_combine_ll_kernel(const __grid_constant__ LLCombineParams p) {
  const LLCombineArgs& a = p.r[blockIdx.y];
  const WsLayout& lay = p.lay;
  const RankCtx& ctx = a.ctx;
  const int P = ctx.world, me = ctx.rank, M = lay.max_tokens, K = lay.topk, H = lay.hidden;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = kLLThreads / 32;
  // consecutive work items go to different SMs, so a short list of items spreads over the whole GPU
  const int gw = warp * gridDim.x + blockIdx.x, total_warps = gridDim.x * nwarps;
  Control* ctl = control_of(ctx.ws[me]);
  const unsigned long long epoch = ctl->epoch[kOpLLCombine] + 1;
  const int aborted = ld_volatile_int(&ctl->abort);    // set: an earlier call gave up, the handle's tensors may never have been written
  const LLLayout ll = make_ll_layout(P, M, K, H);
  const long long bank_off = lay.ll + (long long)(epoch & 1) * ll.bank_bytes;
  const int row_bytes = H * 2;
  // profile instantiation only: phase stamps (nanoseconds since kernel start) of block 0 in Control::dbg[8..15]
  unsigned long long t_start = 0;
  if constexpr (kProfile) t_start = global_timer_ns();
  auto stamp = [&](int i) {
    if constexpr (kProfile)
      if (blockIdx.x == 0 && threadIdx.x == 0) ctl->dbg[8 + i] = global_timer_ns() - t_start;
  };

  int ok = 1;
  if (threadIdx.x < P && threadIdx.x != me && epoch > 2)
    ok = wait_flag_ge(&ctl->ll_comb_ack[threadIdx.x], epoch - 2, ctx, kOpLLCombine, 0, threadIdx.x);
  const int alive = __syncthreads_and(ok);
  stamp(0);

  if (alive) {
    // ---- return every expert row of a peer's token, part by part, to its (token, slot) slot there
    const int R = aborted ? 0 : min(*a.num_rows, a.x_rows);
    PendingFlags pending;
    for (int item = gw; item < R * kLLParts; item += total_warps) {
      const int r = item / kLLParts, part = item % kLLParts;
      const int code = a.recv_row_src[r];
      if (code < 0) continue;
      const int src = code / (M * K), rem = code - src * M * K;
      if (src == me || src >= P) continue;
      const LLPart pr = ll_part(H, part);
      if (pr.v0 >= pr.v1) continue;
      uint8_t* base = ctx.ws[src] + bank_off;
      int4* dst = reinterpret_cast<int4*>(base + ll.ret + (size_t)rem * row_bytes + (size_t)pr.v0 * 2);
      const int4* from = reinterpret_cast<const int4*>(reinterpret_cast<const uint8_t*>(a.x) + (size_t)r * row_bytes + (size_t)pr.v0 * 2);
      warp_copy_row1(dst, from, (pr.v1 - pr.v0) / 8, lane);
      pending.add(reinterpret_cast<unsigned long long*>(base + ll.ret_flag) + (size_t)rem * kLLParts + part, epoch, lane);
    }
    pending.publish(epoch, lane);
    stamp(1);
    // ---- weighted sum at the source, slot order, fp32: a warp takes `step` 16-byte columns of a part of a token.  Rows of
    // this rank's own experts are read from x, the others from the return slots once their flags are set.
    uint8_t* mine = ctx.ws[me] + bank_off;
    const unsigned long long* flags = reinterpret_cast<const unsigned long long*>(mine + ll.ret_flag);
    const int part_units = ll_part(H, 0).v1 / 8;      // the first part is the widest
    const int subs32 = (part_units + 31) / 32;
    const int step = a.T * kLLParts * subs32 <= total_warps ? 32 : 64, subs = (part_units + step - 1) / step;
    for (int item = gw; item < a.T * kLLParts * subs; item += total_warps) {
      const int t = item / (kLLParts * subs), rest = item - t * (kLLParts * subs), part = rest / subs, sub = rest - part * subs;
      const LLPart pr = ll_part(H, part);
      const int u_begin = pr.v0 / 8 + sub * step, u_end = min(pr.v1 / 8, u_begin + step);
      if (u_begin >= u_end) continue;
      // lane k holds slot k: expert, weight, whether it counts (in range, first occurrence), where its row is
      long long e = -1;
      float w = 0.f;
      int local = -1;
      if (lane < K) {
        e = a.topk_idx[(size_t)t * K + lane];
        w = a.topk_w[(size_t)t * K + lane];
        local = a.local_row[(size_t)t * K + lane];
      }
      bool counts = lane < K && e >= 0 && e < a.E;
      for (int z = 0; z < K; ++z) {
        const long long ez = __shfl_sync(0xffffffffu, e, z);
        if (z < lane && ez == e) counts = false;
      }
      const unsigned valid = __ballot_sync(0xffffffffu, counts);
      int got = !aborted;
      if (got && counts && local >= a.x_rows) {        // the handle and x do not belong together
        report_failure(ctx, kStatusBadArgument, kOpLLCombine, 2, me, a.x_rows, local);
        got = 0;
      }
      if (got && counts && local < 0) got = wait_flag_ge(flags + ((size_t)t * K + lane) * kLLParts + part, epoch, ctx, kOpLLCombine, 1, me);
      if (!__all_sync(0xffffffffu, got)) break;
      const unsigned long long my_row = reinterpret_cast<unsigned long long>(
          local >= 0 ? reinterpret_cast<const uint8_t*>(a.x) + (size_t)local * row_bytes
                     : mine + ll.ret + ((size_t)t * K + min(lane, K - 1)) * row_bytes);
      int4* out = reinterpret_cast<int4*>(reinterpret_cast<uint8_t*>(a.out) + (size_t)t * row_bytes);
      const int u0 = u_begin + lane;
      const bool one = u0 < u_end, two = u0 + 32 < u_end;
      float a0[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, a1[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int kb = 0; kb < K; kb += 8) {    // eight slots' loads in flight at a time
        int4 v0[8], v1[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          if (kb + k < K && ((valid >> (kb + k)) & 1u)) {
            const int4* row = reinterpret_cast<const int4*>(__shfl_sync(0xffffffffu, my_row, kb + k));
            if (one) v0[k] = __ldcg(row + u0);
            if (two) v1[k] = __ldcg(row + u0 + 32);
          }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          if (kb + k < K && ((valid >> (kb + k)) & 1u)) {      // warp-uniform
            const float wk = __shfl_sync(0xffffffffu, w, kb + k);
            const __nv_bfloat162* h0 = reinterpret_cast<const __nv_bfloat162*>(&v0[k]);
            const __nv_bfloat162* h1 = reinterpret_cast<const __nv_bfloat162*>(&v1[k]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              // product and sum are rounded separately (no fused multiply-add), as the CPU oracle does
              if (one) {
                a0[2 * i] = __fadd_rn(a0[2 * i], __fmul_rn(wk, __low2float(h0[i])));
                a0[2 * i + 1] = __fadd_rn(a0[2 * i + 1], __fmul_rn(wk, __high2float(h0[i])));
              }
              if (two) {
                a1[2 * i] = __fadd_rn(a1[2 * i], __fmul_rn(wk, __low2float(h1[i])));
                a1[2 * i + 1] = __fadd_rn(a1[2 * i + 1], __fmul_rn(wk, __high2float(h1[i])));
              }
            }
          }
        }
      }
      int4 o;
      __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
      if (one) {
#pragma unroll
        for (int i = 0; i < 4; ++i) oh[i] = __floats2bfloat162_rn(a0[2 * i], a0[2 * i + 1]);
        out[u0] = o;
      }
      if (two) {
#pragma unroll
        for (int i = 0; i < 4; ++i) oh[i] = __floats2bfloat162_rn(a1[2 * i], a1[2 * i + 1]);
        out[u0 + 32] = o;
      }
    }
  }

  stamp(2);
  if (last_block_of_rank(ctl, kOpLLCombine, gridDim.x)) {
    stamp(3);
    if (!ld_volatile_int(&ctl->abort) && threadIdx.x < P)
      st_release_sys(&control_of(ctx.ws[threadIdx.x])->ll_comb_ack[me], epoch);
    if (threadIdx.x == 0) ctl->epoch[kOpLLCombine] = epoch;
  }
}

// One rank: every row is in x, so a warp takes 32 pieces of 16 bytes of a token and there is nothing to wait for.  Launch and two
// dependent rounds of loads (slots, rows) bound it; small blocks, as many as there are pieces, in an ordinary launch.  A captured
// combine of one token of 7168, top-8: 8.4 us as a cooperative launch of the kernel above (2.5 inside), 4.3 here (2.0 inside);
// 128 tokens 10.4 and 6.4 us.
template <bool kProfile>
__global__ void __launch_bounds__(kLLLocalThreads) ep_combine_ll_local_kernel(const __grid_constant__ LLCombineParams p) {
  const LLCombineArgs& a = p.r[0];
  const int K = p.lay.topk, units = p.lay.hidden / 8, spans = (units + 31) / 32, lane = threadIdx.x & 31;
  Control* ctl = control_of(a.ctx.ws[0]);
  unsigned long long t_start = 0;
  if constexpr (kProfile) t_start = global_timer_ns();
  auto stamp = [&](int i) {
    if constexpr (kProfile)
      if (blockIdx.x == 0 && threadIdx.x == 0) ctl->dbg[8 + i] = global_timer_ns() - t_start;
  };
  const int aborted = ld_volatile_int(&ctl->abort);    // set: an earlier call gave up, the handle's tensors may never have been written
  const int item = blockIdx.x * (kLLLocalThreads / 32) + (threadIdx.x >> 5), t = item / spans, u = (item - t * spans) * 32 + lane;
  if (t < a.T) {
    // lane k holds slot k: whether it counts (id in range, first occurrence), its weight, its row
    int e = -1, local = -1;
    float w = 0.f;
    if (lane < K) {
      const size_t at = (size_t)t * K + lane;
      const long long v = __ldg(a.topk_idx + at);
      w = __ldg(a.topk_w + at);
      local = __ldg(a.local_row + at);
      e = (v < 0 || v >= a.E) ? -1 : (int)v;
    }
    stamp(0);
    const unsigned same = __match_any_sync(0xffffffffu, e);
    const bool counts = e >= 0 && (same & ((1u << lane) - 1u)) == 0;
    const unsigned valid = __ballot_sync(0xffffffffu, counts);
    bool ok = !aborted;
    if (ok && counts && (local < 0 || local >= a.x_rows)) {       // the handle and x do not belong together
      report_failure(a.ctx, kStatusBadArgument, kOpLLCombine, 2, 0, a.x_rows, (unsigned long long)(long long)local);
      ok = false;
    }
    stamp(1);
    if (__all_sync(0xffffffffu, ok)) {
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      const int4* x = reinterpret_cast<const int4*>(a.x);
      for (int kb = 0; kb < K; kb += 8) {    // eight slots' loads in flight at a time
        int4 v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (kb + k < K && ((valid >> (kb + k)) & 1u)) {
            const int4* row = x + (size_t)__shfl_sync(0xffffffffu, local, kb + k) * units;
            if (u < units) v[k] = __ldg(row + u);
          }
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (kb + k < K && ((valid >> (kb + k)) & 1u)) {         // warp-uniform
            const float wk = __shfl_sync(0xffffffffu, w, kb + k);
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v[k]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              // product and sum are rounded separately (no fused multiply-add), as the CPU oracle does
              acc[2 * i] = __fadd_rn(acc[2 * i], __fmul_rn(wk, __low2float(h[i])));
              acc[2 * i + 1] = __fadd_rn(acc[2 * i + 1], __fmul_rn(wk, __high2float(h[i])));
            }
          }
      }
      if (u < units) {
        int4 o;
        __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int i = 0; i < 4; ++i) oh[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
        reinterpret_cast<int4*>(a.out)[(size_t)t * units + u] = o;
      }
    }
  }
  stamp(2);
  if (item == 0 && lane == 0) {            // nothing but this thread reads the epoch
    const unsigned long long epoch = ctl->epoch[kOpLLCombine] + 1;
    ctl->ll_comb_ack[0] = epoch;
    ctl->epoch[kOpLLCombine] = epoch;
  }
  stamp(3);
}

cudaError_t launch_ll_combine(const LLCombineParams& p, int nranks, int blocks, cudaStream_t stream) {
  if (p.lay.world == 1 && nranks == 1) {
    const int warps = max(1, p.r[0].T * ((p.lay.hidden / 8 + 31) / 32)), per = kLLLocalThreads / 32, grid = (warps + per - 1) / per;
    if (p.profile) ep_combine_ll_local_kernel<true><<<grid, kLLLocalThreads, 0, stream>>>(p);
    else ep_combine_ll_local_kernel<false><<<grid, kLLLocalThreads, 0, stream>>>(p);
    return cudaGetLastError();
  }
  dim3 grid(blocks, nranks), block(kLLThreads);
  void* args[] = {const_cast<LLCombineParams*>(&p)};
  const void* fn = p.profile ? (const void*)ep_combine_ll_kernel<true> : (const void*)ep_combine_ll_kernel<false>;
  return cudaLaunchCooperativeKernel(fn, grid, block, args, 0, stream);
}

}  // namespace dep
