// ep_dispatch_ht: all-to-all-v token push with rank-level dedup and receive-side expansion.
//
// Every warp works on its own, there is no block-wide step inside the kernel.
//   Sender warps take groups of kGroupTokens source tokens.  A token row is read once into registers
//   (a quarter row per pass) and stored ONCE per destination GPU into that GPU's staging area through
//   the peer mapping (NVLink), optionally quantised to e4m3 with one fp32 scale per 128 values on the
//   way.  Rows whose destination is the sending rank itself are written straight into the output
//   tensor, one copy per local expert.  After a group the warp publishes one release flag per
//   destination: flags cover two tokens, so the receivers follow the senders closely, no sender ever
//   drains a pipeline at a chunk boundary, and there are several groups per sender warp, which keeps
//   the last wave of groups short.
//   Receiver warps take blocks of kRowBlock staged rows of one source, in the order the senders
//   produce them.  Each record names its source token; the warp waits for that token's flag and
//   materialises every output row of the staged row (one per local expert of the token), so a token
//   crosses NVLink once no matter how many experts of the destination it uses.
//   Groups and blocks are handed out by two shared counters; sender warps turn into receivers once
//   the last group is on its way.
//
// Between two GPUs 32 SMs of 16-byte register stores reach the same rate as bulk shared->global copies
// (about 0.69 TB/s per direction with both directions busy); the register form needs no staging in
// shared memory, no proxy fences and no barriers, and lets a block keep 16 rows in flight.
//
// The reference's dispatch (csrc/kernels/dispatch/dispatch.cpp:463-590) has the same three jobs (payload
// scatter, receiver expansion from a forward list, per-source completion flags) spread over 64
// role-specialised vector cores and WQE queues.
#include <algorithm>

#include "api.h"
#include "fanout.cuh"

namespace dep {

// 16 bf16 values (two 16-byte pieces) -> their absolute maximum.
__device__ __forceinline__ float amax16(const int4& a, const int4& b, float v[16]) {
  const __nv_bfloat162* ha = reinterpret_cast<const __nv_bfloat162*>(&a);
  const __nv_bfloat162* hb = reinterpret_cast<const __nv_bfloat162*>(&b);
  float m = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __low2float(ha[i]); v[2 * i + 1] = __high2float(ha[i]);
    v[8 + 2 * i] = __low2float(hb[i]); v[8 + 2 * i + 1] = __high2float(hb[i]);
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) m = fmaxf(m, fabsf(v[i]));
  return m;
}

// Fused quantiser: a bf16 row -> e4m3 bytes and one fp32 scale per 128 values, written to every destination.
// amax over 128 values clamped to 1e-4, scale = amax / 448, q = e4m3(x * ((1 / amax) * 448)): reciprocal, then
// multiply, which is how torch evaluates the recipe's `448.0 / amax` (deep_ep/utils/math.py:45-60 of the reference),
// so results equal the recipe bit for bit.
// Lane l of a pass owns 16 consecutive values; 8 consecutive lanes share a scale.
__device__ __forceinline__ void warp_quant_fanout(const int4* src, int H, unsigned long long dst, unsigned long long dst_sf,
                                                  unsigned mask, int lane) {
  const int units = H / 16, passes = (units + 31) / 32, nsf = H / 128;
  float sf_keep[2] = {0.f, 0.f};   // lane l ends up with the scales of blocks l and 32 + l
  for (int p0 = 0; p0 < passes; p0 += 2) {
    int4 raw[2][2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int u = (p0 + q) * 32 + lane;
      if (p0 + q < passes && u < units) { raw[q][0] = __ldg(src + 2 * u); raw[q][1] = __ldg(src + 2 * u + 1); }
      else { raw[q][0] = make_int4(0, 0, 0, 0); raw[q][1] = make_int4(0, 0, 0, 0); }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int p = p0 + q, u = p * 32 + lane;
      if (p >= passes) break;
      float v[16];
      float amax = amax16(raw[q][0], raw[q][1], v);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
      amax = fmaxf(amax, 1e-4f);
      const float inv = __frcp_rn(amax) * 448.0f;   // torch evaluates `448 / amax` (scalar / tensor) as reciprocal, then multiply
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        w[i] = (uint32_t)__nv_cvt_float_to_fp8(v[4 * i] * inv, __NV_SATFINITE, __NV_E4M3) |
               ((uint32_t)__nv_cvt_float_to_fp8(v[4 * i + 1] * inv, __NV_SATFINITE, __NV_E4M3) << 8) |
               ((uint32_t)__nv_cvt_float_to_fp8(v[4 * i + 2] * inv, __NV_SATFINITE, __NV_E4M3) << 16) |
               ((uint32_t)__nv_cvt_float_to_fp8(v[4 * i + 3] * inv, __NV_SATFINITE, __NV_E4M3) << 24);
      const int4 out = make_int4((int)w[0], (int)w[1], (int)w[2], (int)w[3]);
      // block p * 4 + g lives in lanes 8g..8g+7; lane l keeps the scale of block 32 * (p / 8) + l
      const float g = __shfl_sync(0xffffffffu, amax / 448.0f, (lane & 3) * 8);
      if ((lane >> 2) == (p & 7)) { if ((p >> 3) == 0) sf_keep[0] = g; else sf_keep[1] = g; }
      for (unsigned m = mask; m; m &= m - 1) {
        int4* d = reinterpret_cast<int4*>(shfl_u64(dst, __ffs(m) - 1));
        if (u < units) d[u] = out;
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int b = 32 * q + lane;
    for (unsigned m = mask; m; m &= m - 1) {
      float* d = reinterpret_cast<float*>(shfl_u64(dst_sf, __ffs(m) - 1));
      if (b < nsf) d[b] = sf_keep[q];
    }
  }
}

// Zeroes the rows of this rank's output that no token fills: the padding of every expert's aligned block and the rows behind
// the last block.  (4096 x 8 fp8 rows over 256 experts in blocks of 128 rows: clearing the whole output first took a pass of 95 us,
// these rows add about 12 us to the kernel.)
__device__ __forceinline__ void zero_padding(const DispatchArgs& a, int local_experts, int row_bytes, int nsf, int gw, int warps, int lane) {
  for_padding_rows(a.pad_offsets, a.pad_counts, local_experts, a.recv_rows, gw, warps, [&](int row) {
    zero_row(reinterpret_cast<uint8_t*>(a.recv_x) + (size_t)row * row_bytes, row_bytes, a.recv_sf + (size_t)row * nsf, nsf, lane);
  });
}

// kPieces: one rank that keeps all its rows, the work items are column pieces of tokens.  Several ranks run without: their items
// are groups of tokens with a flag each, and none of the arithmetic of pieces (8 ranks x 512 tokens of 4096 emulated in one launch
// on one GPU: 129 us, 134 with the number of pieces as a variable and a ticket taken ahead).
template <bool kProfile, bool kPieces>
__global__ void __launch_bounds__(kDispatchThreads, 1) ep_dispatch_ht_kernel(const __grid_constant__ DispatchParams p) {
  const DispatchArgs& a = p.r[blockIdx.y];
  const WsLayout& lay = p.lay;
  const RankCtx& ctx = a.ctx;
  const int P = ctx.world, me = ctx.rank, Tmax = lay.max_tokens, H = lay.hidden, K = a.K;
  const int NG = (Tmax + kGroupTokens - 1) / kGroupTokens;
  const int lane = threadIdx.x & 31;
  const int q = lane >> 3, c = lane & 7;      // metadata of a group is fetched by lane = (token of the group) * 8 + field
  Control* ctl = control_of(ctx.ws[me]);
  const unsigned long long epoch = ctl->epoch[kOpDispatch] + 1;
  const bool aborted = ld_volatile_int(&ctl->abort) != 0;   // an earlier call gave up, the plan's tensors may never have been written

  const bool fp8 = a.mode != kDispatchBf16;
  const int nsf = fp8 ? H / 128 : 0;
  const int row_bytes = fp8 ? H : H * 2;     // payload bytes of one output row
  const int units = row_bytes / 16;
  const bool sender = (int)blockIdx.x < p.send_blocks;
  PhaseClock<kProfile> clk;
  clk.start();

  auto pad = [&]() {
    if (a.pad_offsets && !aborted) {
      zero_padding(a, a.E / P, row_bytes, nsf, (int)(threadIdx.x >> 5) * gridDim.x + blockIdx.x, gridDim.x * (kDispatchThreads / 32), lane);
      clk.mark(kProfData);
    }
  };
  // One rank starts with the padding, a fixed share per warp, and the tickets even it out (4096 tokens quantised to fp8, top-8 of
  // 256 experts in blocks of 128 rows, with the launch: 104 us, 110 with the padding last).  With peers the senders serve them
  // first, and receivers, whose rows are not here yet, start with it (2 ranks x 1024 tokens of 7168 over 64 experts, emulated in
  // one launch: 74 us, 98 with the padding first everywhere).
  if constexpr (kPieces) pad();

  if (sender) {
    // ================================================================ sender
    int ok = 1;
    if (lane < P) ok = wait_flag_ge(&ctl->disp_ack[lane], epoch - 1, ctx, kOpDispatch, 0, lane);
    bool alive = __all_sync(0xffffffffu, ok) && !aborted;
    clk.mark(kProfWait);
    // a work item is a group of tokens, or a column piece of one token when no peer waits for flags
    const int Lx = a.E / P, per_item = kPieces ? 1 : kGroupTokens, pieces = kPieces ? p.pieces : 1;
    const int ngroups = (a.T + per_item - 1) / per_item * pieces;
    const int per_piece = kPieces ? ((units + pieces - 1) / pieces + 31) / 32 * 32 : units;   // 16-byte pieces of an output row
    const uint8_t* x = reinterpret_cast<const uint8_t*>(a.x);
    const int src_row_bytes = a.mode == kDispatchFp8Given ? H : H * 2;
    uint8_t* recv_x = reinterpret_cast<uint8_t*>(a.recv_x);
    const int my_first_row = (p.local_direct && !a.expand) ? a.rank_rows[me] : 0;
    // groups are handed out in order by a shared counter, so the warps stay busy whatever the groups' sizes
    int ticket = next_ticket(&ctl->ticket[kOpDispatch][0], lane);
    while (ticket < ngroups && alive) {
      const int gi = ticket, t0 = gi / pieces * per_item, count = min(a.T - t0, per_item);
      const int u_begin = kPieces ? min(units, gi % pieces * per_piece) : 0, u_count = kPieces ? min(units - u_begin, per_piece) : units;
      // its round trip overlaps this item; with peers a warp takes no group while it still sends one
      if constexpr (kPieces) ticket = next_ticket(&ctl->ticket[kOpDispatch][0], lane);
      // routing of the whole group in one round of loads: lane (q, c) holds send_slot[t0 + q][c] and the local output rows
      // of slots c and c + 8 of token t0 + q (-1: the slot's expert lives elsewhere)
      int ss = -1, sr0 = -1, sr1 = -1;
      if (q < count) {
        const int t = t0 + q;
        if (c < P) ss = a.send_slot[(size_t)t * P + c];
        if (p.local_direct && a.expand) {
          if (c < K) {
            const int r = a.slot_row[(size_t)t * K + c];
            const long long e = a.topk_idx[(size_t)t * K + c];
            if (r >= 0 && e >= 0 && e < a.E && (int)(e / Lx) == me) sr0 = r;
          }
          if (c + 8 < K) {
            const int r = a.slot_row[(size_t)t * K + c + 8];
            const long long e = a.topk_idx[(size_t)t * K + c + 8];
            if (r >= 0 && e >= 0 && e < a.E && (int)(e / Lx) == me) sr1 = r;
          }
        }
      }
      clk.mark(kProfMeta);
      for (int qq = 0; qq < count; ++qq) {
        const int t = t0 + qq;
        // lanes 0..P-1: the staged row on every destination rank; lanes P..P+K-1: the output rows on this rank
        const int j = __shfl_sync(0xffffffffu, ss, qq * 8 + (lane & 7));
        const int j_me = __shfl_sync(0xffffffffu, ss, qq * 8 + me);
        const int k = lane - P;
        const int r0 = __shfl_sync(0xffffffffu, sr0, qq * 8 + (k & 7)), r1 = __shfl_sync(0xffffffffu, sr1, qq * 8 + (k & 7));
        unsigned long long dst = 0, dst_sf = 0;
        if (lane < P) {
          if (j >= 0 && !(p.local_direct && lane == me) && DEP_INDEX_OK(ctx, j, Tmax, kOpDispatch, 0)) {
            dst = reinterpret_cast<unsigned long long>(ctx.ws[lane] + lay.stage + ((size_t)me * Tmax + j) * lay.stage_row_bytes);
            dst_sf = dst + H;
          }
        } else if (p.local_direct && k < K) {
          int row = -1;
          if (a.expand) row = k < 8 ? r0 : r1;
          else if (k == 0 && j_me >= 0) row = my_first_row + j_me;
          if (row >= 0 && (a.recv_rows <= 0 || DEP_INDEX_OK(ctx, row, a.recv_rows, kOpDispatch, 1))) {
            dst = reinterpret_cast<unsigned long long>(recv_x + (size_t)row * row_bytes);
            dst_sf = reinterpret_cast<unsigned long long>(a.recv_sf + (size_t)row * nsf);
          }
        }
        const unsigned mask = __ballot_sync(0xffffffffu, dst != 0);
        if (mask == 0) continue;
        const uint8_t* src = x + (size_t)t * src_row_bytes;
        if (a.mode == kDispatchFp8Fused) {
          warp_quant_fanout(reinterpret_cast<const int4*>(src) + 2 * u_begin, u_count * 16, dst + (size_t)u_begin * 16,
                            dst_sf + (size_t)u_begin / 2, mask, lane);      // 8 pieces of codes share a 4-byte scale
        } else {
          warp_fanout<false>(reinterpret_cast<const int4*>(src) + u_begin, u_count, dst + (size_t)u_begin * 16, mask, lane);
          if (fp8 && u_begin == 0) warp_fanout_f32<false>(a.x_sf + (size_t)t * nsf, nsf, dst_sf, mask, lane);
        }
        if (u_begin == 0) clk.add_rows(__popc(mask));      // a row counts once, with its first piece
      }
      clk.mark(kProfData);
      // publish the group: every lane's stores are ordered before the flag by the warp barrier + release
      __syncwarp();
      if (!kPieces && lane < P && !(p.local_direct && lane == me))
        st_release_sys(reinterpret_cast<unsigned long long*>(ctx.ws[lane] + lay.disp_flag) + (size_t)me * NG + gi, epoch);
      clk.mark(kProfPublish);
      if constexpr (!kPieces) ticket = next_ticket(&ctl->ticket[kOpDispatch][0], lane);
    }
  }
  if constexpr (!kPieces) pad();
  {
    // ================================================================ receiver (sender warps join once all groups are sent)
    uint8_t* recv_x = reinterpret_cast<uint8_t*>(a.recv_x);
    const uint8_t* stage = ctx.ws[me] + lay.stage;
    const unsigned long long* flags = reinterpret_cast<const unsigned long long*>(ctx.ws[me] + lay.disp_flag);
    // the sources whose rows pass through the staging area: all ranks, or all but this one
    const int S = aborted ? 0 : p.local_direct ? P - 1 : P, first = p.local_direct ? 1 : 0;
    int max_nb = 0;
    for (int s = 0; s < S; ++s) {
      const int r = (me + first + s) % P;
      max_nb = max(max_nb, (a.rank_rows[r + 1] - a.rank_rows[r] + kRowBlock - 1) / kRowBlock);
    }
    // items are blocks of kRowBlock staged rows, block b of every source before block b + 1 of any: the order in which
    // the senders, which all walk their tokens front to back, complete them
    for (int item = next_ticket(&ctl->ticket[kOpDispatch][1], lane); item < max_nb * S;
         item = next_ticket(&ctl->ticket[kOpDispatch][1], lane)) {
      const int r = (me + first + item % S) % P, j0 = (item / S) * kRowBlock;
      const int rows_r = min(a.rank_rows[r + 1] - a.rank_rows[r], Tmax), T_r = a.rank_tokens[r];
      if (j0 >= rows_r) continue;
      const int cnt = min(kRowBlock, rows_r - j0);
      // the block's records in one round of loads: lane (q, c) holds fields c, 8 + c, 16 + c of record j0 + q
      int f0 = 0, f1 = 0, f2 = 0;
      if (q < cnt) {
        const int* rec = a.stage_meta + ((size_t)r * Tmax + j0 + q) * a.meta_stride;
        if (c < a.meta_stride) f0 = rec[c];
        if (8 + c < a.meta_stride) f1 = rec[8 + c];
        if (16 + c < a.meta_stride) f2 = rec[16 + c];
      }
      clk.mark(kProfMeta);
      int waited = -1;
      bool alive = true;
      for (int qq = 0; qq < cnt && alive; ++qq) {
        const int j = j0 + qq;
        const int t = __shfl_sync(0xffffffffu, f0, qq * 8);
        if (t < 0 || t >= T_r) {   // a record names the source token whose flag covers it: the plan is damaged
          if (lane == 0) report_failure(ctx, kStatusBadArgument, kOpDispatch, 3, r, T_r, (unsigned long long)(unsigned)t);
          alive = false;
          break;
        }
        if (t / kGroupTokens != waited) {
          waited = t / kGroupTokens;
          int ok = 1;
          if (lane == 0) ok = wait_flag_ge(flags + (size_t)r * NG + waited, epoch, ctx, kOpDispatch, 1, r);
          alive = __shfl_sync(0xffffffffu, ok, 0) != 0;
          clk.mark(kProfWait);
          if (!alive) break;
        }
        const int n = min(__shfl_sync(0xffffffffu, f0, qq * 8 + 1), kMaxTopk);
        const int fi = 2 + lane, from = qq * 8 + (fi & 7);
        const int e0 = __shfl_sync(0xffffffffu, f0, from), e1 = __shfl_sync(0xffffffffu, f1, from), e2 = __shfl_sync(0xffffffffu, f2, from);
        unsigned long long dst = 0, dst_sf = 0;
        if (lane < n) {
          const int row = ((fi >> 3) == 0 ? e0 : (fi >> 3) == 1 ? e1 : e2) & kRowMask;
          if (a.recv_rows <= 0 || DEP_INDEX_OK(ctx, row, a.recv_rows, kOpDispatch, 1)) {
            dst = reinterpret_cast<unsigned long long>(recv_x + (size_t)row * row_bytes);
            dst_sf = reinterpret_cast<unsigned long long>(a.recv_sf + (size_t)row * nsf);
          }
        }
        const unsigned mask = __ballot_sync(0xffffffffu, dst != 0);
        const uint8_t* src = stage + ((size_t)r * Tmax + j) * lay.stage_row_bytes;
        warp_fanout<true>(reinterpret_cast<const int4*>(src), units, dst, mask, lane);
        if (fp8) warp_fanout_f32<true>(reinterpret_cast<const float*>(src + H), nsf, dst_sf, mask, lane);
        clk.add_rows(__popc(mask));
        clk.mark(kProfData);
      }
      if (!alive) break;
    }
  }

  clk.finish(a.prof ? a.prof + (size_t)blockIdx.x * kDispatchProfWords : nullptr, sender ? 0 : 1);

  // ---- exit: the last block of this rank tells every source that its staged rows are consumed
  if (last_block_of_rank(ctl, kOpDispatch, gridDim.x)) {
    if (!ld_volatile_int(&ctl->abort) && threadIdx.x < P)
      st_release_sys(&control_of(ctx.ws[threadIdx.x])->disp_ack[me], epoch);
    if (threadIdx.x == 0) { ctl->ticket[kOpDispatch][0] = 0; ctl->ticket[kOpDispatch][1] = 0; ctl->epoch[kOpDispatch] = epoch; }
  }
}

// One rank without a budget of SMs: no peer waits for a flag and no block for another, so every warp takes one piece of a token
// (2 KB of a bf16 row) and is done, and the hardware deals the blocks out.  Written bytes bound it, and a loop over many pieces per
// warp is slower at that whatever its items: SMs write at different speeds, and the slowest one ends last (4096 rows of 14 KB stored
// eight times each, stand-alone: 86 to 88 us in pieces of 1 to 2 KB with 64 to 512 threads per block, 97 to 100 us as 148 blocks of
// 512 threads that stride over the pieces, with plain, streaming or bulk stores alike; kernel above with tickets 94 us).
// The first p.pad_blocks blocks zero the padding rows.
constexpr int kLocalDispatchThreads = 256;
constexpr int kLocalUnroll = 4;       // 16-byte pieces per lane and item

__global__ void __launch_bounds__(kLocalDispatchThreads) ep_dispatch_local_kernel(const __grid_constant__ DispatchParams p) {
  const DispatchArgs& a = p.r[0];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = kLocalDispatchThreads / 32, H = p.lay.hidden, K = a.K;
  Control* ctl = control_of(a.ctx.ws[0]);
  const bool aborted = ld_volatile_int(&ctl->abort) != 0;   // an earlier call gave up, the plan's tensors may never have been written
  const bool fp8 = a.mode != kDispatchBf16;
  const int nsf = fp8 ? H / 128 : 0, row_bytes = fp8 ? H : H * 2, units = row_bytes / 16;
  if (blockIdx.x == 0 && threadIdx.x == 0) {                // nothing else in this kernel reads the epoch
    const unsigned long long epoch = ctl->epoch[kOpDispatch] + 1;
    if (!aborted) ctl->disp_ack[0] = epoch;
    ctl->epoch[kOpDispatch] = epoch;
  }
  if (aborted) return;
  if ((int)blockIdx.x < p.pad_blocks) {
    zero_padding(a, a.E, row_bytes, nsf, warp * p.pad_blocks + blockIdx.x, p.pad_blocks * nwarps, lane);
    return;
  }
  const int item = ((int)blockIdx.x - p.pad_blocks) * nwarps + warp, t = item / p.pieces, piece = item - t * p.pieces;
  if (t >= a.T) return;
  const int per_piece = ((units + p.pieces - 1) / p.pieces + 31) / 32 * 32, u_begin = min(units, piece * per_piece);
  const int u_count = min(units - u_begin, per_piece);
  const uint8_t* src = reinterpret_cast<const uint8_t*>(a.x) + (size_t)t * (a.mode == kDispatchFp8Given ? H : H * 2);
  // lane k: the output row of slot k (rank layout: lane 0, the token's one row)
  int row = -1;
  if (a.expand) { if (lane < K) row = __ldg(a.slot_row + (size_t)t * K + lane); }
  else if (lane == 0) row = __ldg(a.send_slot + t);
  if (row >= 0 && a.recv_rows > 0 && !DEP_INDEX_OK(a.ctx, row, a.recv_rows, kOpDispatch, 1)) row = -1;
  const unsigned mask = __ballot_sync(0xffffffffu, row >= 0);
  if (mask == 0) return;
  const unsigned long long dst = reinterpret_cast<unsigned long long>(reinterpret_cast<uint8_t*>(a.recv_x) + (long long)row * row_bytes);
  const unsigned long long dst_sf = reinterpret_cast<unsigned long long>(a.recv_sf + (long long)row * nsf);
  if (a.mode == kDispatchFp8Fused) {
    warp_quant_fanout(reinterpret_cast<const int4*>(src) + 2 * u_begin, u_count * 16, dst + (size_t)u_begin * 16,
                      dst_sf + (size_t)u_begin / 2, mask, lane);      // 8 pieces of codes share a 4-byte scale
  } else {
    warp_fanout<false, kLocalUnroll>(reinterpret_cast<const int4*>(src) + u_begin, u_count, dst + (size_t)u_begin * 16, mask, lane);
    if (fp8 && piece == 0) warp_fanout_f32<false>(a.x_sf + (size_t)t * nsf, nsf, dst_sf, mask, lane);
  }
}

cudaError_t launch_dispatch(const DispatchParams& params, int nranks, cudaStream_t stream) {
  DispatchParams p = params;
  if (p.lay.hidden > 8192) return cudaErrorInvalidValue;   // the fused quantiser keeps at most 64 scales per row in registers
  p.pieces = 0;
  if (p.lay.world == 1 && nranks == 1 && p.local_direct && p.whole_gpu && !p.profile) {
    const DispatchArgs& a = p.r[0];
    const int units = (a.mode == kDispatchBf16 ? 2 : 1) * p.lay.hidden / 16, warps = kLocalDispatchThreads / 32;
    p.pieces = (units + 32 * kLocalUnroll - 1) / (32 * kLocalUnroll);
    p.pad_blocks = a.pad_offsets ? std::min(592, (a.recv_rows + warps - 1) / warps) : 0;      // 592: four blocks per SM
    const long long blocks = p.pad_blocks + ((long long)a.T * p.pieces + warps - 1) / warps;
    ep_dispatch_local_kernel<<<(unsigned)std::max(1ll, blocks), kLocalDispatchThreads, 0, stream>>>(p);
    return cudaGetLastError();
  }
  if (p.lay.world == 1 && p.local_direct) {
    // No peer waits for a group's flag, so the items can be as small as balances the warps.  4096 rows of 14 KB stored eight times
    // each by 144 blocks: 101 us in whole rows, 98 in halves, 93 in quarters (a quarter is what a warp holds in registers);
    // with a single destination per row (rank layout) a quarter is too little work for its records, two items per warp do.
    const int units = (p.r[0].mode == kDispatchBf16 ? 2 : 1) * p.lay.hidden / 16, warps = (p.send_blocks + p.recv_blocks) * (kDispatchThreads / 32);
    const int wanted = std::max(p.r[0].expand ? 4 : 1, 2 * warps / std::max(1, p.r[0].T));
    const int per_piece = std::max(64, ((units + wanted - 1) / wanted + 31) / 32 * 32);
    p.pieces = (units + per_piece - 1) / per_piece;
  }
  dim3 grid(p.send_blocks + p.recv_blocks, nranks), block(kDispatchThreads);
  void* args[] = {const_cast<DispatchParams*>(&p)};
  const void* fn = p.pieces > 0 ? (p.profile ? (const void*)ep_dispatch_ht_kernel<true, true> : (const void*)ep_dispatch_ht_kernel<false, true>)
                                : (p.profile ? (const void*)ep_dispatch_ht_kernel<true, false> : (const void*)ep_dispatch_ht_kernel<false, false>);
  return cudaLaunchCooperativeKernel(fn, grid, block, args, 0, stream);
}

}  // namespace dep
