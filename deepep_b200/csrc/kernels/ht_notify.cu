// ep_notify: routing layout of one dispatch, computed identically on every rank.
//
// Design (differs from the reference's 47-phase notify, csrc/kernels/notify/notify.cpp:1426-1970,
// which exchanges count tables, forward packets and backward packets in three rounds):
// on one NVSwitch domain the routing table itself is tiny, so every rank pushes its
// [T, K] expert ids and weights to every peer once (P2P stores + one release flag per
// peer), and each rank then derives *all* metadata locally from the gathered table:
//   - per-(source, expert) counts  -> expert row offsets, ordered (expert, source, token, slot)
//   - rank-level dedup             -> one staged row per (source token, destination rank)
//   - receive-side expansion lists -> stage_meta[(source, staged row)] = rows to materialise
// Offsets come from prefix sums over 64-token tiles (bit masks + popcounts), never from
// atomics, so the layout is deterministic and equal to the CPU oracle bit for bit.
//
// The pass moves next to nothing; a chain of short phases between grid barriers bounds it, so each phase is cut over all
// threads: one thread per (token, slot) reads a tile's ids once into shared memory, and the same tile serves the counts
// and the records when every block has one.  One rank on one GPU, before it had a kernel of its own, 1531 x 6 routes over 64
// experts: 37.7 us with one thread per token, 20.9 us since; 4096 x 8 over 256 experts in blocks of 128 rows: 78.9 us (one block
// wrote all padding marks), 26.9 us.
#include <cooperative_groups.h>

#include <algorithm>

#include "api.h"
#include "local_tile.cuh"

namespace cg = cooperative_groups;

namespace dep {

constexpr int kNotifyThreads = 256;

struct TileMasks {
  unsigned expert[kMaxExperts][2];   // bit t: token t of the tile routes to this expert
  unsigned rank[kMaxRanks][2];       // bit t: token t of the tile routes to this rank
};

__device__ __forceinline__ int below(const unsigned m[2], int tl) {
  unsigned lo = tl < 32 ? ((1u << tl) - 1u) : 0xffffffffu;
  unsigned hi = tl < 32 ? 0u : ((1u << (tl - 32)) - 1u);
  return __popc(m[0] & lo) + __popc(m[1] & hi);
}

// One tile of a source's table: its ids, which slots count (id in range, no earlier slot of the token names the same
// expert), which of them live on this rank, and the masks.
struct Tile {
  TileMasks m;
  int id[kChunkTokens * kMaxTopk];          // [token of the tile][slot]
  unsigned valid[kChunkTokens];             // bit k: slot k counts
  unsigned local[kChunkTokens];             // bit k: slot k counts and its expert lives on this rank
};

// One thread per (token, slot): the ids are fetched once, coalesced, and all further work reads shared memory.
// `own` (may be null): the caller's int64 table, read in place of the gathered one for this rank's own tokens.
__device__ void load_tile(Tile& s, const int* table, const long long* own, int tile, int T_r, int K, int E, int Lx, int me) {
  const int first = tile * kChunkTokens, n = min(kChunkTokens, T_r - first) * K;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const size_t at = (size_t)first * K + i;
    const long long v = own ? __ldg(own + at) : (long long)__ldcg(table + at);
    s.id[i] = (v < 0 || v >= E) ? -1 : (int)v;
  }
  for (int i = threadIdx.x; i < E * 2; i += blockDim.x) (&s.m.expert[0][0])[i] = 0u;
  if (threadIdx.x < kMaxRanks * 2) (&s.m.rank[0][0])[threadIdx.x] = 0u;
  if (threadIdx.x < kChunkTokens) { s.valid[threadIdx.x] = 0u; s.local[threadIdx.x] = 0u; }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int tl = i / K, k = i - tl * K, e = s.id[i];
    bool counts = e >= 0;
    for (int j = i - k; j < i; ++j) counts = counts && s.id[j] != e;
    if (counts) {
      const int d = e / Lx;
      atomicOr(&s.m.expert[e][tl >> 5], 1u << (tl & 31));
      atomicOr(&s.m.rank[d][tl >> 5], 1u << (tl & 31));
      atomicOr(&s.valid[tl], 1u << k);
      if (d == me) atomicOr(&s.local[tl], 1u << k);
    }
  }
  __syncthreads();
}

template <bool kProfile>
__global__ void __launch_bounds__(kNotifyThreads) ep_notify_kernel(const __grid_constant__ NotifyParams p) {
  cg::grid_group grid = cg::this_grid();
  const NotifyArgs& a = p.r[blockIdx.y];
  const WsLayout& lay = p.lay;
  const RankCtx& ctx = a.ctx;
  const int P = ctx.world, me = ctx.rank, K = a.K, E = a.E, Lx = E / P, Tmax = lay.max_tokens;
  const int NT = (Tmax + kChunkTokens - 1) / kChunkTokens;
  uint8_t* ws = ctx.ws[me];
  Control* ctl = control_of(ws);
  const unsigned long long epoch = ctl->epoch[kOpNotify] + 1;
  const int gtid = blockIdx.x * blockDim.x + threadIdx.x, gstride = gridDim.x * blockDim.x;

  __shared__ Tile s_tile;
  TileMasks& s_m = s_tile.m;
  __shared__ int s_T[kMaxRanks];
  __shared__ int s_rank_base[kMaxRanks + 1];
  __shared__ int s_off[kMaxExperts];
  __shared__ int s_base[kMaxExperts];                   // scratch: totals, then per-task row bases
  __shared__ int s_rows;

  // profile instantiation only: phase stamps of block 0 (nanoseconds since kernel start) in Control::dbg[16..23]
  unsigned long long t_start = 0;
  if constexpr (kProfile) t_start = global_timer_ns();
  auto stamp = [&](int i) {
    if constexpr (kProfile)
      if (blockIdx.x == 0 && threadIdx.x == 0) ctl->dbg[16 + i] = global_timer_ns() - t_start;
  };

  // ---- A: publish my routing table into every peer (after they consumed the previous one).  My own tokens are read from
  // the caller's tensors.
  int ok = 1;
  if (threadIdx.x < P) ok = wait_flag_ge(&ctl->notify_ack[threadIdx.x], epoch - 1, ctx, kOpNotify, 0, threadIdx.x);
  int alive = __syncthreads_and(ok);
  if (alive) {
    const int n = a.T * K;
    for (int i = gtid; i < (P - 1) * n; i += gstride) {
      const int q = i / n, j = i - q * n, d = (me + 1 + q) % P;
      long long v = a.topk_idx[j];
      int e = (v < 0 || v >= E) ? -1 : (int)v;
      reinterpret_cast<int*>(ctx.ws[d] + lay.gather_idx)[(size_t)me * Tmax * K + j] = e;
      if (a.topk_w) reinterpret_cast<float*>(ctx.ws[d] + lay.gather_w)[(size_t)me * Tmax * K + j] = a.topk_w[j];
    }
    if (blockIdx.x == 0 && threadIdx.x < P) {
      int* hdr = reinterpret_cast<int*>(ctx.ws[threadIdx.x] + lay.gather_hdr) + me * 4;
      hdr[0] = a.T;
      hdr[1] = a.topk_w != nullptr;
    }
    __threadfence_system();
  }
  grid.sync();
  if (alive && blockIdx.x == 0 && threadIdx.x < P)
    st_release_sys(&control_of(ctx.ws[threadIdx.x])->notify_ready[me], epoch);

  stamp(0);
  // ---- B: wait for every rank's table
  const int* ghdr = reinterpret_cast<const int*>(ws + lay.gather_hdr);
  const int* gidx = reinterpret_cast<const int*>(ws + lay.gather_idx);
  const float* gw = reinterpret_cast<const float*>(ws + lay.gather_w);
  ok = 1;
  if (alive && threadIdx.x < P) ok = wait_flag_ge(&ctl->notify_ready[threadIdx.x], epoch, ctx, kOpNotify, 1, threadIdx.x);
  alive = __syncthreads_and(ok) && alive;
  if (threadIdx.x < kMaxRanks) s_T[threadIdx.x] = (alive && threadIdx.x < P) ? __ldcg(ghdr + threadIdx.x * 4) : 0;
  __syncthreads();
  const bool has_w = alive && a.recv_w != nullptr && __ldcg(ghdr + 1) != 0;
  // the ids and weights of source r: this rank's own come from the caller's tensors
  auto own_ids = [&](int r) { return r == me ? a.topk_idx : nullptr; };
  auto weight_of = [&](int r, int i) {
    if (!has_w) return 0.f;
    return r == me ? (a.topk_w ? __ldg(a.topk_w + i) : 0.f) : __ldcg(gw + (size_t)r * Tmax * K + i);
  };

  stamp(1);
  // ---- C: per-(source, tile) histograms
  for (int task = blockIdx.x; task < P * NT; task += gridDim.x) {
    int r = task / NT, tile = task - r * NT;
    if (tile * kChunkTokens >= s_T[r]) continue;
    load_tile(s_tile, gidx + (size_t)r * Tmax * K, own_ids(r), tile, s_T[r], K, E, Lx, me);
    for (int e = threadIdx.x; e < E; e += blockDim.x)
      a.hist[(size_t)task * E + e] = __popc(s_m.expert[e][0]) + __popc(s_m.expert[e][1]);
    if (threadIdx.x == 0) a.hits[task] = __popc(s_m.rank[me][0]) + __popc(s_m.rank[me][1]);
    if (a.rank_matrix && threadIdx.x < P)
      atomicAdd(&a.rank_matrix[r * P + threadIdx.x], __popc(s_m.rank[threadIdx.x][0]) + __popc(s_m.rank[threadIdx.x][1]));
    if (r == me && threadIdx.x < P)
      a.own_hits[tile * P + threadIdx.x] = __popc(s_m.rank[threadIdx.x][0]) + __popc(s_m.rank[threadIdx.x][1]);
    __syncthreads();
  }
  grid.sync();
  // a block whose wait ran out has counted nothing: all blocks give up together and leave an empty plan
  if (__syncthreads_or(threadIdx.x == 0 && ld_volatile_int(&ctl->abort))) {
    alive = 0;
    if (threadIdx.x < kMaxRanks) s_T[threadIdx.x] = 0;
    __syncthreads();
  }

  stamp(2);
  // ---- D1: exclusive scans over tiles
  {   // one warp per (source, expert): the lanes take 32 tiles at a time, exclusive prefix by a warp scan
    const int lane_ = threadIdx.x & 31;
    for (int i = gtid >> 5; i < P * E; i += gstride >> 5) {
      const int r = i / E, e = i - r * E, nt = (s_T[r] + kChunkTokens - 1) / kChunkTokens;
      int run = 0;
      for (int tile0 = 0; tile0 < nt; tile0 += 32) {
        const int tile = tile0 + lane_;
        int* cell = a.hist + ((size_t)r * NT + tile) * E + e;
        const int v = tile < nt ? *cell : 0;
        int incl = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int o = __shfl_up_sync(0xffffffffu, incl, d);
          if (lane_ >= d) incl += o;
        }
        if (tile < nt) *cell = run + incl - v;
        run += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane_ == 0) a.cnt[i] = run;
    }
  }
  {   // staged-row starts of every (source, chunk) and my own per-destination starts: one warp each, same warp scan
    const int w = gtid >> 5, lane_ = threadIdx.x & 31;
    if (w < 2 * P) {
      const bool own = w >= P;
      const int r = own ? me : w, d = w - P, nt = (s_T[r] + kChunkTokens - 1) / kChunkTokens;
      int run = 0;
      for (int tile0 = 0; tile0 < nt; tile0 += 32) {
        const int tile = tile0 + lane_;
        const int v = tile < nt ? (own ? a.own_hits[tile * P + d] : a.hits[r * NT + tile]) : 0;
        int incl = v;
#pragma unroll
        for (int q = 1; q < 32; q <<= 1) {
          const int o = __shfl_up_sync(0xffffffffu, incl, q);
          if (lane_ >= q) incl += o;
        }
        if (tile < nt) {
          if (own) {
            a.own_hits[tile * P + d] = run + incl - v;
            if (a.send_prefix) a.send_prefix[d * max(nt, 1) + tile] = run + incl - v;
          } else a.chunk_start[r * (NT + 1) + tile] = run + incl - v;
        }
        run += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (own && nt == 0 && lane_ == 0 && a.send_prefix) a.send_prefix[d] = 0;
      if (!own)
        for (int tile = nt + lane_; tile <= NT; tile += 32) a.chunk_start[r * (NT + 1) + tile] = run;
    }
  }
  grid.sync();

  stamp(3);
  // ---- D2: expert row offsets of every rank (each block keeps its own copy in shared memory)
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int tot = 0;
    for (int r = 0; r < P; ++r) tot += a.cnt[r * E + e];
    s_base[e] = tot;                                      // total rows of expert e (all sources)
  }
  __syncthreads();
  if ((threadIdx.x >> 5) < P) {    // warp d: aligned exclusive prefix over the local experts of rank d
    const int d = threadIdx.x >> 5, lane_ = threadIdx.x & 31;
    int run = 0;
    for (int l0 = 0; l0 < Lx; l0 += 32) {
      const int l = l0 + lane_, e = d * Lx + l;
      const int tot = l < Lx ? s_base[e] : 0;
      const int al = a.expand ? (tot + a.alignment - 1) / a.alignment * a.alignment : tot;
      int incl = al;
#pragma unroll
      for (int q = 1; q < 32; q <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, incl, q);
        if (lane_ >= q) incl += o;
      }
      if (l < Lx) {
        s_off[e] = run + incl - al;
        if (d == me && blockIdx.x == 0) { a.expert_counts[l] = tot; a.expert_offsets[l] = run + incl - al; }
      }
      run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (d == me && lane_ == 0) { s_rows = run; if (blockIdx.x == 0) a.expert_offsets[Lx] = run; }
  }
  if (threadIdx.x == 0) {
    int run = 0;
    for (int r = 0; r < P; ++r) { s_rank_base[r] = run; run += a.chunk_start[r * (NT + 1) + NT]; }
    s_rank_base[P] = run;
  }
  __syncthreads();
  if (!a.expand && threadIdx.x == 0) s_rows = s_rank_base[P];
  __syncthreads();
  if (blockIdx.x == 0) {
    if (threadIdx.x <= P) a.rank_rows[threadIdx.x] = s_rank_base[threadIdx.x];
    if (threadIdx.x < P) a.rank_tokens[threadIdx.x] = s_T[threadIdx.x];
    if (a.rank_matrix && threadIdx.x < P * P) {
      int run = 0;
      for (int i = threadIdx.x % P; i <= (int)threadIdx.x; i += P) run += a.rank_matrix[i];
      a.rank_prefix[threadIdx.x] = run;
    }
  }
  if (a.expand && a.alignment > 1) {    // padding rows carry no source; the experts are dealt out to the blocks
    for (int l = blockIdx.x; l < Lx; l += gridDim.x) {
      const int e = me * Lx + l, end = (l + 1 < Lx) ? s_off[e + 1] : s_rows;
      for (int row = s_off[e] + s_base[e] + threadIdx.x; row < end && row < a.rcap; row += blockDim.x) {
        a.recv_row_src[row] = -1;
        if (a.recv_w) a.recv_w[row] = 0.f;
      }
    }
    __syncthreads();                    // s_base is about to be reused
  }

  stamp(4);
  // ---- E: per-token records, one thread per (token, slot)
  const bool one_each = P * NT <= (int)gridDim.x;       // every block has one tile at most: phase C left it in shared memory
  for (int task = blockIdx.x; task < P * NT; task += gridDim.x) {
    const int r = task / NT, tile = task - r * NT, T_r = s_T[r];
    if (tile * kChunkTokens >= T_r) continue;
    if (!one_each) load_tile(s_tile, gidx + (size_t)r * Tmax * K, own_ids(r), tile, T_r, K, E, Lx, me);
    {   // first row of expert e for this (source, tile): the expert's block, then earlier sources, then earlier tiles
      const int* hist_task = a.hist + (size_t)task * E;
      for (int e = threadIdx.x; e < E; e += blockDim.x) {
        int b = hist_task[e];
        for (int q = 0; q < r; ++q) b += a.cnt[q * E + e];
        s_base[e] = s_off[e] + b;
      }
      __syncthreads();
    }
    const int t0 = tile * kChunkTokens, live = min(kChunkTokens, T_r - t0);
    const int j0 = a.chunk_start[r * (NT + 1) + tile];  // staged rows of this source before the tile
    for (int i = threadIdx.x; i < live * K; i += blockDim.x) {
      const int tl = i / K, k = i - tl * K, e = s_tile.id[i];
      const unsigned local = s_tile.local[tl];
      const bool counts = (s_tile.valid[tl] >> k) & 1u, here = (local >> k) & 1u;
      const int row = a.expand && counts && (here || r == me) ? s_base[e] + below(s_m.expert[e], tl) : -1;
      if (r == me) a.slot_row[(size_t)t0 * K + i] = row;
      if (local == 0) continue;                         // no slot of the token lives on this rank
      const int j = j0 + below(s_m.rank[me], tl);
      if (a.expand) {
        if (here) {
          a.stage_meta[((size_t)r * Tmax + j) * a.meta_stride + 2 + __popc(local & ((1u << k) - 1u))] = row | (k << kRowSlotShift);
          if (row < a.rcap) {
            a.recv_row_src[row] = (r * Tmax + t0) * K + i;
            if (a.recv_w) a.recv_w[row] = weight_of(r, t0 * K + i);
          }
        }
      } else {
        const long long out = (long long)s_rank_base[r] + j;
        if (out < a.rcap) {
          if (k == 0) {
            a.recv_row_src[out] = (r * Tmax + t0 + tl) * K;
            if (a.recv_src) a.recv_src[out] = t0 + tl;
          }
          if (a.recv_idx) a.recv_idx[(size_t)out * K + k] = here ? e - me * Lx : -1;
          if (a.recv_w) a.recv_w[(size_t)out * K + k] = here ? weight_of(r, t0 * K + i) : 0.f;
        }
      }
    }
    for (int tl = threadIdx.x; tl < live; tl += blockDim.x) {
      const unsigned local = s_tile.local[tl];
      if (local == 0) continue;
      const int j = j0 + below(s_m.rank[me], tl);
      int* rec = a.stage_meta + ((size_t)r * Tmax + j) * a.meta_stride;
      rec[0] = t0 + tl;
      rec[1] = a.expand ? __popc(local) : 1;
      if (!a.expand) { rec[2] = s_rank_base[r] + j; rec[3] = (int)local; }   // which slots of the token live on this rank
    }
    if (r == me)
      for (int i = threadIdx.x; i < live * P; i += blockDim.x) {
        const int tl = i / P, d = i - tl * P;
        const bool hit = (s_m.rank[d][tl >> 5] >> (tl & 31)) & 1u;
        a.send_slot[(size_t)t0 * P + i] = hit ? a.own_hits[tile * P + d] + below(s_m.rank[d], tl) : -1;
      }
    __syncthreads();
  }
  __threadfence();
  grid.sync();

  stamp(5);
  // ---- F: release the gathered table, publish counts to the host, advance the epoch
  if (blockIdx.x == 0) {
    if (threadIdx.x < P) st_release_sys(&control_of(ctx.ws[threadIdx.x])->notify_ack[me], epoch);
    if (a.mailbox) {
      for (int l = threadIdx.x; l < Lx; l += blockDim.x) a.mailbox[4 + l] = a.expert_counts[l];
      __threadfence_system();
      __syncthreads();
      if (threadIdx.x == 0) {
        int maxT = 0;
        for (int r = 0; r < P; ++r) maxT = max(maxT, s_T[r]);
        a.mailbox[0] = alive ? s_rows : -1;
        a.mailbox[1] = s_rank_base[P];
        a.mailbox[2] = maxT;
        __threadfence_system();
        a.mailbox[3] = a.seq ? a.seq : (int)(epoch & 0x7fffffff);
        __threadfence_system();
      }
    }
    if (threadIdx.x == 0) ctl->epoch[kOpNotify] = epoch;
  }
}

// ------------------------------------------------------------------------------------------ one rank
// The same plan for a single rank, by clusters of 16 CTAs.  There is no table to exchange, so what is left is a chain of short steps
// over the own table; the CTAs of a cluster pass their counts through distributed shared memory and meet at cluster barriers, and the
// launch need not be cooperative.  Each CTA owns a range of tokens (whole 64-token tiles), keeps its ids and one bit per (expert,
// token) in shared memory from the first step to the last, and no count passes through memory.  Sixteen SMs would write the records
// of a large table slowly, so several clusters do the first steps alike and each writes its share of every range: clusters never wait
// for one another.  Kernel times as one grid of 128 cooperative blocks (the kernel above) and here: 1531 x 6 routes over 64 experts 20.9
// and 8.0 us, 4096 x 8 over 256 22.7 and 10.6 (13.2 with one cluster), in blocks of 128 rows 26.3 and 10.8, 16384 x 8 over 64 34.9 and
// 16.3 (26.5 with one), 16384 x 16 over 1024 72 and 35 (60 with one, 50 with eight).
constexpr int kLocalNotifyClusters = 4;    // at most, one per 16384 slots: eight do not all fit the GPU at once

template <bool kProfile>
__global__ void __launch_bounds__(kTileThreads) ep_notify_local_kernel(const __grid_constant__ NotifyParams p) {
  cg::cluster_group cluster = cg::this_cluster();
  const NotifyArgs& a = p.r[0];
  constexpr int C = kTileCtas;
  const int c = blockIdx.x % C, share = blockIdx.x / C, shares = gridDim.x / C;
  const int T = a.T, K = a.K, E = a.E, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int per = LocalTile::tokens(T), stride = LocalTile::stride(per);
  const int t0 = min(T, c * per), live = min(per, T - t0), n = live * K;
  const int NT = (p.lay.max_tokens + kChunkTokens - 1) / kChunkTokens;
  extern __shared__ __align__(16) unsigned char smem[];
  const LocalTile s(smem, per, E);
  __shared__ int s_warp[kTileThreads / 32], s_hits[2];
  Control* ctl = control_of(a.ctx.ws[0]);
  unsigned long long t_start = 0;
  if constexpr (kProfile) t_start = global_timer_ns();
  auto stamp = [&](int i) {
    if constexpr (kProfile)
      if (blockIdx.x == 0 && tid == 0) ctl->dbg[16 + i] = global_timer_ns() - t_start;
  };

  // ---- the ids, which tokens every expert gets, and the counts of the other CTAs
  stamp(0);
  s.count(a.topk_idx + (size_t)t0 * K, n, per, K, E);
  stamp(1);
  cluster.sync();
  stamp(2);
  int before, tot;
  s.gather(cluster, c, E, s_hits, before, tot);
  const int rows = tid < E ? (a.expand ? (tot + a.alignment - 1) / a.alignment * a.alignment : tot) : 0;
  const int first = tile_prefix(rows, s_warp);
  if (tid < E) {
    s.tot[tid] = tot; s.off[tid] = first; s.base[tid] = first + before;
    if (tid == E - 1) s.off[E] = first + rows;
    if (blockIdx.x == 0) {
      a.expert_counts[tid] = tot; a.expert_offsets[tid] = first;
      if (a.mailbox) a.mailbox[4 + tid] = tot;
    }
  }
  __syncthreads();
  const int hits_before = s_hits[0], hits = s_hits[1], all_rows = a.expand ? s.off[E] : hits;
  if (blockIdx.x == 0) {
    if (tid == 0) {
      if (a.mailbox) { a.mailbox[0] = all_rows; a.mailbox[1] = hits; a.mailbox[2] = T; }
      a.expert_offsets[E] = s.off[E];
      a.rank_rows[0] = 0; a.rank_rows[1] = hits; a.rank_tokens[0] = T;
      if (a.rank_matrix) {
        a.rank_matrix[0] = a.rank_prefix[0] = hits;
        if (T == 0) a.send_prefix[0] = 0;
      }
    }
    const int nt = (T + kChunkTokens - 1) / kChunkTokens;
    for (int i = nt + tid; i <= NT; i += kTileThreads) a.chunk_start[i] = hits;
    // The last word tells a host that polls it that the counts are there; the records are complete when the launch is.  The fence
    // takes 2 us, which the others spend on the records.
    __syncthreads();
    if (tid == kTileThreads - 1) {
      const unsigned long long epoch = ctl->epoch[kOpNotify] + 1;
      ctl->notify_ack[0] = epoch;
      ctl->epoch[kOpNotify] = epoch;
      if (a.mailbox) {
        __threadfence_system();
        a.mailbox[3] = a.seq ? a.seq : (int)(epoch & 0x7fffffff);
      }
    }
  }
  stamp(3);

  // ---- padding rows carry no source; the experts are dealt out to the CTAs
  const bool has_w = a.recv_w != nullptr && a.topk_w != nullptr;
  if (a.expand && a.alignment > 1)
    for (int e = warp * (int)gridDim.x + blockIdx.x; e < E; e += gridDim.x * (kTileThreads / 32))
      for (int row = s.off[e] + s.tot[e] + lane; row < s.off[e + 1] && row < a.rcap; row += 32) {
        a.recv_row_src[row] = -1;
        if (a.recv_w) a.recv_w[row] = 0.f;
      }

  // ---- per-token records of this cluster's share, one thread per (token, slot)
  const int tokens = (live + shares - 1) / shares, first_token = min(live, share * tokens), last_token = min(live, first_token + tokens);
  for (int i = first_token * K + tid; i < last_token * K; i += kTileThreads) {
    const int tl = i / K, k = i - tl * K, e = s.id[i];
    const unsigned valid = s.valid[tl];
    const bool counts = (valid >> k) & 1u;
    const int row = a.expand && counts ? s.base[e] + LocalTile::below(s.mask + e * stride, tl) : -1;
    a.slot_row[(size_t)t0 * K + i] = row;
    if (valid == 0) continue;
    const int j = hits_before + LocalTile::below(s.hit, tl);
    const float w = has_w && counts ? __ldg(a.topk_w + (size_t)t0 * K + i) : 0.f;
    if (a.expand) {
      if (!counts) continue;
      a.stage_meta[(size_t)j * a.meta_stride + 2 + __popc(valid & ((1u << k) - 1u))] = row | (k << kRowSlotShift);
      if (row < a.rcap) {
        a.recv_row_src[row] = t0 * K + i;
        if (a.recv_w) a.recv_w[row] = w;
      }
    } else if (j < a.rcap) {
      if (k == 0) {
        a.recv_row_src[j] = (t0 + tl) * K;
        if (a.recv_src) a.recv_src[j] = t0 + tl;
      }
      if (a.recv_idx) a.recv_idx[(size_t)j * K + k] = counts ? e : -1;
      if (a.recv_w) a.recv_w[(size_t)j * K + k] = w;
    }
  }
  for (int tl = first_token + tid; tl < last_token; tl += kTileThreads) {
    const unsigned valid = s.valid[tl];
    const int j = hits_before + LocalTile::below(s.hit, tl);
    a.send_slot[t0 + tl] = valid ? j : -1;
    if (tl % kChunkTokens == 0) {
      a.chunk_start[(t0 + tl) / kChunkTokens] = j;
      if (a.send_prefix) a.send_prefix[(t0 + tl) / kChunkTokens] = j;
    }
    if (valid == 0) continue;
    int* rec = a.stage_meta + (size_t)j * a.meta_stride;
    rec[0] = t0 + tl;
    rec[1] = a.expand ? __popc(valid) : 1;
    if (!a.expand) { rec[2] = j; rec[3] = (int)valid; }
  }
  stamp(4);
  cluster.sync();           // nobody reads another CTA's counts any more
  stamp(5);
}

static cudaError_t launch_notify_local(const NotifyParams& p, cudaStream_t stream) {
  const NotifyArgs& a = p.r[0];
  const void* fn = p.profile ? (const void*)ep_notify_local_kernel<true> : (const void*)ep_notify_local_kernel<false>;
  constexpr int kSlots = kTileCtas * kTileThreads;
  const int clusters = std::max(1, std::min(kLocalNotifyClusters, (a.T * a.K + kSlots - 1) / kSlots));
  return launch_tiles(fn, &p, clusters, LocalTile::bytes(LocalTile::tokens(a.T), a.E, a.K), stream);
}

cudaError_t launch_notify(const NotifyParams& p, int nranks, int blocks, cudaStream_t stream) {
  if (p.lay.world == 1 && nranks == 1) return launch_notify_local(p, stream);
  for (int i = 0; i < nranks; ++i) {
    const NotifyArgs& a = p.r[i];
    if (!a.rank_matrix) continue;
    const cudaError_t e = cudaMemsetAsync(a.rank_matrix, 0, sizeof(int) * a.ctx.world * a.ctx.world, stream);
    if (e != cudaSuccess) return e;
  }
  dim3 grid(blocks, nranks), block(kNotifyThreads);
  void* args[] = {const_cast<NotifyParams*>(&p)};
  const void* fn = p.profile ? (const void*)ep_notify_kernel<true> : (const void*)ep_notify_kernel<false>;
  return cudaLaunchCooperativeKernel(fn, grid, block, args, 0, stream);
}

}  // namespace dep
