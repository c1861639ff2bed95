// All-to-all-v fused with a bf16 grouped GEMM: argument blocks and launchers.
//
// Counterpart of the reference's experiments/ep_gmm_fused (csrc/all_to_allv_grouped_mat_mul_udma and
// csrc/grouped_mat_mul_all_to_allv_udma; python ops.py:182-369):
//   a2av_gmm   rows sorted by global expert travel to the expert's rank, which multiplies them by its experts' weights
//   gmm_a2av   the expert rank multiplies its gathered rows by its experts' weights and the results travel back
// Row order on the expert rank: local expert first, source rank second, source order inside a segment.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace dep {

constexpr int kGmmBM = 128;   // rows per accumulator (TMEM lanes); a2av_gmm tiles hold two of them
constexpr int kGmmBN = 256;   // output columns per tile
constexpr int kGmmNarrowBN = 128;   // the same where tiles of 256 columns leave SMs without work
constexpr int kGmmBK = 64;    // K elements per pipeline stage (one 128-byte swizzle row of bf16)
constexpr int kGmmTableInts = 4 + kMaxExperts + 1;   // header (rows, -, -, -) + exclusive prefix of the per-expert row counts

// Byte offsets of the GMM areas inside a workspace (relative to WsLayout::mega); identical on every rank.
struct GmmRegion {
  long long table_a;   // int [kGmmTableInts]   a2av_gmm: where each expert's rows start in this rank's staged x
  long long table_b;   // int [kGmmTableInts]   gmm_a2av: where each expert's rows start in this rank's output
  long long stage;     // bf16 [max_rows][max_k] a2av_gmm: this rank's x, read by the expert ranks
  long long recv;      // bf16 [max_rows][max_n] gmm_a2av: rows returned to this rank, written by the expert ranks
  long long total;
};
__host__ __device__ inline GmmRegion gmm_region(long long max_rows, long long max_k, long long max_n) {
  GmmRegion g;
  long long at = 0;
  auto take = [&](long long b) { long long o = at; at = (at + b + 1023) / 1024 * 1024; return o; };
  g.table_a = take(kGmmTableInts * 4);
  g.table_b = take(kGmmTableInts * 4);
  g.stage = take(max_rows * max_k * 2);
  g.recv = take(max_rows * max_n * 2);
  g.total = at;
  return g;
}

struct GmmArgs {
  RankCtx ctx;
  long long table_off, data_off;   // absolute byte offsets in a workspace: this op's table, its stage / recv area
  const __nv_bfloat16* x;          // a2av_gmm: [rows_in, K] sorted by global expert; gmm_a2av: [rows_in, K] grouped by (local expert, source)
  const void* counts;              // [E] int, or long long (counts64): rows this rank sends to (a2av_gmm) / gets back from (gmm_a2av)
                                   // every global expert, as the caller holds them
  __nv_bfloat16* out;              // a2av_gmm: [out_rows_cap, N] on the expert rank; gmm_a2av: [out_rows_cap, N] on the source rank
  __nv_bfloat16* gathered;         // a2av_gmm: [gathered_cap, K] the all-to-all-v result, A operand of the GEMM
                                   // (single-rank form: a copy for the caller, or null)
  CUtensorMap tmap_a;              // A operand [rows, K] bf16, 3-D with z = 0: box 64 x 128, 128-byte swizzle
  CUtensorMap tmap_b;              // weights [L * K, N] bf16 (N contiguous): box 64 (N) x 64 (K), 128-byte swizzle
  int rows_in, E, K, N;
  int out_rows_cap, gathered_cap, max_tiles, counts64;
  int* tile_info;                  // scratch [max_tiles][4]: local expert, first row, rows, -
  int* num_tiles;                  // [2]: tiles in use, rows on the expert side
  int* pulled;                     // scratch [max_tiles]: rows of each tile that have arrived (a2av_gmm)
  int* error_flag;                 // 1: a pipeline wait ran out; 2: the row counts exceed a capacity or disagree with x
};
struct GmmParams { WsLayout lay; GmmArgs r[kMaxRanks]; };
cudaError_t launch_a2av_gmm(const GmmParams& p, int nranks, int blocks, cudaStream_t stream);
cudaError_t launch_gmm_a2av(const GmmParams& p, int nranks, int blocks, cudaStream_t stream);
// Whether one rank works on tiles of 128 columns instead of 256: `rows` in `row_tiles` tiles of up to 256 rows, the last of `last_rows`.
// Every block decides this from the counts that it lays its tiles out from.  Both widths were timed for 7425 combinations of rows,
// experts, k and n with the weights not in L2; us of a launch in a captured graph, narrow / wide:
//  * Narrow tiles that all start at once (5512 points, 0.60 to 0.91 of the wide ones' time): an SM fills its shared memory with about
//    100 KB/us whatever its neighbours do, and a K step of a narrow tile is 48 KB instead of 64.  8 experts of 256 rows, 2048 x 1536
//    (96 narrow tiles) 20 / 28, 16 of 64 rows, 2048 x 1024 (128) 17 / 22, one of 300 rows, 7168 x 4096 (64) 46 / 71.
//  * A second round of narrow tiles against one of wide tiles: 8 experts of 257 rows, 2048 x 1536 (192) 31 / 28, at k = 7168 88 / 75.
//    Where it holds nothing but short tiles of the last row block, the narrow ones still gain with k up to 2048 (20 points, 0.78 to
//    0.91): one expert of 1025 rows, 2048 x 4096 (160) 25 / 28, of 1100 rows at k = 7168 74 / 73.
//  * More rounds: the wide ones.  They are the faster by more than 5 % at 1013 points behind this line, the narrow ones at 357, most of
//    these three narrow rounds for two wide ones (4 experts of 1100 rows, 2048 x 2048, 39 / 49).
__host__ __device__ inline bool gmm_narrow_tiles(long long row_tiles, long long last_rows, long long rows, long long k, long long n,
                                                 long long blocks) {
  const long long cols = (n + kGmmNarrowBN - 1) / kGmmNarrowBN, tiles = row_tiles * cols;
  const bool short_end = tiles <= blocks + cols && last_rows <= kGmmBM && rows > kGmmBM * row_tiles && k <= 2048;   // some tile is full
  return tiles <= blocks || short_end;
}
// Either op on one rank (world 1) whose x, output, gathered rows and weights do not overlap: p.r[0] with tmap_a over x.
cudaError_t launch_gmm_local(const GmmParams& p, int blocks, cudaStream_t stream);

// Tensor map of bf16 [rows, cols], `cols` contiguous, 128-byte swizzle, box {64 columns, box_rows}.  `shared_rows`: the operand whose
// boxes many blocks load at once, as a 3-D map with a second plane behind the first; boxes are taken at z = 0 alone, nothing of the
// second plane is read.  It is there for the extent that the map states: boxes of a map over less than 128 KB came slowly when 60 blocks
// or more loaded them at once.  8 experts of 1 row, 7168 x 1536, 112 KB of x, by the tensor's address and by the GPU: tiles of
// 128 columns 70 to 81 us, of 256 columns 57 to 86; as planes 41 and 57, like 16 rows (229 KB) either way.
constexpr unsigned long long kGmmMapBytes = 128 * 1024;
bool encode_bf16_map(CUtensorMap* map, const void* base, long long rows, long long cols, int box_rows, bool shared_rows,
                     const char** error);

}  // namespace dep
