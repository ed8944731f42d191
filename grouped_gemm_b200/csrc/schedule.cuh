// Tile schedule shared by the persistent kernel (device) and its host replay.
//
// The reference builds per-expert GEMM problems with a one-block kernel
// (csrc/fill_arguments.cuh:34-98), sorts them by k for wgrad (:80-86) and leaves
// the walk over tiles to CUTLASS' device-only group scheduler.  Here all of it is
// a few integers per CTA: an exclusive prefix sum of batch_sizes (row_start), an
// order of the experts (perm), an exclusive prefix sum of per-expert tile counts
// in that order (tile_start), and pure functions from a position in the launch
// order to (expert, rows, columns, k-range).
#pragma once

#include <stdint.h>

#if defined(__CUDACC__)
#define B200GMM_HD __host__ __device__ __forceinline__
#else
#define B200GMM_HD inline
#endif

namespace b200gmm {

enum Mode : int {
  kNN = 0,  // c[rows_i] = a[rows_i] @ b[i]       (forward)
  kNT = 1,  // c[rows_i] = a[rows_i] @ b[i]^T     (dgrad, or forward with trans_b)
  kTN = 2,  // c[i]      = a[rows_i]^T @ b[rows_i] (wgrad)
};

constexpr int kBlockM = 128;  // output rows per CTA (UMMA M per CTA)
constexpr int kBlockN = 256;  // output tile cols   (UMMA N)
constexpr int kBlockK = 64;   // k depth per pipeline stage = one 128-byte swizzle row of bf16

// Transposed ("swap-AB") tiles of the forward / dgrad layouts: an expert with at
// most kLightRows rows does not get a 128-row tile.  Instead 128 output COLUMNS
// ride the UMMA M dimension and the few rows ride UMMA N (a multiple of 16), so a
// 5-row expert costs an N=16 instruction instead of a padded 128 x 256 one.  Such a
// tile is kLightCols columns wide and takes kLightK of the contraction per pipeline
// stage.  (Larger experts keep 128-row tiles for their last rows too: a transposed
// tile for the remainder would sweep the expert's weights a second time.)
constexpr int kLightRows = 64;
constexpr int kLightCols = 128;
constexpr int kLightK = 128;

struct Problem {
  int mode;
  int z;
  int64_t tokens;  // rows of a
  int64_t d1;      // a.shape[1]: k for NN/NT, m for TN
  int64_t n;       // output columns
  int tile_m;      // output rows per scheduled tile: 128 (one CTA) or 256 (a CTA pair)
  int tile_n;      // output columns per scheduled tile: 256, or 512 (a CTA pair: two accumulators of 256)
  int group_m;     // row-tiles swept together across the columns (L2 reuse of b)
  int light;       // 1: experts of <= kLightRows rows run as transposed tiles (NN/NT, tile_m 128)
  int order;       // 0: experts in index order.  1: experts sorted by rows, largest first
  int64_t wait_ns; // limit of every wait inside the kernel, in nanoseconds
  // Derived on the host so that decoding a tile needs no 64-bit division:
  int nt;          // column tiles: ceil(n / tile_n)
  int nt1;         // column tiles of one accumulator: ceil(n / 256)
  int mt;          // TN: row tiles of c[i]: ceil(d1 / tile_m)
  int lt;          // column tiles of a transposed tile's width: ceil(n / 128)
  int wide_a;      // TN: a's columns are a multiple of 64, one TMA load brings all 64-column boxes of a stage
  int wide_b;      // TN: same for b
  int single_wave; // every tile there can be is some cluster's first: no position is drawn from the counter
  int pair_sum;    // NN/NT: a is [2, tokens, d1] and the contraction runs over a[0] x b, then a[1] x b2.
                   // (The gated product's input gradient as one launch: no second product to
                   // write, read back and add, and one rounding instead of three.  With zero_rest
                   // instead of a zeroed [2, tokens, n] a training step of 16384 rows, 8 experts of
                   // 4096 x 14336, went from 13.73 to 13.27 ms, the gradient's error from 3.0e-3 to 2.3e-3.)
  int dest_indexed;  // row_dest holds rows of a [dest_rows, n] destination at dest_lo, not addresses
  int64_t dest_rows;
  int zero_rest;   // gated backward: rows past the last expert's of both halves of c become zeros
  int swap_rows;   // NN/NT: a tile of at most this many rows (rounded up, swapped_rows) runs with its operands swapped
  // A pair's launch (narrow_tiles): up to this many rounds of tiles of one accumulator it has no wide ones, and
  // it has them if they cost less at this percentage.
  int narrow_rounds;
  int wide_cost;
  int swap_units;  // ... if it has this many accumulators (a pair's gated tile: 2, gate and up, else 1)
};

// Fills the derived fields of a Problem whose shape fields are set.
B200GMM_HD void derive(Problem* p) {
  p->nt = static_cast<int>((p->n + p->tile_n - 1) / p->tile_n);
  p->nt1 = static_cast<int>((p->n + kBlockN - 1) / kBlockN);
  p->mt = static_cast<int>((p->d1 + p->tile_m - 1) / p->tile_m);
  p->lt = static_cast<int>((p->n + kLightCols - 1) / kLightCols);
}

struct Tile {
  int expert;
  int row0;        // NN/NT: first row of a/c (global); TN: first row of c[expert]
  int col0;        // first output column
  int valid_rows;  // rows of this tile that exist in the output
  int k_row0;      // TN: first contraction row in a/b (global); else 0
  int k_len;       // contraction length (k, or batch_sizes[expert] for TN)
  int kind;        // 0: tile_m x 256 tile; 1: transposed tile (valid_rows <= kLightRows, kLightCols columns)
  int units;       // accumulators of kBlockN columns: 1, or 2 (a CTA pair's tile of 512 columns; the last may be half)
};

B200GMM_HD int ceil_div_i(int a, int b) { return (a + b - 1) / b; }

// Row-tiles of tile_m rows an expert with `rows` rows gets, and the rows that go
// to transposed tiles instead (0 if none).
B200GMM_HD int heavy_row_tiles(const Problem& p, int rows) {
  if (p.light && rows <= kLightRows) return 0;
  return ceil_div_i(rows, p.tile_m);
}
B200GMM_HD int light_rows(const Problem& p, int rows) {
  return (p.light && rows <= kLightRows) ? rows : 0;
}

// Tiles of one expert; of a pair's launch, whose columns may be cut in two ways (TileGrid), row
// tiles.  TN always has the full c[i] grid (empty experts still need their zeros written,
// csrc/fill_arguments.cuh:100-119).
B200GMM_HD int expert_tiles(const Problem& p, int rows) {
  if (p.tile_n > kBlockN) return p.mode == kTN ? p.mt : ceil_div_i(rows, p.tile_m);
  if (p.mode == kTN) return p.mt * p.nt;
  return heavy_row_tiles(p, rows) * p.nt + (light_rows(p, rows) > 0 ? p.lt : 0);
}

// Most tiles of one accumulator a launch can have, whatever batch_sizes holds (B200GMM_LIGHT off).
B200GMM_HD int64_t max_tiles(const Problem& p) {
  if (p.mode == kTN) return int64_t(p.z) * p.mt * p.nt1;
  return (p.tokens / p.tile_m + (p.z < p.tokens ? p.z : p.tokens)) * p.nt1;
}

// Pipeline stages (ring slots) one tile consumes.
B200GMM_HD int tile_stages(const Tile& t) {
  return t.kind ? (t.k_len + kLightK - 1) / kLightK : (t.k_len + kBlockK - 1) / kBlockK;
}

// Swapped tiles (NN/NT): a tile with few rows is computed as its transpose, from the same
// loads.  The tile's weight columns ride UMMA M (one CTA: two MMAs of 128 columns; a pair: one
// MMA of 2 x 128 for each accumulator) and its rows ride UMMA N, rounded up to the step that N
// allows, so that the tensor core works for the rows that exist and not for tile_m of
// them, and only those rows are fetched.  Which launches, and up to how many rows a tile:
// Problem::swap_rows (b200gmm.cu: swap_rows).
// Returns the rounded row count, 0 for a plain tile.
B200GMM_HD int swapped_rows(const Problem& p, const Tile& t) {
  if (p.swap_rows == 0 || t.kind != 0 || t.units < p.swap_units) return 0;
  const int step = p.tile_m == kBlockM ? 16 : 32;  // (a power of two: no division before every tile)
  const int rows = (t.valid_rows + step - 1) & ~(step - 1);
  return rows <= p.swap_rows ? rows : 0;
}

// Within one expert: walk group_m row-tiles down, then step one column-tile
// right, so that concurrently running CTAs share a and b panels in L2.
B200GMM_HD void decode_in_expert(int local, int row_tiles, int nt, int group_m, int* mi, int* ni) {
  const int group_span = group_m * nt;
  const int g = local / group_span;
  const int first = g * group_m;
  const int gm = (row_tiles - first) < group_m ? (row_tiles - first) : group_m;
  const int r = local - g * group_span;
  *mi = first + r % gm;
  *ni = r / gm;
}

// Rounds that `tiles` tiles take on `clusters`; and, counted in rounds of tiles of one accumulator, that
// `tiles` tiles of two do, where what is left after whole rounds is taken as halves if these fit
// one round (tile_order).
template <class Int>
B200GMM_HD Int rounds_narrow(Int tiles, Int clusters) { return (tiles + clusters - 1) / clusters; }
template <class Int>
B200GMM_HD Int rounds_wide(Int tiles, Int clusters) {
  const Int whole = tiles / clusters, left = tiles - whole * clusters;
  return 2 * whole + (left == 0 ? 0 : (2 * left <= clusters ? 1 : 2));
}

// Whether a pair's launch takes its tiles one accumulator wide.  A wide tile brings its rows
// once for two accumulators, which makes a round of it cost Problem::wide_cost percent of two
// narrow ones; but it is coarse, and half idle where the last column tile is one accumulator wide.
B200GMM_HD bool narrow_tiles(const Problem& p, int row_tiles, int clusters) {
  if (p.n <= kBlockN) return true;
  const int narrow = rounds_narrow(row_tiles * p.nt1, clusters), wide = rounds_wide(row_tiles * p.nt, clusters);
  return narrow <= 1 || narrow <= p.narrow_rounds || int64_t(100) * narrow <= int64_t(p.wide_cost) * wide;
}

// How a launch cuts the columns, and the row tiles swept together.
struct TileGrid {
  int nt;
  int tile_n;
  int group_m;
};
// Launch order of a pair's `row_tiles` in positions, which is what the grid's `clusters` draw: tiles,
// and what is left over after whole rounds of wide ones as halves when the halves fit one
// round, which then lasts half as long.  A half that does not exist (the last column tile
// may be one accumulator wide) is a position of no units; a launch of narrow tiles has none, since
// clusters whose draws hit them are left with fewer tiles than others (11 experts, 16933 rows,
// 2792 x 592, two wide column tiles of which the second is one accumulator: 71 us as narrow tiles, 87 as
// halves).  (clusters == 0: whole wide tiles.)
struct TileOrder {
  TileGrid grid;
  int whole;  // positions before the halves
  int total;
};
B200GMM_HD TileOrder tile_order(const Problem& p, int row_tiles, int clusters) {
  TileOrder o;
  if (clusters > 0 && narrow_tiles(p, row_tiles, clusters)) {
    // half as many row tiles together keep what is in flight about square
    o.grid = TileGrid{p.nt1, kBlockN, p.group_m > 1 ? p.group_m / 2 : 1};
    o.whole = o.total = row_tiles * p.nt1;
    return o;
  }
  o.grid = TileGrid{p.nt, p.tile_n, p.group_m};
  const int tiles = row_tiles * p.nt;
  const int left = clusters > 0 ? tiles % clusters : 0;
  const int halves = 2 * left <= clusters ? left : 0;
  o.whole = tiles - halves;
  o.total = tiles + halves;
  return o;
}
// Tile of a position, and which half of it (-1: all).
B200GMM_HD int tile_of_position(const TileOrder& o, int position, int* half) {
  *half = position < o.whole ? -1 : (position - o.whole) & 1;
  return position < o.whole ? position : o.whole + ((position - o.whole) >> 1);
}

// Accumulators that a tile of tile_n columns fills at column col0.
B200GMM_HD int tile_units(const Problem& p, int tile_n, int col0) {
  return tile_n > kBlockN && p.n - col0 > kBlockN ? 2 : 1;
}

// `local` = tile index relative to the expert's first tile; rs/re = row_start[expert],
// row_start[expert+1] (already clamped to tokens).
B200GMM_HD Tile make_tile(const Problem& p, const TileGrid& grid, int expert, int local, int rs, int re) {
  Tile t;
  t.expert = expert;
  t.kind = 0;
  const int nt = grid.nt;
  int mi, ni;
  if (p.mode == kTN) {
    decode_in_expert(local, p.mt, nt, grid.group_m, &mi, &ni);
    t.row0 = mi * p.tile_m;
    const int left = static_cast<int>(p.d1) - t.row0;
    t.valid_rows = left < p.tile_m ? left : p.tile_m;
    t.k_row0 = rs;
    t.k_len = re - rs;
    t.col0 = ni * grid.tile_n;
    t.units = tile_units(p, grid.tile_n, t.col0);
    return t;
  }
  t.k_row0 = 0;
  // (the two parts of a pair sum start at a k-block of their own)
  t.k_len = static_cast<int>(p.d1);
  if (p.pair_sum) t.k_len = (t.k_len + kBlockK - 1) / kBlockK * kBlockK * 2;
  const int mt = heavy_row_tiles(p, re - rs);
  if (local < mt * nt) {
    decode_in_expert(local, mt, nt, grid.group_m, &mi, &ni);
    t.row0 = rs + mi * p.tile_m;
    const int left = re - t.row0;
    t.valid_rows = left < p.tile_m ? left : p.tile_m;
    t.col0 = ni * grid.tile_n;
    t.units = tile_units(p, grid.tile_n, t.col0);
  } else {
    t.units = 1;
    t.kind = 1;
    t.row0 = rs + mt * kBlockM;
    t.valid_rows = re - t.row0;
    t.col0 = (local - mt * nt) * kLightCols;
  }
  return t;
}

// What a position that is half a tile (tile_of_position) leaves of it.
B200GMM_HD void take_half(Tile* t, int half) {
  if (half < 0) return;
  t->units = half < t->units ? 1 : 0;
  t->col0 += half * kBlockN;
}

// The nine per-expert values of the reference's GemmProblem
// (csrc/fill_arguments.cuh:13-18, :66-78), in int64.  `start` is the exclusive
// prefix sum of batch_sizes at expert `e`, `size` is batch_sizes[e].
B200GMM_HD void fill_fields(const Problem& p, int e, int64_t start, int64_t size, int64_t* out9) {
  if (p.mode == kTN) {
    const int64_t m = p.d1, n = p.n, k = size;
    out9[0] = m; out9[1] = n; out9[2] = k;
    out9[3] = m;  // a is read as column-major m x k: leading dimension = rows
    out9[4] = n; out9[5] = n;
    out9[6] = m * start; out9[7] = start * n; out9[8] = static_cast<int64_t>(e) * m * n;
  } else {
    const int64_t m = size, n = p.n, k = p.d1;
    out9[0] = m; out9[1] = n; out9[2] = k;
    out9[3] = k;
    out9[4] = (p.mode == kNT) ? k : n;  // NT reads b[i] as column-major k x n
    out9[5] = n;
    out9[6] = start * k; out9[7] = static_cast<int64_t>(e) * k * n; out9[8] = start * n;
  }
}

}  // namespace b200gmm
