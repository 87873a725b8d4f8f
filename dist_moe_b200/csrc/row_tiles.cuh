// How the forward and input-gradient GEMMs split an expert's routed rows into tiles, and which gathered row blocks a BF16
// tile needs.  Plain arithmetic, for the kernels and for host code.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define DM_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define DM_HOST_DEVICE inline
#endif

namespace dm {

constexpr int kRwMaxN = 256;          // routed rows per tile (N side of the MMA)
constexpr int kRwGatherBlock = 128;   // rows per readiness counter of the fused dispatch
constexpr int kRwBoxes = 5;           // heights of the row boxes: the smallest one that covers half a tile is loaded

// Rows of a gather unit, 1 to 8: as few as leave no gather warp more than one unit of a launch, for at least that many rows.
DM_HOST_DEVICE constexpr int rw_gather_unit_rows(int total_rows, int warps) {
  return total_rows <= warps ? 1 : total_rows <= 2 * warps ? 2 : total_rows <= 4 * warps ? 4 : 8;
}

// Whether a dispatch GEMM's `num_sms` says that its flags are kept clear: the mark with a bound on the SMs of up to 16 bits, zero for
// none.  Larger numbers are bounds and nothing else, as they are to the other GEMMs (all of the device).
constexpr int kRwKeptClear = 1 << 30;
DM_HOST_DEVICE constexpr bool rw_flags_kept_clear(int num_sms) { return (num_sms & ~0xffff) == kRwKeptClear; }

// A CTA of the pair loads half of a tile's rows.
DM_HOST_DEVICE constexpr int rw_box_rows(int i) { return i == 0 ? 16 : 32 * i; }
DM_HOST_DEVICE constexpr int rw_box_index(int n) { return n <= 32 ? 0 : (n + 63) >> 6; }

// Row tiles of an expert and the rows each of them takes (the last one what is left): equal tiles, multiples of 32.
DM_HOST_DEVICE constexpr int rw_row_tiles(int rows) { return (rows + kRwMaxN - 1) / kRwMaxN; }
DM_HOST_DEVICE constexpr int rw_rows_per_tile(int rows) {
  return rows > 0 ? ((rows + rw_row_tiles(rows) - 1) / rw_row_tiles(rows) + 31) & ~31 : 32;
}

struct RowsTile {
  int e, pair, row0, rows, n;  // rows: real rows of the tile, n: the MMA's N (rows rounded up to 32)
};

// `rows_per_tile[e]` rows per tile of an expert; consecutive tiles share the weight block (`pair` of column blocks).
DM_HOST_DEVICE RowsTile rw_decode(int tile, int& e, const int* tile_start, const int* off, const uint16_t* rows_per_tile) {
  while (tile >= tile_start[e + 1]) ++e;
  const int local = tile - tile_start[e];
  const int rows = off[e + 1] - off[e];
  const int per = rows_per_tile[e];
  const int nt = rw_row_tiles(rows);
  RowsTile t;
  t.e = e;
  t.pair = local / nt;
  const int first = (local - t.pair * nt) * per;
  t.row0 = off[e] + first;
  const int left = rows - first;
  t.rows = left < per ? left : per;
  if (t.rows < 0) t.rows = 0;
  t.n = t.rows > 0 ? (t.rows + 31) & ~31 : 32;
  return t;
}

// Row blocks [first, last] that hold the tile's rows.  Nothing about a tile's blocks follows from what an earlier tile of
// the same CTA waited for: a CTA's next tile may lie in a later column block and start at an earlier row, and the blocks
// between two tiles of one CTA are pulled for other CTAs.
struct RowsBlocks {
  int first, last;
};
DM_HOST_DEVICE RowsBlocks rw_tile_blocks(const RowsTile& t, int total_rows) {
  const int end = t.row0 + t.n < total_rows ? t.row0 + t.n : total_rows;
  RowsBlocks b;
  b.first = t.row0 / kRwGatherBlock;
  b.last = (end - 1) / kRwGatherBlock;
  return b;
}

// Pairs that take tiles where tiles are short of rows and the launch streams weights: as few as need the rounds that all of them
// would need.  A last round with a part of the pairs has too few loads in flight for HBM; with these all rounds are alike, and the
// pairs that are left out were not missed.  `rows` is the launch's largest tile, `limit` the kernel's line, `workers` all pairs.
// `heavy`: where the epilogue counts (SwiGLU and quantisation), two or three rounds stay as they are if the last one has more
// than half of the pairs.
DM_HOST_DEVICE constexpr int balanced_pairs(int tiles, int workers, int rows, int limit, bool heavy = false) {
  const int rounds = (tiles + workers - 1) / workers;
  if (rows > limit || rounds <= 1) return workers;
  if (heavy && rounds <= 3 && 2 * (tiles - (rounds - 1) * workers) > workers) return workers;
  return (tiles + rounds - 1) / rounds;
}

// Rows of the group [off, next) that a block-scaled GEMM works on, `count` of them real.  None where the group does not
// start on a scale atom of 128 rows: the caller has broken the padding rule, and the MMA would take the rows' scales from an
// odd TMEM column, which is a misaligned address.
DM_HOST_DEVICE constexpr bool bs_group_aligned(int off) { return (off & 127) == 0; }
DM_HOST_DEVICE int bs_group_rows(int off, int next, int count) {
  const int room = next - off, rows = count < room ? count : room;
  return rows > 0 && bs_group_aligned(off) ? rows : 0;
}

// Row tiles of an expert in the MXFP8 pair kernel: one of its rows rounded up to 32, or several nearly equal ones that start
// at multiples of 64 rows, because the MMA takes its scale columns (32 rows each) from an even column on.
DM_HOST_DEVICE constexpr int bs_rows_per_tile(int rows) {
  return rows <= kRwMaxN ? rw_rows_per_tile(rows) : ((rows + rw_row_tiles(rows) - 1) / rw_row_tiles(rows) + 63) & ~63;
}

// Scale atoms (128 rows) that the rows of a tile touch at most, in a launch whose largest tile has `n_max` rows: only experts
// of more than 256 rows have several tiles, of 192 or 256 rows each, and those of 192 that start inside an atom end with one.
DM_HOST_DEVICE constexpr int bs_tile_atoms(int n_max) { return n_max <= 128 ? 1 : 2; }

}  // namespace dm
