// Which shape of the SpMM kernels a product takes, and how its rows are handed out.  Plain host
// C++: spmm.cu launches what this file decides, and the rules can be checked without a GPU.
#pragma once
#include <cstdint>

namespace csg {

constexpr int M_THREADS = 256;
constexpr int M_WARPS = M_THREADS / 32;
constexpr int M_BLOCKS_PER_SM = 3;
constexpr int SPLIT = 1024;      // longest row one lane group walks alone in a large product ...
constexpr int SPLIT_MIN = 128;   // ... and in a small one
constexpr int ROW_COST = 4;      // cost of a row beside its nonzeros, in nonzeros
constexpr int UNIT_MIN = 128;    // smallest and largest cost of a unit
constexpr int UNIT_MAX = 2048;
// Staging room per warp: rows of a unit and (column, value) pairs.  Less where a whole warp takes a
// row, four columns to a lane: what a block does not hold stays with the L1, and neighbouring rows of a mesh
// share rows of B there (9-point mesh, 1.05 M rows, four blocks per SM: width 96 341 us with 512 rows and 448 pairs,
// 318 with 256 and 256; width 128 477 and 446).  Two panels in four blocks keep the pairs (the mesh at 256: 727 us
// with 256 pairs, 714 with 448).
constexpr int batch_rows(int lanes, int vec) { return lanes == 32 && vec == 4 ? 256 : UNIT_MAX / ROW_COST; }
constexpr int batch_pairs(int lanes, int vec, int panels, int blocks) {
  return lanes == 32 && vec == 4 && (panels == 1 || blocks == 3) ? 256 : 448;
}

// lanes   lanes of a group
// vec     columns per lane
// panels  panels of lanes * vec columns walked at once
// masked  the last panel is ragged
// whole   rows outside units of short rows go to the whole warp
// even    lanes of a group in units of short rows of much the same length
// blocks  per SM
struct SpmmShape {
  int lanes, vec, panels, masked, whole, even, blocks;
  constexpr bool operator==(const SpmmShape &o) const {
    return lanes == o.lanes && vec == o.vec && panels == o.panels && masked == o.masked && whole == o.whole &&
           even == o.even && blocks == o.blocks;
  }
};

// every shape that spmm_shape() returns
#define CSG_SPMM_SHAPES(X)                                                                        \
  X(1, 1, 1, 0, 0, 1, 3) X(1, 2, 1, 0, 0, 1, 3) X(1, 4, 1, 0, 0, 1, 3) X(2, 4, 1, 0, 0, 2, 3)       \
  X(4, 4, 1, 0, 0, 4, 3) X(8, 4, 1, 0, 0, 8, 3) X(8, 4, 1, 0, 1, 8, 3) X(16, 4, 1, 0, 1, 16, 3)     \
  X(4, 1, 1, 1, 0, 4, 3) X(8, 1, 1, 1, 0, 8, 3) X(16, 1, 1, 1, 0, 16, 3)                            \
  X(4, 2, 1, 1, 0, 4, 3) X(8, 2, 1, 1, 0, 8, 3) X(16, 2, 1, 1, 0, 16, 3)                            \
  X(4, 4, 1, 1, 0, 4, 3) X(8, 4, 1, 1, 0, 8, 3) X(16, 4, 1, 1, 1, 16, 3) X(16, 4, 1, 1, 1, 4, 3)    \
  X(32, 1, 1, 1, 1, 32, 4) X(32, 1, 2, 1, 1, 32, 4) X(32, 2, 1, 1, 1, 32, 4) X(32, 2, 2, 1, 1, 32, 4) \
  X(32, 4, 1, 0, 1, 32, 3) X(32, 4, 1, 0, 1, 32, 4) X(32, 4, 2, 0, 1, 32, 3) X(32, 4, 2, 0, 1, 32, 4) \
  X(32, 4, 1, 1, 1, 4, 3) X(32, 4, 1, 1, 1, 8, 3) X(32, 4, 1, 1, 1, 16, 3) X(32, 4, 1, 1, 1, 32, 3) \
  X(32, 4, 2, 1, 1, 8, 3) X(32, 4, 2, 1, 1, 16, 3) X(32, 4, 2, 1, 1, 32, 3)                         \
  X(32, 4, 2, 1, 1, 8, 4) X(32, 4, 2, 1, 1, 16, 4) X(32, 4, 2, 1, 1, 32, 4)

// Lane groups by dense width: four or two columns per lane where the width and the alignment of B
// and C (`align`, in bytes: 16, 8 or 4) allow, single floats otherwise, and as many lanes as the row has such
// pieces (up to 32); two panels per walk when the panel count is even.  (Groups of one to eight lanes
// for widths without a power-of-two factor, one float per lane, left a group walking the row once
// per column: 5.5 ms for 0.28 M nonzeros at width 41 on a B200, 0.095 ms with the masked panels.)
inline SpmmShape spmm_shape(int32_t n, int32_t nnz, int32_t w, int align) {
  const long long b_bytes = static_cast<long long>(n) * w * 4;
  const int vec = w % 4 == 0 && align % 16 == 0 ? 4 : w % 2 == 0 && align % 8 == 0 ? 2 : 1;
  const int cols = w / vec;
  auto narrow = [&](int lanes, int masked, int whole) { return SpmmShape{lanes, vec, 1, masked, whole, lanes, M_BLOCKS_PER_SM}; };
  if (vec == 4) {
    // At 32 columns a lane of the whole warp has a single float per gather, which saves power-law graphs the
    // idle lanes of groups that wait for the longest row, and tells against it once most of B is not in the L2.
    // By the warp over walked, R-MAT of 9 to 16 edges a row: 0.78 to 0.97 with 8 MiB of B, 0.62 to 0.87 with 32, 0.87
    // to 0.98 with 128, 0.87 to 0.94 with 183, 0.91 to 0.95 with 256, 0.92 to 1.00 with 366, 0.93 to 1.07 with 512.  (4 edges
    // would gain as well, but their lengths on average are those of meshes, which lose a percent.)
    if (w == 32) return narrow(8, 0, nnz > 12ll * n && b_bytes <= (256ll << 20));
    if (w == 64) return narrow(16, 0, 1);
    if (w == 16 || w == 8 || w == 4) return narrow(cols, 0, 0);
  }
  if (cols == 1) return narrow(1, 0, 0);
  if (cols <= 4) return narrow(4, 1, 0);
  if (cols <= 8) return narrow(8, 1, 0);
  if (cols <= 16) {
    SpmmShape s = narrow(16, 1, vec == 4);
    // (a large mesh in grid order; the others gain nothing: 1.05 M rows 211 us by sixteen lanes, 182 by groups of four;
    // relabelled 320 and 336)
    if (vec == 4 && w == 48 && b_bytes > (128ll << 20)) s.even = 4;
    return s;
  }
  SpmmShape s{32, vec, (cols + 31) / 32 % 2 == 0 ? 2 : 1, cols % 32 != 0 || vec < 4, 1, 32, M_BLOCKS_PER_SM};
  if (vec < 4) {  // little in flight per lane: more warps (R-MAT scale 20 at 41: 572 us with three blocks, 501 with four)
    s.blocks = 4;
    return s;
  }
  // Units of rows of one length go to lane groups that fill the width without a rest, as many panels as
  // it takes: a mesh wastes neither lanes nor gathers there (9-point mesh, 1.05 M rows, width 96: 493 us with 24 of
  // 32 lanes on, 286 by groups of eight; at 192 643 and 540).  Smaller groups read too little of a row of B at a
  // time where rows are far apart (relabelled, width 176: 1.17 ms by the warp, 1.61 by groups of four), ragged ones
  // gain nothing.  Width 144 stays at 550 us, 474 by groups of four, for the same reason.
  if (s.masked) s.even = w % 64 == 0 ? 16 : w % 32 == 0 ? 8 : w == 80 ? 4 : 32;
  // Three blocks per SM leave the L1 larger, four have more gathers under way.  One panel: while B is mostly in the
  // L2 three (65,536 rows of R-MAT at 128: 103 us and 112 with four), beyond it four (scale 22 3.26 and 3.13 ms; road
  // network of 1.05 M rows 422 and 381 us); a ragged panel stays with three (the mesh at 96: 286 and 311 us).  Two
  // panels are enough in flight where rows are long (131,072 Zipf rows at 256: 326 us and 370; R-MAT scale 18 351 and
  // 367); short rows want four (the mesh at 256: 805 us and 714; road network of 250,000 rows at 192 149 and 139).
  const bool long_rows = nnz > 12ll * n;
  if (s.panels == 1)
    s.blocks = !s.masked && b_bytes > (192ll << 20) ? 4 : 3;
  else
    s.blocks = !long_rows && b_bytes > ((s.masked ? 96ll : 192ll) << 20) ? 4 : 3;
  return s;
}

struct SpmmPlan {
  SpmmShape shape;
  int32_t rows_grid, long_grid;  // blocks of the two launches
  int32_t unit;                  // cost per unit of rows
  int32_t split, piece;          // longest row one group walks alone, nonzeros per piece of a longer one
};

inline SpmmPlan spmm_plan(int32_t n, int32_t nnz, int32_t w, int align, int num_sms, int32_t queue_cap) {
  SpmmPlan p;
  p.shape = spmm_shape(n, nnz, w, align);
  p.long_grid = num_sms * M_BLOCKS_PER_SM;
  p.rows_grid = num_sms * p.shape.blocks;
  const long long total = static_cast<long long>(ROW_COST) * n + nnz;
  const bool wide = p.shape.lanes == 32 && p.shape.vec == 4;
  const long long warps = static_cast<long long>(wide ? p.rows_grid : p.long_grid) * M_WARPS;
  long long unit;
  if (wide) {
    // Units of at least UNIT_MIN, up to eight of them for each warp of the grid, the same number for all: with
    // a few more units than warps, most warps wait for those that draw a second one (9-point mesh, 40,000 rows,
    // width 192: 41.0 us so, 32.8 with one unit each).  Where there are fewer units than warps, no more blocks than
    // SMs are started, or than find a unit.
    long long rounds = total / (warps * UNIT_MIN);
    rounds = rounds < 1 ? 1 : rounds > 8 ? 8 : rounds;
    unit = total / (warps * rounds) + 1;
  } else {
    unit = total / (warps * 8);  // enough units that every warp of the grid draws several of them
  }
  const long long most = static_cast<long long>(batch_rows(p.shape.lanes, p.shape.vec)) * ROW_COST;
  unit = unit < UNIT_MIN ? UNIT_MIN : unit > most ? most : unit;
  p.unit = static_cast<int32_t>(unit);
  if (wide) {
    long long blocks = (total / unit + 1 + M_WARPS - 1) / M_WARPS;
    if (blocks < num_sms) blocks = num_sms;
    if (blocks < p.rows_grid) p.rows_grid = static_cast<int32_t>(blocks);
  }
  // A row walked alone is a serial chain of gathers: it should not outlast what the other
  // groups do meanwhile, twice the average share of a group here.  Large products keep the
  // upper limit (fewer atomics), small ones would otherwise wait for their longest row: one
  // of 1024 nonzeros is 128 dependent steps of gathers.
  const long long groups = static_cast<long long>(p.long_grid) * M_WARPS * (32 / p.shape.lanes);
  const long long share = nnz / groups;
  p.split = SPLIT_MIN;
  while (p.split < SPLIT && (p.split < 2 * share || nnz / p.split + 1 > queue_cap)) p.split *= 2;
  p.piece = p.split / 4;
  return p;
}

}  // namespace csg
