// Apply a permutation to a CSR matrix: rows only, or rows and columns
// (P A P^T) with every output row re-sorted.
//
// Semantics of sporder/src/reorder.cu:72-149: new row p is old row
// new_order[p]; in symmetric mode column c becomes old2new[c] and the row is
// sorted by its new column ids, values moving with their columns; ptr_new is
// the inclusive scan of the gathered row lengths with ptr_new[0] = 0.
//
// The reference gathers into scratch and runs a device-wide segmented sort.  Here
// a row is gathered, remapped and sorted by as much hardware as it needs:
//   * rows of up to 32 entries (the bulk) in registers: a warp reads the descriptors of 32
//     consecutive new rows with coalesced loads, then sorts four rows of up to 8 entries,
//     two of up to 16 or one of up to 32 at a time in segments of the warp (bitonic
//     network over shuffles);
//   * rows of up to 256 entries by one warp each, two, four or eight entries per lane in
//     registers (strides of 32 and more are exchanges between a lane's own registers);
//   * rows of up to 4096 entries by one thread block: every warp sorts runs of 256 in
//     registers, the runs are merged in shared memory by rank (an entry's place in the
//     merged run is its own index plus the number of smaller entries in the partner run,
//     found by binary search - keys are distinct), the last merge writes the output;
//   * longer rows - on power-law inputs single rows hold 10^5 entries - as tiles of 4096
//     sorted the same way into a scratch copy by as many blocks as there are tiles, then one
//     pass that places every entry at the sum of its ranks in all tiles of its row.
// A permutation that keeps every row and column inside its block of 1024 (every csg order
// with the default chunk size does) needs none of this: the old row is sorted by column, so the
// new row is already sorted block by block and only the entries of one block have to be ordered
// among themselves.  len_block_sums_kernel notices such a permutation and tells the host, which then
// launches apply_flat_kernel instead of the kernels above.  That one, which also does the copy
// of the rows-only mode, cuts the output into tiles of 128 entries whatever rows they belong to.
#include <algorithm>
#include <cstddef>

#include "common.cuh"

namespace csg {

namespace {

constexpr int R_THREADS = 256;
constexpr int R_SCAN_IPT = 8;
constexpr int R_SCAN_TILE = R_THREADS * R_SCAN_IPT;  // rows per scan block
constexpr int LOCAL_BITS = 10;                       // blocks of 1024 rows / columns: the default csg chunk
constexpr int FLAT_TILE = 128;                       // output entries per tile of apply_flat_kernel
constexpr int R_WARP = 256;                          // longest row sorted by one warp in registers
constexpr int R_MED = 4096;                          // longest row (and tile of a longer row) sorted in shared memory

// What lies in front of a row: entries in the low half, rows that have any in the high one.
using RowCount = unsigned long long;
__device__ __forceinline__ RowCount row_count(uint32_t entries, uint32_t rows) {
  return static_cast<RowCount>(rows) << 32 | entries;
}

// Entries and rows with entries that each block of new rows takes.  With `outcome`, the last block also tells the host
// whether any row leaves its block of 1024: here and not in ptr_new_kernel, so that the host reads it and
// launches the rest while the scan still runs (a random order of a 65,536-row mesh: 90 us with the
// wait behind ptr_new_kernel, 84 here).  The kernels behind it are programmatic dependent launches: 8 us less a call.
__global__ void __launch_bounds__(R_THREADS) len_block_sums_kernel(
    int32_t n, const int32_t *__restrict__ ptr_old, const int32_t *__restrict__ new_order,
    RowCount *__restrict__ block_sums, uint32_t *__restrict__ leaves_block, volatile uint32_t *outcome, uint32_t ticket) {
  let_next_kernel_start();
  __shared__ RowCount sm[R_THREADS / 32];
  const int32_t base = blockIdx.x * R_SCAN_TILE;
  uint32_t s = 0, rows = 0;
  int moved = 0;
#pragma unroll
  for (int i = 0; i < R_SCAN_IPT; ++i) {
    const int32_t p = base + i * R_THREADS + threadIdx.x;
    if (p < n) {
      const int32_t src = new_order[p];
      const uint32_t len = static_cast<uint32_t>(ptr_old[src + 1] - ptr_old[src]);
      s += len;
      rows += len ? 1u : 0u;
      moved |= (src >> LOCAL_BITS) != (p >> LOCAL_BITS);
    }
  }
  moved = __syncthreads_or(moved);
  if (outcome && threadIdx.x == 0) {
    if (moved) atomicExch(leaves_block, 1u);
    __threadfence();
    if (atomicAdd(leaves_block + 1, 1u) == gridDim.x - 1) {
      __threadfence();
      outcome[1] = atomicAdd(leaves_block, 0u);
      __threadfence_system();
      outcome[0] = ticket;
    }
  }
  s = __reduce_add_sync(FULL, s);
  rows = __reduce_add_sync(FULL, rows);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = row_count(s, rows);
  __syncthreads();
  if (threadIdx.x == 0) {
    RowCount total = 0;
#pragma unroll
    for (int w = 0; w < R_THREADS / 32; ++w) total += sm[w];
    block_sums[blockIdx.x] = total;
  }
}

__global__ void __launch_bounds__(1024) scan_block_sums_kernel(int32_t nb, RowCount *block_sums) {
  let_next_kernel_start();
  wait_for_kernels_before();
  // exclusive scan in place, one block, any nb
  __shared__ RowCount sm[32];
  __shared__ RowCount carry_s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  for (int32_t base = 0; base < nb; base += 1024) {
    const int32_t i = base + threadIdx.x;
    const RowCount v = i < nb ? block_sums[i] : 0;
    RowCount incl = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const RowCount t = __shfl_up_sync(FULL, incl, off);
      if (lane >= off) incl += t;
    }
    if (lane == 31) sm[warp] = incl;
    __syncthreads();
    RowCount wbase = 0, tot = 0;
    for (int w = 0; w < 32; ++w) {
      const RowCount t = sm[w];
      if (w < warp) wbase += t;
      tot += t;
    }
    const RowCount carry = carry_s;
    if (i < nb) block_sums[i] = carry + wbase + incl - v;
    __syncthreads();
    if (threadIdx.x == 0) carry_s = carry + tot;
    __syncthreads();
  }
}

// Up to this many blocks of rows, ptr_new_kernel adds up the sums in front of its own block itself: one kernel less in the
// chain of launches (power-law band of 65,536 rows, rows only 58.2 and 53.4 us, mesh of 1,048,576 rows 88.7 and 83.1).
constexpr int32_t SCAN_IN_PLACE = 2048;

constexpr int TILES_BY_THREAD = 16;  // further tiles of a row that its thread names

// Row pointers of the new matrix, and for the tiles of apply_flat_kernel the list of the rows that have entries (first
// entry, where it was less where it is; one more entry behind the last) with the place in it that each tile begins at.
__global__ void __launch_bounds__(R_THREADS) ptr_new_kernel(
    int32_t n, int32_t nnz, const int32_t *__restrict__ ptr_old, const int32_t *__restrict__ new_order,
    const RowCount *block_sums, int32_t *__restrict__ ptr_new,
    int32_t *__restrict__ old2new, int32_t *__restrict__ tile_row, int2 *__restrict__ row_at, uint32_t rows_max) {
  let_next_kernel_start();
  constexpr int WARPS = R_THREADS / 32;
  __shared__ RowCount sums[R_SCAN_IPT * WARPS];  // of 32 rows each, in row order
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int32_t first = blockIdx.x * R_SCAN_TILE + threadIdx.x;
  int32_t len[R_SCAN_IPT], from[R_SCAN_IPT], incl[R_SCAN_IPT];
  uint32_t filled[R_SCAN_IPT];  // rows of the 32 that have entries
#pragma unroll
  for (int i = 0; i < R_SCAN_IPT; ++i) {
    const int32_t p = first + i * R_THREADS;
    len[i] = from[i] = 0;
    if (p < n) {
      const int32_t src = new_order[p];
      from[i] = ptr_old[src];
      len[i] = ptr_old[src + 1] - from[i];
      if (old2new) old2new[src] = p;
    }
    incl[i] = len[i];
  }
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
#pragma unroll
    for (int i = 0; i < R_SCAN_IPT; ++i) {
      const int32_t t = __shfl_up_sync(FULL, incl[i], off);
      if (lane >= off) incl[i] += t;
    }
  }
#pragma unroll
  for (int i = 0; i < R_SCAN_IPT; ++i) {
    filled[i] = __ballot_sync(FULL, len[i] != 0);
    if (lane == 31) sums[i * WARPS + warp] = row_count(static_cast<uint32_t>(incl[i]), __popc(filled[i]));
  }
  __syncthreads();
  if (warp == 0) {  // sums -> what lies in front of each 32 rows of the block
    static_assert(R_SCAN_IPT * WARPS == 64, "two per lane");
    const RowCount x = sums[2 * lane], y = sums[2 * lane + 1];
    RowCount run = x + y;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const RowCount t = __shfl_up_sync(FULL, run, off);
      if (lane >= off) run += t;
    }
    sums[2 * lane] = run - x - y;
    sums[2 * lane + 1] = run - y;
  }
  __syncthreads();
  wait_for_kernels_before();  // (all so far is the caller's)
  RowCount block_front;
  if (gridDim.x > SCAN_IN_PLACE) {
    block_front = __ldcg(block_sums + blockIdx.x);
  } else {
    constexpr int EACH = SCAN_IN_PLACE / R_THREADS;
    RowCount part[EACH];
#pragma unroll
    for (int u = 0; u < EACH; ++u) {
      const uint32_t b = u * R_THREADS + threadIdx.x;
      part[u] = b < blockIdx.x ? __ldcg(block_sums + b) : 0;
    }
#pragma unroll
    for (int u = 1; u < EACH; ++u) part[0] += part[u];
    const uint32_t entries = __reduce_add_sync(FULL, static_cast<uint32_t>(part[0]));
    const uint32_t rows = __reduce_add_sync(FULL, static_cast<uint32_t>(part[0] >> 32));
    __shared__ RowCount front_of_block[WARPS];
    if (lane == 0) front_of_block[warp] = row_count(entries, rows);
    __syncthreads();
    block_front = 0;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) block_front += front_of_block[w];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) ptr_new[0] = 0;
  bool several = false;
  uint32_t tile[R_SCAN_IPT], end[R_SCAN_IPT], place[R_SCAN_IPT];
#pragma unroll
  for (int i = 0; i < R_SCAN_IPT; ++i) {
    const int32_t p = first + i * R_THREADS;
    const RowCount front = block_front + sums[i * WARPS + warp];
    const uint32_t run = static_cast<uint32_t>(front) + static_cast<uint32_t>(incl[i] - len[i]);
    place[i] = static_cast<uint32_t>(front >> 32) + __popc(filled[i] & ((1u << lane) - 1u));
    end[i] = run + static_cast<uint32_t>(len[i]);
    if (p < n) {
      ptr_new[p + 1] = static_cast<int32_t>(end[i]);
      if (len[i] && place[i] < rows_max) row_at[place[i]] = make_int2(static_cast<int32_t>(run), from[i] - static_cast<int32_t>(run));
      const uint32_t rows = place[i] + (len[i] ? 1u : 0u);
      if (p == n - 1 && rows < rows_max) row_at[rows] = make_int2(static_cast<int32_t>(end[i]), 0);
    }
    // the row that holds the first entry of a tile
    end[i] = min(end[i], static_cast<uint32_t>(nnz));
    tile[i] = (run + FLAT_TILE - 1) / FLAT_TILE;
    if (tile[i] * FLAT_TILE < end[i]) tile_row[tile[i]] = static_cast<int32_t>(place[i]);
    several |= (++tile[i]) * FLAT_TILE < end[i];
  }
  // the further tiles of a row: the first of them by its own thread, since where one row has some its neighbours often
  // have them too (symmetrised R-MAT of 120,000 rows: 83 us the call, 89 with all of them by the warp), those of the longest
  // by its warp (a row of 98,000 entries in front of R-MAT scale 22 has 768)
  for (int step = 0; step < TILES_BY_THREAD && several; ++step) {
    several = false;
#pragma unroll
    for (int i = 0; i < R_SCAN_IPT; ++i) {
      if (tile[i] * FLAT_TILE >= end[i]) continue;
      tile_row[tile[i]] = static_cast<int32_t>(place[i]);
      several |= (++tile[i]) * FLAT_TILE < end[i];
    }
  }
  if (!__any_sync(FULL, several)) return;
#pragma unroll
  for (int i = 0; i < R_SCAN_IPT; ++i)
    for (uint32_t more = __ballot_sync(FULL, tile[i] * FLAT_TILE < end[i]); more; more &= more - 1u) {
      const int l = __ffs(static_cast<int>(more)) - 1;
      const uint32_t last = __shfl_sync(FULL, end[i], l), at = __shfl_sync(FULL, place[i], l);
      for (uint32_t t = __shfl_sync(FULL, tile[i], l) + lane; t * FLAT_TILE < last; t += 32)
        tile_row[t] = static_cast<int32_t>(at);
    }
}

struct ApplyArgs {
  int32_t n, nnz;
  const int32_t *ptr_old, *ind_old;
  const float *val_old;      // nullptr: pattern only
  const int32_t *new_order;
  const int32_t *old2new;    // nullptr: rows only (apply_flat_kernel<true>)
  const int32_t *ptr_new;
  int32_t *ind_new;
  float *val_new;
  int32_t *queue_warp, *queue_block;  // new rows of 33..R_WARP entries / of up to R_MED
  int2 *queue_long;                   // longer rows: (new row, number of its first tile)
  const int2 *row_at;                 // the rows that have entries: first entry, where it was less where it is
  const int32_t *tile_row;            // per tile of the output: place in row_at of the row its first entry belongs to
  int32_t rows_max;                   // entries of row_at
  uint32_t *counters;                 // [0] warp rows, [1] block rows, [2..3] packed (long rows, tiles),
                                      // [4] set when the permutation leaves blocks of 1024, [5] blocks that looked
  int32_t *tmp_key;                   // scratch copy of the long rows' sorted tiles, indexed like ind_new
  float *tmp_val;
};
constexpr int CNT_WARP = 0, CNT_BLOCK = 1, CNT_LONG = 2, CNT_MOVED = 4;

// Rows of up to W entries, 32 / W of them at a time: each row in a segment of W lanes.
// `mask` names the lanes whose row (src, len, dst) belongs to this size class.
template <int W>
__device__ __forceinline__ void apply_class(const ApplyArgs &a, unsigned mask, int32_t src, int32_t len,
                                            int32_t dst, int lane) {
  constexpr int PER_PASS = 32 / W;
  const int sub = lane / W, j = lane % W;
  while (mask) {
    const unsigned bit = __fns(mask, 0, sub + 1);  // the (sub+1)-th row of the class, if any
    const bool have = bit < 32u;
    const int from = have ? static_cast<int>(bit) : 0;
    const int32_t s = __shfl_sync(FULL, src, from);
    const int32_t l = __shfl_sync(FULL, len, from);
    const int32_t d = __shfl_sync(FULL, dst, from);
#pragma unroll
    for (int r = 0; r < PER_PASS; ++r) mask &= mask - 1u;  // (0 & anything stays 0)
    const bool mine = have && j < l;
    int32_t key = 0x7FFFFFFF;
    float v = 0.0f;
    if (mine) {
      key = a.old2new[a.ind_old[s + j]];
      if (a.val_new) v = a.val_old[s + j];
    }
#pragma unroll
    for (int k = 2; k <= W; k <<= 1) {
#pragma unroll
      for (int x = k >> 1; x > 0; x >>= 1) {
        const int32_t ok = __shfl_xor_sync(FULL, key, x);
        const float ov = __shfl_xor_sync(FULL, v, x);
        const bool up = (j & k) == 0;
        const bool lower = (j & x) == 0;
        const bool take = (up == lower) ? (ok < key) : (ok > key);
        if (take) {
          key = ok;
          v = ov;
        }
      }
    }
    if (mine) {
      a.ind_new[d + j] = key;
      if (a.val_new) a.val_new[d + j] = v;
    }
  }
}

// One warp per 32 consecutive new rows: descriptors with coalesced loads, rows of up to 32
// entries finished here, longer rows queued for the kernels behind.  Latency of its gathers: eight
// blocks per SM, 32 registers (road network of 2.1 M rows, random order: 162 us with 40 registers and
// six blocks, 136 with eight).
__global__ void __launch_bounds__(R_THREADS, 8) apply_short_kernel(ApplyArgs a) {
  const int lane = threadIdx.x & 31;
  const int32_t warps = (gridDim.x * blockDim.x) >> 5;
  const int32_t batches = (a.n + 31) / 32;
  for (int32_t batch = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; batch < batches; batch += warps) {
    const int32_t p = batch * 32 + lane;
    int32_t src = 0, len = 0, dst = 0;
    if (p < a.n) {
      const int32_t src_row = a.new_order[p];
      src = a.ptr_old[src_row];
      len = a.ptr_old[src_row + 1] - src;
      dst = a.ptr_new[p];
    }
    if (len > 32) {
      if (len <= R_WARP) {
        a.queue_warp[atomicAdd(&a.counters[CNT_WARP], 1u)] = p;
      } else if (len <= R_MED) {
        a.queue_block[atomicAdd(&a.counters[CNT_BLOCK], 1u)] = p;
      } else {
        const unsigned long long tiles = static_cast<unsigned long long>((len + R_MED - 1) / R_MED);
        const unsigned long long old = atomicAdd(
            reinterpret_cast<unsigned long long *>(a.counters + CNT_LONG), (1ull << 32) | tiles);
        a.queue_long[old >> 32] = make_int2(p, static_cast<int32_t>(old & 0xFFFFFFFFu));
      }
    }
    apply_class<8>(a, __ballot_sync(FULL, len > 0 && len <= 8), src, len, dst, lane);
    apply_class<16>(a, __ballot_sync(FULL, len > 8 && len <= 16), src, len, dst, lane);
    apply_class<32>(a, __ballot_sync(FULL, len > 16 && len <= 32), src, len, dst, lane);
  }
}

// Bitonic network over the 32 * EPL entries of a warp, ascending.  Entry e sits in register
// e / 32 of lane e % 32: partners at a distance below 32 are reached by shuffles, partners
// further away are the lane's own registers.  The stages are a loop, not unrolled code: fully
// unrolled, the three instances of the network were so much code that the warps of a block,
// each at another stage, spent most of their time waiting for instructions to be fetched.
template <int EPL, int DR>
__device__ __forceinline__ void local_exchange(int32_t (&key)[EPL], float (&val)[EPL], int k) {
#pragma unroll
  for (int r = 0; r < EPL; ++r) {
    if ((r & DR) == 0 && r + DR < EPL) {
      const bool up = ((r * 32) & k) == 0;  // k >= 64 here: the bit lies in r
      const bool swap = up ? (key[r + DR] < key[r]) : (key[r + DR] > key[r]);
      const int32_t k0 = key[r], k1 = key[r + DR];
      const float v0 = val[r], v1 = val[r + DR];
      key[r] = swap ? k1 : k0;
      key[r + DR] = swap ? k0 : k1;
      val[r] = swap ? v1 : v0;
      val[r + DR] = swap ? v0 : v1;
    }
  }
}

template <int EPL>
__device__ __forceinline__ void warp_sort(int32_t (&key)[EPL], float (&val)[EPL], int lane) {
#pragma unroll 1
  for (int k = 2; k <= 32 * EPL; k <<= 1) {
#pragma unroll 1
    for (int x = k >> 1; x > 0; x >>= 1) {
      if (x >= 32) {
        if (x == 128) local_exchange<EPL, 4>(key, val, k);
        if (x == 64) local_exchange<EPL, 2>(key, val, k);
        if (x == 32) local_exchange<EPL, 1>(key, val, k);
      } else {
        const bool lower = (lane & x) == 0;
#pragma unroll
        for (int r = 0; r < EPL; ++r) {
          const int e = r * 32 + lane;
          const int32_t ok = __shfl_xor_sync(FULL, key[r], x);
          const float ov = __shfl_xor_sync(FULL, val[r], x);
          const bool up = (e & k) == 0;
          const bool take = (up == lower) ? (ok < key[r]) : (ok > key[r]);
          key[r] = take ? ok : key[r];
          val[r] = take ? ov : val[r];
        }
      }
    }
  }
}

// One row of up to 32 * EPL entries, gathered, remapped, sorted and written by one warp.
template <int EPL>
__device__ __forceinline__ void warp_row(const ApplyArgs &a, int32_t src, int32_t L, int32_t dst, int lane) {
  int32_t key[EPL];
  float val[EPL];
#pragma unroll
  for (int r = 0; r < EPL; ++r) {
    const int32_t i = r * 32 + lane;
    key[r] = 0x7FFFFFFF;
    val[r] = 0.0f;
    if (i < L) {
      key[r] = a.old2new[a.ind_old[src + i]];
      if (a.val_new) val[r] = a.val_old[src + i];
    }
  }
  warp_sort<EPL>(key, val, lane);
#pragma unroll
  for (int r = 0; r < EPL; ++r) {
    const int32_t i = r * 32 + lane;
    if (i < L) {
      a.ind_new[dst + i] = key[r];
      if (a.val_new) a.val_new[dst + i] = val[r];
    }
  }
}

// ---- tiles of the output ---------------------------------------------------------------------
// A warp per tile of FLAT_TILE consecutive output entries, rows in order.  ROWS: a copy of the
// old rows in their new order.  Otherwise (a permutation that keeps rows and columns in their
// blocks of 1024) an entry's place is the start of its run - the entries of its row in its column's
// block - plus the number of smaller entries in the run, found by comparing where the run is
// short and in a bit map of the block where it is long.  Runs belong to the tile that holds their
// first entry; a tile reads on behind its end as far as its last run goes.
// All rows cost the same per entry this way.  By blocks of 256 threads on tiles of 2048 entries, with ten barriers a
// tile, the reordered R-MAT scale 22 took 955 us here, now 522; mesh of 1,048,576 rows 94 and 48.  Bound by the
// gathers and by the tiles' own instructions about equally at 45 warps per SM (scale 20: 7.2 warp instructions an entry, L1
// 63 %, DRAM 18 %; 40 registers; 11 KB of shared memory a block leave the L1 its space: with 27 KB 677 us).  Tiles of 64 / 96 / 256 entries: 10 / 4 / 30 % slower.
// A tile finds its rows in the list of those that have entries: at most 128, whatever lies between them.  Walked row by
// row, 32 at a time, 4 M empty rows between two entries took one warp 88 ms (the whole call now 0.07), and half of the
// rows of an R-MAT matrix are empty (scale 22 rows only 319 -> 258 us).
constexpr int FLAT_PER = FLAT_TILE / 32;    // windows of 32 entries
// longest run ranked by comparing: 20 took 624 us for the whole call, 28 606, 48 581, 72 579, 128 585 (a bit map costs a
// warp two trips over the run and a scan)
constexpr int FLAT_LONG = 72;
constexpr int FLAT_WARPS = R_THREADS / 32;
// whether a run is ranked by comparing: short, and its last entries no further behind the tile than one window
__device__ __forceinline__ bool flat_short(int32_t s, int32_t end) {
  return end - s <= FLAT_LONG && end <= FLAT_TILE + 32;
}

struct FlatWarp {
  uint32_t row_head[FLAT_PER];    // entries that begin a row
  int32_t delta[FLAT_TILE];       // at these: where the row was less where it is
  int32_t key[FLAT_TILE + 32];    // new columns, and those behind the tile as far as its last run goes
  uint32_t map[32];               // a long run's columns, and how many lie in front of each word
  uint16_t map_before[32];
};

// Runs of more than FLAT_DEFER entries wait until the block is through with its tiles and are then ranked by all its
// warps, eight runs at a time (a warp by itself needed 9 us for 1,000 entries, nearly half of a small call's kernel).
constexpr int FLAT_DEFER = 128, FLAT_QUEUE = 64, FLAT_BATCH = 4;
struct FlatRun {
  int32_t at, len, delta;  // first entry of the output, entries, where they were less where they go
};
struct FlatBlock {
  int32_t queued;
  FlatRun run[FLAT_QUEUE];
};

__device__ __forceinline__ void flat_mark(FlatWarp &sh, int32_t k) { atomicOr(&sh.map[(k >> 5) & 31], 1u << (k & 31)); }
// columns in front of each word of the map, by one warp
__device__ __forceinline__ void flat_count(FlatWarp &sh, int lane) {
  const int c = __popc(sh.map[lane]);
  int incl = c;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int x = __shfl_up_sync(FULL, incl, off);
    if (lane >= off) incl += x;
  }
  sh.map_before[lane] = static_cast<uint16_t>(incl - c);
}
__device__ __forceinline__ void flat_put(const ApplyArgs &a, const FlatWarp &sh, const FlatRun &run, int32_t i, int32_t k) {
  const int32_t w = (k >> 5) & 31;
  const int32_t at = run.at + sh.map_before[w] + __popc(sh.map[w] & ((1u << (k & 31)) - 1u));
  a.ind_new[at] = k;
  if (a.val_new) a.val_new[at] = a.val_old[run.at + run.delta + i];
}

// A run that begins at entry s of the tile, by one warp.
__device__ __forceinline__ void flat_run_by_warp(const ApplyArgs &a, FlatWarp &sh, const FlatRun &run, int32_t s, int lane) {
  auto key = [&](int32_t i) {
    return s + i < FLAT_TILE ? sh.key[s + i] : a.old2new[a.ind_old[run.at + run.delta + i]];
  };
  sh.map[lane] = 0u;
  __syncwarp();
  for (int32_t i = lane; i < run.len; i += 32) flat_mark(sh, key(i));
  __syncwarp();
  flat_count(sh, lane);
  __syncwarp();
  for (int32_t i = lane; i < run.len; i += 32) flat_put(a, sh, run, i, key(i));
  __syncwarp();
}

// The runs that waited, by all warps: a map each, the entries of all of them side by side.
__device__ __forceinline__ void flat_runs_by_block(const ApplyArgs &a, FlatWarp *shared, const FlatRun *run, int runs) {
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  int32_t total = 0;
  for (int r = 0; r < runs; ++r) total += run[r].len;
  shared[warp].map[lane] = 0u;
  __syncthreads();
  for (int pass = 0; pass < 2; ++pass) {
    for (int32_t i0 = 0; i0 < total; i0 += FLAT_BATCH * R_THREADS) {
      int32_t key[FLAT_BATCH], at[FLAT_BATCH], of[FLAT_BATCH];
#pragma unroll
      for (int b = 0; b < FLAT_BATCH; ++b) {
        at[b] = i0 + b * R_THREADS + threadIdx.x;
        of[b] = 0;
        if (at[b] >= total) {
          of[b] = -1;
          continue;
        }
        while (at[b] >= run[of[b]].len) at[b] -= run[of[b]++].len;
        key[b] = a.ind_old[run[of[b]].at + run[of[b]].delta + at[b]];
      }
#pragma unroll
      for (int b = 0; b < FLAT_BATCH; ++b)
        if (of[b] >= 0) key[b] = a.old2new[key[b]];
#pragma unroll
      for (int b = 0; b < FLAT_BATCH; ++b) {
        if (of[b] < 0) continue;
        if (pass == 0)
          flat_mark(shared[of[b]], key[b]);
        else
          flat_put(a, shared[of[b]], run[of[b]], at[b], key[b]);
      }
    }
    __syncthreads();
    if (pass == 0) {
      flat_count(shared[warp], lane);
      __syncthreads();
    }
  }
}

template <bool ROWS, bool VALUES>
__global__ void __launch_bounds__(R_THREADS, 6) apply_flat_kernel(ApplyArgs a) {
  __shared__ FlatWarp shared[FLAT_WARPS];
  __shared__ FlatBlock later;
  constexpr int PER = FLAT_PER;
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  FlatWarp &sh = shared[warp];
  const uint32_t upto = FULL >> (31 - lane);
  wait_for_kernels_before();
  const int32_t nnz = min(a.ptr_new[a.n], a.nnz);
  const int32_t tiles = nnz / FLAT_TILE + (nnz % FLAT_TILE ? 1 : 0);
  if (!ROWS) {
    if (threadIdx.x == 0) later.queued = 0;
    __syncthreads();
  }
  for (int32_t t = blockIdx.x * FLAT_WARPS + warp; t < tiles; t += gridDim.x * FLAT_WARPS) {
    const int32_t t0 = t * FLAT_TILE, cnt = nnz - t0 < FLAT_TILE ? nnz - t0 : FLAT_TILE, t1 = t0 + cnt;
    const int32_t ra = a.tile_row[t];
    if (lane < PER) sh.row_head[lane] = 0u;
    __syncwarp();
    int32_t row_end, delta0 = 0;  // end of the row that holds the tile's last entry; of the row that holds its first
    for (int32_t p0 = ra;; p0 += 32) {  // (at most five times)
      const int2 r = p0 < a.rows_max - lane ? a.row_at[p0 + lane] : make_int2(nnz, 0);
      if (p0 == ra) delta0 = __shfl_sync(FULL, r.y, 0);
      const unsigned behind = __ballot_sync(FULL, r.x >= t1);
      const int rows = behind ? __ffs(static_cast<int>(behind)) - 1 : 32;
      if (lane < rows && r.x >= t0) {
        sh.delta[r.x - t0] = r.y;
        atomicOr(&sh.row_head[(r.x - t0) >> 5], 1u << ((r.x - t0) & 31));
      }
      if (behind) {
        row_end = min(__shfl_sync(FULL, r.x, rows), nnz);
        break;
      }
    }
    __syncwarp();
    int32_t key[PER], from[PER];
    uint32_t rows[PER];
    int32_t last = -1;  // entry that begins the row in hand
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int e = u * 32 + lane;
      rows[u] = sh.row_head[u];
      const uint32_t m = rows[u] & upto;
      const int32_t h = m ? u * 32 + 31 - __clz(static_cast<int>(m)) : last;
      from[u] = t0 + e + (h >= 0 ? sh.delta[h] : delta0);
      key[u] = e < cnt ? a.ind_old[from[u]] : 0;
      if (rows[u]) last = u * 32 + 31 - __clz(static_cast<int>(rows[u]));
    }
    float val[PER];
    if (VALUES) {
#pragma unroll
      for (int u = 0; u < PER; ++u) val[u] = u * 32 + lane < cnt ? a.val_old[from[u]] : 0.0f;
    }
    if (ROWS) {
#pragma unroll
      for (int u = 0; u < PER; ++u) {
        const int e = u * 32 + lane;
        if (e < cnt) {
          a.ind_new[t0 + e] = key[u];
          if (VALUES) a.val_new[t0 + e] = val[u];
        }
      }
      __syncwarp();
      continue;
    }
    // in the same trip: the entry in front of the tile, if its row goes on here, and 32 behind it, as far as its
    // last row goes
    const int32_t last_delta = last >= 0 ? sh.delta[last] : delta0;
    const bool comes_in = (rows[0] & 1u) == 0u, in = lane < row_end - t1;
    int32_t prev = comes_in ? a.ind_old[t0 - 1 + delta0] : 0;
    int32_t more = in ? a.ind_old[t1 + lane + last_delta] : 0;
    float more_val = 0.0f;
    if (VALUES && in) more_val = a.val_old[t1 + lane + last_delta];
#pragma unroll
    for (int u = 0; u < PER; ++u) key[u] = u * 32 + lane < cnt ? a.old2new[key[u]] : 0;
    if (comes_in) prev = a.old2new[prev];
    if (in) more = a.old2new[more];
    // first entries of runs; entries behind the matrix count as such
    uint32_t heads[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int e = u * 32 + lane;
      int32_t front = __shfl_up_sync(FULL, key[u], 1);
      const int32_t across = u > 0 ? __shfl_sync(FULL, key[u > 0 ? u - 1 : 0], 31) : prev;
      if (lane == 0) front = across;
      const bool head = (front >> LOCAL_BITS) != (key[u] >> LOCAL_BITS) || (u == 0 && lane == 0 && !comes_in) || e >= cnt;
      heads[u] = __ballot_sync(FULL, head) | rows[u];
      sh.key[e] = key[u];
    }
    // the last run's entries behind the tile
    int32_t ext = 0;
    if (row_end > t1) {  // (only a full tile has something behind it)
      const int32_t blk = __shfl_sync(FULL, key[PER - 1], 31) >> LOCAL_BITS;
      unsigned other = __ballot_sync(FULL, !in || (more >> LOCAL_BITS) != blk);
      ext = other ? __ffs(static_cast<int>(other)) - 1 : 32;
      sh.key[FLAT_TILE + lane] = more;
      while (other == 0u) {
        const int32_t at = t1 + ext + lane;
        other = __ballot_sync(FULL, lane >= row_end - t1 - ext || (a.old2new[a.ind_old[at + last_delta]] >> LOCAL_BITS) != blk);
        ext += other ? __ffs(static_cast<int>(other)) - 1 : 32;
      }
    }
    __syncwarp();
    int32_t next[PER];  // first head behind each window
    next[PER - 1] = FLAT_TILE + ext;
#pragma unroll
    for (int u = PER - 2; u >= 0; --u)
      next[u] = heads[u + 1] ? (u + 1) * 32 + __ffs(static_cast<int>(heads[u + 1])) - 1 : next[u + 1];
    int32_t run = -1;  // first entry of the run in hand; -1: the tile before does it
    bool any_long = false;
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int e = u * 32 + lane;
      const uint32_t m = heads[u] & upto, after = heads[u] & ~upto;
      const int32_t s = m ? u * 32 + 31 - __clz(static_cast<int>(m)) : run;
      const int32_t end = after ? u * 32 + __ffs(static_cast<int>(after)) - 1 : next[u];
      if (heads[u]) run = u * 32 + 31 - __clz(static_cast<int>(heads[u]));
      if (s >= 0 && e < cnt) {
        if (flat_short(s, end)) {
          int32_t at = t0 + s;
          for (int32_t j = s; j < end; ++j) at += sh.key[j] < key[u] ? 1 : 0;
          a.ind_new[at] = key[u];
          if (VALUES) a.val_new[at] = val[u];
        } else {
          any_long = true;
        }
      }
    }
    if (run >= 0 && lane < ext && flat_short(run, FLAT_TILE + ext)) {
      int32_t at = t0 + run;
      for (int32_t j = run; j < FLAT_TILE + ext; ++j) at += sh.key[j] < more ? 1 : 0;
      a.ind_new[at] = more;
      if (VALUES) a.val_new[at] = more_val;
    }
    if (__any_sync(FULL, any_long)) {
#pragma unroll 1
      for (int u = 0; u < PER; ++u) {
        uint32_t h = 0u;
        int32_t behind = 0;
#pragma unroll
        for (int v = 0; v < PER; ++v)
          if (v == u) {
            h = heads[v];
            behind = next[v];
          }
        while (h) {
          const int32_t s = u * 32 + __ffs(static_cast<int>(h)) - 1;
          h &= h - 1u;
          const int32_t end = h ? u * 32 + __ffs(static_cast<int>(h)) - 1 : behind;
          if (s >= cnt || flat_short(s, end)) continue;
          int32_t row = -1;  // where the run's row begins in the tile
          for (int v = 0; v <= u; ++v) {
            const uint32_t m = v < u ? sh.row_head[v] : sh.row_head[v] & (FULL >> (31 - (s & 31)));
            if (m) row = v * 32 + 31 - __clz(static_cast<int>(m));
          }
          const FlatRun long_run = {t0 + s, end - s, row >= 0 ? sh.delta[row] : delta0};
          int32_t place = FLAT_QUEUE;
          if (long_run.len > FLAT_DEFER) {
            if (lane == 0) place = atomicAdd(&later.queued, 1);
            place = __shfl_sync(FULL, place, 0);
          }
          if (place < FLAT_QUEUE) {
            if (lane == 0) later.run[place] = long_run;
          } else {
            flat_run_by_warp(a, sh, long_run, s, lane);
          }
        }
      }
    }
    __syncwarp();
  }
  if (ROWS) return;
  __syncthreads();
  const int queued = min(later.queued, FLAT_QUEUE);
  for (int i = 0; i < queued; i += FLAT_WARPS)
    flat_runs_by_block(a, shared, later.run + i, min(queued - i, FLAT_WARPS));
}

// One warp per queued row of 33..R_WARP entries.
__global__ void __launch_bounds__(R_THREADS) apply_warp_kernel(ApplyArgs a) {
  const int lane = threadIdx.x & 31;
  const uint32_t count = a.counters[CNT_WARP];
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t item = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; item < count; item += warps) {
    const int32_t p = a.queue_warp[item];
    const int32_t src_row = a.new_order[p];
    const int32_t src = a.ptr_old[src_row], L = a.ptr_old[src_row + 1] - src;
    const int32_t dst = a.ptr_new[p];
    if (L <= 64) {
      warp_row<2>(a, src, L, dst, lane);
    } else if (L <= 128) {
      warp_row<4>(a, src, L, dst, lane);
    } else {
      warp_row<8>(a, src, L, dst, lane);
    }
  }
}

// ---- up to R_MED entries by one block ---------------------------------------------------
// Shared memory: two copies of (keys, values).  Sorts the L <= R_MED entries that
// fetch(i) delivers (remapped key and value of entry i) and hands entry number q of the
// sorted order to put(q, key, value).  Runs of 256 are sorted in registers by the warps;
// merges by rank: an entry moves to its own index in its run plus the number of smaller
// entries in the partner run.
struct BlockSortShared {
  int32_t key[2][R_MED];
  float val[2][R_MED];
};

// number of entries of run[0..len) below x (keys are distinct)
__device__ __forceinline__ int32_t rank_in_run(const int32_t *run, int32_t len, int32_t x) {
  int32_t lo = 0, hi = len;
  while (lo < hi) {
    const int32_t mid = (lo + hi) >> 1;
    if (run[mid] < x)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

template <typename Fetch, typename Put>
__device__ void block_sort(BlockSortShared &sh, int32_t L, bool with_val, Fetch fetch, Put put) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int WARPS = R_THREADS / 32;
  __syncthreads();  // the buffers may still be read by the previous use
  for (int32_t base = warp * R_WARP; base < L; base += WARPS * R_WARP) {
    int32_t key[8];
    float val[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int32_t i = base + r * 32 + lane;
      key[r] = 0x7FFFFFFF;
      val[r] = 0.0f;
      if (i < L) fetch(i, key[r], val[r]);
    }
    warp_sort<8>(key, val, lane);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int32_t i = base + r * 32 + lane;
      if (i < L) {  // the padding sorts behind every entry: the run's entries come first
        sh.key[0][i] = key[r];
        if (with_val) sh.val[0][i] = val[r];
      }
    }
  }
  __syncthreads();
  int cur = 0;
  for (int32_t run = R_WARP; run < L || run == R_WARP; run <<= 1) {
    const bool last = (run << 1) >= L;  // the merge that leaves one run: it delivers the result
    for (int32_t i = threadIdx.x; i < L; i += R_THREADS) {
      const int32_t q = i / run, o = i - q * run;
      const int32_t partner = (q ^ 1) * run;
      int32_t plen = L - partner;
      plen = plen < 0 ? 0 : (plen > run ? run : plen);
      const int32_t x = sh.key[cur][i];
      const int32_t at = (q >> 1) * (run << 1) + o + rank_in_run(sh.key[cur] + partner, plen, x);
      const float v = with_val ? sh.val[cur][i] : 0.0f;
      if (last) {
        put(at, x, v);
      } else {
        sh.key[cur ^ 1][at] = x;
        if (with_val) sh.val[cur ^ 1][at] = v;
      }
    }
    __syncthreads();
    if (last) break;
    cur ^= 1;
  }
}

// One block per queued row of R_WARP + 1 .. R_MED entries.
__global__ void __launch_bounds__(R_THREADS) apply_block_kernel(ApplyArgs a) {
  extern __shared__ __align__(16) unsigned char apply_smem[];
  BlockSortShared &sh = *reinterpret_cast<BlockSortShared *>(apply_smem);
  const uint32_t count = a.counters[CNT_BLOCK];
  for (uint32_t item = blockIdx.x; item < count; item += gridDim.x) {
    const int32_t p = a.queue_block[item];
    const int32_t src_row = a.new_order[p];
    const int32_t src = a.ptr_old[src_row], L = a.ptr_old[src_row + 1] - src;
    const int32_t dst = a.ptr_new[p];
    block_sort(
        sh, L, a.val_new != nullptr,
        [&](int32_t i, int32_t &k, float &v) {
          k = a.old2new[a.ind_old[src + i]];
          if (a.val_new) v = a.val_old[src + i];
        },
        [&](int32_t q, int32_t k, float v) {
          a.ind_new[dst + q] = k;
          if (a.val_new) a.val_new[dst + q] = v;
        });
  }
}

// ---- rows longer than R_MED ----------------------------------------------------------------
struct LongTile {
  int32_t src, L, dst, tile, tiles;
};
// tile number -> its row (binary search on the queue entries' first tile numbers, ascending
// by construction) and its place in the row
__device__ __forceinline__ LongTile long_tile(const ApplyArgs &a, int32_t id, int32_t queued) {
  int32_t lo = 0, hi = queued;  // queue_long[lo].y <= id < queue_long[hi].y
  while (hi - lo > 1) {
    const int32_t mid = (lo + hi) >> 1;
    if (a.queue_long[mid].y <= id)
      lo = mid;
    else
      hi = mid;
  }
  const int2 q = a.queue_long[lo];
  const int32_t src_row = a.new_order[q.x];
  LongTile t;
  t.src = a.ptr_old[src_row];
  t.L = a.ptr_old[src_row + 1] - t.src;
  t.dst = a.ptr_new[q.x];
  t.tile = id - q.y;
  t.tiles = (t.L + R_MED - 1) / R_MED;
  return t;
}

// One block per tile of R_MED entries of a long row: remapped and sorted into the scratch copy.
__global__ void __launch_bounds__(R_THREADS) apply_tiles_kernel(ApplyArgs a) {
  extern __shared__ __align__(16) unsigned char apply_smem[];
  BlockSortShared &sh = *reinterpret_cast<BlockSortShared *>(apply_smem);
  const int32_t queued = static_cast<int32_t>(a.counters[CNT_LONG + 1]);
  const int32_t total = static_cast<int32_t>(a.counters[CNT_LONG]);
  for (int32_t id = blockIdx.x; id < total; id += gridDim.x) {
    const LongTile t = long_tile(a, id, queued);
    const int32_t off = t.tile * R_MED;
    const int32_t len = t.L - off < R_MED ? t.L - off : R_MED;
    block_sort(
        sh, len, a.val_new != nullptr,
        [&](int32_t i, int32_t &k, float &v) {
          k = a.old2new[a.ind_old[t.src + off + i]];
          if (a.val_new) v = a.val_old[t.src + off + i];
        },
        [&](int32_t q, int32_t k, float v) {
          a.tmp_key[t.dst + off + q] = k;
          if (a.val_new) a.tmp_val[t.dst + off + q] = v;
        });
  }
}

// One block per tile again: every entry goes to the sum of its ranks in all tiles of its row
// (its own index in its own tile).
__global__ void __launch_bounds__(R_THREADS) apply_merge_kernel(ApplyArgs a) {
  const int32_t queued = static_cast<int32_t>(a.counters[CNT_LONG + 1]);
  const int32_t total = static_cast<int32_t>(a.counters[CNT_LONG]);
  for (int32_t id = blockIdx.x; id < total; id += gridDim.x) {
    const LongTile t = long_tile(a, id, queued);
    const int32_t off = t.tile * R_MED;
    const int32_t len = t.L - off < R_MED ? t.L - off : R_MED;
    const int32_t *row = a.tmp_key + t.dst;
    for (int32_t i = threadIdx.x; i < len; i += R_THREADS) {
      const int32_t x = row[off + i];
      int32_t at = i;
      for (int32_t other = 0; other < t.tiles; ++other) {
        if (other == t.tile) continue;
        const int32_t oo = other * R_MED;
        at += rank_in_run(row + oo, t.L - oo < R_MED ? t.L - oo : R_MED, x);
      }
      a.ind_new[t.dst + at] = x;
      if (a.val_new) a.val_new[t.dst + at] = a.tmp_val[t.dst + off + i];
    }
  }
}


// Scratch of one call.  The list of rows that apply_flat_kernel reads and the sorted tiles of the other route share
// their place: no call needs both.
struct ReorderScratch {
  size_t block_sums, counters, queue_warp, queue_block, queue_long, tile_row, old2new, row_at, tmp_key, tmp_val, bytes;
  int32_t rows_max;
  ReorderScratch(int32_t n, int32_t nnz, bool symmetric) {
    const size_t rows = static_cast<size_t>(n), z = static_cast<size_t>(nnz > 0 ? nnz : 1);
    rows_max = std::min(std::min(n, nnz), INT32_MAX - 1) + 1;  // and one behind the last
    Arena ar;
    block_sums = ar.take(sizeof(RowCount) * ((rows + R_SCAN_TILE - 1) / R_SCAN_TILE));
    counters = ar.take(256);
    queue_warp = ar.take(sizeof(int32_t) * (static_cast<size_t>(nnz) / 32 + 1));       // rows of 33..R_WARP entries
    queue_block = ar.take(sizeof(int32_t) * (static_cast<size_t>(nnz) / R_WARP + 1));  // rows of up to R_MED
    queue_long = ar.take(sizeof(int2) * (static_cast<size_t>(nnz) / R_MED + 1));       // longer rows
    tile_row = ar.take(sizeof(int32_t) * (static_cast<size_t>(nnz) / FLAT_TILE + 2));
    old2new = symmetric ? ar.take(sizeof(int32_t) * rows) : 0;
    Arena tiles = ar;
    tmp_key = symmetric ? tiles.take(sizeof(int32_t) * z) : 0;
    tmp_val = symmetric ? tiles.take(sizeof(float) * z) : 0;
    row_at = ar.take(sizeof(int2) * static_cast<size_t>(rows_max));
    bytes = std::max(ar.off, tiles.off);
  }
};

}  // namespace

bool launch_reorder(Context &ctx, int32_t n, int32_t nnz, const int32_t *d_ptr_old,
                    const int32_t *d_ind_old, const float *d_val_old, const int32_t *d_new_order,
                    int mode, int32_t *d_ptr_new, int32_t *d_ind_new, float *d_val_new) {
  const bool symmetric = mode == 1;
  const bool with_vals = d_val_old != nullptr && d_val_new != nullptr;
  const ReorderScratch lay(n, nnz, symmetric);
  if (!ensure_workspace(ctx, lay.bytes)) return false;
  const int32_t nb = (n + R_SCAN_TILE - 1) / R_SCAN_TILE;
  RowCount *block_sums = reinterpret_cast<RowCount *>(ctx.ws + lay.block_sums);
  ApplyArgs a;
  a.n = n;
  a.nnz = nnz;
  a.ptr_old = d_ptr_old;
  a.ind_old = d_ind_old;
  a.val_old = with_vals ? d_val_old : nullptr;
  a.new_order = d_new_order;
  a.ptr_new = d_ptr_new;
  a.ind_new = d_ind_new;
  a.val_new = with_vals ? d_val_new : nullptr;
  a.counters = reinterpret_cast<uint32_t *>(ctx.ws + lay.counters);
  a.queue_warp = reinterpret_cast<int32_t *>(ctx.ws + lay.queue_warp);
  a.queue_block = reinterpret_cast<int32_t *>(ctx.ws + lay.queue_block);
  a.queue_long = reinterpret_cast<int2 *>(ctx.ws + lay.queue_long);
  int32_t *tile_row = reinterpret_cast<int32_t *>(ctx.ws + lay.tile_row);
  int2 *row_at = reinterpret_cast<int2 *>(ctx.ws + lay.row_at);
  a.tile_row = tile_row;
  a.row_at = row_at;
  a.rows_max = lay.rows_max;
  int32_t *old2new = symmetric ? reinterpret_cast<int32_t *>(ctx.ws + lay.old2new) : nullptr;
  a.old2new = old2new;
  a.tmp_key = symmetric ? reinterpret_cast<int32_t *>(ctx.ws + lay.tmp_key) : nullptr;
  a.tmp_val = symmetric ? reinterpret_cast<float *>(ctx.ws + lay.tmp_val) : nullptr;
  CSG_CUDA(cudaMemsetAsync(a.counters, 0, 8 * sizeof(uint32_t), ctx.stream));
  volatile uint32_t *const outcome = outcome_words(ctx, OUTCOME_WORD);
  ++ctx.outcome_ticket;
  len_block_sums_kernel<<<nb, R_THREADS, 0, ctx.stream>>>(n, d_ptr_old, d_new_order, block_sums, a.counters + CNT_MOVED,
                                                          symmetric ? outcome : nullptr, ctx.outcome_ticket);
  CSG_CUDA(cudaGetLastError());
  if (nb > SCAN_IN_PLACE) {
    CSG_CUDA(launch_behind(true, scan_block_sums_kernel, 1, 1024, 0, ctx.stream, nb, block_sums));
    count_launches(1);
  }
  CSG_CUDA(launch_behind(true, ptr_new_kernel, nb, R_THREADS, 0, ctx.stream, n, nnz, d_ptr_old, d_new_order, block_sums,
                         d_ptr_new, old2new, tile_row, row_at, lay.rows_max));
  count_launches(2);
  if (nnz == 0) return true;
  bool local = false;
  if (symmetric) {
    if (!wait_outcome(ctx, ctx.stream, OUTCOME_WORD, ctx.outcome_ticket)) return false;
    local = outcome[1] == 0u;
  }
  if (!symmetric || local) {
    constexpr int64_t block = static_cast<int64_t>(FLAT_TILE) * FLAT_WARPS;
    int64_t grid = (static_cast<int64_t>(nnz) + block - 1) / block;
    if (grid > ctx.num_sms * 32) grid = ctx.num_sms * 32;
    auto kernel = symmetric ? (with_vals ? apply_flat_kernel<false, true> : apply_flat_kernel<false, false>)
                            : (with_vals ? apply_flat_kernel<true, true> : apply_flat_kernel<true, false>);
    CSG_CUDA(launch_behind(true, kernel, static_cast<int>(grid), R_THREADS, 0, ctx.stream, a));
    count_launches(1);
    return true;
  }
  const int sort_smem = static_cast<int>(sizeof(BlockSortShared));
  CSG_CUDA(cudaFuncSetAttribute(apply_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sort_smem));
  CSG_CUDA(cudaFuncSetAttribute(apply_tiles_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sort_smem));
  int64_t want = ((static_cast<int64_t>(n) + 31) / 32 * 32 + R_THREADS - 1) / R_THREADS;
  int grid = static_cast<int>(want < ctx.num_sms * 8 ? want : ctx.num_sms * 8);
  if (grid < 1) grid = 1;
  apply_short_kernel<<<grid, R_THREADS, 0, ctx.stream>>>(a);
  CSG_CUDA(cudaGetLastError());
  apply_warp_kernel<<<ctx.num_sms * 6, R_THREADS, 0, ctx.stream>>>(a);
  CSG_CUDA(cudaGetLastError());
  apply_block_kernel<<<ctx.num_sms * 3, R_THREADS, sort_smem, ctx.stream>>>(a);
  CSG_CUDA(cudaGetLastError());
  apply_tiles_kernel<<<ctx.num_sms * 3, R_THREADS, sort_smem, ctx.stream>>>(a);
  CSG_CUDA(cudaGetLastError());
  apply_merge_kernel<<<ctx.num_sms * 4, R_THREADS, 0, ctx.stream>>>(a);
  CSG_CUDA(cudaGetLastError());
  count_launches(5);
  return true;
}

}  // namespace csg
