// Per-row Space-Saving sketch over the in-chunk candidate stream, then top-k.
//
// Semantics restated from the reference, bit for bit:
//   stream order  sporder/src/common/chunk_similarity_top_k.cu:52-84
//                 (columns of the row ascending; rows of a column ascending;
//                 only rows of the row's own chunk, never the row itself)
//   Dice term     :73-75  alpha = 2.0f / float(|r| + |s|), IEEE fp32 divide
//   container     sporder/src/common/warp_spacesaving.cuh:31-44,109-150
//                 (hit: w += alpha; else first empty slot in (lane, cell) order;
//                 else evict the slot with the least (weight, cell, lane) and
//                 give it weight min + alpha)
//   top-k         :46-66,71-90 (per-lane selection sort by weight, then k rounds
//                 of arg-max over the lanes' cursors, ties to the smaller lane)
//
// What differs is the machinery:
//  * rows come from a work list ordered by the length of their stream, longest first: a
//    stream is an order-dependent chain;
//  * the longest rows (65536 candidates or more, and of the shorter ones as many as let both kernels end
//    soonest) set the run time.  Their streams are written out to memory by the whole grid (heavy_expand_kernel,
//    one warp per 128 columns); then a group of warps works on each row and resolves up to 64
//    candidates per round (see "the chains in rounds" below);
//  * all other rows run side by side, one per LANE: the container of a row is a column of
//    shared memory, a step of 32 rows costs a warp little more than a step of one row did, and
//    further warps of the block produce the streams (see "a row per lane" below).  This
//    kernel follows the chain kernel as a programmatic dependent launch, so that its blocks
//    settle beside that kernel's on the same SMs;
//  * sketches of more than 128 slots keep one warp per row, its slots in the lanes' registers;
//    a step on a full sketch costs three redux.sync (see Sketch::add_full), and their heaviest
//    rows run one warp per scheduler (heavy_consume_kernel);
//  * a large call runs in two parts (see run_csg): the longest rows of the chunk with the most
//    nonzeros on a stream of their own, ahead of the rest.  Both parts go through launch_cells
//    with their own lists and control words.
#include "common.cuh"

namespace csg {

namespace {

constexpr int S_WARPS = 4;
constexpr int S_THREADS = 32 * S_WARPS;
constexpr int S_RING = 256;    // stream elements per batch, light rows
constexpr int H_PART = SKETCH_PART_COLS;  // columns of a heavy row expanded by one warp: small enough
                                         // that a slice of hub columns (up to chunk-1 candidates
                                         // each) does not become the last warp to finish
constexpr int LANE_CELLS = 4;  // largest sketch (cells per lane) kept by one lane (rows_in_lanes_kernel)
constexpr int S_LONG = 48;     // groups with at least this many pending entries are copied by the whole warp

struct SketchArgs {
  int32_t n, nnz, k, row_base, chunk;
  const int32_t *ptr;
  const int2 *seg;
  const int32_t *seg_rank, *row_seg, *row_cols;
  const int2 *cand;
  const int32_t *row_list;
  const uint32_t *row_work;
  uint32_t *ctrl;
  uint64_t *table;
  // materialised streams of the heavy rows
  int2 *hstream;
  uint32_t *heavy_off;
  int32_t *heavy_state;
  uint32_t stream_cap, heavy_max;
  uint32_t *part_base;  // first part of each heavy row, plus the total
  uint32_t *part_off;   // per part: entries it produces
};

// The sketch of one row: CELLS slots per lane, all in registers.  Slot (lane, cell) is
// the (lane*CELLS + cell)-th to be filled; its number is lane*CELLS + cell.
template <int CELLS>
struct Sketch {
  int32_t key[CELLS];
  float w[CELLS];
  int32_t filled;      // warp-uniform
  // valid while the sketch is full:
  uint32_t gmin;       // weight bits of the slot the next miss evicts (same in all lanes)
  int32_t gown;        // its lane
  int32_t gcell;       // its cell
  uint32_t l1w, l2w;   // this lane's smallest and second smallest weight (bits) ...
  int32_t l1c, l2c;    // ... and their cells, ordered by (weight, cell)
  int32_t lane;        // read once through volatile asm: a re-read of the special
                       // register inside the dependent chain costs ~25 cycles each time

  __device__ __forceinline__ void bind_lane() {
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));
  }

  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int c = 0; c < CELLS; ++c) {
      key[c] = -1;
      w[c] = 0.0f;
    }
    filled = 0;
    gmin = 0;
    gown = gcell = 0;
    l1w = l2w = 0;
    l1c = l2c = 0;
  }

  // Weights are positive, so their bit patterns order like the values.  Strict
  // comparisons keep the smaller cell first among equal weights.
  __device__ __forceinline__ void lane_top2() {
    l1w = __float_as_uint(w[0]);
    l1c = 0;
    l2w = 0xFFFFFFFFu;
    l2c = CELLS;  // "none": loses every tie
#pragma unroll
    for (int c = 1; c < CELLS; ++c) {
      const uint32_t x = __float_as_uint(w[c]);
      const bool first = x < l1w, second = x < l2w;
      l2w = first ? l1w : (second ? x : l2w);
      l2c = first ? l1c : (second ? c : l2c);
      l1w = first ? x : l1w;
      l1c = first ? c : l1c;
    }
  }

  // Victim of the next eviction given every lane's smallest (weight, cell): the least
  // (weight, cell, lane).  Two dependent redux.sync.
  __device__ __forceinline__ void find_victim(uint32_t lw, int32_t lc, uint32_t &vmin, int32_t &vown,
                                              int32_t &vcell) const {
    vmin = __reduce_min_sync(FULL, lw);
    const uint32_t t = (lw == vmin) ? static_cast<uint32_t>((lc << 5) | lane) : 0xFFFFFFFFu;
    const uint32_t win = __reduce_min_sync(FULL, t);
    vown = static_cast<int32_t>(win & 31u);
    vcell = static_cast<int32_t>(win >> 5);
  }

  __device__ __forceinline__ void refresh_victim() {
    lane_top2();
    find_victim(l1w, l1c, gmin, gown, gcell);
  }

  // slot (lane, cell) holding key s, or -1.  Warp-uniform result.
  __device__ __forceinline__ int32_t find_slot(int32_t s) const {
    int hit_cell = -1;
#pragma unroll
    for (int c = 0; c < CELLS; ++c) hit_cell = (key[c] == s) ? c : hit_cell;
    const uint32_t hs = __reduce_min_sync(
        FULL, hit_cell >= 0 ? static_cast<uint32_t>(lane * CELLS + hit_cell) : 0xFFFFFFFFu);
    return static_cast<int32_t>(hs);
  }

  __device__ __forceinline__ void add_weight(int32_t slot, float a) {
    const int hl = slot / CELLS, hc = slot % CELLS;
    const bool me = lane == hl;
#pragma unroll
    for (int c = 0; c < CELLS; ++c) w[c] = (me & (c == hc)) ? w[c] + a : w[c];
  }

  __device__ __forceinline__ void put(int32_t slot, int32_t s, float wv) {
    const int ol = slot / CELLS, oc = slot % CELLS;
    const bool me = lane == ol;
#pragma unroll
    for (int c = 0; c < CELLS; ++c) {
      const bool p = me & (c == oc);
      w[c] = p ? wv : w[c];
      key[c] = p ? s : key[c];
    }
  }

  // one stream element while the sketch still has empty slots
  __device__ __forceinline__ void add_filling(int32_t s, float a) {
    const int32_t slot = find_slot(s);
    if (slot >= 0) {
      add_weight(slot, a);
      return;
    }
    put(filled, s, a);
    ++filled;
    if (filled == 32 * CELLS) refresh_victim();
  }

  // One stream element with the sketch full.  Only the victim's lane can change its
  // smallest weight on a miss, and its new smallest is either the re-inserted slot or
  // its cached second smallest: the speculative victim search therefore starts after one
  // add, one compare and one select, and the bookkeeping of the lane's own top-2 runs
  // beside the reductions instead of in front of them.  Written with selects only: a
  // lane-divergent branch here costs more than the rest of the step.
  __device__ __forceinline__ void add_full(int32_t s, float a) {
    const bool own = lane == gown;
    const float wnew = __uint_as_float(gmin) + a;
    const uint32_t nb = __float_as_uint(wnew);
    const int32_t slot = find_slot(s);
    // speculation: this element misses and replaces the cached victim
    const bool new_first = (nb < l2w) | ((nb == l2w) & (gcell < l2c));
    const uint32_t sw = own ? (new_first ? nb : l2w) : l1w;
    const int32_t sc = own ? (new_first ? gcell : l2c) : l1c;
    uint32_t smin;
    int32_t sown, scell;
    find_victim(sw, sc, smin, sown, scell);
    if (slot < 0) {  // miss (warp-uniform): commit
      const int32_t gslot = gown * CELLS + gcell;
      put(gslot, s, wnew);
      if (CELLS <= 2) {  // the lane's pair, reordered
        l2w = own ? (new_first ? l2w : nb) : l2w;
        l2c = own ? (new_first ? l2c : gcell) : l2c;
        l1w = sw;
        l1c = sc;
      } else {
        lane_top2();
      }
      gmin = smin;
      gown = sown;
      gcell = scell;
    } else {  // hit: the speculation is void
      add_weight(slot, a);
      lane_top2();
      if (slot / CELLS == gown) find_victim(l1w, l1c, gmin, gown, gcell);
    }
  }

  __device__ __forceinline__ void local_sort_descending() {
    // the reference's selection sort, including where it stops
#pragma unroll
    for (int i = 0; i < CELLS - 1; ++i) {
      if (key[i] == -1) break;
      int best = i;
      float best_w = w[i];
#pragma unroll
      for (int j = i + 1; j < CELLS; ++j) {
        if (key[j] == -1) break;
        if (w[j] > best_w) {
          best = j;
          best_w = w[j];
        }
      }
      if (best != i) {
        // dynamic register index: resolved with selects after unrolling
        int32_t bk = key[i];
        float bw = w[i];
#pragma unroll
        for (int j = i + 1; j < CELLS; ++j) {
          if (j == best) {
            const int32_t tk = key[j];
            const float tw = w[j];
            key[j] = bk;
            w[j] = bw;
            bk = tk;
            bw = tw;
          }
        }
        key[i] = bk;
        w[i] = bw;
      }
    }
  }

  // writes the row's k entries: the valid prefix, then zeros
  __device__ __forceinline__ void select_top_k(int32_t k, uint64_t *out, int32_t row_base) {
    local_sort_descending();
    int pos = 0;
    uint64_t mine = 0;
    int i = 0;
    for (; i < k; ++i) {
      float wc = 0.0f;
      int32_t kc = -1;
#pragma unroll
      for (int c = 0; c < CELLS; ++c) {
        if (c == pos) {
          wc = w[c];
          kc = key[c];
        }
      }
      const uint32_t wb = __float_as_uint(wc);
      const uint32_t g = __reduce_max_sync(FULL, wb);
      if (g == 0u) break;  // every lane is past its last filled slot
      const int wl = __ffs(__ballot_sync(FULL, wb == g)) - 1;
      const int32_t ek = __shfl_sync(FULL, kc, wl);
      if (lane == (i & 31)) mine = pack_entry(ek + row_base, __uint_as_float(g));
      if (lane == wl) ++pos;
      if ((i & 31) == 31) {
        out[(i - 31) + lane] = mine;
        mine = 0;
      }
    }
    if ((i & 31) != 0 && lane < (i & 31)) out[(i & ~31) + lane] = mine;
    for (int j = i + lane; j < k; j += 32) out[j] = 0;  // the stages behind stop at the first empty entry
  }
};

// Producer side of one row: walks the row's column groups 32 at a time (one per lane)
// and writes the stream, in order and without the row itself, into the warp's ring.
template <int RING>
struct Producer {
  const SketchArgs &a;
  int32_t r, rb, re, rs;
  int32_t pb;         // CSR position of lane 0's column in the current window
  int32_t gst, glen;  // this lane's group: first entry, length (0 when it has no candidates)
  int32_t grank;      // index of row r inside the group
  int32_t done;       // stream entries of this lane's group already produced
  int2 nsg;           // next window, requested one window ahead
  int32_t nrank;

  __device__ __forceinline__ Producer(const SketchArgs &args) : a(args) {}

  // cand[idx], idx from a group descriptor the transpose wrote (checked build: tested)
  __device__ __forceinline__ int2 cand_at(int32_t idx) const {
    return index_ok(a.ctrl, CHK_CAND, idx, a.nnz) ? a.cand[idx] : make_int2(r, 1);
  }

  __device__ __forceinline__ void load_next(int32_t p) {
    nsg = make_int2(0, 0);
    nrank = 0;
    if (p < re) {
      nsg = a.seg[p];
      nrank = a.seg_rank[p];
    }
  }
  __device__ __forceinline__ void take_window() {
    gst = nsg.x;
    glen = nsg.y >= 2 ? nsg.y : 0;
    grank = nrank;
    done = 0;
  }
  // columns [row_begin, row_end) of row `row` (CSR positions), which has row_size entries
  __device__ __forceinline__ void begin(int32_t row, int32_t row_begin, int32_t row_end,
                                        int32_t row_size) {
    r = row;
    rb = row_begin;
    re = row_end;
    rs = row_size;
    pb = rb;
    load_next(pb + lane_id());
    take_window();
    load_next(pb + 32 + lane_id());
  }

  // entry q of this lane's group with the row itself skipped -> (row, alpha)
  __device__ __forceinline__ void emit(int32_t q, int32_t *ring_s, float *ring_a, int32_t at) const {
    const int2 e = cand_at(gst + q + (q >= grank ? 1 : 0));
    ring_s[at] = e.x;
    ring_a[at] = 2.0f / static_cast<float>(rs + e.y);
  }

  // Fills the ring with up to RING elements; returns how many.  0 = stream finished.
  __device__ __forceinline__ int produce(int32_t *ring_s, float *ring_a) {
    const int lane = lane_id();
    int fill = 0;
    for (;;) {
      const int32_t rem = glen > 0 ? glen - 1 - done : 0;
      const unsigned pending = __ballot_sync(FULL, rem > 0);
      if (pending == 0u) {  // window exhausted: next 32 columns
        pb += 32;
        if (pb >= re) break;
        take_window();
        load_next(pb + 32 + lane);
        continue;
      }
      if (fill >= RING) break;
      const unsigned longs = __ballot_sync(FULL, rem >= S_LONG);
      const int first = __ffs(pending) - 1;
      if ((longs >> first) & 1u) {
        // the next group in stream order is a long one: whole warp, coalesced
        const int32_t g_st = __shfl_sync(FULL, gst, first);
        const int32_t g_rank = __shfl_sync(FULL, grank, first);
        const int32_t g_done = __shfl_sync(FULL, done, first);
        const int32_t g_rem = __shfl_sync(FULL, rem, first);
        const int32_t take = g_rem < RING - fill ? g_rem : RING - fill;
        for (int32_t i0 = 0; i0 < take; i0 += 128) {
          int2 e[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int32_t q = g_done + i0 + u * 32 + lane;
            if (i0 + u * 32 + lane < take) e[u] = cand_at(g_st + q + (q >= g_rank ? 1 : 0));
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int32_t i = i0 + u * 32 + lane;
            if (i < take && index_ok(a.ctrl, CHK_RING, fill + i, RING)) {
              ring_s[fill + i] = e[u].x;
              ring_a[fill + i] = 2.0f / static_cast<float>(rs + e[u].y);
            }
          }
        }
        if (lane == first) done += take;
        fill += take;
        continue;
      }
      // leading run of short groups, from `first` up to (not including) the first long
      // group: lane-parallel, ring positions from a prefix sum
      const unsigned later_longs = longs & ~((1u << first) - 1u);
      const int stop = later_longs ? __ffs(later_longs) - 1 : 32;
      const int32_t mine = (lane >= first && lane < stop) ? rem : 0;
      int32_t incl = mine;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int32_t t = __shfl_up_sync(FULL, incl, off);
        if (lane >= off) incl += t;
      }
      const int32_t space = RING - fill;
      const int32_t before = incl - mine;
      int32_t take = space - before;
      take = take < 0 ? 0 : (take > mine ? mine : take);
      {
        // eight independent loads in flight per lane: the copy is latency bound otherwise
        const int32_t at0 = fill + before;
        int32_t i = 0;
        for (; i + 8 <= take; i += 8) {
          int2 e[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int32_t q = done + i + u;
            e[u] = cand_at(gst + q + (q >= grank ? 1 : 0));
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            if (index_ok(a.ctrl, CHK_RING, at0 + i + u, RING)) {
              ring_s[at0 + i + u] = e[u].x;
              ring_a[at0 + i + u] = 2.0f / static_cast<float>(rs + e[u].y);
            }
          }
        }
        int2 e[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int32_t q = done + i + u;
          if (i + u < take) e[u] = cand_at(gst + q + (q >= grank ? 1 : 0));
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          if (i + u < take && index_ok(a.ctrl, CHK_RING, at0 + i + u, RING)) {
            ring_s[at0 + i + u] = e[u].x;
            ring_a[at0 + i + u] = 2.0f / static_cast<float>(rs + e[u].y);
          }
        }
      }
      done += take;
      const int32_t total = __shfl_sync(FULL, incl, 31);
      fill += total < space ? total : space;
    }
    __syncwarp();
    return fill;
  }
};

// Feeds `cnt` staged stream elements to the sketch.
template <int CELLS>
__device__ __forceinline__ void consume(Sketch<CELLS> &sk, const int32_t *bs, const float *ba,
                                        int cnt) {
  int t = 0;
  for (; t < cnt && sk.filled < 32 * CELLS; ++t) sk.add_filling(bs[t], ba[t]);
  if (t < cnt) {  // full sketch: the dependent chain, next element requested one step ahead
    int32_t ns = bs[t];
    float na = ba[t];
#pragma unroll 1
    for (; t < cnt; ++t) {
      const int32_t cs = ns;
      const float cf = na;
      const int nt = t + 1 < cnt ? t + 1 : t;
      ns = bs[nt];
      na = ba[nt];
      sk.add_full(cs, cf);
    }
  }
}

// A stream key as an index into a table over the chunk's rows: in the checked build a key
// outside the chunk is recorded and replaced by the chunk's first row.
__device__ __forceinline__ int32_t key_in_chunk(uint32_t *ctrl, int32_t s, int32_t cbase, int32_t span) {
  return index_ok(ctrl, CHK_KEY, static_cast<long long>(s) - cbase, span) ? s : cbase;
}

__device__ __forceinline__ bool row_bounds_ok(const SketchArgs &a, int32_t rb, int32_t re) {
  if (rb < 0 || re < rb || re > a.nnz) {  // malformed row pointers: flag and skip
    if (lane_id() == 0) atomicExch(&a.ctrl[CTRL_BAD_INPUT], 1u);
    return false;
  }
  return true;
}

// Rows [ticket, end) of the list, one warp per row, producing and consuming in turn.
template <int CELLS>
__device__ __forceinline__ void rows_by_warp(const SketchArgs &a, uint32_t end, int32_t *bs, float *ba) {
  const int lane = lane_id();
  Sketch<CELLS> sk;
  sk.bind_lane();
  Producer<S_RING> prod(a);
  for (;;) {
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(&a.ctrl[CTRL_ROW_TICKET], 1u);  // starts after the heavy rows
    item = __shfl_sync(FULL, item, 0);
    if (item >= end) break;
    const int32_t r = a.row_list[item];
    if (!index_ok(a.ctrl, CHK_LIST, r, a.n)) continue;
    const int32_t rb = a.ptr[r], re = a.ptr[r + 1];
    if (!row_bounds_ok(a, rb, re)) continue;
    sk.clear();
    prod.begin(r, a.row_seg[r], a.row_seg[r] + a.row_cols[r], re - rb);
    for (;;) {
      const int cnt = prod.produce(bs, ba);
      if (cnt == 0) break;
      consume<CELLS>(sk, bs, ba, cnt);
      __syncwarp();
    }
    sk.select_top_k(a.k, a.table + static_cast<size_t>(r) * a.k, a.row_base);
  }
}

// all: every row the chain kernel leaves (sketches of more than LANE_CELLS cells per lane; the
// others go to rows_in_lanes_kernel).  Otherwise only the rows of heavy weight that did not fit
// the stream buffer.
template <int CELLS>
__global__ void __launch_bounds__(S_THREADS) sketch_kernel(SketchArgs a, int all, int after_primary) {
  __shared__ int32_t ring_s[S_WARPS][S_RING];
  __shared__ float ring_a[S_WARPS][S_RING];
  const int warp = threadIdx.x >> 5;
  rows_by_warp<CELLS>(a, a.ctrl[all ? CTRL_ROWS_LISTED : CTRL_MID_END], ring_s[warp], ring_a[warp]);
  // Launched as the programmatic dependent of the heavy-chain kernel, this kernel starts
  // while that one is still running; it must not be seen as finished before it.
  if (after_primary) wait_for_kernels_before();
}

// ---- a row per lane -----------------------------------------------------------------------
// Most candidates of a large call belong to rows of middling length, far more rows than the
// GPU has warps.  What counts for them is instructions per candidate, and a warp that works on
// one row spends all its 32 lanes on one candidate (56 warp instructions each, measured).  Here
// every LANE has a row of its own: 32 sequential containers side by side, each in a column of
// shared memory (word i of lane l at [i * 32 + l], so that lanes reading different places never
// meet in a bank), some 170 instructions per step of up to 32 candidates.
//   * W[code]: weight bits of slot `code` (cell * 32 + lane in the container's terms, so that
//     the eviction order (weight, cell, lane) is (weight, code)), ~0 while the slot is empty;
//   * an index from key to slot: a byte per row of the chunk (TableIndex), or for chunks whose
//     tables would leave room for too few warps a chained hash table (ChainIndex);
//   * the least weight of every eight slots, its slot, and the least of those in registers, so
//     that a miss knows its victim.  Hits and misses then recompute one group's least and the
//     least of all in the same way: lanes that do either run together.
// 32 consecutive rows of the list differ by at most a quarter in length, so lanes idle little.
// The containers belong to one warp of a block; four more warps produce the streams, 32
// candidates of a row at a time, into a ring the first warp reads a phase later (a lane that
// walks its row's columns by itself spends a memory latency per candidate: ten times slower).
// At the end of a batch all warps select the rows' top k, by counting ranks.
// What bounds it: the latency of a step (some 550 cycles; a warp alone on a scheduler issues
// every other cycle, and the producing warps take slots as well), then the tail of the longest
// rows.  R-MAT scale 22, everything but the heavy rows (297 M candidates): 25 ms of the GPU with a
// warp per row, 11 ms this way.
constexpr int L_RING = 32;         // candidates produced per row and phase, one per lane of a producing warp
constexpr int L_PRODUCERS = 4;     // producing warps ...
constexpr int L_WARPS = 1 + L_PRODUCERS;
constexpr int L_ROWS = 32 / L_PRODUCERS;  // ... and rows of each
constexpr int L_TABLE_MAX = LANE_TABLE_ROWS;

// Key -> slot by one byte per row of the chunk (0 = not there, else slot + 1).  Keys travel as
// the byte's place in the lane's column of the table; those of the slots, 16 bits each, are
// kept for evictions and for the selection.
template <int CELLS>
struct TableIndex {
  static constexpr int M = 32 * CELLS;
  static __host__ __device__ int quads(int64_t span) { return static_cast<int>((span + 3) / 4); }
  static int words(int64_t span) { return M * 16 + (quads(span) + 1) * 32; }  // (one word more: what an empty slot's key names)
  uint32_t *mem;  // this lane's column of the index's words
  static __device__ __forceinline__ uint32_t encode(uint32_t s) { return (s >> 2) * 128u + (s & 3u); }
  static __device__ __forceinline__ uint32_t decode(uint32_t e) { return (e >> 7) * 4u + (e & 3u); }
  __device__ __forceinline__ uint8_t &place(uint32_t e) { return reinterpret_cast<uint8_t *>(mem + M * 16)[e]; }
  __device__ __forceinline__ uint16_t &stored(int c) { return reinterpret_cast<uint16_t *>(mem + (c >> 1) * 32)[c & 1]; }
  __device__ __forceinline__ uint32_t key(int c) { return decode(stored(c)); }
  __device__ __forceinline__ void init(int64_t span) {
    for (int i = 0; i <= quads(span); ++i) mem[M * 16 + i * 32] = 0u;
    for (int c = 0; c < M; ++c) stored(c) = static_cast<uint16_t>(quads(span) * 128);
  }
  __device__ __forceinline__ int find(uint32_t e) { return static_cast<int>(place(e)); }
  __device__ __forceinline__ void replace(int c, uint32_t e, bool) {
    place(stored(c)) = 0;
    stored(c) = static_cast<uint16_t>(e);
    place(e) = static_cast<uint8_t>(c + 1);
  }
  __device__ __forceinline__ void forget(int c, int64_t span) {
    place(stored(c)) = 0;
    stored(c) = static_cast<uint16_t>(quads(span) * 128);
  }
  __device__ __forceinline__ void forget_all() {}
};

// Key -> slot by hashing: one byte per bucket names the first slot of its chain, a slot's word
// holds its key (24 bits) and the next slot of the chain.  Four to sixteen buckets per slot: the 32
// lanes of a warp wait for the longest chain among them.
template <int CELLS>
struct ChainIndex {
  static constexpr int M = 32 * CELLS;
  static constexpr int BITS = CELLS <= 2 ? 10 : 9;
  static constexpr uint32_t NONE = 0xFFu;
  static int words(int64_t) { return M * 32 + (1 << BITS) / 4 * 32; }
  uint32_t *mem;
  static __device__ __forceinline__ uint32_t encode(uint32_t s) { return s; }
  __device__ __forceinline__ uint8_t &head(uint32_t s) {
    const uint32_t b = (s * 0x9E3779B1u) >> (32 - BITS);
    return reinterpret_cast<uint8_t *>(mem + M * 32 + (b >> 2) * 32)[b & 3u];
  }
  __device__ __forceinline__ uint32_t &entry(uint32_t c) { return mem[c * 32]; }
  __device__ __forceinline__ uint32_t key(int c) { return entry(c) >> 8; }
  __device__ __forceinline__ void init(int64_t) { forget_all(); }
  __device__ __forceinline__ int find(uint32_t s) {  // slot + 1, 0 when the key is not there
    uint32_t c = head(s);
    while (c != NONE) {
      const uint32_t e = entry(c);
      if (e >> 8 == s) return static_cast<int>(c) + 1;
      c = e & 0xFFu;
    }
    return 0;
  }
  __device__ __forceinline__ void replace(int c, uint32_t s, bool used) {
    if (used) {  // out of its chain
      const uint32_t e = entry(c), next = e & 0xFFu;
      uint8_t &first = head(e >> 8);
      uint32_t at = first;
      if (at == static_cast<uint32_t>(c)) {
        first = static_cast<uint8_t>(next);
      } else {
        while (at != NONE) {
          const uint32_t f = entry(at);
          if ((f & 0xFFu) == static_cast<uint32_t>(c)) {
            entry(at) = (f & ~0xFFu) | next;
            break;
          }
          at = f & 0xFFu;
        }
      }
    }
    uint8_t &first = head(s);
    entry(c) = (s << 8) | first;
    first = static_cast<uint8_t>(c);
  }
  __device__ __forceinline__ void forget(int, int64_t) {}
  __device__ __forceinline__ void forget_all() {
    for (int i = 0; i < (1 << BITS) / 4; ++i) mem[M * 32 + i * 32] = 0xFFFFFFFFu;
  }
};

struct LaneShared {
  uint32_t first;          // place in the list of the batch's first row
  int32_t count[2][32];    // candidates in each row's part of the ring's buffers
};

// shared memory of a block, in words: weights, two buffers of the ring (keys, Dice terms), what
// the warps tell one another, then the index.  Outside the phases the ring's words serve the
// top-k selection.
template <int CELLS>
struct LaneLayout {
  static constexpr int M = 32 * CELLS;
  static constexpr int RING_OFF = M * 32;
  static constexpr int BUFFER = 2 * L_RING * 32;
  static constexpr int SHARED_OFF = RING_OFF + 2 * BUFFER;
  static constexpr int I_OFF = SHARED_OFF + sizeof(LaneShared) / 4;
  static_assert(L_WARPS * 2 * S_RING <= I_OFF, "rows_by_warp borrows the memory in front of the index for its rings");
  static_assert(L_WARPS * M <= 2 * BUFFER, "the selection's copies of the weights fit the ring");
};

// Least of N values with what goes with it; the first of equal ones.  A tree, so that a step's
// chain of dependent compares is three or four deep.
template <int N>
__device__ __forceinline__ void least_of(const uint32_t (&v)[N], const int32_t (&tag)[N], uint32_t &best,
                                         int32_t &best_tag) {
  if constexpr (N == 1) {
    best = v[0];
    best_tag = tag[0];
  } else {
    constexpr int H = (N + 1) / 2;
    uint32_t h[H];
    int32_t t[H];
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      bool first;
      h[i] = __vibmin_u32(v[2 * i], v[2 * i + 1], &first);  // minimum and which one it was, one instruction
      t[i] = first ? tag[2 * i] : tag[2 * i + 1];
    }
    if constexpr (N % 2 == 1) {
      h[H - 1] = v[N - 1];
      t[H - 1] = tag[N - 1];
    }
    least_of<H>(h, t, best, best_tag);
  }
}

template <int CELLS, typename Index>
struct LaneSketch {
  static constexpr int M = 32 * CELLS;
  static constexpr int GROUPS = M / 8;
  uint32_t *mem;         // this lane's column of the weights
  Index index;
  uint32_t gw[GROUPS];   // least weight of every eight slots ...
  int32_t gc[GROUPS];    // ... and the first slot that has it
  uint32_t low;          // the least of all of them, which the next miss takes ...
  int32_t victim;        // ... and its slot

  __device__ __forceinline__ uint32_t &weight(int c) { return mem[c * 32]; }
  // The j-th slot to be filled.  While it is empty its weight is the j-th smallest bit pattern:
  // a miss then takes the empty slots in order like any other victim, and that weight vanishes
  // in the first Dice term added to it.
  static __device__ __forceinline__ int code_of(int j) { return (j % CELLS) * 32 + j / CELLS; }

  __device__ __forceinline__ void init(int64_t span) {
    for (int j = 0; j < M; ++j) weight(code_of(j)) = static_cast<uint32_t>(j);
    index.init(span);
    fresh();
  }
  __device__ __forceinline__ void fresh() {
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) {
      gw[g] = static_cast<uint32_t>((g * 8 % 32) * CELLS + g * 8 / 32);
      gc[g] = g * 8;
    }
    low = 0;
    victim = 0;
  }
  __device__ __forceinline__ void clear(int64_t span) {  // back to empty, at the price of what was filled
    for (int j = 0; j < M && weight(code_of(j)) >= static_cast<uint32_t>(M); ++j) {
      weight(code_of(j)) = static_cast<uint32_t>(j);
      index.forget(code_of(j), span);
    }
    index.forget_all();
    fresh();
  }

  // One candidate (e: its key as the index has it, p: what find(e) said), then the look-up of the
  // next one, whose latency passes while this one's group and victim are worked out.
  __device__ __forceinline__ int step(uint32_t e, float al, int p, uint32_t next) {
    const int c = p ? p - 1 : victim;
    const uint32_t held = weight(c);
    if (p == 0) index.replace(c, e, low >= static_cast<uint32_t>(M));
    weight(c) = __float_as_uint(__uint_as_float(held) + al);
    const int found = index.find(next);
    const int g8 = c & ~7;
    uint32_t w[8];
    int32_t tags[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      w[i] = weight(g8 + i);
      tags[i] = i;
    }
    uint32_t least;
    int32_t first;
    least_of<8>(w, tags, least, first);
    first += g8;
#pragma unroll
    for (int i = 0; i < GROUPS; ++i) {
      gw[i] = 8 * i == g8 ? least : gw[i];
      gc[i] = 8 * i == g8 ? first : gc[i];
    }
    least_of<GROUPS>(gw, gc, low, victim);
    return found;
  }
};

// The rows between the chain kernel's and the lanes' own, before those: the long ones of chunks without a
// byte table (bucket_scan_kernel says which), and rows that did not fit the stream buffer (rare: more than
// 2^28 candidates, little memory left, or a caller's bound on the buffer).
template <int CELLS>
__device__ __noinline__ void rows_before_the_lanes(const SketchArgs &a, uint32_t end, uint32_t *mem) {
  mem += (threadIdx.x >> 5) * 2 * S_RING;
  rows_by_warp<CELLS>(a, end, reinterpret_cast<int32_t *>(mem), reinterpret_cast<float *>(mem + S_RING));
}

// A row as a producing warp keeps it: columns [p, re) are left, `q` candidates of column p are
// produced already; rs is the row's length, cbase its chunk's first row.
struct LaneRow {
  int32_t r, p, re, q, rs, cbase;
};
__device__ __forceinline__ LaneRow lane_row(const SketchArgs &a, uint32_t item, uint32_t listed) {
  LaneRow w = {-1, 0, 0, 0, 0, 0};
  if (item < listed) {
    w.r = a.row_list[item];
    if (!index_ok(a.ctrl, CHK_LIST, w.r, a.n)) w.r = -1;
  }
  if (w.r >= 0) {
    w.p = a.ptr[w.r];
    w.re = a.ptr[w.r + 1];
    if (w.p < 0 || w.re < w.p || w.re > a.nnz) {  // malformed row pointers: flag and skip
      atomicExch(&a.ctrl[CTRL_BAD_INPUT], 1u);
      w.r = -1;
      w.p = w.re = 0;
    }
    w.rs = w.re - w.p;
    if (w.r >= 0) {
      w.p = a.row_seg[w.r];
      w.re = w.p + a.row_cols[w.r];
    }
    w.cbase = (w.r / a.chunk) * a.chunk;
  }
  return w;
}

// Place of element u of row l in a ring buffer: shifted by u, so that neither a lane per row
// (the reader) nor a lane per element (the producer) meets another in a bank.
__device__ __forceinline__ int ring_at(int u, int l) { return u * 32 + ((l + u) & 31); }

// A row while its part of a ring buffer is filled: the state of LaneRow, the columns in hand (one
// per lane: group and place of the row in it) and the candidates produced so far.
struct LaneFill {
  int32_t p, q, re, rs, cbase, total;
  int2 sg;
  int32_t rank;
};
__device__ __forceinline__ void load_columns(const SketchArgs &a, LaneFill &f, int lane) {
  f.sg = make_int2(0, 0);
  f.rank = 0;
  if (f.p + lane < f.re) {
    f.sg = a.seg[f.p + lane];
    f.rank = a.seg_rank[f.p + lane];
  }
}
// One window of 32 columns for each of K rows (rows first, first + 1, .. of the batch), side by
// side so that their latencies overlap: lengths, prefix sums, then lane t fetches candidate t,
// whose column it finds by a search over the prefix sums.
template <typename Index, int K>
__device__ __forceinline__ void fill_window(const SketchArgs &a, LaneFill (&f)[K], int first, uint32_t span,
                                            uint32_t *buffer, int lane) {
  int32_t left[K], incl[K], all[K], take[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    left[k] = f[k].sg.y >= 2 ? f[k].sg.y - 1 : 0;  // candidates of this lane's column
    if (lane == 0) left[k] -= f[k].q;
    incl[k] = left[k];
  }
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int32_t t = __shfl_up_sync(FULL, incl[k], off);
      if (lane >= off) incl[k] += t;
    }
  }
  int j[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    all[k] = __shfl_sync(FULL, incl[k], 31);
    take[k] = min(all[k], L_RING - f[k].total);
    j[k] = 0;
  }
#pragma unroll
  for (int step = 16; step > 0; step >>= 1) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int32_t v = __shfl_sync(FULL, incl[k], j[k] + step - 1);
      j[k] += v <= lane - f[k].total ? step : 0;  // this lane fetches candidate lane - total of the window
    }
  }
  int2 e[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int x = lane - f[k].total;
    int32_t ord = x - __shfl_sync(FULL, incl[k] - left[k], j[k]) + (j[k] == 0 ? f[k].q : 0);
    const int32_t start = __shfl_sync(FULL, f[k].sg.x, j[k]), own = __shfl_sync(FULL, f[k].rank, j[k]);
    ord += ord >= own ? 1 : 0;  // the row itself is not its candidate
    e[k] = make_int2(f[k].cbase, 1);
    if (x >= 0 && x < take[k] && index_ok(a.ctrl, CHK_CAND, start + ord, a.nnz)) e[k] = a.cand[start + ord];
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    if (take[k] < all[k]) {  // the window holds more: go on from here next time
      const int jj = __ffs(static_cast<int>(__ballot_sync(FULL, incl[k] > take[k]))) - 1;
      f[k].q = take[k] - __shfl_sync(FULL, incl[k] - left[k], jj) + (jj == 0 ? f[k].q : 0);
      f[k].p += jj;
    } else {
      f[k].p += 32;
      f[k].q = 0;
    }
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int x = lane - f[k].total;
    if (x >= 0 && x < take[k]) {
      const int at = ring_at(lane, first + k);
      // (a key outside the chunk only comes from rows that are not sorted: kept in bounds)
      buffer[at] = Index::encode(
          min(static_cast<uint32_t>(key_in_chunk(a.ctrl, e[k].x, f[k].cbase, a.chunk) - f[k].cbase), span - 1u));
      buffer[L_RING * 32 + at] = __float_as_uint(2.0f / static_cast<float>(f[k].rs + e[k].y));
    }
    f[k].total += take[k];
  }
}

// One phase of a producing warp: the next L_RING candidates of each of its rows.  `mine` is the
// row of lane i < L_ROWS (row number first_row + i of the batch).  The descriptors of the next rows'
// columns are on their way while a pair of rows is worked on.
template <typename Index>
__device__ __forceinline__ void produce_phase(const SketchArgs &a, LaneRow &mine, int first_row, uint32_t span,
                                              uint32_t *buffer, int32_t *count) {
  constexpr int K = 2;
  const int lane = lane_id();
  auto take_rows = [&](int i, LaneFill (&f)[K]) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      f[k].p = __shfl_sync(FULL, mine.p, i + k);
      f[k].q = __shfl_sync(FULL, mine.q, i + k);
      f[k].re = __shfl_sync(FULL, mine.re, i + k);
      f[k].total = 0;
      load_columns(a, f[k], lane);
    }
  };
  LaneFill next[K];
  take_rows(0, next);
#pragma unroll 1
  for (int i = 0; i < L_ROWS; i += K) {
    LaneFill f[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      f[k] = next[k];
      f[k].rs = __shfl_sync(FULL, mine.rs, i + k);
      f[k].cbase = __shfl_sync(FULL, mine.cbase, i + k);
    }
    if (i + K < L_ROWS) take_rows(i + K, next);
    fill_window<Index, K>(a, f, first_row + i, span, buffer, lane);
#pragma unroll
    for (int k = 0; k < K; ++k) {  // few candidates per column: more windows
      while (f[k].total < L_RING && f[k].p < f[k].re) {
        LaneFill one[1] = {f[k]};
        load_columns(a, one[0], lane);
        fill_window<Index, 1>(a, one, first_row + i + k, span, buffer, lane);
        f[k] = one[0];
      }
      if (lane == i + k) {
        mine.p = f[k].p;
        mine.q = f[k].q;
      }
      if (lane == 0) count[first_row + i + k] = f[k].total;
    }
  }
}

// Top k of the rows owner = warp, warp + L_WARPS, ... of the batch.
template <int CELLS, typename Index>
__device__ __forceinline__ void select_phase(const SketchArgs &a, uint32_t *mem, const LaneRow &row_of_lane) {
  using L = LaneLayout<CELLS>;
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  uint32_t *const tw = mem + L::RING_OFF + warp * L::M;
  for (int owner = warp; owner < 32; owner += L_WARPS) {
    const int32_t row = __shfl_sync(FULL, row_of_lane.r, owner);
    if (row < 0) continue;
    const int32_t base = __shfl_sync(FULL, row_of_lane.cbase, owner) + a.row_base;
    Sketch<CELLS> top;  // slot (lane, cell) of the container, as select_top_k has it
    Index theirs;
    theirs.mem = mem + L::I_OFF + owner;
#pragma unroll
    for (int c = 0; c < CELLS; ++c) {
      const int code = c * 32 + lane;
      const uint32_t bits = mem[code * 32 + owner];
      const bool on = bits >= static_cast<uint32_t>(L::M);  // (below: an empty slot)
      top.key[c] = on ? static_cast<int32_t>(theirs.key(code)) : -1;
      top.w[c] = on ? __uint_as_float(bits) : 0.0f;
    }
    int have = 0;
#pragma unroll
    for (int c = 0; c < CELLS; ++c) have += __popc(__ballot_sync(FULL, top.key[c] >= 0));
    top.local_sort_descending();
    // Entry i of lane l is number l * CELLS + i; the selection takes the heaviest first, on
    // ties the smaller number: an entry's place is how many come before it.
    __syncwarp();
#pragma unroll
    for (int c = 0; c < CELLS; ++c) tw[lane * CELLS + c] = __float_as_uint(top.w[c]);
    __syncwarp();
    int place[CELLS];
#pragma unroll
    for (int c = 0; c < CELLS; ++c) place[c] = 0;
    for (int i4 = 0; i4 * 4 < have; ++i4) {
      const uint4 v = reinterpret_cast<const uint4 *>(tw)[i4];
      const uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e4 = 0; e4 < 4; ++e4)
#pragma unroll
        for (int c = 0; c < CELLS; ++c)
          place[c] += x[e4] + (i4 * 4 + e4 < lane * CELLS + c ? 1u : 0u) > __float_as_uint(top.w[c]) ? 1 : 0;
    }
    uint64_t *const out = a.table + static_cast<size_t>(row) * a.k;
#pragma unroll
    for (int c = 0; c < CELLS; ++c)
      if (top.key[c] >= 0 && place[c] < a.k) out[place[c]] = pack_entry(top.key[c] + base, top.w[c]);
    for (int j = have + lane; j < a.k; j += 32) out[j] = 0;  // the stages behind stop at the first empty entry
  }
}

template <int CELLS, typename Index>
// (four blocks per SM by registers, so that one also fits beside the 18 warps of a chain block at 128 slots)
__global__ void __launch_bounds__(32 * L_WARPS, 4) rows_in_lanes_kernel(SketchArgs a, int wait_first) {
  if (wait_first) wait_for_kernels_before();
  let_next_kernel_start();
  using L = LaneLayout<CELLS>;
  extern __shared__ __align__(16) uint32_t lanes_mem[];
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  const uint32_t listed = a.ctrl[CTRL_ROWS_LISTED], mid_end = a.ctrl[CTRL_MID_END];
  const uint32_t span = static_cast<uint32_t>(a.chunk < a.n ? a.chunk : a.n);
  if (a.ctrl[CTRL_HEAVY_ROWS] < mid_end) rows_before_the_lanes<CELLS>(a, mid_end, lanes_mem);
  __syncthreads();
  LaneShared &sh = *reinterpret_cast<LaneShared *>(lanes_mem + L::SHARED_OFF);
  uint32_t *const ring = lanes_mem + L::RING_OFF;
  LaneSketch<CELLS, Index> sk;
  sk.mem = lanes_mem + lane;
  sk.index.mem = lanes_mem + L::I_OFF + lane;
  if (warp == 0) sk.init(span);
  for (;;) {
    if (threadIdx.x == 0) sh.first = atomicAdd(&a.ctrl[CTRL_LANE_TICKET], 32u);
    __syncthreads();
    const uint32_t first = sh.first;
    if (first >= listed) break;
    // (every warp reads all 32 rows: the producers need their own, the selection needs any)
    const LaneRow row = lane_row(a, first + lane, listed);
    const int first_row = (warp - 1) * L_ROWS;
    LaneRow mine = row;
    if (warp > 0) {
      const int from = (first_row + lane) & 31;
      mine.r = __shfl_sync(FULL, row.r, from);
      mine.p = __shfl_sync(FULL, row.p, from);
      mine.re = __shfl_sync(FULL, row.re, from);
      mine.rs = __shfl_sync(FULL, row.rs, from);
      mine.cbase = __shfl_sync(FULL, row.cbase, from);
      produce_phase<Index>(a, mine, first_row, span, ring, sh.count[0]);
    }
    __syncthreads();
    for (int b = 0;; b ^= 1) {
      const int cnt = sh.count[b][lane];
      const int most = __reduce_max_sync(FULL, cnt);
      if (most == 0) break;  // the same in every warp: all rows are through
      if (warp > 0) {
        produce_phase<Index>(a, mine, first_row, span, ring + (b ^ 1) * L::BUFFER, sh.count[b ^ 1]);
      } else {
        const uint32_t *const in = ring + b * L::BUFFER;
        uint32_t key = in[ring_at(0, lane)], term = in[L_RING * 32 + ring_at(0, lane)];
        if (cnt == 0) key = 0;  // (no candidate: nothing was written here)
        int found = sk.index.find(key);
#pragma unroll 1
        for (int u = 0; u < most; ++u) {
          const uint32_t e = key;
          const float al = __uint_as_float(term);
          const int next = ring_at(u + 1 < L_RING ? u + 1 : u, lane);  // requested a step ahead
          key = u + 1 < cnt ? in[next] : 0u;
          term = in[L_RING * 32 + next];
          if (u < cnt) found = sk.step(e, al, found, key);
        }
      }
      __syncthreads();
    }
    select_phase<CELLS, Index>(a, lanes_mem, row);
    __syncthreads();
    if (warp == 0) sk.clear(span);
  }
  // Launched as the programmatic dependent of the heavy-chain kernel (see launch_cells): it must
  // not be seen as finished before that one.
  wait_for_kernels_before();
}

// ---- heavy rows through materialised streams ------------------------------------------
// part -> (heavy row, column range).  Uniform over the warp.
struct PartRef {
  uint32_t item, first;  // heavy row, and its first part
  int32_t r, pb, pe, row_size;
};
__device__ __forceinline__ PartRef part_ref(const SketchArgs &a, uint32_t part, uint32_t heavy) {
  uint32_t lo = 0, hi = heavy;  // part_base[lo] <= part < part_base[hi]
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (a.part_base[mid] <= part)
      lo = mid;
    else
      hi = mid;
  }
  PartRef p;
  p.item = lo;
  p.first = a.part_base[lo];
  p.r = a.row_list[lo];
  const int32_t rb = a.row_seg[p.r], re = rb + a.row_cols[p.r];
  p.row_size = a.ptr[p.r + 1] - a.ptr[p.r];
  p.pb = rb + static_cast<int32_t>(part - p.first) * H_PART;
  p.pe = p.pb + H_PART < re ? p.pb + H_PART : re;
  return p;
}

// Offsets of the heavy rows' streams in hstream; trims the heavy set to what fits.
__global__ void __launch_bounds__(1024) heavy_offsets_kernel(SketchArgs a) {
  let_next_kernel_start();
  wait_for_kernels_before();
  __shared__ unsigned long long sm[32];
  __shared__ unsigned long long carry_s;
  __shared__ uint32_t count_s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t H = a.ctrl[CTRL_HEAVY_ROWS];
  if (H > a.heavy_max) H = a.heavy_max;
  if (threadIdx.x == 0) {
    carry_s = 0;
    count_s = H;
  }
  __syncthreads();
  for (uint32_t base = 0; base < H; base += 1024) {
    const uint32_t i = base + threadIdx.x;
    uint32_t v = 0, np = 0;
    if (i < H) {
      const int32_t r = a.row_list[i];
      v = a.row_work[r];
      np = static_cast<uint32_t>((a.row_cols[r] + H_PART - 1) / H_PART);
    }
    // parts first (same scan, second value packed in the high half of 64 bits)
    unsigned long long pk = (static_cast<unsigned long long>(np) << 43) | v;  // sums: < 2^21 parts, < 2^43 entries
    unsigned long long incl = pk;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned long long t = __shfl_up_sync(FULL, incl, off);
      if (lane >= off) incl += t;
    }
    if (lane == 31) sm[warp] = incl;
    __syncthreads();
    unsigned long long wbase = 0, tot = 0;
    for (int w = 0; w < 32; ++w) {
      const unsigned long long t = sm[w];
      if (w < warp) wbase += t;
      tot += t;
    }
    const unsigned long long carry = carry_s;
    const unsigned long long excl = carry + wbase + incl - pk;
    if (i < H) {
      const unsigned long long e_off = excl & ((1ull << 43) - 1);
      a.heavy_off[i] = static_cast<uint32_t>(e_off > 0xFFFFFFFFull ? 0xFFFFFFFFull : e_off);
      a.part_base[i] = static_cast<uint32_t>(excl >> 43);
      // first row that does not fit the stream buffer, or whose slices would overflow the
      // 21 bits the scan has for their count: it and the rows behind it stay with the light rows
      if (e_off + v > a.stream_cap || (excl >> 43) + np >= (1ull << 21)) atomicMin(&count_s, i);
    }
    __syncthreads();
    if (threadIdx.x == 0) carry_s = carry + tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const uint32_t Hc = count_s;
    // parts of the rows that stay heavy: part_base[Hc] closes the table
    if (Hc == H)
      a.part_base[H] = static_cast<uint32_t>(carry_s >> 43);
    // (when trimmed, part_base[Hc] already holds the first dropped row's base)
    a.ctrl[CTRL_HEAVY_PARTS] = Hc == H ? static_cast<uint32_t>(carry_s >> 43) : a.part_base[Hc];
    a.ctrl[CTRL_HEAVY_ROWS] = count_s;
    a.ctrl[CTRL_ROW_TICKET] = count_s;  // the other rows' tickets start behind the heavy ones
    a.ctrl[CTRL_HEAVY_TICKET] = 0;
    a.ctrl[CTRL_HEAVY_TICKET + 1] = 0;
  }
}

// stream entries each part (H_PART columns of a heavy row) will produce; one warp per part.  Whoever expands a part
// adds up the parts of the row in front of it: one block that scanned all counts took 18 us of a call of
// 360 (65,536 rows, some 300 parts) and 48 of one of 28 ms, the parts' own sums nothing that shows.
__global__ void __launch_bounds__(256) heavy_part_count_kernel(SketchArgs a) {
  let_next_kernel_start();
  wait_for_kernels_before();
  const int lane = lane_id();
  const uint32_t heavy = a.ctrl[CTRL_HEAVY_ROWS], parts = a.ctrl[CTRL_HEAVY_PARTS];
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t part = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; part < parts; part += warps) {
    const PartRef p = part_ref(a, part, heavy);
    uint32_t cnt = 0;
    for (int32_t q = p.pb + lane; q < p.pe; q += 32) {
      const int32_t len = a.seg[q].y;
      cnt += len >= 2 ? static_cast<uint32_t>(len - 1) : 0u;
    }
    cnt = __reduce_add_sync(FULL, cnt);
    if (lane == 0) a.part_off[part] = cnt;
  }
}

// one warp per part: its slice of the row's stream, written out in order
__global__ void __launch_bounds__(S_THREADS) heavy_expand_kernel(SketchArgs a) {
  let_next_kernel_start();
  wait_for_kernels_before();
  __shared__ int32_t ring_s[S_WARPS][S_RING];
  __shared__ float ring_a[S_WARPS][S_RING];
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  const uint32_t heavy = a.ctrl[CTRL_HEAVY_ROWS], parts = a.ctrl[CTRL_HEAVY_PARTS];
  int32_t *bs = ring_s[warp];
  float *ba = ring_a[warp];
  Producer<S_RING> prod(a);
  for (;;) {
    uint32_t part = 0;
    if (lane == 0) part = atomicAdd(&a.ctrl[CTRL_HEAVY_TICKET], 1u);
    part = __shfl_sync(FULL, part, 0);
    if (part >= parts) break;
    const PartRef p = part_ref(a, part, heavy);
    if (p.pe <= p.pb) continue;
    if (!index_ok(a.ctrl, CHK_LIST, p.r, a.n)) continue;
    uint32_t before = 0;
    for (uint32_t q = p.first + lane; q < part; q += 32) before += a.part_off[q];
    uint32_t at = a.heavy_off[p.item] + __reduce_add_sync(FULL, before);
    int2 *out = a.hstream + at;
    prod.begin(p.r, p.pb, p.pe, p.row_size);
    for (;;) {
      const int cnt = prod.produce(bs, ba);
      if (cnt == 0) break;
      // The offsets were laid out from the rows' work counters; a slice that would pass the
      // end of the buffer all the same (counters and groups out of step) is refused, not written.
      if (cnt > static_cast<int>(a.stream_cap) || at > a.stream_cap - static_cast<uint32_t>(cnt)) {
        if (lane == 0) atomicExch(&a.ctrl[CTRL_STREAM_OVERRUN], 1u);
        break;
      }
      for (int i = lane; i < cnt; i += 32) out[i] = make_int2(bs[i], __float_as_int(ba[i]));
      out += cnt;
      at += static_cast<uint32_t>(cnt);
      __syncwarp();
    }
  }
}

// The dependent chains: one warp per heavy row, one warp per scheduler (one block per SM,
// kept alone there by its shared-memory request), reading the stream back in batches.
// The finished sketch goes to memory; the top-k selection is a kernel of its own, because
// with it in the same function the compiler schedules this loop 1.5x slower.
template <int CELLS>
__global__ void __launch_bounds__(S_THREADS, 1) heavy_consume_kernel(SketchArgs a) {
  extern __shared__ __align__(16) unsigned char heavy_pad[];  // only there to fill the SM
  __shared__ int32_t ring_s[S_WARPS][S_RING];
  __shared__ float ring_a[S_WARPS][S_RING];
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  if (heavy_pad[0] == 255 && a.n < 0) return;  // keeps the padding referenced
  // every block of this grid is resident now (one per SM): let the kernel of the other
  // rows, launched behind this one in the same stream, start on whatever is left
  wait_for_kernels_before();  // (first: the kernel of the other rows, which starts now, does not wait for the ones before)
  let_next_kernel_start();
  const uint32_t heavy = a.ctrl[CTRL_HEAVY_ROWS];
  int32_t *bs = ring_s[warp];
  float *ba = ring_a[warp];
  Sketch<CELLS> sk;
  sk.bind_lane();
  for (;;) {
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(&a.ctrl[CTRL_HEAVY_TICKET + 1], 1u);
    item = __shfl_sync(FULL, item, 0);
    if (item >= heavy) break;
    const int32_t r = a.row_list[item];
    const uint32_t total = a.row_work[r];
    const int2 *in = a.hstream + a.heavy_off[item];
    sk.clear();
    for (uint32_t base = 0; base < total; base += S_RING) {
      const int cnt = static_cast<int>(total - base < S_RING ? total - base : S_RING);
      for (int i = lane; i < cnt; i += 32) {
        const int2 e = in[base + i];
        bs[i] = e.x;
        ba[i] = __int_as_float(e.y);
      }
      __syncwarp();
      consume<CELLS>(sk, bs, ba, cnt);
      __syncwarp();
    }
    int32_t *st = a.heavy_state + static_cast<size_t>(item) * (2 * CELLS * 32);
#pragma unroll
    for (int c = 0; c < CELLS; ++c) {
      st[(2 * c) * 32 + lane] = sk.key[c];
      st[(2 * c + 1) * 32 + lane] = __float_as_int(sk.w[c]);
    }
  }
}

// ---- the chains in rounds ---------------------------------------------------------------
// A full sketch behaves like a queue ordered by (weight, slot code): a miss takes the
// least entry and puts it back heavier, so within a short stretch of the stream the i-th
// miss takes the i-th entry of the order as it stood at the start of the stretch.  A round
// looks at the next 32 or 64 stream elements, one or two per lane, and resolves the whole window:
//   * the misses take the entries of the order S0 at the start of the round one after the other, but skip an
//     entry that a hit has made heavier before they reached it ("held");
//   * an element whose key S0 holds in an entry that was taken before the element's turn is
//     a miss, not a hit ("gone"), and takes the next entry like any other miss;
//   * a second element with the key of an earlier one is a hit on the entry the first one ("leader")
//     left, whichever kind the first one was.
// Only leaders with their entry among the window's lightest ("open") can go either way.  Let r be an open element's
// entry's place in the order, P the leaders in front of it that S0 does not hold and A the open elements in front of
// it with places below r.  The entry is gone iff P + A > r: of the entries below, A are taken or held for certain, and
// an open element in front with a place above r counts only if it is gone itself - but then
// P' + A' > r' for it, at most r' - r - 1 of its A' lie between r and r', so P + A >= P' + A' - (r' - r - 1) > r.
// P alone, and P plus all leaders in front that S0 holds, settle most open elements; the others count A by a ballot
// each (1.5 a window of the longest row of R-MAT scale 20).
// All this holds as long as no entry put back or made heavier is light enough to be taken again: the window ends
// before the first miss whose entry is not below the least weight the window has left in any ("least"; equal weights
// count as not below).  One element alone is always resolved exactly.  Of 64 elements, a round resolves 59.2 on the
// longest row of R-MAT scale 20 (64 slots), 64.0 on that of its symmetrised form (128 slots); 20 to 30 where the
// Dice terms vary widely, as a window of 32 does: rounds_row times both widths on every row.
// While the sketch has empty slots, miss number i fills the next i-th slot, and the window ends at the second
// element of a key.
// A group of warps works on one row: its first warp walks the stream and decides the rounds, the other
// warps order the slots for it (rank_slots); meanwhile the first warp looks the window up.  State lives in
// shared memory: weights and keys by slot code, a key -> slot table over the chunk's rows, and
// the order of the round.  What bounds it is the dependent instructions of the first warp, some 450 a round of 64
// (1,850 cycles) and 300 a round of 32 (1,090): no pipe is busy.  ns per candidate with windows of 32 and strict
// rounds that ended at the first open element that is not held, and now: R-MAT scale 20, 64 slots, longest row
// 23.4 -> 15.9, rows of 166,000 / 76,000 / 30,000 candidates 51 -> 20.8, 89 -> 27.0, 184 -> 39.2; symmetrised scale 19,
// 128 slots, longest 29.4 -> 18.2, 146,000 / 61,000 candidates 41 -> 26.5, 78 -> 31.7; power-law band of 4,096 rows
// 26.7 -> 16.4.  32 slots, by windows of 32, which had a warp per row and strict rounds: whole calls 33.5 -> 12.0 ms (R-MAT
// scale 20, k = 8), 5.3 -> 2.1 (top-k graph of an R-MAT matrix of 13,400 rows), 71.6 -> 21.9 (symmetrised, 262,144 rows
// in chunks of 4,096).
constexpr int H_RING = 1024;     // stream elements in a row's ring ...
constexpr int H_SEG = 256;       // ... staged this many at a time
constexpr int ROUND_CELLS = 4;   // largest sketch (cells per lane) resolved in rounds
constexpr int MATES = 1024;      // words of the duplicate detector (two for 64 elements)
constexpr int ROUND_TAB_MAX = 65536;  // largest chunk (rows) with a key -> slot table
constexpr int TRIAL_ROUNDS = 8;     // rounds of each width a row times before it settles on one ...
constexpr int COMMIT_ROUNDS = 160;  // ... for this many rounds
template <int CELLS>
struct Helpers {
  static constexpr int N = 2 * CELLS;                    // warps that order the slots, sixteen slots each
  // Groups (rows) per block, one block per SM: with two the registers of an SM still hold two
  // blocks of rows_in_lanes_kernel (one at 96 slots and more), which does most of the work of a large call.
  static constexpr int ROWS = CELLS == 1 ? 4 : 2;
  static constexpr int THREADS = 32 * (1 + N);           // of a group
};
// named barriers of a group: row in hand, state is ready to be ordered, the order is ready
constexpr int BAR_ROW = 1, BAR_STATE = 2, BAR_ORDER = 3;

template <int CELLS>
struct RoundState {
  static constexpr int M = 32 * CELLS;
  static constexpr int W = M < 64 ? M : 64;  // widest window, and entries of the order that are kept
  __align__(16) uint32_t w[M + 4];   // weight bits by slot code (cell * 32 + lane); the last for who has none
  __align__(16) int32_t key[M + 4];
  int32_t rank[M];               // position of each slot in ascending (weight, code) order
  uint2 order[W];                // the lightest in that order: weight bits, key << 8 | slot code
  uint2 takes[W + 2];            // the same without the entries that hits hold back
  int32_t row_done;              // tells the other warps that the row is through
  uint32_t item;                 // the row in hand (place in the list)
  uint32_t spare;                // where stores of lanes without one go
};

// A group's shared memory: state, the ring of stream elements (a segment lands while the ones before it are
// consumed), the duplicate detector (all zero between windows), then the key -> slot table (slot
// + 1, one byte per row of the chunk; none for very large chunks).  The rounds are functions of
// their own; they get an offset and build their pointers from the array itself, so that the
// compiler sees shared memory and not a generic address (slower by some ten cycles a load).
extern __shared__ __align__(16) unsigned char heavy_dyn[];
template <int CELLS>
struct GroupMemory {
  static constexpr int RING = (sizeof(RoundState<CELLS>) + 15) / 16 * 16;
  static constexpr int MATE = RING + H_RING * 8;
  // (chunks of more than MATES rows share half as many words: their tables are the larger part)
  static constexpr __host__ __device__ int tab_offset(bool hash) { return MATE + (hash ? MATES / 2 : MATES) * 8; }
  static constexpr int SPARE = static_cast<int>(offsetof(RoundState<CELLS>, spare));
  static __device__ __forceinline__ RoundState<CELLS> &state(int base) {
    return *reinterpret_cast<RoundState<CELLS> *>(heavy_dyn + base);
  }
  static __device__ __forceinline__ int2 *ring(int base) {
    return reinterpret_cast<int2 *>(heavy_dyn + base + RING);
  }
  static __device__ __forceinline__ uint2 *mates(int base) {
    return reinterpret_cast<uint2 *>(heavy_dyn + base + MATE);
  }
  template <bool HASH>
  static __device__ __forceinline__ uint8_t *tab(int base) { return heavy_dyn + base + tab_offset(HASH); }
};

// what the rounds of a row need to know
struct RoundRow {
  int base;           // the group's place in shared memory
  int32_t cbase;      // first row of the chunk
  uint32_t *ctrl;     // checked build: where a key outside its chunk is recorded ...
  int32_t span;       // ... and the rows of a chunk
  int bars;           // the group's named barriers are bars + BAR_*
};

template <int CELLS>
__device__ __forceinline__ void bar_arrive(int id) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(Helpers<CELLS>::THREADS) : "memory");
}
template <int CELLS>
__device__ __forceinline__ void bar_wait(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(Helpers<CELLS>::THREADS) : "memory");
}

// Slot that holds key s (relative to the chunk), or -1.  With TAB from the key -> slot table;
// without it by comparing s with every slot's key (unique in a sketch, empty slots hold -1).
template <int CELLS, bool TAB, bool HASH>
__device__ __forceinline__ int slot_of(const RoundRow &row, int32_t s) {
  if (TAB) return static_cast<int>(GroupMemory<CELLS>::template tab<HASH>(row.base)[s]) - 1;
  const RoundState<CELLS> &st = GroupMemory<CELLS>::state(row.base);
  int q = -1;
#pragma unroll
  for (int i4 = 0; i4 < 8 * CELLS; ++i4) {
    const int4 kk = reinterpret_cast<const int4 *>(st.key)[i4];
    q = kk.x == s ? 4 * i4 : q;
    q = kk.y == s ? 4 * i4 + 1 : q;
    q = kk.z == s ? 4 * i4 + 2 : q;
    q = kk.w == s ? 4 * i4 + 3 : q;
  }
  return q;
}

// One of the other warps: the place of its sixteen slots in the (weight, code) order, the
// number of entries (x, i) below (mine, slot).  Eight lanes to four slots, as many parts of the entries.
// "x < mine" is counted as sat((mine - x) * 2^90), one fused multiply-add that is exactly 1 or 0:
// weights lie in [2^-31, 2^32], so two different ones are at least 2^-54 apart.  An equal entry
// is below for a smaller code: then the bar is the next float above.
// Returns false once the row is through.
template <int CELLS>
__device__ __forceinline__ bool rank_slots(int base, int helper, int lane) {
  RoundState<CELLS> &st = GroupMemory<CELLS>::state(base);
  constexpr float BIG = 1.2379400392853803e27f;  // 2^90
  constexpr float ZERO = 8388608.0f;             // 2^23: counts are read off its last bits
  constexpr int GROUP = 8, SLOTS = 4, QUADS = CELLS;
  const int sub = lane % GROUP, first = helper * 16 + lane / GROUP * SLOTS, slot = first + sub % SLOTS, own = first / 4;
  const float4 *const v4 = reinterpret_cast<const float4 *>(st.w);
  float4 all[QUADS];  // (loaded in one go: left to itself the compiler waits for every load)
  float m[SLOTS];
#pragma unroll
  for (int b = 0; b < QUADS; ++b) all[b] = v4[b * GROUP + sub];
#pragma unroll
  for (int i = 0; i < SLOTS; ++i) m[i] = __uint_as_float(st.w[first + i]);
  const uint32_t bits = st.w[slot];
  const int32_t key = st.key[slot];
  const bool done = *static_cast<volatile int32_t *>(&st.row_done);
  float acc[SLOTS];
#pragma unroll
  for (int i = 0; i < SLOTS; ++i) {
    const float lt = m[i] * BIG, le = __uint_as_float(__float_as_uint(m[i]) + 1u) * BIG;
    acc[i] = ZERO;
#pragma unroll
    for (int b = 0; b < QUADS; ++b) {
      // entries of the slots' own block of four in front of this slot, and others, have the bar of their block
      const bool before = b * GROUP + sub < own, upto = b * GROUP + sub <= own;
      const float bar = before ? le : lt, front = upto ? le : lt;
      const float x[4] = {all[b].x, all[b].y, all[b].z, all[b].w};
      float c[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) c[k] = __saturatef(fmaf(x[k], -BIG, k < i ? front : bar));
      acc[i] += (c[0] + c[1]) + (c[2] + c[3]);
    }
  }
  // counts of the slots in the bytes of one word
  uint32_t counts = __byte_perm(__float_as_uint(acc[0]), __float_as_uint(acc[1]), 0x0040) & 0xFFFFu;
  counts = __byte_perm(counts, __byte_perm(__float_as_uint(acc[2]), __float_as_uint(acc[3]), 0x0040), 0x5410);
#pragma unroll
  for (int d = 1; d < GROUP; d <<= 1) counts += __shfl_xor_sync(FULL, counts, d);
  const int pos = static_cast<int>(counts >> (8 * (sub % SLOTS)) & 255u);
  if (done) return false;
  if (sub < SLOTS)
    st.rank[slot] = pos;
  else if (pos < RoundState<CELLS>::W)
    st.order[pos] = make_uint2(bits, static_cast<uint32_t>(key) << 8 | static_cast<uint32_t>(slot));
  return true;
}

// The window of a round, E elements per lane (element 32 e + lane of the window in place e).
template <int E>
struct Window {
  bool valid[E];
  int32_t s[E];   // key, relative to the chunk
  float al[E];    // Dice term
};

// bits of a mask over the window (32 to a word) in front of this lane's element e
template <int E>
__device__ __forceinline__ int count_before(const uint32_t (&mask)[E], int e, uint32_t below) {
  int c = __popc(mask[e] & below);
#pragma unroll
  for (int f = 0; f < E; ++f)
    if (f < e) c += __popc(mask[f]);
  return c;
}

// elements of `same` among the first L of the window
template <int E>
__device__ __forceinline__ int count_prefix(const uint32_t (&same)[E], int L) {
  int c = 0;
#pragma unroll
  for (int f = 0; f < E; ++f) {
    const int l = L - 32 * f;
    c += __popc(same[f] & (l >= 32 ? FULL : l <= 0 ? 0u : (1u << l) - 1u));
  }
  return c;
}

template <int CELLS, int E>
__device__ __forceinline__ void window_load(const RoundRow &row, uint32_t p, uint32_t end, int lane, Window<E> &w) {
  const int2 *const ring = GroupMemory<CELLS>::ring(row.base);
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int2 elem = ring[(p + e * 32 + lane) & (H_RING - 1)];
    w.valid[e] = p + e * 32 + lane < end;
    const int32_t key = w.valid[e] ? elem.x : row.cbase;
    // (a key outside the chunk only comes from rows that are not sorted: kept in bounds)
    w.s[e] = static_cast<int32_t>(min(static_cast<uint32_t>(key_in_chunk(row.ctrl, key, row.cbase, row.span) - row.cbase),
                                      static_cast<uint32_t>(row.span) - 1u));
    w.al[e] = __int_as_float(elem.y);
  }
}

// Elements with the same key, part one: every lane sets its bit in a word of shared memory under its key.
// match.any, the instruction made for this, takes some 380 cycles here.
template <bool HASH>
__device__ __forceinline__ int mate_word(int32_t s) {
  return HASH ? static_cast<int>((static_cast<uint32_t>(s) * 0x9E3779B1u) >> 23) : s;
}
template <int CELLS, int E, bool HASH>
__device__ __forceinline__ void window_mark(const RoundRow &row, int lane, const Window<E> &w) {
  uint2 *const mates = GroupMemory<CELLS>::mates(row.base);
#pragma unroll
  for (int e = 0; e < E; ++e) {
    uint2 &word = mates[mate_word<HASH>(w.s[e])];
    if (w.valid[e]) atomicOr(e == 0 ? &word.x : &word.y, 1u << lane);
  }
}
// Part two (after a __syncwarp): the marks, 32 elements of the window to a word; the words are clear again.
template <int CELLS, int E, bool HASH>
__device__ __forceinline__ void window_collect(const RoundRow &row, uint32_t p, int lane, const Window<E> &w,
                                               uint32_t (&same)[E][E]) {
  uint2 *const mates = GroupMemory<CELLS>::mates(row.base);
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const uint2 both = mates[mate_word<HASH>(w.s[e])];
    same[e][0] = w.valid[e] ? both.x : 0u;
    if (E > 1) same[e][E - 1] = w.valid[e] ? both.y : 0u;
  }
  if (HASH) {  // a word may stand for several keys: the others are taken out one by one
    const int2 *const ring = GroupMemory<CELLS>::ring(row.base);
#pragma unroll
    for (int e = 0; e < E; ++e)
#pragma unroll
      for (int f = 0; f < E; ++f)
        for (uint32_t rest = same[e][f] & (e == f ? ~(1u << lane) : FULL); rest; rest &= rest - 1u) {
          const int b = __ffs(static_cast<int>(rest)) - 1;
          if (ring[(p + f * 32 + b) & (H_RING - 1)].x - row.cbase != w.s[e]) same[e][f] &= ~(1u << b);
        }
  }
  __syncwarp();
#pragma unroll
  for (int e = 0; e < E; ++e)
    if (w.valid[e]) mates[mate_word<HASH>(w.s[e])] = make_uint2(0u, 0u);
}

// One more Dice term for a key that comes again in the window; the element of `rest` (later elements of the key) that
// brought it is taken out.
template <int E>
__device__ __forceinline__ void add_later(uint32_t (&rest)[E], float al, uint32_t &weight) {
  uint32_t any = rest[0];
#pragma unroll
  for (int f = 1; f < E; ++f) any |= rest[f];
  weight = any ? __float_as_uint(__uint_as_float(weight) + al) : weight;
  if (E > 1) rest[E - 1] = rest[0] ? rest[E - 1] : rest[E - 1] & (rest[E - 1] - 1u);
  rest[0] &= rest[0] - 1u;  // (0 stays 0)
}

// One round on a full sketch: resolves the window at p (loaded and marked), moves p on and loads and marks the next
// one.  Lanes without a store write to a spare place instead of branching around it, and a window's look-ups by key
// are made while the other warps order the slots: a branch costs the lone warp some 25 cycles.
template <int CELLS, int E, bool TAB, bool HASH>
__device__ __forceinline__ void round_window(const RoundRow &row, uint32_t &p, uint32_t end, int lane, Window<E> &w) {
  using G = GroupMemory<CELLS>;
  RoundState<CELLS> &st = G::state(row.base);
  constexpr int M = 32 * CELLS, W = 32 * E;
  static_assert(W <= RoundState<CELLS>::W, "a window takes entries of the order");
  const uint32_t below = (1u << lane) - 1u;
  bar_arrive<CELLS>(row.bars + BAR_STATE);
  // while the other warps order the slots: what S0 says about the window
  int q[E], absent_before[E], kept_before[E];
  bool present[E], leader[E];
  uint32_t absent[E], kept[E], same[E][E];
  uint32_t one[E], all[E];  // weight with the first, with every Dice term of the key in the window
#pragma unroll
  for (int e = 0; e < E; ++e) q[e] = w.valid[e] ? slot_of<CELLS, TAB, HASH>(row, w.s[e]) : -1;
  window_collect<CELLS, E, HASH>(row, p, lane, w, same);
#pragma unroll
  for (int e = 0; e < E; ++e) {
    present[e] = q[e] >= 0;  // S0 holds the key
    q[e] = present[e] ? q[e] : 0;
    one[e] = st.w[q[e]];
    leader[e] = w.valid[e] && (same[e][e] & below) == 0u && (e == 0 || same[e][0] == 0u);  // first element of its key
    absent[e] = __ballot_sync(FULL, leader[e] && !present[e]);
    kept[e] = __ballot_sync(FULL, leader[e] && present[e]);
  }
  Window<E> nx;
  window_load<CELLS, E>(row, p + W, end, lane, nx);
  uint32_t rest[E][E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    absent_before[e] = count_before<E>(absent, e, below);
    kept_before[e] = count_before<E>(kept, e, below);
    one[e] = all[e] = __float_as_uint(__uint_as_float(one[e]) + w.al[e]);
#pragma unroll
    for (int f = 0; f < E; ++f) rest[e][f] = f == e ? same[e][f] & ~(below | 1u << lane) : f > e ? same[e][f] : 0u;
    add_later<E>(rest[e], w.al[e], all[e]);
  }
  for (;;) {
    bool later = false;
#pragma unroll
    for (int e = 0; e < E; ++e)
#pragma unroll
      for (int f = 0; f < E; ++f) later |= present[e] && rest[e][f];
    if (!__any_sync(FULL, later)) break;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      add_later<E>(rest[e], w.al[e], all[e]);
      add_later<E>(rest[e], w.al[e], all[e]);
    }
  }
  bar_wait<CELLS>(row.bars + BAR_ORDER);
  int rho[E];
  uint2 mine[E];  // the entries of rank 32 e + lane
#pragma unroll
  for (int e = 0; e < E; ++e) rho[e] = st.rank[q[e]];
#pragma unroll
  for (int e = 0; e < E; ++e) mine[e] = st.order[e * 32 + lane];
  bool open[E], gone[E], unsure[E], either = false;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    open[e] = leader[e] && present[e] && rho[e] < W;
    gone[e] = open[e] && absent_before[e] > rho[e];
    unsure[e] = open[e] && !gone[e] && absent_before[e] + kept_before[e] > rho[e];
    either |= unsure[e];
  }
  if (__any_sync(FULL, either)) {  // count the open elements in front with lower places, one such element per word at a time
    uint32_t left[E], any = 0u;
#pragma unroll
    for (int e = 0; e < E; ++e) any |= left[e] = __ballot_sync(FULL, unsure[e]);
    while (any) {
      int j[E], r[E], lower[E];
      any = 0u;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        j[e] = 31 - __clz(static_cast<int>(left[e] | 1u));
        r[e] = __shfl_sync(FULL, rho[e], j[e]);
        lower[e] = 0;
      }
#pragma unroll
      for (int e = 0; e < E; ++e) {
#pragma unroll
        for (int f = 0; f <= e; ++f) {
          const uint32_t front = __ballot_sync(FULL, open[f] && rho[f] < r[e]);
          lower[e] += __popc(f == e ? front & ((1u << j[e]) - 1u) : front);
        }
        if (lane == j[e]) gone[e] = open[e] && absent_before[e] + lower[e] > r[e];
        left[e] &= ~(1u << j[e]);
        any |= left[e];
      }
    }
  }
  // the elements that miss, and the entries that hits hold back
  uint32_t missing[E], held[E], flipped = 0u;
  bool miss[E];
  int turn[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    uint32_t h = 0u;
#pragma unroll
    for (int f = 0; f < E; ++f) h |= open[f] && !gone[f] && (E == 1 || rho[f] >> 5 == e) ? 1u << (rho[f] & 31) : 0u;
    held[e] = __reduce_or_sync(FULL, h);
    const uint32_t f = __ballot_sync(FULL, gone[e]);
    missing[e] = absent[e] | f;
    flipped |= f;
    miss[e] = (leader[e] && !present[e]) || gone[e];
  }
#pragma unroll
  for (int e = 0; e < E; ++e)
    st.takes[(held[e] >> lane) & 1u ? W : e * 32 + lane - count_before<E>(held, e, below)] = mine[e];
#pragma unroll
  for (int e = 0; e < E; ++e) turn[e] = flipped ? count_before<E>(missing, e, below) : absent_before[e];
  __syncwarp();
  uint2 take[E];
#pragma unroll
  for (int e = 0; e < E; ++e) take[e] = st.takes[miss[e] ? turn[e] : 0];
  // the least weight that the window leaves in an entry: a miss whose entry is not below may have to
  // take that one instead
  uint32_t least = 0xFFFFFFFFu;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    one[e] = miss[e] ? __float_as_uint(__uint_as_float(take[e].x) + w.al[e]) : one[e];
    least = miss[e] || open[e] ? min(least, one[e]) : least;
  }
  least = __reduce_min_sync(FULL, least);
  int L = W;
#pragma unroll
  for (int e = E - 1; e >= 0; --e) {
    const uint32_t again = __ballot_sync(FULL, miss[e] && take[e].x >= least);
    L = again ? e * 32 + __ffs(static_cast<int>(again)) - 1 : L;
  }
  L = max(1, min(L, static_cast<int>(end - p)));  // one element alone is always resolved exactly
  bool later = false;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    all[e] = miss[e] ? one[e] : all[e];
#pragma unroll
    for (int f = 0; f < E; ++f) {
      rest[e][f] = miss[e] ? (f == e ? same[e][f] & ~(below | 1u << lane) : f > e ? same[e][f] : 0u) : 0u;
      later |= rest[e][f] != 0u;
    }
  }
  p += L;
  if (L < W) {
    window_load<CELLS, E>(row, p, end, lane, nx);
    later = false;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      bool cut = false;
      leader[e] = leader[e] && e * 32 + lane < L;
#pragma unroll
      for (int f = 0; f < E; ++f) {
        const int l = L - 32 * f;
        const uint32_t in = l >= 32 ? FULL : l <= 0 ? 0u : (1u << l) - 1u;
        const uint32_t whole = f == e ? same[e][f] & ~(below | 1u << lane) : f > e ? same[e][f] : 0u;
        cut |= (whole & ~in) != 0u;
        rest[e][f] = whole & in;
      }
      all[e] = cut ? one[e] : all[e];
#pragma unroll
      for (int f = 0; f < E; ++f) {
        rest[e][f] = leader[e] && (cut || miss[e]) ? rest[e][f] : 0u;
        later |= rest[e][f] != 0u;
      }
    }
  }
  window_mark<CELLS, E, HASH>(row, lane, nx);
  while (__any_sync(FULL, later)) {
    later = false;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      add_later<E>(rest[e], w.al[e], all[e]);
#pragma unroll
      for (int f = 0; f < E; ++f) later |= rest[e][f] != 0u;
    }
  }
#pragma unroll
  for (int e = 0; e < E; ++e)
    if (TAB) heavy_dyn[row.base + (leader[e] && miss[e] ? G::tab_offset(HASH) + static_cast<int>(take[e].y >> 8) : G::SPARE)] = 0;
  // (a key taken by one miss may be put back by a later one, which then is a flipped lane:
  // clear first, then set)
  __syncwarp();
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const bool put = leader[e] && miss[e];
    const int slot = static_cast<int>(take[e].y & 255u);
    st.key[put ? slot : M] = w.s[e];
    if (TAB) heavy_dyn[row.base + (put ? G::tab_offset(HASH) + w.s[e] : G::SPARE)] = static_cast<uint8_t>(slot + 1);
    st.w[leader[e] ? (miss[e] ? slot : q[e]) : M] = all[e];
  }
  __syncwarp();
  w = nx;
}

// One round while the sketch has empty slots; `filled` is updated.  (No order needed.)
template <int CELLS, bool TAB, bool HASH>
__device__ __forceinline__ int round_fill(const RoundRow &row, uint32_t p, uint32_t end, int lane, int &filled) {
  RoundState<CELLS> &st = GroupMemory<CELLS>::state(row.base);
  uint8_t *const tab = GroupMemory<CELLS>::template tab<HASH>(row.base);
  constexpr int M = 32 * CELLS;
  const uint32_t below = (1u << lane) - 1u;
  Window<1> w;
  window_load<CELLS, 1>(row, p, end, lane, w);
  window_mark<CELLS, 1, HASH>(row, lane, w);
  __syncwarp();
  uint32_t mates[1][1];
  window_collect<CELLS, 1, HASH>(row, p, lane, w, mates);
  const int q = w.valid[0] ? slot_of<CELLS, TAB, HASH>(row, w.s[0]) : -1;
  const bool miss = w.valid[0] && q < 0, hit = w.valid[0] && q >= 0;
  const uint32_t missing = __ballot_sync(FULL, miss);
  const int mrank = __popc(missing & below);
  const unsigned same = mates[0][0];
  int lim = w.valid[0] ? 32 : lane;
  if (miss && ((same & below) || mrank >= M - filled)) lim = lane;
  const int L = static_cast<int>(__reduce_min_sync(FULL, static_cast<uint32_t>(lim)));
  const unsigned prefix = L >= 32 ? FULL : (1u << L) - 1u;
  if (lane < L) {
    if (miss) {
      const int j = filled + mrank;  // j-th slot to be filled: lane j / CELLS, cell j % CELLS
      const int code = (j % CELLS) * 32 + j / CELLS;
      st.key[code] = w.s[0];
      st.w[code] = __float_as_uint(w.al[0]);
      if (TAB) tab[w.s[0]] = static_cast<uint8_t>(code + 1);
    } else if (hit && ((same & prefix) & below) == 0u) {
      float wv = __uint_as_float(st.w[q]);
      for (int t = __popc(same & prefix); t > 0; --t) wv += w.al[0];
      st.w[q] = __float_as_uint(wv);
    }
  }
  filled += __popc(missing & prefix);
  __syncwarp();
  return L;
}

// copies the H_SEG stream elements from `from` on (those in front of `total`) into the ring without passing
// through registers
__device__ __forceinline__ void stage_segment(int2 *ring, const int2 *in, uint32_t from, uint32_t total, int lane) {
  const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(ring + (from & (H_RING - 1)))) + lane * 8;
  const int2 *src = in + from + lane;
  const int left = static_cast<int>(min(total - min(from, total), static_cast<uint32_t>(H_SEG))) - lane;
#pragma unroll
  for (int i = 0; i < H_SEG / 32; ++i)
    if (i * 32 < left)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + i * 256), "l"(src + i * 32) : "memory");
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// where a row's stream has got to: [p, ...), elements in front of `seg` + 2 H_SEG are in the ring or on their way
struct RowStream {
  const int2 *in;
  uint32_t total, p, seg;
};

// Windows that start in a segment may reach into the next, so that one has to be here; the one behind it is
// on its way meanwhile.
__device__ __forceinline__ void next_segment(int2 *ring, RowStream &s, int lane) {
  stage_segment(ring, s.in, s.seg + 2 * H_SEG, s.total, lane);
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  __syncwarp();
}

// At most `left` rounds of one width.  Functions of their own:
// compiled into one body each kind loses speed to the other's registers and schedule.
template <int CELLS, int E, bool TAB, bool HASH>
__device__ __noinline__ uint2 window_rounds(const RoundRow row, RowStream s, int left) {
  int2 *const ring = GroupMemory<CELLS>::ring(row.base);
  const int lane = lane_id();
  uint32_t end = min(s.total, s.seg + 2 * H_SEG);
  Window<E> w;
  window_load<CELLS, E>(row, s.p, end, lane, w);
  window_mark<CELLS, E, HASH>(row, lane, w);
  __syncwarp();
  while (s.p < s.total && left > 0) {
    if (s.p >= s.seg + H_SEG) {
      s.seg += H_SEG;
      next_segment(ring, s, lane);
      end = min(s.total, s.seg + 2 * H_SEG);
    }
    round_window<CELLS, E, TAB, HASH>(row, s.p, end, lane, w);
    --left;
  }
  {  // the marks of the window that does not come here
    uint32_t same[E][E];
    window_collect<CELLS, E, HASH>(row, s.p, lane, w, same);
    __syncwarp();
  }
  return make_uint2(s.p, s.seg);
}

// One heavy row, start to finish, by the first warp: stream batches in, rounds, final sketch out.
template <int CELLS, bool TAB, bool HASH>
__device__ __noinline__ void rounds_row(const int2 *in, uint32_t total, const RoundRow row, int32_t *out) {
  RoundState<CELLS> &st = GroupMemory<CELLS>::state(row.base);
  uint8_t *const tab = GroupMemory<CELLS>::template tab<HASH>(row.base);
  int2 *const ring = GroupMemory<CELLS>::ring(row.base);
  constexpr int M = 32 * CELLS;
  const int lane = lane_id();
#pragma unroll
  for (int c = 0; c < CELLS; ++c) {
    st.key[c * 32 + lane] = -1;
    st.w[c * 32 + lane] = 0u;
  }
  int filled = 0;
  __syncwarp();
  RowStream s = {in, total, 0u, 0u};
  stage_segment(ring, in, 0, total, lane);
  stage_segment(ring, in, H_SEG, total, lane);
  next_segment(ring, s, lane);
  while (s.p < total && filled < M) {
    if (s.p >= s.seg + H_SEG) {
      s.seg += H_SEG;
      next_segment(ring, s, lane);
    }
    s.p += round_fill<CELLS, TAB, HASH>(row, s.p, min(total, s.seg + 2 * H_SEG), lane, filled);
  }
  // Which width is faster depends on the row: windows of 64 cost more and pay where most of them are resolved
  // whole - rows whose own length dominates their Dice terms.  Where the terms vary widely, entries put back light
  // are taken again soon and either width ends after the same few elements.  So the row measures: a few rounds of
  // each width against the clock, then a long stretch of the one that resolved more elements per cycle, and again.
  int wide = 1, left = TRIAL_ROUNDS, trial = 1;  // width in use, rounds of the stretch, width on trial (-1 none)
  long long got[2] = {0, 0}, took[2] = {0, 0};
  int streak = 0, last = -1;
  while (s.p < total) {
    const uint32_t from = s.p;
    const long long t0 = clock64();
    uint2 at;
    if constexpr (CELLS == 1)  // (a window of 64 would need more entries than there are)
      at = window_rounds<CELLS, 1, TAB, HASH>(row, s, 1 << 20);
    else
      at = wide ? window_rounds<CELLS, 2, TAB, HASH>(row, s, left) : window_rounds<CELLS, 1, TAB, HASH>(row, s, left);
    s.p = at.x;
    s.seg = at.y;
    if (trial >= 0) {
      got[trial] = s.p - from;
      took[trial] = clock64() - t0;
    }
    if (trial == 1) {  // wide windows tried: now the others
      trial = wide = 0;
      left = TRIAL_ROUNDS;
    } else if (trial == 0) {  // both tried: elements per cycle, compared without dividing
      wide = got[1] * took[0] >= got[0] * took[1] ? 1 : 0;
      // the stretch grows while the same width keeps winning (up to 16 times as long)
      streak = wide == last ? (streak < 4 ? streak + 1 : 4) : 0;
      last = wide;
      trial = -1;
      left = COMMIT_ROUNDS << streak;
    } else {  // a stretch is over: measure again
      trial = wide = 1;
      left = TRIAL_ROUNDS;
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int c = 0; c < CELLS; ++c) {
    const int32_t kk = st.key[c * 32 + lane];
    out[(2 * c) * 32 + lane] = kk >= 0 ? kk + row.cbase : -1;
    out[(2 * c + 1) * 32 + lane] = static_cast<int32_t>(st.w[c * 32 + lane]);
    if (TAB && kk >= 0) tab[kk] = 0;  // the table is empty again for the next row
  }
  __syncwarp();
}

// A group of warps per heavy row, in list order (longest first).  Several groups to a block, so
// that the chains of a call that runs one chunk ahead fill few SMs while the rest of the call
// is transposed on the others.
template <int CELLS>
__global__ void __launch_bounds__(Helpers<CELLS>::THREADS *Helpers<CELLS>::ROWS) __maxnreg__(CELLS <= 2 ? 88 : 72)
    heavy_rounds_kernel(SketchArgs a, int tab_bytes) {
  constexpr int THREADS = Helpers<CELLS>::THREADS;
  using G = GroupMemory<CELLS>;
  const int group = threadIdx.x / THREADS, in_group = threadIdx.x % THREADS;
  const int32_t span = a.chunk < a.n ? a.chunk : a.n;
  const int base = group * (G::tab_offset(span > MATES) + tab_bytes);
  RoundState<CELLS> &st = G::state(base);
  const int lane = lane_id(), warp = in_group >> 5, bars = 3 * group;
  wait_for_kernels_before();  // (first: the kernel of the other rows, which starts now, does not wait for the ones before)
  let_next_kernel_start();
  const uint32_t heavy = a.ctrl[CTRL_HEAVY_ROWS];
  for (int i = G::MATE + in_group * 16; i < G::tab_offset(span > MATES) + tab_bytes; i += THREADS * 16)
    *reinterpret_cast<uint4 *>(heavy_dyn + base + i) = make_uint4(0, 0, 0, 0);
  for (;;) {
    if (in_group == 0) {
      st.item = atomicAdd(&a.ctrl[CTRL_HEAVY_TICKET + 1], 1u);
      st.row_done = 0;
    }
    bar_wait<CELLS>(bars + BAR_ROW);
    const uint32_t item = st.item;
    if (item >= heavy) break;
    const int32_t r = a.row_list[item];
    // checked build: the row, its place in the state array and its stream's extent
    const bool ok = index_ok(a.ctrl, CHK_LIST, r, a.n) && index_ok(a.ctrl, CHK_STATE, item, a.heavy_max) &&
                    index_ok(a.ctrl, CHK_STREAM, static_cast<long long>(a.heavy_off[item]) + a.row_work[r],
                             static_cast<long long>(a.stream_cap) + 1);
    if (warp > 0) {
      for (;;) {
        bar_wait<CELLS>(bars + BAR_STATE);
        if (!rank_slots<CELLS>(base, warp - 1, lane)) break;
        bar_arrive<CELLS>(bars + BAR_ORDER);
      }
    } else {
      if (ok) {
        const RoundRow row = {base, (r / a.chunk) * a.chunk, a.ctrl, span, bars};
        int32_t *out = a.heavy_state + static_cast<size_t>(item) * (2 * CELLS * 32);
        const int2 *in = a.hstream + a.heavy_off[item];
        if (tab_bytes > 0 && span <= MATES)
          rounds_row<CELLS, true, false>(in, a.row_work[r], row, out);
        else if (tab_bytes > 0)
          rounds_row<CELLS, true, true>(in, a.row_work[r], row, out);
        else
          rounds_row<CELLS, false, true>(in, a.row_work[r], row, out);
      }
      if (lane == 0) st.row_done = 1;
      __syncwarp();
      bar_arrive<CELLS>(bars + BAR_STATE);
    }
    bar_wait<CELLS>(bars + BAR_ROW);
  }
}

template <int CELLS>
__global__ void __launch_bounds__(S_THREADS) heavy_topk_kernel(SketchArgs a) {
  wait_for_kernels_before();
  let_next_kernel_start();
  const int lane = lane_id();
  const uint32_t heavy = a.ctrl[CTRL_HEAVY_ROWS];
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  Sketch<CELLS> sk;
  sk.bind_lane();
  for (uint32_t item = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; item < heavy; item += warps) {
    const int32_t *st = a.heavy_state + static_cast<size_t>(item) * (2 * CELLS * 32);
    sk.clear();
#pragma unroll
    for (int c = 0; c < CELLS; ++c) {
      sk.key[c] = st[(2 * c) * 32 + lane];
      sk.w[c] = __int_as_float(st[(2 * c + 1) * 32 + lane]);
    }
    const int32_t r = a.row_list[item];
    sk.select_top_k(a.k, a.table + static_cast<size_t>(r) * a.k, a.row_base);
  }
}

// shared memory of a block of heavy_rounds_kernel: as many groups as their key tables leave room for
struct ChainBlock {
  int groups, group_bytes, tab_bytes, room;
};
template <int CELLS>
ChainBlock chain_block(const Context &ctx, int64_t span) {
  ChainBlock b;
  b.tab_bytes = span <= ROUND_TAB_MAX ? static_cast<int>((span + 15) / 16 * 16) : 0;
  b.group_bytes = GroupMemory<CELLS>::tab_offset(span > MATES) + b.tab_bytes;
  b.room = ctx.smem_optin - 1024;
  b.groups = Helpers<CELLS>::ROWS;
  while (b.groups > 1 && b.groups * b.group_bytes > b.room) --b.groups;
  return b;
}

template <int CELLS>
bool launch_cells(Context &ctx, const SketchArgs &a, int phase, bool no_heavy_rows) {
  // A call that runs one chunk ahead has two of these sequences in flight: the chunk ahead on
  // the side stream, the rest on the context's stream.  Where a chain block takes a whole SM
  // (sketches beyond ROUND_CELLS) the two share the SMs, since the kernel of the other rows starts
  // only when every chain block has one.
  cudaStream_t st = phase == PHASE_PRIO ? ctx.side_stream : ctx.stream;
  const bool behind = phase == PHASE_ALL;
  constexpr bool in_rounds = CELLS <= ROUND_CELLS;
  if (!no_heavy_rows) {
    CSG_CUDA(launch_behind(behind, heavy_offsets_kernel, 1, 1024, 0, st, a));
    CSG_CUDA(launch_behind(behind, heavy_part_count_kernel, ctx.num_sms * 4, 256, 0, st, a));
    CSG_CUDA(launch_behind(behind, heavy_expand_kernel, ctx.num_sms * 8, S_THREADS, 0, st, a));
    // (the rest of the call starts its own chains only behind this point: by then the chains
    // ahead, next in their stream, hold their SMs, and the kernel of the other rows cannot
    // settle on them first)
    if (phase == PHASE_PRIO) CSG_CUDA(cudaEventRecord(ctx.ev[8], st));
    // Sketches of up to ROUND_CELLS cells per lane are resolved in rounds, a group of warps per row.
    if constexpr (in_rounds) {
      const ChainBlock block = chain_block<CELLS>(ctx, a.chunk < a.n ? a.chunk : a.n);
      CSG_CUDA(cudaFuncSetAttribute(heavy_rounds_kernel<CELLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, block.room));
      // (all of an SM's memory as shared: a block of another split cannot move in beside this one)
      CSG_CUDA(cudaFuncSetAttribute(heavy_rounds_kernel<CELLS>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                    cudaSharedmemCarveoutMaxShared));
      // (a plain launch: started beside the end of the expansion, blocks gather on the SMs that are through first, and
      // symmetrised R-MAT of scale 20 takes 29.4 ms instead of 27.7)
      CSG_CUDA(launch_behind(false, heavy_rounds_kernel<CELLS>, ctx.num_sms, Helpers<CELLS>::THREADS * block.groups,
                             block.groups * block.group_bytes, st, a, block.tab_bytes));
    }
    if constexpr (CELLS > ROUND_CELLS) {
      const int pad = ctx.smem_optin - 1024 - 2 * S_WARPS * S_RING * 4;
      CSG_CUDA(cudaFuncSetAttribute(heavy_consume_kernel<CELLS>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, pad));
      const int ahead = prio_chain_blocks(ctx.num_sms);
      const int blocks = phase == PHASE_PRIO ? ahead : phase == PHASE_REST ? ctx.num_sms - ahead : ctx.num_sms;
      CSG_CUDA(launch_behind(false, heavy_consume_kernel<CELLS>, blocks, S_THREADS, pad, st, a));
    }
  }
  // The other rows run beside the heavy chains: their kernel follows in the same stream
  // as a programmatic dependent launch, so its blocks are placed only after every block
  // of the chain kernel is running (and has its SM to itself), and it fills the SMs that
  // stay or fall free.  It waits for the chain kernel before it ends (see sketch_kernel).
  auto launch_light = [&](auto kernel, int threads, int smem, bool dependent, auto... args) -> bool {
    if (smem > 48 * 1024)
      CSG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    CSG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    int per_sm = 0;
    CSG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
    if (per_sm < 1) per_sm = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctx.num_sms * per_sm);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dependent ? 1 : 0;
    CSG_CUDA(cudaLaunchKernelEx(&cfg, kernel, a, args...));
    return true;
  };
  // The chunk ahead has listed only its heavy rows: there is other work only if some of them did
  // not fit the stream buffer.  That runs behind the chains in plain stream order, where its
  // idle blocks would otherwise sit on the SMs until the chains end.
  const int64_t span = a.chunk < a.n ? a.chunk : a.n;
  if (phase == PHASE_PRIO || CELLS > LANE_CELLS || span > (1 << 24)) {
    if (!launch_light(sketch_kernel<CELLS>, S_THREADS, 0, phase != PHASE_PRIO && !no_heavy_rows, phase == PHASE_PRIO ? 0 : 1,
                      phase == PHASE_PRIO ? 0 : 1))
      return false;
  } else if constexpr (CELLS <= LANE_CELLS) {
    auto lanes = [&](auto kernel, int index_words) {
      return launch_light(kernel, 32 * L_WARPS, (LaneLayout<CELLS>::I_OFF + index_words) * 4, behind || !no_heavy_rows,
                          no_heavy_rows ? 1 : 0);
    };
    if (span <= L_TABLE_MAX) {
      if (!lanes(rows_in_lanes_kernel<CELLS, TableIndex<CELLS>>, TableIndex<CELLS>::words(span))) return false;
    } else if (!lanes(rows_in_lanes_kernel<CELLS, ChainIndex<CELLS>>, ChainIndex<CELLS>::words(span))) {
      return false;
    }
  }
  count_launches(1);
  if (no_heavy_rows) return true;
  CSG_CUDA(launch_behind(behind, heavy_topk_kernel<CELLS>, ctx.num_sms, S_THREADS, 0, st, a));
  count_launches(5);
  return true;
}

}  // namespace

int chain_groups(const Context &ctx, int slots, int64_t span) {
  static_assert(ROUND_CELLS == 4, "a case each");
  switch (slots / 32) {
    case 1: return chain_block<1>(ctx, span).groups;
    case 2: return chain_block<2>(ctx, span).groups;
    case 3: return chain_block<3>(ctx, span).groups;
    case 4: return chain_block<4>(ctx, span).groups;
    default: return 0;
  }
}

bool launch_sketch(Context &ctx, int32_t n, int32_t nnz, const CsgParams &p, const int32_t *d_ptr,
                   CsgScratch &s, int32_t row_base, bool zero_table, int phase) {
  if (!s.no_heavy_rows && !plan_chains(ctx, nnz, s, phase)) return false;
  SketchArgs a;
  a.n = n;
  a.nnz = nnz;
  a.k = p.k;
  a.row_base = row_base;
  a.chunk = p.chunk;
  a.ptr = d_ptr;
  a.seg = s.seg;
  a.seg_rank = s.seg_rank;
  a.row_seg = s.row_seg;
  a.row_cols = s.row_cols;
  a.cand = s.cand;
  a.row_list = s.row_list;
  a.row_work = s.row_work;
  a.hstream = s.hstream;
  a.heavy_off = s.heavy_off;
  a.heavy_state = s.heavy_state;
  a.stream_cap = s.stream_cap;
  a.heavy_max = s.heavy_max;
  a.part_base = s.part_base;
  a.part_off = s.part_off;
  a.ctrl = s.ctrl;
  a.table = s.table;
  // Rows without candidates are never visited.  The greedy stage knows them from their work
  // count and never reads their entries; whoever reads the whole table (its export, the
  // statistics) needs them to read as empty.
  if (zero_table)
    CSG_CUDA(cudaMemsetAsync(s.table, 0, sizeof(uint64_t) * static_cast<size_t>(n) * p.k, ctx.stream));
  switch (p.M / 32) {
#define CSG_CASE(C) \
  case C:           \
    return launch_cells<C>(ctx, a, phase, s.no_heavy_rows);
    CSG_CASE(1) CSG_CASE(2) CSG_CASE(3) CSG_CASE(4) CSG_CASE(5) CSG_CASE(6) CSG_CASE(7) CSG_CASE(8)
    CSG_CASE(9) CSG_CASE(10) CSG_CASE(11) CSG_CASE(12) CSG_CASE(13) CSG_CASE(14) CSG_CASE(15)
    CSG_CASE(16)
#undef CSG_CASE
    default:
      set_error("sketch capacity %d is not a multiple of 32 in [32, 512]", p.M);
      return false;
  }
}

}  // namespace csg
