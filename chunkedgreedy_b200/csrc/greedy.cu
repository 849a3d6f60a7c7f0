// Greedy chaining inside each chunk, and the optional table statistics.
//
// Semantics restated from sporder/src/csg/chunk_similarity_greedy.cu:14-96: the
// chain starts at the chunk's first row; the next row is the unvisited in-chunk
// entry of the current row's top-k list with the largest weight (ties: smaller
// index); with none left the chain restarts at the smallest unvisited row
// (sporder/src/common/warp_visited_bitmap.cuh:99-111).  The visiting order is the
// permutation (new2old).
//
// One warp runs a chunk's chain as in the reference; what changes: rows whose candidate
// stream was empty are known from the transpose (row_work == 0) and never enter the chain
// (see greedy_lists_kernel), the chain runs on short lists in shared memory, and the order
// leaves the block in one coalesced copy.
#include "common.cuh"

namespace csg {

namespace {

constexpr int G_WARPS = 4;

struct GreedyArgs {
  int32_t n, k, chunk, num_chunks, row_base;
  const uint64_t *table;
  const uint32_t *row_work;
  int32_t *order;
  uint32_t *ctrl;      // stats block, or nullptr
  uint32_t *ctrl_all;  // the control words (checked build: where a bad index is recorded)
  uint32_t *gbitmaps;  // global bitmaps when a chunk's bitmaps do not fit shared memory
  int32_t words;       // bitmap words per chunk
};

struct ChainStats {  // lives at ctrl[CTRL_STATS ...]
  unsigned long long total_degree;
  double total_weight;
  double link_weight_sum;
  int32_t zero_degree_rows;
  int32_t restarts;
  int32_t links;
  int32_t pad;
  double in_chunk_weight;  // table weights whose candidate lies in the row's own chunk
};

// The chain of rows [start, end), run by one warp on the table itself.
__device__ __forceinline__ void chain_chunk(const GreedyArgs &a, int32_t start, int32_t end, uint32_t *visited) {
  const int lane = lane_id();
  const int32_t size = end - start;
  const int32_t words = (size + 31) >> 5;
  uint32_t *nonempty = visited + a.words;
  for (int32_t w = lane; w < words; w += 32) visited[w] = 0;
  for (int32_t base = 0; base < size; base += 32) {
    const int32_t i = base + lane;
    const bool ne = (i < size) && a.row_work[start + i] != 0;
    const unsigned m = __ballot_sync(FULL, ne);
    if (lane == 0) nonempty[base >> 5] = m;
  }
  __syncwarp();

  int32_t cur = start, emitted = 0, scan = 0, mine = 0;
  int32_t restarts = 0, links = 0;
  float link_w = 0.0f;
  for (;;) {
    const int32_t loc = cur - start;
    if (lane == 0) visited[loc >> 5] |= 1u << (loc & 31);
    if (lane == (emitted & 31)) mine = cur + a.row_base;
    ++emitted;
    if ((emitted & 31) == 0 && index_ok(a.ctrl_all, CHK_ORDER, emitted, size + 1))
      a.order[start + emitted - 32 + lane] = mine;
    __syncwarp();

    int32_t best_c = -1;
    if (nonempty[loc >> 5] & (1u << (loc & 31))) {
      const uint64_t *row = a.table + static_cast<size_t>(cur) * a.k;
      uint32_t best_w = 0;  // weight bits; real weights are positive
      for (int32_t j = lane; j < a.k; j += 32) {
        const uint64_t e = row[j];
        if (e == 0) break;  // valid entries form a prefix
        const int32_t cand = entry_index(e) - a.row_base;
        if (cand < start || cand >= end) continue;
        const int32_t cl = cand - start;
        if (visited[cl >> 5] & (1u << (cl & 31))) continue;
        // The next row of the chain is one of these candidates, and its list is needed as
        // soon as the arg-max below is known: ask for every candidate's list now, so that the
        // one dependent load per step finds it in L1 instead of waiting on L2.
        asm volatile("prefetch.global.L1 [%0];" ::"l"(a.table + static_cast<size_t>(cand) * a.k));
        const uint32_t wb = entry_weight_bits(e);
        if (wb > best_w || (wb == best_w && cand < best_c)) {
          best_w = wb;
          best_c = cand;
        }
      }
      const uint32_t g = __reduce_max_sync(FULL, best_w);
      if (g != 0u) {
        const uint32_t c = (best_w == g) ? static_cast<uint32_t>(best_c) : 0xFFFFFFFFu;
        best_c = static_cast<int32_t>(__reduce_min_sync(FULL, c));
        links += 1;
        link_w += __uint_as_float(g);
      } else {
        best_c = -1;
      }
    }
    if (best_c >= 0) {
      cur = best_c;
      continue;
    }
    // Restart at the smallest unvisited row; `scan` only moves forward.  A row without a
    // list (no bit in `nonempty`) would be emitted, find no neighbour and restart again, one
    // dependent step each - and on many inputs most rows are like that.  They change nothing
    // for the rows behind them, so all unvisited rows without a list in front of the first
    // unvisited row WITH a list are emitted here at once, in index order, as the chain
    // would have emitted them one by one (each of them counts as one restart).
    int32_t nxt = -1;
    for (int32_t base = scan; base < words; base += 32) {
      const int32_t w = base + lane;
      uint32_t fr = 0, ne = 0;
      if (w < words) {
        fr = ~visited[w];
        if (w == words - 1 && (size & 31)) fr &= (1u << (size & 31)) - 1u;
        ne = nonempty[w];
      }
      const uint32_t listed = fr & ne, bare = fr & ~ne;
      const unsigned mb = __ballot_sync(FULL, listed != 0);
      const int lb = mb ? __ffs(mb) - 1 : 32;  // lane of the first word that holds a row with a list
      const uint32_t fb = __shfl_sync(FULL, listed, lb & 31);
      const int bitb = mb ? __ffs(fb) - 1 : 0;
      uint32_t take = lane < lb ? bare : (lane == lb ? bare & ((1u << bitb) - 1u) : 0u);
      if (__any_sync(FULL, take != 0)) {
        const int32_t cnt = __popc(take);
        int32_t incl = cnt;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const int32_t t = __shfl_up_sync(FULL, incl, off);
          if (lane >= off) incl += t;
        }
        const int32_t total = __shfl_sync(FULL, incl, 31);
        // entries still waiting in registers go out first, then the run, in place
        if (lane < (emitted & 31)) a.order[start + (emitted & ~31) + lane] = mine;
        int32_t at = start + emitted + incl - cnt;
        if (w < words) visited[w] |= take;
        while (take) {
          const int b = __ffs(take) - 1;
          take &= take - 1;
          if (index_ok(a.ctrl_all, CHK_ORDER, at - start, size)) a.order[at] = start + (w << 5) + b + a.row_base;
          ++at;
        }
        emitted += total;
        restarts += total;
        __syncwarp();
        // the block of 32 that is being filled now: its first entries are already in memory
        if (lane < (emitted & 31)) mine = a.order[start + (emitted & ~31) + lane];
      }
      if (mb) {
        scan = base + lb;
        nxt = (scan << 5) + bitb;
        break;
      }
    }
    if (nxt < 0) break;
    cur = start + nxt;
    restarts += 1;
  }
  if ((emitted & 31) != 0 && lane < (emitted & 31)) a.order[start + (emitted & ~31) + lane] = mine;

  if (a.ctrl && lane == 0) {
    ChainStats *st = reinterpret_cast<ChainStats *>(a.ctrl + CTRL_STATS);
    atomicAdd(&st->restarts, restarts);
    atomicAdd(&st->links, links);
    atomicAdd(&st->link_weight_sum, static_cast<double>(link_w));
  }
}

// Chunks whose lists do not fit shared memory: a warp each.
__global__ void __launch_bounds__(G_WARPS * 32) greedy_kernel(GreedyArgs a) {
  wait_for_kernels_before();
  extern __shared__ uint32_t g_smem[];
  const int warp = threadIdx.x >> 5;
  const int32_t q = blockIdx.x * G_WARPS + warp;
  if (q >= a.num_chunks) return;
  const int64_t start64 = static_cast<int64_t>(q) * a.chunk;
  const int32_t start = static_cast<int32_t>(start64);
  const int32_t end = (start64 + a.chunk > a.n) ? a.n : static_cast<int32_t>(start64 + a.chunk);
  // two bitmaps per chunk: visited, and "row has a non-empty top-k list"
  uint32_t *visited = a.gbitmaps ? a.gbitmaps + static_cast<size_t>(q) * 2 * a.words
                                 : g_smem + static_cast<size_t>(warp) * 2 * a.words;
  chain_chunk(a, start, end, visited);
}

// A block per chunk.  A chunk is one dependent chain of up to 1024 steps, so what counts is the
// latency of a step.
//  * Rows without a list ("bare") stay out of the chain: the chain would emit one only when it
//    restarts there, and change nothing by it.  The rows with a list are numbered 0 .. m-1 in
//    index order.  Restarts go to ascending rows, and a bare row comes out just before
//    the first restart at a row behind it: once the chain is known, every bare row's place
//    follows from the number of rows the chain had emitted at that restart.
//  * The block first writes every list out as 16-bit row numbers in the order in which the chain
//    would try them (weight, on ties the smaller index; the table has the weights in order, only
//    ties have to be put right), candidates outside the chunk as a row that counts as visited.
//  * A step is then: read the current row's list, read those rows' flags, one warp minimum over
//    (place in the list, row) of the free ones.  Lanes without a list entry look at the rows behind
//    the restart cursor meanwhile, and the same minimum says where to restart if no entry is free.
//    All else is kept out of the loop: a lone warp waits four to six cycles for every instruction
//    that needs the one before it, and written without care the step takes 460 cycles instead of 135.
// On a B200, per call: power-law band of 65,536 rows 320 -> 74 us (64 chains, the longest of 900
// steps), R-MAT scale 22 646 -> 258 us (4096 chains).
// A candidate without a list of its own (a caller's own table can hold one) would let the
// chain reach bare rows: such a chunk runs on the table.
constexpr int GS_MAX_SPAN = 32768;   // rows of a chunk: their numbers must fit 15 bits
constexpr uint32_t BARE = 0x8000u;   // in `place`: a bare row's place in the chunk, else a numbered row
constexpr int GS_WINDOW = 32;        // flags behind the last row that read as visited

struct ListLayout {  // shared memory, in bytes
  int flags, row_of, place, mark, window, words, lists, total;
};
__host__ __device__ inline ListLayout list_layout(int32_t span, int32_t k) {
  ListLayout l;
  int at = 0;
  auto take = [&](int bytes) {
    const int o = at;
    at += (bytes + 15) & ~15;
    return o;
  };
  const int words = (span + 31) / 32;
  l.flags = take(span + GS_WINDOW + 1);  // per numbered row: emitted
  l.row_of = take(2 * (span + 1));       // its place in the chunk
  l.place = take(2 * span);              // the order: who goes to each place
  l.mark = take(2 * (span + 1));         // per numbered row: 1 + rows emitted before the restart at it, 0 without one
  l.window = take(2 * 32);               // what lanes without a list entry look at
  l.words = take(8 * words);             // per 32 rows: which have a list; how many in front have one
  l.lists = take(2 * span * k);
  l.total = at;
  return l;
}

// Shared memory by its own 32-bit addresses, in program order.
__device__ __forceinline__ uint32_t lds_u16(uint32_t at) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(at));
  return v;
}
__device__ __forceinline__ uint32_t lds_s8(uint32_t at) {  // sign-extended
  int32_t v;
  asm volatile("ld.shared.s8 %0, [%1];" : "=r"(v) : "r"(at));
  return static_cast<uint32_t>(v);
}
__device__ __forceinline__ void sts_u8(uint32_t at, uint32_t v) {
  asm volatile("st.shared.u8 [%0], %1;" ::"r"(at), "r"(v));
}
__device__ __forceinline__ void sts_u16(uint32_t at, uint32_t v) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(at), "h"(static_cast<uint16_t>(v)));
}

// Out of line for greedy_lists_kernel, whose registers it would cost and which hardly ever calls it.  greedy_kernel,
// which does nothing else, has it inlined: called, it read its arguments from memory at every step (mesh of
// 262,144 rows in chunks of 8,192, k = 16: 3.95 ms per csg call, 3.72 inlined).
__device__ __noinline__ void chain_chunk_rare(const GreedyArgs &a, int32_t start, int32_t end, uint32_t *visited) {
  chain_chunk(a, start, end, visited);
}

// LONG: lists of more than 32 entries.
template <bool STATS, bool LONG>
__global__ void greedy_lists_kernel(GreedyArgs a) {
  wait_for_kernels_before();
  extern __shared__ __align__(16) unsigned char gl_smem[];
  __shared__ int32_t odd, count;
  const int lane = lane_id(), warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int32_t q = blockIdx.x;
  const int64_t start64 = static_cast<int64_t>(q) * a.chunk;
  const int32_t start = static_cast<int32_t>(start64);
  const int32_t end = (start64 + a.chunk > a.n) ? a.n : static_cast<int32_t>(start64 + a.chunk);
  const int32_t size = end - start, words = (size + 31) >> 5;
  const int k = a.k;
  const ListLayout lay = list_layout(a.chunk < a.n ? a.chunk : a.n, k);
  uint8_t *const flags = gl_smem + lay.flags;
  uint16_t *const row_of = reinterpret_cast<uint16_t *>(gl_smem + lay.row_of);
  uint16_t *const place = reinterpret_cast<uint16_t *>(gl_smem + lay.place);
  uint16_t *const mark = reinterpret_cast<uint16_t *>(gl_smem + lay.mark);
  uint32_t *const has = reinterpret_cast<uint32_t *>(gl_smem + lay.words);
  uint32_t *const before = has + words;
  uint16_t *const lists = reinterpret_cast<uint16_t *>(gl_smem + lay.lists);
  if (threadIdx.x == 0) odd = 0;
  for (int32_t w = warp; w < words; w += warps) {
    const int32_t i = (w << 5) + lane;
    const unsigned m = __ballot_sync(FULL, i < size && a.row_work[start + i] != 0);
    if (lane == 0) has[w] = m;
  }
  __syncthreads();
  if (warp == 0) {  // numbers: exclusive sums over the words
    int32_t run = 0;
    for (int32_t w0 = 0; w0 < words; w0 += 32) {
      const int32_t v = w0 + lane < words ? __popc(has[w0 + lane]) : 0;
      int32_t incl = v;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int32_t t = __shfl_up_sync(FULL, incl, off);
        if (lane >= off) incl += t;
      }
      if (w0 + lane < words) before[w0 + lane] = run + incl - v;
      run += __shfl_sync(FULL, incl, 31);
    }
    if (lane == 0) count = run;
  }
  __syncthreads();
  const int32_t m = count;
  for (int32_t i = threadIdx.x; i < size; i += blockDim.x) {
    const uint32_t w = has[i >> 5], bit = 1u << (i & 31);
    if (w & bit) row_of[before[i >> 5] + __popc(w & (bit - 1u))] = static_cast<uint16_t>(i);
  }
  for (int32_t i = threadIdx.x; i < m + GS_WINDOW + 1; i += blockDim.x)
    if (i <= a.chunk + GS_WINDOW) flags[i] = i < m ? 0 : 0xFF;
  for (int32_t i = threadIdx.x; i <= m; i += blockDim.x) mark[i] = static_cast<uint16_t>(i < m ? 0 : m + 1);
  __syncthreads();
  // lists: G lanes a row (16 while a list fits them), U rows of a group in flight
  {
    constexpr int U = 4;
    const int G = k <= 16 ? 16 : 32, groups = blockDim.x / G, group = threadIdx.x / G, gl = threadIdx.x % G;
    bool strange = false;
    for (int32_t r0 = 0; r0 < m; r0 += groups * U) {
      for (int j0 = 0; j0 < k; j0 += G) {
        const int j = j0 + gl;
        uint64_t e[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int32_t r = r0 + u * groups + group;
          e[u] = r < m && j < k ? a.table[static_cast<size_t>(start + row_of[r]) * k + j] : 0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int32_t r = r0 + u * groups + group;
          const uint32_t wb = entry_weight_bits(e[u]), id = static_cast<uint32_t>(e[u]);
          int pos = j;
          // among equal weights the smaller index comes first
          if (k <= G) {
            for (int d = 1; d < G; ++d) {
              const uint32_t uw = __shfl_up_sync(FULL, wb, d, 32), ui = __shfl_up_sync(FULL, id, d, 32);
              const uint32_t dw = __shfl_down_sync(FULL, wb, d, 32), di = __shfl_down_sync(FULL, id, d, 32);
              const bool up = gl >= d && wb && uw == wb, down = gl + d < G && wb && dw == wb;
              if (!__any_sync(FULL, up || down)) break;
              pos += (down && di < id ? 1 : 0) - (up && ui > id ? 1 : 0);
            }
          } else if (wb) {
            const uint64_t *row = a.table + static_cast<size_t>(start + row_of[r]) * k;
            for (int t = j - 1; t >= 0 && entry_weight_bits(row[t]) == wb; --t)
              pos -= static_cast<uint32_t>(row[t]) > id ? 1 : 0;
            for (int t = j + 1; t < k && entry_weight_bits(row[t]) == wb; ++t)
              pos += static_cast<uint32_t>(row[t]) < id ? 1 : 0;
          }
          if (r < m && j < k) {
            const int32_t cand = entry_index(e[u]) - a.row_base - start;
            uint32_t number = static_cast<uint32_t>(m);  // reads as visited
            if (wb && cand >= 0 && cand < size) {
              const uint32_t w = has[cand >> 5], bit = 1u << (cand & 31);
              number = before[cand >> 5] + __popc(w & (bit - 1u));
              strange |= (w & bit) == 0u;
            }
            lists[r * k + pos] = static_cast<uint16_t>(number);
          }
        }
      }
    }
    if (strange) odd = 1;
  }
  __syncthreads();
  if (odd) {
    if (warp == 0) chain_chunk_rare(a, start, end, has);  // (its two bitmaps fit the words)
    return;
  }
  if (warp == 0 && m > 0) {
    const uint32_t s_flags = static_cast<uint32_t>(__cvta_generic_to_shared(flags));
    const uint32_t s_place = static_cast<uint32_t>(__cvta_generic_to_shared(place));
    const uint32_t s_mark = static_cast<uint32_t>(__cvta_generic_to_shared(mark));
    const uint32_t s_row_of = static_cast<uint32_t>(__cvta_generic_to_shared(row_of));
    // a lane reads its entry of the list, or behind the list its place of the cursor's window
    const bool mine = lane < k;
    const uint32_t s_list =
        static_cast<uint32_t>(__cvta_generic_to_shared(gl_smem + (mine ? lay.lists : lay.window))) + 2 * lane;
    const uint32_t stride = mine ? 2 * k : 0;
    const uint32_t tag = mine ? static_cast<uint32_t>(lane) << 15 : 0x80000000u;
    int32_t segments = 0, t = 0;
    float link_w = 0.0f;
    uint32_t c = 0;  // the chain begins with a restart at number 0
    for (;;) {
      // a restart at c: everything in front of it that is not emitted yet is bare
      const uint32_t shift = lds_u16(s_row_of + 2 * c) - c;
      sts_u16(s_mark + 2 * c, t + 1);
      uint32_t cursor = c + 1, next;
      if (!mine) sts_u16(s_list, min(cursor + lane - k, m));
      ++segments;
      const uint32_t out0 = s_place + 2 * shift;
      uint32_t out = out0 + 2 * t;
      for (;;) {
        // (all lanes store the same values, so each sees its own and no barrier is needed)
        sts_u8(s_flags + c, 0xFFu);
        uint32_t at = lds_u16(s_list + c * stride);
        sts_u16(out, c);
        out += 2;
        uint32_t found = lds_s8(s_flags + at) | (tag | at);  // all ones when that row is out already
        if (LONG)
          for (int j = lane + 32; j < k && found == 0xFFFFFFFFu; j += 32) {
            at = lds_u16(s_list + c * stride + 2 * (j - lane));
            found = lds_s8(s_flags + at) | (static_cast<uint32_t>(j) << 15 | at);
          }
        next = __reduce_min_sync(FULL, found);
        if (next >= 0x80000000u) break;
        if (STATS)
          link_w += __uint_as_float(
              entry_weight_bits(a.table[static_cast<size_t>(start + row_of[c]) * k + (next >> 15)]));
        c = next & 0x7FFFu;
      }
      t = static_cast<int32_t>(out - out0) >> 1;
      while (next == 0xFFFFFFFFu && static_cast<int32_t>(cursor) < m) {  // nobody free in the cursor's window
        const uint32_t at = min(cursor + lane, m);
        next = __reduce_min_sync(FULL, lds_s8(s_flags + at) | (0x80000000u | at));
        cursor += 32;
      }
      if (next == 0xFFFFFFFFu) break;
      c = next & 0x7FFFFFFFu;
    }
    if (STATS && lane == 0) {
      ChainStats *st = reinterpret_cast<ChainStats *>(a.ctrl + CTRL_STATS);
      atomicAdd(&st->restarts, size - m + segments - 1);  // every bare row is one; the first row is none
      atomicAdd(&st->links, m - segments);
      atomicAdd(&st->link_weight_sum, static_cast<double>(link_w));
    }
  } else if (STATS && warp == 0 && lane == 0) {
    atomicAdd(&reinterpret_cast<ChainStats *>(a.ctrl + CTRL_STATS)->restarts, size - 1);
  }
  __syncthreads();
  for (int32_t i = threadIdx.x; i < size; i += blockDim.x) {  // the bare rows' places
    const uint32_t w = has[i >> 5], bit = 1u << (i & 31);
    if (w & bit) continue;
    const int32_t number = before[i >> 5] + __popc(w & (bit - 1u));
    int32_t x = number;  // the first restart behind it (the mark behind the last row ends the search)
    while (mark[x] == 0) ++x;
    const int32_t at = i - number + mark[x] - 1;
    if (index_ok(a.ctrl_all, CHK_ORDER, at, size)) place[at] = static_cast<uint16_t>(i | BARE);
  }
  __syncthreads();
  for (int32_t i = threadIdx.x; i < size; i += blockDim.x) {
    const uint32_t v = place[i];
    a.order[start + i] = start + static_cast<int32_t>(v & BARE ? v & ~BARE : row_of[v]) + a.row_base;
  }
}

// sporder/src/common/similarity_top_k.cu:120-157
__global__ void table_stats_kernel(int32_t n, int32_t k, const uint64_t *__restrict__ table,
                                   uint32_t *ctrl) {
  unsigned long long deg = 0;
  double wsum = 0.0;
  int32_t zero = 0;
  for (int32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const uint64_t *row = table + static_cast<size_t>(r) * k;
    int32_t d = 0;
    float rw = 0.0f;
    for (int32_t j = 0; j < k; ++j) {
      const uint64_t e = row[j];
      if (entry_index(e) == -1) break;
      d += 1;
      rw += __uint_as_float(entry_weight_bits(e));
    }
    deg += d;
    wsum += rw;
    zero += (d == 0);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    deg += __shfl_down_sync(FULL, deg, off);
    wsum += __shfl_down_sync(FULL, wsum, off);
    zero += __shfl_down_sync(FULL, zero, off);
  }
  if (lane_id() == 0) {
    ChainStats *st = reinterpret_cast<ChainStats *>(ctrl + CTRL_STATS);
    if (deg) {
      atomicAdd(&st->total_degree, deg);
      atomicAdd(&st->total_weight, wsum);
    }
    if (zero) atomicAdd(&st->zero_degree_rows, zero);
  }
}

// Weight of the table entries that stay inside their row's chunk, for the fraction of the
// graph a chunked ordering cuts (sporder/src/cg/chunk_greedy.cu:66-68,111-112;
// cg/stats_collector.cu:66-72).  Summed in fp64.
__global__ void __launch_bounds__(256) in_chunk_weight_kernel(int32_t n, int32_t k, int32_t chunk,
                                                              const uint64_t *__restrict__ table,
                                                              uint32_t *ctrl) {
  double mine = 0.0;
  for (int32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const int64_t start = static_cast<int64_t>(r / chunk) * chunk;
    const int64_t end = start + chunk < n ? start + chunk : n;
    const uint64_t *row = table + static_cast<size_t>(r) * k;
    for (int32_t j = 0; j < k; ++j) {
      const uint64_t e = row[j];
      if (e == 0) break;
      const int32_t cand = entry_index(e);
      if (cand >= start && cand < end) mine += static_cast<double>(__uint_as_float(entry_weight_bits(e)));
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) mine += __shfl_down_sync(FULL, mine, off);
  if ((threadIdx.x & 31) == 0 && mine != 0.0)
    atomicAdd(&reinterpret_cast<ChainStats *>(ctrl + CTRL_STATS)->in_chunk_weight, mine);
}

}  // namespace

bool launch_in_chunk_weight(Context &ctx, int32_t n, int32_t k, int32_t chunk, const uint64_t *table,
                            uint32_t *ctrl) {
  int grid = (n + 255) / 256;
  if (grid > ctx.num_sms * 8) grid = ctx.num_sms * 8;
  in_chunk_weight_kernel<<<grid, 256, 0, ctx.stream>>>(n, k, chunk, table, ctrl);
  CSG_CUDA(cudaGetLastError());
  count_launches(1);
  return true;
}

bool launch_greedy(Context &ctx, int32_t n, const CsgParams &p, CsgScratch &s,
                   int32_t *d_new_order, bool with_stats, int32_t row_base) {
  GreedyArgs a;
  a.n = n;
  a.k = p.k;
  a.chunk = p.chunk;
  a.row_base = row_base;
  a.num_chunks = static_cast<int32_t>((static_cast<int64_t>(n) + p.chunk - 1) / p.chunk);
  a.table = s.table;
  a.row_work = s.row_work;
  a.order = d_new_order;
  a.ctrl = with_stats ? s.ctrl : nullptr;
  a.ctrl_all = s.ctrl;
  const int32_t span = p.chunk < n ? p.chunk : n;
  a.words = (span + 31) / 32;
  size_t smem = static_cast<size_t>(G_WARPS) * 2 * a.words * sizeof(uint32_t);
  a.gbitmaps = nullptr;
  if (smem > 48 * 1024) {  // very large chunks: bitmaps in global memory
    CSG_REQUIRE(s.gbitmaps != nullptr, "greedy: no global bitmap space was reserved");
    a.gbitmaps = s.gbitmaps;
    smem = 0;
  }
  // a block per chunk on lists in shared memory, if they fit
  if (span <= GS_MAX_SPAN && p.k <= 256) {
    const int bytes = list_layout(span, p.k).total;
    if (bytes + 1024 <= ctx.smem_optin) {
      const bool lng = p.k > 32;
      auto kernel = with_stats ? (lng ? greedy_lists_kernel<true, true> : greedy_lists_kernel<true, false>)
                               : (lng ? greedy_lists_kernel<false, true> : greedy_lists_kernel<false, false>);
      CSG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
      // many chunks: several blocks to an SM; few: more warps to write the lists of each (64 chunks 83.8 us with 512
      // threads, 81.6 with 1024; 4 chunks 91.6 and 87.4)
      const int threads = a.num_chunks <= ctx.num_sms ? 1024 : a.num_chunks <= 2 * ctx.num_sms ? 512 : 256;
      CSG_CUDA(launch_behind(s.one_stream, kernel, a.num_chunks, threads, bytes, ctx.stream, a));
      count_launches(1);
      return true;
    }
  }
  const int grid = (a.num_chunks + G_WARPS - 1) / G_WARPS;
  CSG_CUDA(launch_behind(s.one_stream, greedy_kernel, grid, G_WARPS * 32, static_cast<int>(smem), ctx.stream, a));
  count_launches(1);
  return true;
}

bool launch_table_stats(Context &ctx, int32_t n, int32_t k, const uint64_t *table, uint32_t *ctrl) {
  int grid = (n + 255) / 256;
  if (grid > ctx.num_sms * 8) grid = ctx.num_sms * 8;
  table_stats_kernel<<<grid, 256, 0, ctx.stream>>>(n, k, table, ctrl);
  CSG_CUDA(cudaGetLastError());
  count_launches(1);
  return true;
}

}  // namespace csg
