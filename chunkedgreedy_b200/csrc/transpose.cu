// Chunk-local transpose.
//
// The reference builds a full CSC with a device-wide radix sort
// (sporder/src/common/csr2csc.cu:38-115) and then, per row, scans whole column
// lists to pick out the rows of the row's own chunk
// (sporder/src/common/chunk_similarity_top_k.cu:52-84).  Candidates never leave
// the chunk, so this library transposes every chunk on its own, and only the part of it
// that matters: a column that a single row of the chunk holds brings no candidate.  The
// kernels emit, with "group" for the rows of a chunk that share a column,
//   cand[]  : the rows of every group, ascending, each with its row length (what the Dice term
//             needs);
//   seg[]   : per row, one after the other and columns ascending, its groups: (first, length);
//             and seg_rank[], the place of the row itself inside the group;
//   row_seg, row_cols: where a row's groups are in seg[], and how many;
//   row_work: how many candidates the row's stream will hold.
// Chunks of up to C_NNZ nonzeros in which few enough of them lie in groups are handled start
// to finish by one thread block, without a sort (compact_kernel).  Heavier chunks - on power-law
// inputs a handful of chunks hold millions of nonzeros, and the rows with the longest streams
// live in exactly those - are cut into tiles and sorted by the whole grid: per pass a tile
// histogram, a per-chunk scan and a stable tile scatter, then a group search per element (there
// every column of a row gets an entry of seg[]).
// The reference can be promised a symmetric pattern and then reads the CSR arrays as the CSC
// (sporder/src/common/csr2csc.h:52-54); nothing here needs the promise.
#include "common.cuh"

namespace csg {

namespace {

constexpr int T_THREADS = 512;
constexpr int T_WARPS = T_THREADS / 32;
constexpr int T_IPT = 8;
constexpr int T_TILE = T_THREADS * T_IPT;  // 4096
constexpr int C_NNZ = 65536;               // largest chunk (nonzeros) that compact_kernel looks at ...
constexpr int C_ROWS = 2048;               // ... and its rows
constexpr int C_TALL_ROWS = 4096;          // ... where chunks have more,
constexpr int C_TALL_NNZ = 28672;          // with so many nonzeros

struct TransposeArgs {
  int32_t n, nnz, chunk, num_chunks, passes;
  const int32_t *ptr, *ind;
  uint32_t *keyA, *keyB, *payA, *payB;
  int2 *cand, *seg;
  int32_t *seg_rank, *row_seg, *row_cols;
  uint32_t *row_work;
  uint32_t *ctrl;
  unsigned long long *count;  // only count the groups, rows alone in a column included (nullptr: transpose)
  int32_t *next_chunk;        // chunks compact_kernel's small form passed on to the large one
  // heavy chunks (those that compact_kernel passes on)
  int32_t *heavy_chunk;      // chunk ids, in arrival order
  int32_t *heavy_tile_base;  // first tile of each heavy chunk, plus the total
  uint32_t *tile_hist;       // [tile][256] digit counts, then offsets
  uint32_t *digit_base;      // [heavy chunk][256]
  // a call that runs one chunk ahead: the control words that name the chunk, and whether this
  // pass leaves that chunk out (nullptr / false otherwise)
  const uint32_t *ctrl_main;
  bool skip_prio;
};

struct ChunkSpan {
  int32_t cs, rows, b, L;
};

__device__ __forceinline__ ChunkSpan chunk_span(const TransposeArgs &a, int32_t q) {
  ChunkSpan c;
  const int64_t cs64 = static_cast<int64_t>(q) * a.chunk;
  c.cs = static_cast<int32_t>(cs64);
  const int32_t ce = (cs64 + a.chunk > a.n) ? a.n : static_cast<int32_t>(cs64 + a.chunk);
  c.rows = ce - c.cs;
  c.b = a.ptr[c.cs];
  c.L = a.ptr[ce] - c.b;
  if (c.b < 0 || c.L < 0 || c.L > a.nnz - c.b) {  // malformed row pointers: flag and skip
    atomicExch(&a.ctrl[CTRL_BAD_INPUT], 1u);
    c.L = 0;
  }
  return c;
}

// Row that owns CSR position x: largest row with ptr[row] <= x, searched in
// [row_lo, row_hi] over either the shared copy of the chunk's row pointers or the
// global array.
__device__ __forceinline__ int32_t row_of(const int32_t *p, int32_t lo, int32_t hi, int32_t x) {
  // invariant: p[lo] <= x < p[hi]
  while (hi - lo > 1) {
    const int32_t mid = lo + ((hi - lo) >> 1);
    if (p[mid] <= x)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// One block per chunk, no sort:
//  1. every column sets a bit of a hashed bit map, and a second time a bit of another map: what
//     has not set the second bit is alone in its column (most nonzeros of a mesh or a road);
//  2. the others are numbered in CSR order and entered into a hash table, which counts each
//     column's rows;
//  3. the table's counts of two and more become places in cand[];
//  4. every member writes its row to its group, in any order, and then counts the smaller rows
//     of the group: its place.  (That is one comparison per candidate the sketch stage will have to
//     work through, so it never dominates.)
//  5. members go out with their groups in CSR order, which is the order seg[] wants.
// Chunks of up to 2,048 rows: blocks of 512 threads, two to an SM, for up to 6144 numbered nonzeros (in up to 3072
// columns); chunks with more go on to blocks of 1024 threads for up to 22,528 (in up to 6144 columns), those with
// more again to the tiled sort.  Taller ones: blocks of 1024 threads for up to 16,384 (launch_compact).
// On a B200, 1.05 M rows of the shuffled mesh: 227 us with the groups read off the promised
// symmetry, 115 without any promise; 65,536 rows of the power-law band: 173 -> 84 us.
template <int THREADS_, int CAP_, int TABLE_BITS_, int FILTER_BITS_, int ROWS_>
struct CompactSize {
  static constexpr int ROWS = ROWS_, NNZ = ROWS_ == C_ROWS ? C_NNZ : C_TALL_NNZ, GROUP_BITS = ROWS_ < 4096 ? 12 : 13;
  static constexpr uint32_t GROUP = (1u << GROUP_BITS) - 1u;  // rows of a column
  static constexpr int THREADS = THREADS_, WARPS = THREADS / 32, CAP = CAP_, TABLE_BITS = TABLE_BITS_, FILTER_BITS = FILTER_BITS_;
  static constexpr int TABLE = 1 << TABLE_BITS, FILTER = (1 << FILTER_BITS) / 32;  // entries; words of each map
  // columns from which on a thread gives up: they cannot fill the table, however many are on their way
  static constexpr int COLUMNS = TABLE - 2 * THREADS;
  struct Shared {
    uint32_t key[TABLE];          // columns, then how many members wrote their row
    uint32_t cnt[TABLE];          // rows per column, then (place << GROUP_BITS) | rows, 0 for a column with one
    union {
      uint32_t filter[2][FILTER];
      uint16_t member[CAP];       // rows of the groups
    };
    uint16_t slot[CAP];           // table entry of each numbered nonzero
    uint16_t row[CAP];            // its position, then its row
    int32_t sptr[ROWS + 1];
    uint32_t work[ROWS];
    uint32_t cols[ROWS / 2];      // 16 bits a row
    int32_t warp_sum[32];
    int32_t ticket, columns;
  };
};
using CompactSmall = CompactSize<512, 6144, 12, 17, C_ROWS>;
using CompactLarge = CompactSize<1024, 22528, 13, 17, C_ROWS>;
using CompactTall = CompactSize<1024, 16384, 13, 17, C_TALL_ROWS>;

// exclusive sum over the block's threads; *total is the sum of all
template <int WARPS>
__device__ __forceinline__ int32_t block_sum(int32_t v, int32_t *warp_sum, int32_t *total) {
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  int32_t incl = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int32_t t = __shfl_up_sync(FULL, incl, off);
    if (lane >= off) incl += t;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  const int32_t w = lane < WARPS ? warp_sum[lane] : 0;
  int32_t wi = w;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int32_t t = __shfl_up_sync(FULL, wi, off);
    if (lane >= off) wi += t;
  }
  *total = __shfl_sync(FULL, wi, 31);
  const int32_t base = __shfl_sync(FULL, wi - w, warp);
  __syncthreads();
  return base + incl - v;
}

__device__ __forceinline__ uint32_t column_hash(uint32_t c) { return c * 0x9E3779B1u; }

// NEXT: the chunks that the form before left (ctrl[CTRL_NEXT_COUNT] of them).  LAST: what does not fit
// goes to the tiled sort.
template <typename S, bool NEXT, bool LAST>
__global__ void __launch_bounds__(S::THREADS) compact_kernel(TransposeArgs a) {
  let_next_kernel_start();
  wait_for_kernels_before();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  typename S::Shared &sh = *reinterpret_cast<typename S::Shared *>(smem_raw);
  constexpr int THREADS = S::THREADS, U = 8;
  const int tid = threadIdx.x, lane = tid & 31;
  for (;;) {
    __syncthreads();
    if (tid == 0) sh.ticket = static_cast<int32_t>(atomicAdd(&a.ctrl[NEXT ? CTRL_NEXT_TICKET : CTRL_CHUNK_TICKET], 1u));
    __syncthreads();
    if (sh.ticket >= (NEXT ? static_cast<int32_t>(a.ctrl[CTRL_NEXT_COUNT]) : a.num_chunks)) break;
    const int32_t q = NEXT ? a.next_chunk[sh.ticket] : sh.ticket;
    if (a.skip_prio && static_cast<uint32_t>(q) == a.ctrl_main[CTRL_PRIO]) continue;
    const ChunkSpan c = chunk_span(a, q);
    const int32_t b = c.b, rows = c.rows;
    const int L = c.L;
    if (L > S::NNZ || rows > S::ROWS) {
      if (tid == 0) a.heavy_chunk[atomicAdd(&a.ctrl[CTRL_HEAVY_COUNT], 1u)] = q;
      for (int i = tid; i < rows; i += THREADS) a.row_work[c.cs + i] = 0;  // (the tiled sort adds to it)
      continue;
    }
    if (tid == 0) sh.columns = 0;
    bool ordered = true;
    for (int i = tid; i < rows; i += THREADS) {
      const int32_t x = a.ptr[c.cs + i], y = a.ptr[c.cs + i + 1];
      sh.sptr[i] = x;
      if (i == rows - 1) sh.sptr[rows] = y;
      ordered &= x <= y;
      sh.work[i] = 0;
      if (i < S::ROWS / 2) sh.cols[i] = 0;
    }
    if (!ordered) atomicExch(&a.ctrl[CTRL_BAD_INPUT], 1u);
    for (int i = tid * 4; i < S::TABLE; i += THREADS * 4) {
      *reinterpret_cast<uint4 *>(sh.key + i) = make_uint4(FULL, FULL, FULL, FULL);
      *reinterpret_cast<uint4 *>(sh.cnt + i) = make_uint4(0, 0, 0, 0);
    }
    for (int i = tid * 4; i < 2 * S::FILTER; i += THREADS * 4)
      *reinterpret_cast<uint4 *>(&sh.filter[0][0] + i) = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const uint32_t *const ind = reinterpret_cast<const uint32_t *>(a.ind + b);
    for (int i0 = tid; i0 < L; i0 += THREADS * U) {
      uint32_t col[U];
#pragma unroll
      for (int u = 0; u < U; ++u) col[u] = i0 + u * THREADS < L ? __ldg(ind + i0 + u * THREADS) : 0u;
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (i0 + u * THREADS < L) {
          const uint32_t h = column_hash(col[u]) >> (32 - S::FILTER_BITS), bit = 1u << (h & 31);
          if (atomicOr(&sh.filter[0][h >> 5], bit) & bit) atomicOr(&sh.filter[1][h >> 5], bit);
        }
    }
    __syncthreads();
    // number what may share its column, in CSR order: a warp's elements are consecutive
    int32_t numbered = 0;
    for (int tb = 0; tb < L && numbered <= S::CAP; tb += THREADS * U) {
      const int first = tb + (tid >> 5) * (32 * U) + lane;
      uint32_t col[U];
      unsigned on[U];
      int32_t mine = 0;
#pragma unroll
      for (int u = 0; u < U; ++u) col[u] = first + u * 32 < L ? __ldg(ind + first + u * 32) : 0u;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t h = column_hash(col[u]) >> (32 - S::FILTER_BITS);
        on[u] = __ballot_sync(FULL, first + u * 32 < L && ((sh.filter[1][h >> 5] >> (h & 31)) & 1u) != 0u);
        mine += __popc(on[u]);
      }
      int32_t tile_total;
      int32_t at = numbered + block_sum<S::WARPS>(lane == 0 ? mine : 0, sh.warp_sum, &tile_total);
      at = __shfl_sync(FULL, at, 0);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int32_t s = at + __popc(on[u] & ((1u << lane) - 1u));
        at += __popc(on[u]);
        if (((on[u] >> lane) & 1u) && s < S::CAP) sh.row[s] = static_cast<uint16_t>(first + u * 32);
      }
      numbered += tile_total;
    }
    __syncthreads();
    const int inserted = numbered <= S::CAP ? numbered : 0;
    for (int i0 = tid; i0 < inserted; i0 += THREADS * 4) {
      uint32_t col[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) col[u] = i0 + u * THREADS < inserted ? __ldg(ind + sh.row[i0 + u * THREADS]) : 0u;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (i0 + u * THREADS >= inserted || *static_cast<volatile int32_t *>(&sh.columns) > S::COLUMNS) continue;
        uint32_t t = column_hash(col[u]) >> (32 - S::TABLE_BITS);
        for (;;) {
          const uint32_t seen = atomicCAS(&sh.key[t], FULL, col[u]);
          if (seen == FULL) atomicAdd(&sh.columns, 1);
          if (seen == FULL || seen == col[u]) break;
          t = (t + 1) & (S::TABLE - 1);
        }
        atomicAdd(&sh.cnt[t], 1u);
        sh.slot[i0 + u * THREADS] = static_cast<uint16_t>(t);
      }
    }
    __syncthreads();
    if (numbered > S::CAP || sh.columns > S::COLUMNS) {  // (the same in all threads)
      if (tid == 0) {
        if (LAST)
          a.heavy_chunk[atomicAdd(&a.ctrl[CTRL_HEAVY_COUNT], 1u)] = q;
        else
          a.next_chunk[atomicAdd(&a.ctrl[CTRL_NEXT_COUNT], 1u)] = q;
      }
      if (LAST)
        for (int i = tid; i < rows; i += THREADS) a.row_work[c.cs + i] = 0;  // (the tiled sort adds to it)
      continue;
    }
    // places of the groups, in any order
    {
      constexpr int PER = S::TABLE / THREADS;
      uint32_t v[PER];
      int32_t mine = 0, repeats = 0;
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        v[i] = sh.cnt[i * THREADS + tid];
        if (v[i] > S::GROUP) {  // (only with columns repeated inside rows)
          atomicExch(&a.ctrl[CTRL_BAD_INPUT], 1u);
          v[i] = 0;
        }
        mine += v[i] >= 2 ? static_cast<int32_t>(v[i]) : 0;
        repeats += v[i] >= 2 ? static_cast<int32_t>(v[i]) - 1 : 0;
      }
      if (a.count) {
        repeats = __reduce_add_sync(FULL, repeats);
        if (lane == 0 && repeats) atomicAdd(a.count, static_cast<unsigned long long>(-static_cast<long long>(repeats)));
        if (tid == 0) atomicAdd(a.count, static_cast<unsigned long long>(L));
        continue;
      }
      int32_t total;
      int32_t run = block_sum<S::WARPS>(mine, sh.warp_sum, &total);
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const uint32_t n = v[i];
        sh.cnt[i * THREADS + tid] = n >= 2 ? (static_cast<uint32_t>(run) << S::GROUP_BITS) | n : 0u;
        sh.key[i * THREADS + tid] = 0u;
        run += n >= 2 ? static_cast<int32_t>(n) : 0;
      }
    }
    __syncthreads();
    for (int s = tid; s < numbered; s += THREADS) {
      const uint32_t t = sh.slot[s], g = sh.cnt[t];
      if (g == 0u) continue;
      const int32_t r = row_of(sh.sptr, 0, rows, b + sh.row[s]);
      sh.row[s] = static_cast<uint16_t>(r);
      const uint32_t at = (g >> S::GROUP_BITS) + atomicAdd(&sh.key[t], 1u);
      if (index_ok(a.ctrl, CHK_GROUP, at, S::CAP)) sh.member[at] = static_cast<uint16_t>(r);
      atomicAdd(&sh.work[r], (g & S::GROUP) - 1u);
    }
    __syncthreads();
    int32_t written = 0;
    for (int tb = 0; tb < numbered; tb += THREADS) {
      const int s = tb + tid;
      uint32_t g = 0;
      int32_t r = 0, rank = 0;
      if (s < numbered) {
        g = sh.cnt[sh.slot[s]];
        r = sh.row[s];
      }
      const int32_t start = static_cast<int32_t>(g >> S::GROUP_BITS), len = static_cast<int32_t>(g & S::GROUP);
      for (int32_t i = 0; i < len; ++i) rank += sh.member[start + i] < r ? 1 : 0;
      int32_t tile_total;
      const int32_t at = written + block_sum<S::WARPS>(g ? 1 : 0, sh.warp_sum, &tile_total);
      written += tile_total;
      if (g) {
        a.cand[b + start + rank] = make_int2(c.cs + r, sh.sptr[r + 1] - sh.sptr[r]);
        a.seg[b + at] = make_int2(b + start, len);
        a.seg_rank[b + at] = rank;
        atomicAdd(&sh.cols[r >> 1], 1u << (16 * (r & 1)));
      }
    }
    __syncthreads();
    int32_t before = 0;  // (rows come in order: where a row's groups start is the sum of the rows in front)
    for (int r0 = 0; r0 < rows; r0 += THREADS) {
      const int r = r0 + tid;
      const int32_t n = r < rows ? static_cast<int32_t>((sh.cols[r >> 1] >> (16 * (r & 1))) & 0xFFFFu) : 0;
      int32_t tile_total;
      const int32_t at = before + block_sum<S::WARPS>(n, sh.warp_sum, &tile_total);
      before += tile_total;
      if (r < rows) {
        a.row_seg[c.cs + r] = b + at;
        a.row_cols[c.cs + r] = n;
        a.row_work[c.cs + r] = sh.work[r];
      }
    }
  }
}

// ---- heavy chunks: tiled, whole-grid sort ----------------------------------------

// The chunk that runs ahead of the rest: the one with the most nonzeros, if it is a heavy
// chunk of at least min_nnz nonzeros (a row that streams 65,536 candidates or more needs a
// chunk about that big).  It becomes the only entry of `ap`'s list of heavy chunks.
__global__ void __launch_bounds__(1024) pick_priority_kernel(TransposeArgs a, TransposeArgs ap, int32_t min_nnz,
                                                             volatile uint32_t *outcome, uint32_t ticket) {
  __shared__ unsigned long long best[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long mine = 0;  // (nonzeros << 32) | ~chunk: the first of equally heavy chunks wins
  for (int32_t q = threadIdx.x; q < a.num_chunks; q += blockDim.x) {
    const ChunkSpan c = chunk_span(a, q);
    const unsigned long long v = (static_cast<unsigned long long>(c.L) << 32) | (0xFFFFFFFFu - static_cast<uint32_t>(q));
    mine = v > mine ? v : mine;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const unsigned long long t = __shfl_down_sync(FULL, mine, off);
    mine = t > mine ? t : mine;
  }
  if (lane == 0) best[warp] = mine;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 32; ++w) mine = best[w] > mine ? best[w] : mine;
    const int32_t L = static_cast<int32_t>(mine >> 32);
    const uint32_t q = 0xFFFFFFFFu - static_cast<uint32_t>(mine);
    const bool on = L > 8192 && L >= min_nnz;
    a.ctrl[CTRL_PRIO] = on ? q : PRIO_NONE;
    ap.ctrl[CTRL_PRIO] = on ? q : PRIO_NONE;
    ap.ctrl[CTRL_HEAVY_COUNT] = on ? 1u : 0u;
    ap.heavy_chunk[0] = on ? static_cast<int32_t>(q) : 0;
    outcome[1] = on ? 1u : 0u;
    __threadfence_system();
    outcome[0] = ticket;
  }
}

// what the lists tell the host (read_lists)
__device__ __forceinline__ void tell_lists(volatile uint32_t *outcome, uint32_t ticket, uint32_t chain_rows, uint32_t heavy_chunks,
                                           unsigned long long need) {
  outcome[1] = chain_rows;
  outcome[2] = heavy_chunks;
  outcome[3] = static_cast<uint32_t>(need);
  outcome[4] = static_cast<uint32_t>(need >> 32);
  __threadfence_system();
  outcome[0] = ticket;
}

// Work list of the chunk ahead: its rows within a factor of four of its longest stream (and of
// HEAVY_WORK candidates or more), longest first.  Those can decide when the call ends; the other
// rows of the chunk go with everybody else's.  One block; a chunk has at most PRIO_MAX_CHUNK rows.
constexpr int PRIO_MAX_CHUNK = 4096;
__global__ void __launch_bounds__(1024) priority_rows_kernel(TransposeArgs ap, int32_t *row_list, volatile uint32_t *outcome,
                                                             uint32_t ticket) {
  __shared__ int32_t s_row[PRIO_MAX_CHUNK];
  __shared__ uint32_t s_work[PRIO_MAX_CHUNK];
  __shared__ uint32_t count, longest;
  __shared__ unsigned long long need;
  if (threadIdx.x == 0) {
    count = 0;
    need = 0;
    longest = 0;
  }
  __syncthreads();
  const uint32_t prio = ap.ctrl[CTRL_PRIO];
  uint32_t least = 0;
  if (prio != PRIO_NONE && ap.chunk <= PRIO_MAX_CHUNK) {
    const int64_t start = static_cast<int64_t>(prio) * ap.chunk;
    const int64_t end = start + ap.chunk < ap.n ? start + ap.chunk : ap.n;
    uint32_t top = 0;
    for (int64_t r = start + threadIdx.x; r < end; r += blockDim.x) top = max(top, ap.row_work[r]);
    top = __reduce_max_sync(FULL, top);
    if ((threadIdx.x & 31) == 0 && top) atomicMax(&longest, top);
    __syncthreads();
    least = longest / 4 > HEAVY_WORK ? longest / 4 : HEAVY_WORK;
    for (int64_t r = start + threadIdx.x; r < end; r += blockDim.x) {
      const uint32_t t = ap.row_work[r];
      if (t >= least) {
        const uint32_t at = atomicAdd(&count, 1u);
        s_row[at] = static_cast<int32_t>(r);
        s_work[at] = t;
        atomicAdd(&need, static_cast<unsigned long long>(t));
      }
    }
    __syncthreads();
    const uint32_t H = count;
    // place of every row in the order (longer stream first, then smaller row id)
    for (uint32_t i = threadIdx.x; i < H; i += blockDim.x) {
      const uint32_t w = s_work[i];
      const int32_t r = s_row[i];
      uint32_t before = 0;
      for (uint32_t j = 0; j < H; ++j) {
        const uint32_t wj = s_work[j];
        before += (wj > w || (wj == w && s_row[j] < r)) ? 1u : 0u;
      }
      row_list[before] = r;
    }
  }
  if (threadIdx.x == 0) {
    ap.ctrl[CTRL_ROWS_LISTED] = count;
    ap.ctrl[CTRL_HEAVY_ROWS] = count;
    ap.ctrl[CTRL_MID_END] = count;
    ap.ctrl[CTRL_LANE_TICKET] = count;
    ap.ctrl[CTRL_PRIO_WORK] = least;
    ap.ctrl[CTRL_ROW_TICKET] = count;
    ap.ctrl[CTRL_HEAVY_TICKET] = 0;
    ap.ctrl[CTRL_HEAVY_TICKET + 1] = 0;
    tell_lists(outcome, ticket, count, 0, need);
  }
}

// exclusive scan of the heavy chunks' tile counts (one block)
__global__ void __launch_bounds__(1024) heavy_tiles_kernel(TransposeArgs a) {
  __shared__ int32_t sm[32];
  __shared__ int32_t carry_s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int32_t H = static_cast<int32_t>(a.ctrl[CTRL_HEAVY_COUNT]);
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  for (int32_t base = 0; base < H; base += 1024) {
    const int32_t i = base + threadIdx.x;
    int32_t v = 0;
    if (i < H) v = (chunk_span(a, a.heavy_chunk[i]).L + T_TILE - 1) / T_TILE;
    int32_t incl = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int32_t t = __shfl_up_sync(FULL, incl, off);
      if (lane >= off) incl += t;
    }
    if (lane == 31) sm[warp] = incl;
    __syncthreads();
    int32_t wbase = 0, tot = 0;
    for (int w = 0; w < 32; ++w) {
      const int32_t t = sm[w];
      if (w < warp) wbase += t;
      tot += t;
    }
    const int32_t carry = carry_s;
    if (i < H) a.heavy_tile_base[i] = carry + wbase + incl - v;
    __syncthreads();
    if (threadIdx.x == 0) carry_s = carry + tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    a.heavy_tile_base[H] = carry_s;
    a.ctrl[CTRL_HEAVY_TILES] = static_cast<uint32_t>(carry_s);
  }
}

struct TileRef {
  int32_t h, b, L, off, cnt, cs, rows;
};

// tile t -> its heavy chunk and range (uniform over the block)
__device__ __forceinline__ TileRef tile_ref(const TransposeArgs &a, int32_t t, int32_t H) {
  int32_t lo = 0, hi = H;  // heavy_tile_base[lo] <= t < heavy_tile_base[hi]
  while (hi - lo > 1) {
    const int32_t mid = (lo + hi) >> 1;
    if (a.heavy_tile_base[mid] <= t)
      lo = mid;
    else
      hi = mid;
  }
  const ChunkSpan c = chunk_span(a, a.heavy_chunk[lo]);
  TileRef r;
  r.h = lo;
  r.b = c.b;
  r.L = c.L;
  r.cs = c.cs;
  r.rows = c.rows;
  r.off = (t - a.heavy_tile_base[lo]) * T_TILE;
  r.cnt = c.L - r.off < T_TILE ? c.L - r.off : T_TILE;
  return r;
}

__device__ __forceinline__ const uint32_t *pass_src_keys(const TransposeArgs &a, int ps, int32_t b) {
  if (ps == 0) return reinterpret_cast<const uint32_t *>(a.ind + b);
  return ((ps - 1) & 1 ? a.keyB : a.keyA) + b;
}

__global__ void __launch_bounds__(T_THREADS) heavy_hist_kernel(TransposeArgs a, int ps) {
  __shared__ uint32_t hist[256];
  const int32_t TT = static_cast<int32_t>(a.ctrl[CTRL_HEAVY_TILES]);
  const int32_t H = static_cast<int32_t>(a.ctrl[CTRL_HEAVY_COUNT]);
  const int shift = 8 * ps;
  for (int32_t t = blockIdx.x; t < TT; t += gridDim.x) {
    const TileRef r = tile_ref(a, t, H);
    const uint32_t *kin = pass_src_keys(a, ps, r.b) + r.off;
    if (threadIdx.x < 256) hist[threadIdx.x] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < r.cnt; i += T_THREADS) atomicAdd(&hist[(kin[i] >> shift) & 255u], 1u);
    __syncthreads();
    if (threadIdx.x < 256) a.tile_hist[static_cast<size_t>(t) * 256 + threadIdx.x] = hist[threadIdx.x];
    __syncthreads();
  }
}

// per heavy chunk: counts -> offsets of every (tile, digit) inside the digit's run,
// and the start of every digit's run
__global__ void __launch_bounds__(256) heavy_scan_kernel(TransposeArgs a) {
  __shared__ uint32_t sm[8];
  const int32_t H = static_cast<int32_t>(a.ctrl[CTRL_HEAVY_COUNT]);
  const int d = threadIdx.x, lane = d & 31, warp = d >> 5;
  for (int32_t h = blockIdx.x; h < H; h += gridDim.x) {
    const int32_t t0 = a.heavy_tile_base[h], t1 = a.heavy_tile_base[h + 1];
    // a chunk of millions of nonzeros has hundreds of tiles: sixteen loads in flight per
    // thread, or the walk costs one memory latency per tile
    uint32_t run = 0;
    for (int32_t tb = t0; tb < t1; tb += 16) {
      uint32_t v[16];
#pragma unroll
      for (int u = 0; u < 16; ++u)
        v[u] = tb + u < t1 ? a.tile_hist[static_cast<size_t>(tb + u) * 256 + d] : 0u;
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        if (tb + u < t1) a.tile_hist[static_cast<size_t>(tb + u) * 256 + d] = run;
        run += v[u];
      }
    }
    uint32_t incl = run;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t t = __shfl_up_sync(FULL, incl, off);
      if (lane >= off) incl += t;
    }
    __syncthreads();
    if (lane == 31) sm[warp] = incl;
    __syncthreads();
    uint32_t wbase = 0;
    for (int w = 0; w < warp; ++w) wbase += sm[w];
    a.digit_base[static_cast<size_t>(h) * 256 + d] = wbase + incl - run;
  }
}

__global__ void __launch_bounds__(T_THREADS) heavy_scatter_kernel(TransposeArgs a, int ps) {
  __shared__ uint32_t wc[T_WARPS * 256];
  const int32_t TT = static_cast<int32_t>(a.ctrl[CTRL_HEAVY_TILES]);
  const int32_t H = static_cast<int32_t>(a.ctrl[CTRL_HEAVY_COUNT]);
  const int shift = 8 * ps;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int32_t t = blockIdx.x; t < TT; t += gridDim.x) {
    const TileRef r = tile_ref(a, t, H);
    const uint32_t *kin = pass_src_keys(a, ps, r.b) + r.off;
    const uint32_t *pin = ps == 0 ? nullptr : ((ps - 1) & 1 ? a.payB : a.payA) + r.b + r.off;
    uint32_t *kout = (ps & 1 ? a.keyB : a.keyA) + r.b;
    uint32_t *pout = (ps & 1 ? a.payB : a.payA) + r.b;
    for (int j = tid; j < T_WARPS * 256; j += T_THREADS) wc[j] = 0;
    __syncthreads();
    uint32_t key[T_IPT], rk[T_IPT], pay[T_IPT];
    const int wbase = warp * (32 * T_IPT);
#pragma unroll
    for (int i = 0; i < T_IPT; ++i) {
      const int idx = wbase + i * 32 + lane;
      const bool valid = idx < r.cnt;
      key[i] = valid ? kin[idx] : 0u;
      pay[i] = ps == 0 ? static_cast<uint32_t>(r.off + idx) : (valid ? pin[idx] : 0u);
      const uint32_t d = valid ? ((key[i] >> shift) & 255u) : 256u;
      const unsigned peers = match_digit(d);
      const int leader = __ffs(peers) - 1;
      uint32_t pre = 0;
      if (lane == leader && valid) {
        pre = wc[warp * 256 + d];
        wc[warp * 256 + d] = pre + __popc(peers);
      }
      pre = __shfl_sync(FULL, pre, leader);
      rk[i] = pre + __popc(peers & ((1u << lane) - 1u));
      __syncwarp();
    }
    __syncthreads();
    if (tid < 256) {
      uint32_t run = a.digit_base[static_cast<size_t>(r.h) * 256 + tid] +
                     a.tile_hist[static_cast<size_t>(t) * 256 + tid];
#pragma unroll
      for (int w = 0; w < T_WARPS; ++w) {
        const uint32_t v = wc[w * 256 + tid];
        wc[w * 256 + tid] = run;
        run += v;
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < T_IPT; ++i) {
      const int idx = wbase + i * 32 + lane;
      if (idx < r.cnt) {
        const uint32_t d = (key[i] >> shift) & 255u;
        const uint32_t dst = wc[warp * 256 + d] + rk[i];
        if (index_ok(a.ctrl, CHK_SORT, dst, r.L)) {
          kout[dst] = key[i];
          pout[dst] = pay[i];
        }
      }
    }
    __syncthreads();
  }
}

// Group of every sorted element by two bounded binary searches: a column group
// has at most one entry per row of the chunk, so its ends lie within `rows`
// positions of the element.  For chunks of up to E_ROWS rows the searches run on
// shared-memory copies - the tile's keys with a halo of rows-1 on either side and the
// chunk's row pointers - and the rows' work counters are summed in shared memory first:
// on global memory the kernel was bound by the latency of some thirty dependent loads per
// element and by atomics of a whole tile landing on the same few hub rows.
constexpr int E_ROWS = 1024;
__global__ void __launch_bounds__(T_THREADS) heavy_emit_kernel(TransposeArgs a) {
  __shared__ uint32_t skey[T_TILE + 2 * (E_ROWS - 1)];
  __shared__ int32_t sptr[E_ROWS + 1];
  __shared__ uint32_t swork[E_ROWS];
  const int32_t TT = static_cast<int32_t>(a.ctrl[CTRL_HEAVY_TILES]);
  const int32_t H = static_cast<int32_t>(a.ctrl[CTRL_HEAVY_COUNT]);
  const int f = (a.passes - 1) & 1;
  for (int32_t t = blockIdx.x; t < TT; t += gridDim.x) {
    const TileRef r = tile_ref(a, t, H);
    const uint32_t *K = (f ? a.keyB : a.keyA) + r.b;
    const uint32_t *P = (f ? a.payB : a.payA) + r.b;
    const bool staged = r.rows <= E_ROWS;
    int32_t w0 = 0;  // first sorted position held in skey
    if (!a.count) {  // every column of a row of such a chunk has an entry of seg[]
      // (each tile tells its share of the rows: by the first alone, a road network of 1.05 M rows as one
      // chunk waited 400 us for it)
      const int32_t tiles = (r.L + T_TILE - 1) / T_TILE, k = r.off / T_TILE;
      const int32_t j0 = static_cast<int32_t>(static_cast<int64_t>(r.rows) * k / tiles);
      const int32_t j1 = static_cast<int32_t>(static_cast<int64_t>(r.rows) * (k + 1) / tiles);
      for (int32_t j = j0 + threadIdx.x; j < j1; j += T_THREADS) {
        const int32_t x = a.ptr[r.cs + j], y = a.ptr[r.cs + j + 1];
        const bool ok = x >= r.b && x <= y && y <= r.b + r.L;
        if (!ok) atomicExch(&a.ctrl[CTRL_BAD_INPUT], 1u);
        a.row_seg[r.cs + j] = ok ? x : r.b;
        a.row_cols[r.cs + j] = ok ? y - x : 0;
      }
    }
    int32_t firsts = 0;
    if (staged) {
      w0 = r.off - (r.rows - 1) < 0 ? 0 : r.off - (r.rows - 1);
      const int32_t w1 = r.off + r.cnt + (r.rows - 1) < r.L ? r.off + r.cnt + (r.rows - 1) : r.L;
      for (int32_t j = threadIdx.x; j < w1 - w0; j += T_THREADS) skey[j] = K[w0 + j];
      for (int32_t j = threadIdx.x; j <= r.rows; j += T_THREADS) sptr[j] = a.ptr[r.cs + j];
      for (int32_t j = threadIdx.x; j < r.rows; j += T_THREADS) swork[j] = 0u;
      __syncthreads();
    }
    for (int li = threadIdx.x; li < r.cnt; li += T_THREADS) {
      const int32_t i = r.off + li;
      const uint32_t key = staged ? skey[i - w0] : K[i];
      int32_t lo = i - (r.rows - 1) < 0 ? 0 : i - (r.rows - 1), hi = i;  // first index with K >= key
      while (lo < hi) {
        const int32_t mid = (lo + hi) >> 1;
        if ((staged ? skey[mid - w0] : K[mid]) < key)
          lo = mid + 1;
        else
          hi = mid;
      }
      const int32_t st = lo;
      if (a.count) {
        firsts += i == st ? 1 : 0;
        continue;
      }
      lo = i + 1;
      hi = i + r.rows < r.L ? i + r.rows : r.L;  // first index with K > key
      while (lo < hi) {
        const int32_t mid = (lo + hi) >> 1;
        if ((staged ? skey[mid - w0] : K[mid]) <= key)
          lo = mid + 1;
        else
          hi = mid;
      }
      const int32_t len = lo - st;
      const int32_t p = static_cast<int32_t>(P[i]);
      if (!index_ok(a.ctrl, CHK_GROUP, p, r.L)) continue;
      int32_t row, rl;
      if (staged) {
        const int32_t lr = row_of(sptr, 0, r.rows, r.b + p);
        row = r.cs + lr;
        rl = sptr[lr + 1] - sptr[lr];
        if (len >= 2) saturating_add(&swork[lr], static_cast<uint32_t>(len - 1));
      } else {
        row = row_of(a.ptr, r.cs, r.cs + r.rows, r.b + p);
        rl = a.ptr[row + 1] - a.ptr[row];
        if (len >= 2) saturating_add(&a.row_work[row], static_cast<uint32_t>(len - 1));
      }
      a.cand[r.b + i] = make_int2(row, rl);
      a.seg[r.b + p] = make_int2(r.b + st, len);
      a.seg_rank[r.b + p] = i - st;
    }
    if (a.count) {
      firsts = __reduce_add_sync(FULL, firsts);
      if (lane_id() == 0 && firsts) atomicAdd(a.count, static_cast<unsigned long long>(firsts));
    }
    if (staged) {
      __syncthreads();
      for (int32_t j = threadIdx.x; j < r.rows; j += T_THREADS)
        if (swork[j]) saturating_add(&a.row_work[r.cs + j], swork[j]);
      __syncthreads();
    }
  }
}

// rows of the chunk that runs ahead which that part of the call takes itself
__device__ __forceinline__ bool taken_ahead(uint32_t prio, uint32_t least, int32_t chunk, int32_t r, uint32_t work) {
  return prio != PRIO_NONE && work >= least && static_cast<uint32_t>(r / chunk) == prio;
}

// rows and candidates per bucket of row_work
__global__ void __launch_bounds__(256) bucket_count_kernel(int32_t n, const uint32_t *row_work,
                                                           uint32_t *ctrl, int32_t chunk, const uint32_t *ctrl_ahead) {
  let_next_kernel_start();
  wait_for_kernels_before();
  __shared__ uint32_t bucket[WORK_BUCKETS];
  __shared__ unsigned long long work[WORK_BUCKETS];  // (of rows that may get a chain)
  if (threadIdx.x < WORK_BUCKETS) {
    bucket[threadIdx.x] = 0;
    work[threadIdx.x] = 0;
  }
  __syncthreads();
  const uint32_t prio = ctrl_ahead ? ctrl_ahead[CTRL_PRIO] : PRIO_NONE;
  const uint32_t least = ctrl_ahead ? ctrl_ahead[CTRL_PRIO_WORK] : 0u;
  for (int32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    uint32_t t = __ldcg(row_work + r);
    if (taken_ahead(prio, least, chunk, r, t)) t = 0;
    if (t) atomicAdd(&bucket[work_bucket(t)], 1u);
    if (t >= CHAIN_WORK_MIN) atomicAdd(&work[work_bucket(t)], static_cast<unsigned long long>(t));
  }
  __syncthreads();
  if (threadIdx.x < WORK_BUCKETS && bucket[threadIdx.x]) {
    atomicAdd(&ctrl[CTRL_BUCKET_COUNT + threadIdx.x], bucket[threadIdx.x]);
    if (work[threadIdx.x])
      atomicAdd(reinterpret_cast<unsigned long long *>(ctrl + CTRL_BUCKET_WORK) + threadIdx.x, work[threadIdx.x]);
  }
}

// What the two kernels take, in microseconds: `groups` chains at a time with `chain` per candidate each when all are
// busy, `alone` for the longest, `row` for every row; a lane `lane` per candidate of its row, all of them together
// `lanes`; `start` for the launches that a call without chains leaves out, `list` and `expand` for what they do per row and
// candidate.  chain = 0: no such times, FEW_CHAIN_ROWS rows.
// `forced` > 0: the caller's rule instead, every row in the buckets from that of so many candidates on.
struct ChainCosts {
  float groups, chain, alone, row, lane, lanes, start, list, expand;
  uint32_t rows_max, stream_cap, forced;
};

// Measured: csg and top-k graphs of R-MAT matrices and their symmetrised forms, rows listed down to 2^12 .. 2^17
// candidates, times of both kernels; chains as their own benchmark has them.  A call's time with the rule below
// and with chains for rows of 2^16 candidates or 296 rows, ms: R-MAT scale 22 21.4 and 23.5, top-k graph of scale 16
// 22.8 and 27.3, scale 19 in chunks of 2,048 10.7 and 12.9; symmetrised R-MAT of scale 20 27.9 and 28.0, of 262,144
// rows 12.2 and 16.2, of 65,536 rows 3.3 and 4.1.
// Key tables of tall chunks leave room for three groups of 32 slots (from 44,600 rows on) or two (from 63,900): a chain is
// the faster the fewer share its SM, but beside two the lanes get on, too.  Top-k graphs of 65,536 rows with k = 14, rule for four groups
// and for those there are, ms: R-MAT 16 edges a row 26.8 and 20.0, 6 edges 8.5 and 5.8, symmetrised 23.6 and 14.6, power-law
// band 1.27 both; of 50,000 rows the same.
ChainCosts chain_costs(const Context &ctx, int slots, int32_t span, uint32_t rows_max, uint32_t stream_cap) {
  const bool key_table = span <= LANE_TABLE_ROWS;
  ChainCosts c = {};
  c.rows_max = rows_max;
  c.stream_cap = stream_cap;
  if (ctx.chain_min_work) c.forced = ctx.chain_min_work > CHAIN_WORK_MIN ? ctx.chain_min_work : CHAIN_WORK_MIN;
  const int groups = chain_groups(ctx, slots, span);
  if (groups == 0) return c;
  c.groups = static_cast<float>(groups * ctx.num_sms);
  c.alone = slots == 32 ? 0.028f : slots == 64 ? 0.018f : 0.021f;
  c.chain = slots == 32 ? (groups > 2 ? 0.0125f * groups : 0.040f) : slots == 64 ? 0.030f : slots == 96 ? 0.035f : 0.052f;
  c.row = 3.0f;
  c.lane = key_table ? 0.24f : 0.40f;
  c.lanes = (key_table ? (slots <= 64 ? 5.5e-5f : 7.5e-5f) : 1.0e-4f) * 148.0f / static_cast<float>(ctx.num_sms);
  c.start = 30.0f;
  c.list = 0.015f;
  c.expand = 6.0e-6f;
  return c;
}

// Longest bucket first (one warp, lane l counts the buckets 127 - 4 l .. 124 - 4 l).
// Which rows get a group of warps of the chain kernel each: all rows of HEAVY_WORK candidates or more,
// and below that as many buckets as make the later of the two kernels end soonest (a tenth of the other's time, which
// runs beside it, added).  A chain takes 40 to 80 cycles per candidate and a good part of an SM, a lane among 32 some
// 500 and a sixth of the SM time: too few chains and the lanes wait for their longest row, too many and the chains
// queue.  Without times: the longest buckets that keep the list within FEW_CHAIN_ROWS rows.
// `octaves` > 0: the lanes find their keys by a chained hash table and take some 680 cycles per candidate.
// Of the rows that are left, those within so many octaves of the longest go to a warp each first (four octaves, three
// in very large chunks).  R-MAT scale 19 with chunks of 2,048, chains for 296 rows: 30.0 ms without, 16.9 with three, 13.4
// with four, 14.2 with five.
__global__ void bucket_scan_kernel(uint32_t *ctrl, volatile uint32_t *outcome, uint32_t ticket, int octaves,
                                   const uint32_t *ctrl_ahead, ChainCosts cost) {
  let_next_kernel_start();
  wait_for_kernels_before();
  const int lane = threadIdx.x;
  uint32_t c[4], sum = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    c[j] = ctrl[CTRL_BUCKET_COUNT + WORK_BUCKETS - 1 - (4 * lane + j)];
    sum += c[j];
  }
  uint32_t incl = sum;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t t = __shfl_up_sync(FULL, incl, off);
    if (lane >= off) incl += t;
  }
  uint32_t run = incl - sum;
  const uint32_t listed = __shfl_sync(FULL, incl, 31);
  int longest = 0;
#pragma unroll
  for (int j = 3; j >= 0; --j)
    if (c[j]) longest = WORK_BUCKETS - 1 - (4 * lane + j);
  longest = __reduce_max_sync(FULL, longest);
  const float top = bucket_floor(longest + 1);
  // (the chunk ahead lists its rows down to a quarter of its longest)
  if (ctrl_ahead && ctrl_ahead[CTRL_PRIO] != PRIO_NONE && ctrl_ahead[CTRL_PRIO_WORK] > 0)
    longest = max(longest, work_bucket(4u * ctrl_ahead[CTRL_PRIO_WORK]));
  const int least = max(work_bucket(WARP_WORK_MIN), longest - 4 * octaves);
  uint32_t heavy = 0, mid = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int b = WORK_BUCKETS - 1 - (4 * lane + j);
    ctrl[CTRL_BUCKET_BASE + b] = run;
    run += c[j];
    ctrl[CTRL_BUCKET_FILL + b] = 0;
    const bool few = cost.chain == 0.0f && b >= work_bucket(CHAIN_WORK_MIN) && run <= FEW_CHAIN_ROWS;
    if (cost.forced ? b >= work_bucket(cost.forced) : b >= work_bucket(HEAVY_WORK) || few) heavy = run;
    if (octaves > 0 && b >= least) mid = run;
  }
  heavy = __reduce_max_sync(FULL, heavy);
  // (where the lanes end their longest row before a chain kernel would have begun, there is nothing to weigh)
  const bool weigh = cost.forced == 0 && cost.chain > 0.0f && top * cost.lane > cost.start;
  unsigned long long need = 0;
  if (weigh || heavy > 0) {
    const unsigned long long *const bucket_work = reinterpret_cast<const unsigned long long *>(ctrl + CTRL_BUCKET_WORK);
    unsigned long long work[4], work_sum = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      work[j] = bucket_work[WORK_BUCKETS - 1 - (4 * lane + j)];
      work_sum += work[j];
    }
    unsigned long long work_run = work_sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned long long u = __shfl_up_sync(FULL, work_run, off);
      if (lane >= off) work_run += u;
    }
    const float all = static_cast<float>(__shfl_sync(FULL, work_run, 31));
    work_run -= work_sum;
    run = incl - sum;
    // time with the chains down to this bucket, and the least of them
    float best = 3.0e38f;
    uint32_t rows = 0;
    uint32_t upto[4];
    unsigned long long work_upto[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int b = WORK_BUCKETS - 1 - (4 * lane + j);
      run += c[j];
      work_run += work[j];
      upto[j] = run;
      work_upto[j] = work_run;
      if (!weigh || c[j] == 0 || b < work_bucket(CHAIN_WORK_MIN) || run > cost.rows_max || work_run > cost.stream_cap) continue;
      // (the times hold up to CHAIN_ROWS rows: more of them slow a top-k graph of 20,000 rows from 5.65 to 6.01 ms)
      if (run > CHAIN_ROWS + work_run / HEAVY_WORK) continue;
      const float s = static_cast<float>(work_run), r = static_cast<float>(run);
      const float chains = fmaxf(top * cost.alone, (s * cost.chain + r * cost.row) / cost.groups);
      const float lanes = run < listed ? fmaxf(bucket_floor(b) * cost.lane, (all - s) * cost.lanes) : 0.0f;
      const float time = fmaxf(chains, lanes) + 0.1f * fminf(chains, lanes) + r * cost.list + s * cost.expand;
      if (time < best) {
        best = time;
        rows = run;
      }
    }
    if (weigh) {
      const uint32_t time = __reduce_min_sync(FULL, __float_as_uint(best));
      heavy = max(heavy, __reduce_max_sync(FULL, __float_as_uint(best) == time ? rows : 0u));
    }
    // what their streams take, which the host makes room for (as far as it may: heavy_offsets_kernel)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (c[j] && upto[j] <= heavy) need = work_upto[j];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) need = max(need, __shfl_xor_sync(FULL, need, off));
  }
  mid = __reduce_max_sync(FULL, mid);
  if (mid < heavy) mid = heavy;
  if (lane == 0) {
    ctrl[CTRL_ROWS_LISTED] = listed;
    ctrl[CTRL_HEAVY_ROWS] = heavy;
    ctrl[CTRL_MID_END] = mid;
    ctrl[CTRL_LANE_TICKET] = mid;
    ctrl[CTRL_HEAVY_TICKET] = 0;
    ctrl[CTRL_ROW_TICKET] = heavy;
    tell_lists(outcome, ticket, heavy, ctrl[CTRL_HEAVY_COUNT], need);
  }
}

// The list itself.  A block draws the places of a step's rows bucket by bucket: with an atomic per warp and bucket
// on the few counters that all rows share, the kernel took 15.3 us at 1,048,576 rows of a mesh, now 9.5.
constexpr int LIST_ROWS = 4;  // rows per thread and step
__global__ void __launch_bounds__(256) row_list_kernel(int32_t n, const uint32_t *row_work, uint32_t *ctrl,
                                                       int32_t *row_list, int32_t chunk,
                                                       const uint32_t *ctrl_ahead) {
  let_next_kernel_start();
  wait_for_kernels_before();
  __shared__ uint32_t bucket[WORK_BUCKETS];  // rows of the step, then the place of its first
  const int lane = threadIdx.x & 31;
  const int32_t step = blockDim.x * LIST_ROWS;
  const uint32_t prio = ctrl_ahead ? ctrl_ahead[CTRL_PRIO] : PRIO_NONE;
  const uint32_t least = ctrl_ahead ? ctrl_ahead[CTRL_PRIO_WORK] : 0u;
  for (int64_t base = static_cast<int64_t>(blockIdx.x) * step; base < n; base += static_cast<int64_t>(gridDim.x) * step) {
    if (threadIdx.x < WORK_BUCKETS) bucket[threadIdx.x] = 0;
    __syncthreads();
    int bkt[LIST_ROWS];
    uint32_t at[LIST_ROWS];
#pragma unroll
    for (int i = 0; i < LIST_ROWS; ++i) {
      const int64_t r = base + i * blockDim.x + threadIdx.x;
      uint32_t t = r < n ? __ldcg(row_work + r) : 0u;
      if (r < n && taken_ahead(prio, least, chunk, static_cast<int32_t>(r), t)) t = 0;
      bkt[i] = t ? work_bucket(t) : -1;
    }
#pragma unroll
    for (int i = 0; i < LIST_ROWS; ++i) {
      const unsigned peers = match_digit(bkt[i] >= 0 ? static_cast<uint32_t>(bkt[i]) : 256u);
      if (bkt[i] >= 0) {
        const int leader = __ffs(peers) - 1;
        uint32_t pre = 0;
        if (lane == leader) pre = atomicAdd(&bucket[bkt[i]], __popc(peers));
        at[i] = __shfl_sync(peers, pre, leader) + __popc(peers & ((1u << lane) - 1u));
      }
    }
    __syncthreads();
    if (threadIdx.x < WORK_BUCKETS && bucket[threadIdx.x])
      bucket[threadIdx.x] = ctrl[CTRL_BUCKET_BASE + threadIdx.x] + atomicAdd(&ctrl[CTRL_BUCKET_FILL + threadIdx.x], bucket[threadIdx.x]);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < LIST_ROWS; ++i)
      if (bkt[i] >= 0) row_list[bucket[bkt[i]] + at[i]] = static_cast<int32_t>(base + i * blockDim.x + threadIdx.x);
    __syncthreads();
  }
}

}  // namespace

namespace {
TransposeArgs transpose_args(int32_t n, int32_t ncols, int32_t nnz, int32_t chunk, const int32_t *d_ptr,
                             const int32_t *d_ind, const CsgScratch &s) {
  TransposeArgs a;
  a.n = n;
  a.nnz = nnz;
  a.chunk = chunk;
  a.num_chunks = static_cast<int32_t>((static_cast<int64_t>(n) + chunk - 1) / chunk);
  int bits = 1;
  while (bits < 32 && (static_cast<int64_t>(1) << bits) < ncols) ++bits;  // column ids < ncols
  a.passes = (bits + 7) / 8;
  a.ptr = d_ptr;
  a.ind = d_ind;
  a.keyA = s.keyA;
  a.keyB = s.keyB;
  a.payA = s.payA;
  a.payB = s.payB;
  a.cand = s.cand;
  a.seg = s.seg;
  a.seg_rank = s.seg_rank;
  a.row_seg = s.row_seg;
  a.row_cols = s.row_cols;
  a.row_work = s.row_work;
  a.ctrl = s.ctrl;
  a.count = nullptr;
  a.next_chunk = s.next_chunk;
  a.heavy_chunk = s.heavy_chunk;
  a.heavy_tile_base = s.heavy_tile_base;
  a.tile_hist = s.tile_hist;
  a.digit_base = s.digit_base;
  a.ctrl_main = nullptr;
  a.skip_prio = false;
  return a;
}
}  // namespace

bool launch_priority_pick(Context &ctx, int32_t n, int32_t nnz, int32_t chunk, const int32_t *d_ptr,
                          CsgScratch &s, CsgScratch &prio, int32_t min_chunk_nnz, bool *on) {
  const TransposeArgs a = transpose_args(n, n, nnz, chunk, d_ptr, nullptr, s);
  const TransposeArgs ap = transpose_args(n, n, nnz, chunk, d_ptr, nullptr, prio);
  cudaStream_t st = ctx.stream;
  CSG_CUDA(cudaMemsetAsync(s.ctrl, 0, sizeof(uint32_t) * CTRL_WORDS, st));
  CSG_CUDA(cudaMemsetAsync(prio.ctrl, 0, sizeof(uint32_t) * CTRL_WORDS, st));
  prio.ticket = ++ctx.outcome_ticket;
  pick_priority_kernel<<<1, 1024, 0, st>>>(a, ap, min_chunk_nnz, outcome_words(ctx, OUTCOME_WORD_PRIO), prio.ticket);
  CSG_CUDA(cudaGetLastError());
  count_launches(1);
  if (!wait_outcome(ctx, st, OUTCOME_WORD_PRIO, prio.ticket)) return false;
  *on = outcome_words(ctx, OUTCOME_WORD_PRIO)[1] != 0;
  if (*on) CSG_CUDA(cudaMemsetAsync(s.row_work, 0, sizeof(uint32_t) * static_cast<size_t>(n), st));
  return true;
}

namespace {
bool launch_heavy(Context &ctx, const TransposeArgs &a, bool one_chunk, cudaStream_t st) {
  heavy_tiles_kernel<<<1, 1024, 0, st>>>(a);
  CSG_CUDA(cudaGetLastError());
  const int hgrid = ctx.num_sms * 2;
  const int sgrid = one_chunk ? 1 : a.num_chunks < ctx.num_sms ? a.num_chunks : ctx.num_sms;
  for (int ps = 0; ps < a.passes; ++ps) {
    heavy_hist_kernel<<<hgrid, T_THREADS, 0, st>>>(a, ps);
    CSG_CUDA(cudaGetLastError());
    heavy_scan_kernel<<<sgrid, 256, 0, st>>>(a);
    CSG_CUDA(cudaGetLastError());
    heavy_scatter_kernel<<<hgrid, T_THREADS, 0, st>>>(a, ps);
    CSG_CUDA(cudaGetLastError());
  }
  heavy_emit_kernel<<<hgrid * 2, T_THREADS, 0, st>>>(a);
  CSG_CUDA(cudaGetLastError());
  count_launches(2 + 3 * a.passes);
  return true;
}

bool launch_compact(Context &ctx, const TransposeArgs &a, cudaStream_t st) {
  auto launch = [&](auto kernel, int threads, size_t smem, int per_sm) -> bool {
    CSG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    const int grid = a.num_chunks < ctx.num_sms * per_sm ? a.num_chunks : ctx.num_sms * per_sm;
    CSG_CUDA(launch_behind(!a.skip_prio, kernel, grid, threads, static_cast<int>(smem), st, a));
    return true;
  };
  const int32_t rows = a.chunk < a.n ? a.chunk : a.n;
  // Taller chunks, if there are enough of them for a block each to keep the chip busy: 64 chunks of 4,096
  // rows of a road network 355 -> 159 us, 88 of 3,000 rows of a mesh 567 -> 276.  One chunk of 3,500 rows
  // by itself took 763 us with it and 713 without; 4,096 rows of a mesh (36,800 nonzeros) are looked at only
  // to find that they do not fit, 723 and 595: C_TALL_NNZ.
  if (rows > C_ROWS && rows <= C_TALL_ROWS && a.num_chunks >= ctx.num_sms / 4) {
    if (!launch(compact_kernel<CompactTall, false, true>, CompactTall::THREADS, sizeof(CompactTall::Shared), 1)) return false;
    count_launches(1);
    return true;
  }
  // No more chunks than SMs: the large form at once, one trip over each chunk instead of two for those the small one
  // cannot hold (power-law band of 65,536 rows, 64 chunks: 123 us by both forms, 46 so; 4,096 rows 88 and 77).
  if (a.num_chunks <= ctx.num_sms && rows <= C_ROWS) {
    if (!launch(compact_kernel<CompactLarge, false, true>, CompactLarge::THREADS, sizeof(CompactLarge::Shared), 1)) return false;
    count_launches(1);
    return true;
  }
  if (!launch(compact_kernel<CompactSmall, false, false>, CompactSmall::THREADS, sizeof(CompactSmall::Shared), 2)) return false;
  if (!launch(compact_kernel<CompactLarge, true, true>, CompactLarge::THREADS, sizeof(CompactLarge::Shared), 1)) return false;
  count_launches(2);
  return true;
}

}  // namespace

// the rows with candidates, longest stream first
bool launch_lists(Context &ctx, int32_t n, int32_t chunk, CsgScratch &s, const uint32_t *ctrl_ahead) {
  int grid = (n + 255) / 256;
  if (grid > ctx.num_sms * 8) grid = ctx.num_sms * 8;
  CSG_CUDA(launch_behind(s.one_stream, bucket_count_kernel, grid, 256, 0, ctx.stream, n, s.row_work, s.ctrl, chunk, ctrl_ahead));
  const int32_t span = chunk < n ? chunk : n;
  const int octaves = span <= LANE_TABLE_ROWS ? 0 : span <= WARP_FEW_ROWS ? 4 : 3;
  s.ticket = ++ctx.outcome_ticket;
  CSG_CUDA(launch_behind(s.one_stream, bucket_scan_kernel, 1, 32, 0, ctx.stream, s.ctrl,
                         outcome_words(ctx, OUTCOME_WORD), s.ticket, octaves, ctrl_ahead,
                         chain_costs(ctx, s.slots, span, s.heavy_max, s.stream_cap)));
  int steps = static_cast<int>((static_cast<int64_t>(n) + 256 * LIST_ROWS - 1) / (256 * LIST_ROWS));
  if (steps > ctx.num_sms * 32) steps = ctx.num_sms * 32;
  CSG_CUDA(launch_behind(s.one_stream, row_list_kernel, steps, 256, 0, ctx.stream, n, s.row_work, s.ctrl, s.row_list, chunk,
                         ctrl_ahead));
  count_launches(3);
  return true;
}

// phase PHASE_ALL: the whole transposition on the context's stream.  PHASE_PRIO (on the side
// stream, `s` = the scratch of the part that runs ahead): the one chunk launch_priority_pick
// named, then that chunk's list of heavy rows; ctx.ev[6] marks the end of its transposition.
// PHASE_REST (context's stream): every other chunk; what follows in the stream is behind ev[6], because the lists
// (launch_lists, once the chunk ahead has told what its streams take) read the work counters of all rows.
// A PHASE_ALL call looks at the outcome of compact_kernel on the host: without chunks for the
// tiled sort (none on meshes, roads and most small matrices) its dozen launches are left out.
// d_count: only the number of (chunk, column) pairs is wanted, and added there.
bool launch_transpose(Context &ctx, int32_t n, int32_t ncols, int32_t nnz, int32_t chunk, const int32_t *d_ptr,
                      const int32_t *d_ind, CsgScratch &s, int phase, uint32_t *ctrl_other,
                      unsigned long long *d_count) {
  // ctrl_other: the control words of the other part of a call that runs one chunk ahead
  TransposeArgs a = transpose_args(n, ncols, nnz, chunk, d_ptr, d_ind, s);
  a.ctrl_main = phase == PHASE_PRIO && ctrl_other ? ctrl_other : s.ctrl;
  a.skip_prio = phase == PHASE_REST;
  a.count = d_count;
  if (phase == PHASE_PRIO) {
    cudaStream_t st = ctx.side_stream;
    if (!launch_heavy(ctx, a, true, st)) return false;
    s.ticket = ++ctx.outcome_ticket;
    priority_rows_kernel<<<1, 1024, 0, st>>>(a, s.row_list, outcome_words(ctx, OUTCOME_WORD_PRIO), s.ticket);
    CSG_CUDA(cudaGetLastError());
    count_launches(1);
    CSG_CUDA(cudaEventRecord(ctx.ev[6], st));  // the rest may read this chunk's work counters and its longest stream
    return true;
  }
  cudaStream_t st = ctx.stream;
  if (phase == PHASE_REST) {
    if (!launch_compact(ctx, a, st) || !launch_heavy(ctx, a, false, st)) return false;
    CSG_CUDA(cudaStreamWaitEvent(st, ctx.ev[6], 0));
    return true;
  }
  CSG_CUDA(cudaMemsetAsync(s.ctrl, 0, sizeof(uint32_t) * CTRL_WORDS, st));
  if (!launch_compact(ctx, a, st)) return false;
  if (d_count) return launch_heavy(ctx, a, false, st);
  if (!launch_lists(ctx, n, chunk, s, nullptr)) return false;
  // (the row list is still being written then, and the launches behind it are queued in time)
  if (!read_lists(ctx, s, PHASE_ALL)) return false;
  if (outcome_words(ctx, OUTCOME_WORD)[2] != 0) {
    if (!launch_heavy(ctx, a, false, st)) return false;
    CSG_CUDA(cudaMemsetAsync(s.ctrl + CTRL_BUCKET_COUNT, 0, 3 * sizeof(uint32_t) * WORK_BUCKETS, st));
    return launch_lists(ctx, n, chunk, s, nullptr) && read_lists(ctx, s, PHASE_ALL);
  }
  return true;
}

}  // namespace csg
