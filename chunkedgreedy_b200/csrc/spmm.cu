// fp32 CSR SpMM, C[n x w] = A[n x n] * B[n x w], B and C row-major.
//
// The reference has no first-party SpMM: it times third-party tensor-core kernels
// through bench/spmm/spmm_bench/base.py:48-59 and cuSPARSE through
// sporder/src/bench_cusparse_spmm.cu:64-90.  This kernel is the fp32 CUDA-core
// SpMM the reordered matrix is fed to: the work is the gather of one B row per
// nonzero (4*w bytes), so the kernel is a bandwidth kernel and its job is to keep
// many row gathers in flight.
//
// Row tiling: a group of G lanes owns one row and walks its nonzeros up to eight at a
// time; every lane of the group loads its VEC columns of B[col] (one coalesced segment per
// group), for PAN panels of G*VEC columns at once, and accumulates in registers.  A warp
// therefore handles 32/G rows at once.  Rows are handed out in two levels.  The rows are cut
// into units of equal cost, where a row costs ROW_COST plus its nonzeros: unit u holds the
// rows r with ROW_COST * r + ptr[r] in [u * T, (u + 1) * T), found by searching the row
// pointers, so a stretch of hub rows and a stretch of empty rows make equally many units.  A
// warp draws a unit from one global counter (one atomic per unit), stages the unit's row
// pointers in shared memory with one coalesced read, and its groups take the rows of the
// unit one by one as they finish, so uneven row lengths idle no lanes and no counter is
// hammered once per row.  (Batches of a fixed number of rows left the SMs idle 60 % of the
// kernel on a power-law matrix: one warp drew 128 hub rows.)  Rows longer than a limit are cut
// into pieces that all groups share and that are added with atomics (C is zeroed first for
// those rows), so a hub row never serialises on one warp.  The matrix is read once and marked as streaming data (evict
// first), so that it does not push rows of B out of the L2 cache.
#include <mutex>

#include "../../include/sporder_b200.h"
#include "common.cuh"
#include "spmm_plan.h"

namespace csg {

namespace {

// Columns of the lane's panel pn that exist: with MASK the last panel of a width that is not a
// multiple of G * VEC is ragged, and the lanes behind the last column load and store nothing.
template <int G, int VEC, bool MASK>
__device__ __forceinline__ bool panel_on(int32_t col0, int pn, int32_t w) {
  return !MASK || col0 + pn * (G * VEC) < w;
}

template <int VEC>
__device__ __forceinline__ void load_b(const float *p, float (&out)[VEC]) {
  if (VEC == 4) {
    const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
    out[0] = t.x;
    out[1] = t.y;
    out[2] = t.z;
    out[3] = t.w;
  } else if (VEC == 2) {
    const float2 t = __ldg(reinterpret_cast<const float2 *>(p));
    out[0] = t.x;
    out[1] = t.y;
  } else {
    out[0] = __ldg(p);
  }
}

// base + c * wbytes as one 32 x 32 -> 64 bit multiply-add (written as a 64-bit product of
// converted operands the compiler builds it from four multiplies and two shifts, which on
// short rows was a third of all instructions executed)
__device__ __forceinline__ const float *b_row(const char *base, int32_t c, int32_t wbytes) {
  long long out;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(out) : "r"(c), "r"(wbytes), "l"(reinterpret_cast<long long>(base)));
  return reinterpret_cast<const float *>(out);
}

struct SpmmArgs {
  int32_t n, w, nnz, unit;  // unit: cost per unit of rows (T)
  int32_t split, piece;     // longest row one group walks alone, nonzeros per piece of a longer one
  int32_t queue_cap;        // entries long_rows has room for
  const int32_t *ptr, *ind;
  const float *val;
  const float *B;
  float *C;
  // scratch: [0] row ticket, [2..3] packed (long rows, pieces) counter, then the queue
  uint32_t *ctrl;
  int2 *long_rows;  // (row, first piece number), in piece order
};

// First row r in [0, n] with ROW_COST * r + ptr[r] >= target, n + 1 when there is none.  Two
// searches at once: lanes 0-15 look for target_lo, lanes 16-31 for target_hi, sixteen probes
// per step, so a search costs log16(n) dependent loads instead of log2(n).
__device__ __forceinline__ void unit_bounds(const SpmmArgs &a, long long target_lo, long long target_hi,
                                            int32_t *first, int32_t *last) {
  const int lane = threadIdx.x & 31, i = lane & 15;
  const long long target = lane < 16 ? target_lo : target_hi;
  long long lo = 0, hi = static_cast<long long>(a.n) + 1;  // the answer lies in [lo, hi]
  while (__any_sync(FULL, lo < hi)) {
    const long long len = hi - lo;
    const long long step = (len + 15) / 16;
    long long idx = lo + (i + 1) * step - 1;
    if (idx > hi - 1) idx = hi - 1;
    bool pred = false;
    if (lo < hi) pred = ROW_COST * idx + __ldg(a.ptr + idx) >= target;
    const unsigned votes = (__ballot_sync(FULL, pred) >> (lane & 16)) & 0xFFFFu;
    if (lo < hi) {
      if (votes) {
        const int f = __ffs(votes) - 1;
        long long top = lo + (f + 1) * step - 1;
        if (top > hi - 1) top = hi - 1;
        lo = lo + f * step;
        hi = top;
      } else {
        lo = hi;
      }
    }
  }
  *first = static_cast<int32_t>(__shfl_sync(FULL, lo, 0));
  *last = static_cast<int32_t>(__shfl_sync(FULL, lo, 16));
}

constexpr int CTRL_TICKET = 0;
constexpr int CTRL_PACKED = 2;  // 64-bit: high word = long rows queued, low word = pieces so far
constexpr int CTRL_SCRATCH_WORDS = 64;

// gathers in flight per group and step: eight rows of B, four where a lane already
// fetches two panels of each
template <int PAN>
struct Step {
  static constexpr int U = PAN >= 2 ? 4 : 8;
};

// FMA of up to U nonzeros [p, p + cnt) of one row into acc, for the panels
// pn0 .. pn0 + PAN - 1, all loads of a kind issued together.
template <int G, int VEC, int PAN, bool MASK, int U = Step<PAN>::U>
__device__ __forceinline__ void fma_step(const SpmmArgs &a, int32_t p, int cnt, int32_t col0,
                                         float (&acc)[PAN][VEC]) {
  int32_t c[U];
  float x[U];
  float b[U][PAN][VEC];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const bool on = u < cnt;
    c[u] = on ? __ldcs(a.ind + p + u) : 0;
    x[u] = on ? __ldcs(a.val + p + u) : 0.0f;
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (u < cnt) {
      const float *src = b_row(reinterpret_cast<const char *>(a.B + col0), c[u], a.w * 4);
#pragma unroll
      for (int pn = 0; pn < PAN; ++pn) {
#pragma unroll
        for (int v = 0; MASK && v < VEC; ++v) b[u][pn][v] = 0.0f;
        if (panel_on<G, VEC, MASK>(col0, pn, a.w)) load_b<VEC>(src + pn * G * VEC, b[u][pn]);
      }
    } else {
#pragma unroll
      for (int pn = 0; pn < PAN; ++pn)
#pragma unroll
        for (int v = 0; v < VEC; ++v) b[u][pn][v] = 0.0f;
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int pn = 0; pn < PAN; ++pn)
#pragma unroll
      for (int v = 0; v < VEC; ++v) acc[pn][v] = fmaf(x[u], b[u][pn][v], acc[pn][v]);
}

template <int VEC>
__device__ __forceinline__ void store_c(float *out, const float (&acc)[VEC], bool accumulate) {
  if (accumulate) {
#pragma unroll
    for (int v = 0; v < VEC; ++v) atomicAdd(out + v, acc[v]);
  } else if (VEC == 4) {
    __stcs(reinterpret_cast<float4 *>(out), make_float4(acc[0], acc[1], acc[2], acc[3]));
  } else if (VEC == 2) {
    __stcs(reinterpret_cast<float2 *>(out), make_float2(acc[0], acc[1]));
  } else {
    __stcs(out, acc[0]);
  }
}

// ---- units of short rows ---------------------------------------------------------------
// A unit whose rows all have at most SHORT_MAX nonzeros (every unit of a mesh or a road
// network) needs none of the machinery of spmm_rows_kernel's walk: the warp copies the
// (column, value) pairs of as many rows as fit S_PAIRS into shared memory with coalesced
// loads, its lane groups take those rows in turn, and a row is worked off in pieces of exactly
// as many nonzeros as it has left - no predicates, no padding, one shared-memory read per
// nonzero.  On the 9-point stencil the general walk executes some 470 instructions per four
// rows (opcode counts of a profiler run: a third of them integer multiply-adds for
// addresses, predicates and moves), and the kernel there is bound by instruction issue.
constexpr int SHORT_MAX = 16;

// The warp draws its next unit: rows [*first, *first + *count), their pointers in wp.  False: no
// units are left.  (A unit may hold no row.)
template <int BATCH>
__device__ __forceinline__ bool draw_unit(const SpmmArgs &a, int32_t *wp, int lane, int32_t *first, int32_t *count) {
  uint32_t t = 0;
  if (lane == 0) t = atomicAdd(&a.ctrl[CTRL_TICKET], 1u);
  t = __shfl_sync(FULL, t, 0);
  *count = 0;
  const long long total = static_cast<long long>(ROW_COST) * a.n + a.nnz;
  if (static_cast<long long>(t) * a.unit > total) return false;
  int32_t last;
  unit_bounds(a, static_cast<long long>(t) * a.unit, (static_cast<long long>(t) + 1) * a.unit, first, &last);
  if (last > a.n) last = a.n;
  if (*first < last) {
    *count = last - *first;  // at most unit / ROW_COST <= BATCH rows
    if (*count > BATCH) *count = BATCH;  // (only with row pointers that decrease)
    __syncwarp();
    for (int k = lane; k <= *count; k += 32) wp[k] = __ldg(a.ptr + *first + k);
    __syncwarp();
  }
  return true;
}

// Longest row of the staged unit, SHORT_MAX + 1 when one is malformed (the general path deals with it)
__device__ __forceinline__ int32_t unit_longest(const int32_t *wp, int32_t bcount, int32_t nnz, int lane) {
  int32_t worst = 0;
  for (int k = lane; k < bcount; k += 32) {
    const int32_t b = wp[k], e = wp[k + 1];
    const int32_t len = b < 0 || e < b || e > nnz ? SHORT_MAX + 1 : e - b;
    worst = len > worst ? len : worst;
  }
  return __reduce_max_sync(FULL, worst);
}

// The rows of a short unit are of much the same length (on average 7/8 of the longest: the lane groups of
// a warp then run the same cases), and not of few nonzeros.  A unit of short rows has many of them, and
// by lane groups a row makes more trips than by the warp, which with two panels loses from six nonzeros
// down (5-point mesh of 50,000 rows at width 192: 32 us by the warp, 36 by groups of 16), with one from four.
template <int PAN>
__device__ __forceinline__ bool unit_is_even(const int32_t *wp, int32_t bcount, int32_t longest) {
  const int32_t nonzeros = wp[bcount] - wp[0];
  return 7 * longest * bcount <= 8 * nonzeros && (PAN == 1 ? 4 : 6) * bcount <= nonzeros;
}

// Rows of up to 32 nonzeros, on average a third of the longest or more: at 32 columns, where a lane of the whole
// warp loads a single float, lane groups are still the faster way (24 nonzeros in each of 1.05 M rows: 786 us by
// the warp, 395 by groups; 1 to 31: 607 and 431).  Power-law graphs have few such units (R-MAT scale 20 425 and 421).
constexpr int MILD_MAX = 32;
__device__ __forceinline__ bool unit_is_mild(const int32_t *wp, int32_t bcount, int32_t longest) {
  return longest <= MILD_MAX && longest * bcount <= 3 * (wp[bcount] - wp[0]);
}

// N nonzeros of a row, pairs at sp[0 .. N): gather and FMA
template <int G, int VEC, int PAN, bool MASK, int N>
__device__ __forceinline__ void short_slots(const int2 *sp, const char *bcol, int32_t wbytes, int32_t col0,
                                            float (&acc)[PAN][VEC]) {
  int2 pr[N];
  float b[N][PAN][VEC];
#pragma unroll
  for (int j = 0; j < N; ++j) pr[j] = sp[j];
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const float *src = b_row(bcol, pr[j].x, wbytes);
#pragma unroll
    for (int pn = 0; pn < PAN; ++pn) {
#pragma unroll
      for (int v = 0; MASK && v < VEC; ++v) b[j][pn][v] = 0.0f;
      if (panel_on<G, VEC, MASK>(col0, pn, wbytes / 4)) load_b<VEC>(src + pn * G * VEC, b[j][pn]);
    }
  }
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const float x = __int_as_float(pr[j].y);
#pragma unroll
    for (int pn = 0; pn < PAN; ++pn)
#pragma unroll
      for (int v = 0; v < VEC; ++v) acc[pn][v] = fmaf(x, b[j][pn][v], acc[pn][v]);
  }
}

// The nonzeros sp[0 .. cnt) of one row into acc: pieces of UC while more than CAP are left, then
// all the rest in one piece.
template <int G, int VEC, int PAN, bool MASK, int UC = Step<PAN>::U>
__device__ __forceinline__ void staged_row(const int2 *sp, int32_t cnt, const char *bcol, int32_t wbytes, int32_t col0,
                                           float (&acc)[PAN][VEC]) {
  constexpr int CAP = UC + 1;
  int32_t q = 0;
  for (; cnt - q > CAP; q += UC) short_slots<G, VEC, PAN, MASK, UC>(sp + q, bcol, wbytes, col0, acc);
  switch (cnt - q) {
#define CSG_REST(N)                                              \
  case N:                                                        \
    if constexpr (N <= CAP) short_slots<G, VEC, PAN, MASK, N>(sp + q, bcol, wbytes, col0, acc); \
    break;
    CSG_REST(1) CSG_REST(2) CSG_REST(3) CSG_REST(4) CSG_REST(5) CSG_REST(6) CSG_REST(7) CSG_REST(8) CSG_REST(9)
#undef CSG_REST
    default:
      break;
  }
}

// all rows [bfirst, bfirst + bcount) of a short unit; wp holds their row pointers, sp is the
// warp's buffer of S_PAIRS pairs
template <int G, int VEC, int PAN, bool MASK, int S_PAIRS, int UC = Step<PAN>::U>
__device__ __forceinline__ void short_rows(const SpmmArgs &a, const int32_t *wp, int2 *sp, int32_t bfirst,
                                           int32_t bcount, int lane) {
  constexpr int PER_WARP = 32 / G;
  const int sub = lane / G, gl = lane % G;
  const int panels = (a.w + G * VEC - 1) / (G * VEC);
  const int32_t wbytes = a.w * 4;
  int32_t r0 = 0;
  while (r0 < bcount) {
    // rows [r0, r1): as many as the pair buffer holds (at least S_PAIRS / SHORT_MAX of them)
    const int32_t p0 = wp[r0];
    int32_t lo = r0 + 1, hi = bcount;
    while (lo < hi) {
      const int32_t mid = (lo + hi + 1) >> 1;
      if (wp[mid] - p0 <= S_PAIRS)
        lo = mid;
      else
        hi = mid - 1;
    }
    const int32_t r1 = lo, cnt = wp[r1] - p0;
    __syncwarp();  // the rows before are done with the buffer
    for (int32_t k = lane; k < cnt; k += 32)
      sp[k] = make_int2(__ldcs(a.ind + p0 + k), __float_as_int(__ldcs(a.val + p0 + k)));
    __syncwarp();
    for (int32_t idx = r0 + sub; idx < r1; idx += PER_WARP) {
      const int32_t b = wp[idx] - p0, e = wp[idx + 1] - p0;
      float *out = a.C + static_cast<size_t>(bfirst + idx) * a.w + gl * VEC;
      for (int pn0 = 0; pn0 < panels; pn0 += PAN) {
        float acc[PAN][VEC];
#pragma unroll
        for (int pn = 0; pn < PAN; ++pn)
#pragma unroll
          for (int v = 0; v < VEC; ++v) acc[pn][v] = 0.0f;
        const int32_t col0 = pn0 * (G * VEC) + gl * VEC;
        const char *bcol = reinterpret_cast<const char *>(a.B + col0);
        // (every gather of a piece is issued before its first FMA, so a row of nine costs one
        // trip to memory, not two)
        staged_row<G, VEC, PAN, MASK, UC>(sp + b, e - b, bcol, wbytes, col0, acc);
#pragma unroll
        for (int pn = 0; pn < PAN; ++pn)
          if (panel_on<G, VEC, MASK>(col0, pn, a.w)) store_c<VEC>(out + (pn0 + pn) * (G * VEC), acc[pn], false);
      }
    }
    r0 = r1;
  }
}

template <int VEC>
__device__ __forceinline__ void queue_long_row(const SpmmArgs &a, int32_t r, int32_t len, bool first_lane) {
  if (!first_lane) return;
  const unsigned long long pieces = static_cast<unsigned long long>((len + a.piece - 1) / a.piece);
  const unsigned long long old =
      atomicAdd(reinterpret_cast<unsigned long long *>(a.ctrl + CTRL_PACKED), (1ull << 32) | pieces);
  a.long_rows[old >> 32] = make_int2(r, static_cast<int32_t>(old & 0xFFFFFFFFu));
}

// All rows of a unit where a whole warp takes a row: the nonzeros of as many rows as fit the pair
// buffer are staged with coalesced loads and the rows worked off from there.  Walking the row
// itself, the gathers of every eight nonzeros waited for the trip that fetched their columns
// first, as long as their own.  Without the walk's state there is room for four blocks per SM.
// R-MAT scale 22 at width 128, this launch alone: 3.03 ms walking, 2.37 staged, 2.18 staged with four
// blocks per SM; both launches 4.3 ms walking, 3.1 to 3.3 so.
//
// MG > 0, a product of one panel of MG lanes with MVEC columns each: rows of up to GROUP_MAX nonzeros
// go to lane groups of MG lanes, several rows at a time, the longer ones to the whole warp, VEC columns
// a lane.  Two is where the widths and graphs measured agree best, within a few percent of 1 to 4: symmetrised R-MAT
// scale 20 (half the edges) at 64, 594 us with 0, 537, 534, 536, 537 with 4; R-MAT scale 22 1,942, 1,929, 1,922, 1,916,
// 1,904; scale 20 with 4 edges a row at 40, 237, 246, 246, 253, 252; 131,072 Zipf rows at 48, 118, 117, 118, 123, 124.
constexpr int GROUP_MAX = 2;
template <int VEC, int PAN, bool MASK, int S_PAIRS, int UC, int MG = 0, int MVEC = 1>
__device__ __forceinline__ void whole_unit(const SpmmArgs &a, const int32_t *wp, int2 *sp, int32_t bfirst, int32_t bcount,
                                           int lane) {
  constexpr int G = 32;
  const int panels = (a.w + G * VEC - 1) / (G * VEC);
  const int32_t wbytes = a.w * 4;
  auto stage = [&](int32_t p, int32_t cnt) {
    __syncwarp();  // the rows before are done with the buffer
    for (int32_t k = lane; k < cnt; k += 32) sp[k] = make_int2(__ldcs(a.ind + p + k), __float_as_int(__ldcs(a.val + p + k)));
    __syncwarp();
  };
  for (int32_t r0 = 0; r0 < bcount;) {
    const int32_t p0 = wp[r0];
    bool fits = false;
    if (r0 + lane < bcount) {
      const int32_t b = wp[r0 + lane], e = wp[r0 + lane + 1];
      fits = p0 >= 0 && b >= p0 && e >= b && e <= a.nnz && e - p0 <= S_PAIRS && e - b <= a.split;
    }
    const unsigned m = __ballot_sync(FULL, fits);
    const int take = m == FULL ? 32 : __ffs(static_cast<int>(~m)) - 1;
    // `take` rows in the buffer, or one alone: malformed (empty), too long for the buffer, or queued
    int32_t len0 = 0;
    if (take > 0) {
      stage(p0, wp[r0 + take] - p0);
    } else {
      len0 = wp[r0 + 1] - p0;
      if (p0 < 0 || len0 < 0 || wp[r0 + 1] > a.nnz) len0 = 0;
      if (len0 > a.split) {
        for (int32_t j = lane * VEC; j < a.w; j += G * VEC)
#pragma unroll
          for (int v = 0; v < VEC; ++v) a.C[static_cast<size_t>(bfirst + r0) * a.w + j + v] = 0.0f;
        queue_long_row<VEC>(a, bfirst + r0, len0, lane == 0);
        ++r0;
        continue;
      }
    }
    const int32_t rows = take > 0 ? take : 1;
    unsigned whole = rows >= 32 ? FULL : (1u << rows) - 1u;  // the rows that the whole warp takes
    if constexpr (MG > 0) {
      const unsigned grouped = __ballot_sync(FULL, lane < take && wp[r0 + lane + 1] - wp[r0 + lane] <= GROUP_MAX);
      whole &= ~grouped;
      const int32_t col0 = (lane % MG) * MVEC;
      unsigned mine = grouped;  // group k takes the rows k, k + 32 / MG, ... of them
      for (int k = 0; k < lane / MG; ++k) mine &= mine - 1u;
      while (mine) {
        const int i = __ffs(static_cast<int>(mine)) - 1;
        const int32_t b = wp[r0 + i] - p0, e = wp[r0 + i + 1] - p0;
        float acc[1][MVEC];
#pragma unroll
        for (int v = 0; v < MVEC; ++v) acc[0][v] = 0.0f;
        staged_row<MG, MVEC, 1, MASK>(sp + b, e - b, reinterpret_cast<const char *>(a.B + col0), wbytes, col0, acc);
        if (panel_on<MG, MVEC, MASK>(col0, 0, a.w))
          store_c<MVEC>(a.C + static_cast<size_t>(bfirst + r0 + i) * a.w + col0, acc[0], false);
#pragma unroll
        for (int k = 0; k < 32 / MG; ++k) mine &= mine - 1u;
      }
      __syncwarp();
    }
    for (; whole; whole &= whole - 1u) {
      const int32_t i = __ffs(static_cast<int>(whole)) - 1;
      const int32_t b = wp[r0 + i] - p0, cnt = take > 0 ? wp[r0 + i + 1] - p0 - b : len0;
      float *out = a.C + static_cast<size_t>(bfirst + r0 + i) * a.w + lane * VEC;
      for (int pn0 = 0; pn0 < panels; pn0 += PAN) {
        float acc[PAN][VEC];
#pragma unroll
        for (int pn = 0; pn < PAN; ++pn)
#pragma unroll
          for (int v = 0; v < VEC; ++v) acc[pn][v] = 0.0f;
        const int32_t col0 = pn0 * (G * VEC) + lane * VEC;
        const char *bcol = reinterpret_cast<const char *>(a.B + col0);
        if (take > 0) {
          staged_row<G, VEC, PAN, MASK, UC>(sp + b, cnt, bcol, wbytes, col0, acc);
        } else {
          for (int32_t q = 0; q < cnt; q += S_PAIRS) {
            const int32_t part = cnt - q < S_PAIRS ? cnt - q : S_PAIRS;
            stage(p0 + q, part);
            staged_row<G, VEC, PAN, MASK, UC>(sp, part, bcol, wbytes, col0, acc);
          }
        }
#pragma unroll
        for (int pn = 0; pn < PAN; ++pn)
          if (panel_on<G, VEC, MASK>(col0, pn, a.w)) store_c<VEC>(out + (pn0 + pn) * (G * VEC), acc[pn], false);
      }
    }
    r0 += rows;
  }
}

// First launch: all rows of up to a.split nonzeros.  Every lane group is persistent: it takes
// the next row of its warp's unit as soon as its current row is finished, so the groups of
// a warp never wait for the one with the longest row.  Longer rows are zeroed and
// queued for the second launch.  A row is walked once per PAN panels (w = panels * G * VEC).
// WHOLE, EVEN, BLOCKS: see SpmmShape and whole_unit.
template <int G, int VEC, int PAN, bool MASK, bool WHOLE, int EVEN, int BLOCKS>
__global__ void __launch_bounds__(M_THREADS, BLOCKS) spmm_rows_kernel(SpmmArgs a) {
  constexpr int U = Step<PAN>::U;
  constexpr int ROWS = batch_rows(G, VEC), PAIRS = batch_pairs(G, VEC, PAN, BLOCKS);
  __shared__ int32_t sptr[M_WARPS][ROWS + 1];
  __shared__ int2 spair[M_WARPS][PAIRS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gl = lane % G;
  const unsigned below_group = (1u << (lane - gl)) - 1u;  // lanes of the groups in front of mine
  int32_t *wp = sptr[warp];
  // With four blocks per SM a lane has 64 registers: pieces of six nonzeros fit them, eight do not (R-MAT scale
  // 22 at 128: 3.26 ms with eight, 3.13 with six).
  constexpr int SIX = PAN == 1 ? 6 : U;
  if constexpr (G == 32) {
    constexpr int SPAN = EVEN == G ? PAN : 1;
    constexpr int UC = VEC == 4 && BLOCKS == 4 ? SIX : U, SUC = BLOCKS == 4 && Step<SPAN>::U > 6 ? 6 : Step<SPAN>::U;
    int32_t first = 0, count = 0;
    while (draw_unit<ROWS>(a, wp, lane, &first, &count)) {
      if (count == 0) continue;
      const int32_t longest = VEC == 4 ? unit_longest(wp, count, a.nnz, lane) : SHORT_MAX + 1;
      if (longest <= SHORT_MAX && (EVEN == G || unit_is_even<PAN>(wp, count, longest)))
        short_rows<EVEN, VEC, SPAN, EVEN == G && MASK, PAIRS, SUC>(a, wp, spair[warp], first, count, lane);
      else
        whole_unit<VEC, PAN, MASK, PAIRS, UC>(a, wp, spair[warp], first, count, lane);
    }
    return;
  }
  // Narrower, but with a column or two for each lane of a warp: units of short rows by lane groups, in
  // the others most nonzeros go to the whole warp.  Walked by lane groups, those took trips in turn
  // for columns and gathers, and code for a remainder of each group's own.  At widths 40 and 64: R-MAT
  // scale 22 took 3.09 and 2.34 ms, now 2.00 and 1.87; 65,536 Zipf rows 104 and 75 us, now 56 and 52.
  if constexpr (G < 32 && WHOLE) {
    static_assert(PAN == 1, "one panel covers the row");
    constexpr int UC = EVEN == G ? U : SIX;
    int32_t first = 0, count = 0;
    while (draw_unit<ROWS>(a, wp, lane, &first, &count)) {
      if (count == 0) continue;
      const int32_t longest = unit_longest(wp, count, a.nnz, lane);
      if (EVEN != G && longest <= SHORT_MAX && unit_is_even<PAN>(wp, count, longest))
        short_rows<EVEN, VEC, 1, false, PAIRS>(a, wp, spair[warp], first, count, lane);
      else if (longest <= SHORT_MAX || (G == 8 && unit_is_mild(wp, count, longest)))
        short_rows<G, VEC, PAN, MASK, PAIRS>(a, wp, spair[warp], first, count, lane);
      else
        whole_unit<G * VEC / 32, 1, MASK, PAIRS, UC, G, VEC>(a, wp, spair[warp], first, count, lane);
    }
    return;
  }
  const int panels = (a.w + G * VEC - 1) / (G * VEC);
  // warp-uniform: the rows in hand [bfirst, bfirst + bcount) and how many of them are given out
  int32_t bfirst = 0, bcount = 0, bnext = 0;
  bool exhausted = false;
  bool short_unit = false;  // the unit in hand goes to short_rows once every group is idle
  // group-uniform: the row in hand (-1: none), its extent, the walk's position and panel
  int32_t row = -1, pb = 0, p = 0, pe = 0, pn0 = 0;
  float acc[PAN][VEC];
#pragma unroll
  for (int pn = 0; pn < PAN; ++pn)
#pragma unroll
    for (int v = 0; v < VEC; ++v) acc[pn][v] = 0.0f;
  for (;;) {
    if (row >= 0 && p >= pe) {  // end of a walk: store, then the next panels or a new row
      float *out = a.C + static_cast<size_t>(row) * a.w + pn0 * (G * VEC) + gl * VEC;
#pragma unroll
      for (int pn = 0; pn < PAN; ++pn) {
        if (panel_on<G, VEC, MASK>(pn0 * (G * VEC) + gl * VEC, pn, a.w))
          store_c<VEC>(out + pn * G * VEC, acc[pn], false);
#pragma unroll
        for (int v = 0; v < VEC; ++v) acc[pn][v] = 0.0f;
      }
      pn0 += PAN;
      if (pn0 < panels)
        p = pb;
      else
        row = -1;
    }
    const unsigned want = __ballot_sync(FULL, row < 0 && gl == 0);  // groups without a row
    if (want) {
      if (bnext >= bcount && !exhausted) {
        bnext = 0;
        exhausted = !draw_unit<ROWS>(a, wp, lane, &bfirst, &bcount);
        short_unit = bcount > 0 && unit_longest(wp, bcount, a.nnz, lane) <= SHORT_MAX;
      }
      bool hold = false;  // a short unit in hand: no row of it is handed out one by one
      {
        if (short_unit) {
          hold = true;
          // (groups still walking a row of the unit before finish it first)
          if (__ballot_sync(FULL, row >= 0) == 0u) {
            short_rows<G, VEC, PAN, MASK, PAIRS>(a, wp, spair[warp], bfirst, bcount, lane);
            bnext = bcount;
            short_unit = false;
            // (no group holds a row here: saying so frees the walk's registers for short_rows)
            row = -1;
            pb = p = pe = pn0 = 0;
#pragma unroll
            for (int pn = 0; pn < PAN; ++pn)
#pragma unroll
              for (int v = 0; v < VEC; ++v) acc[pn][v] = 0.0f;
          }
        }
      }
      if (!hold && row < 0) {
        const int idx = bnext + __popc(want & below_group);
        if (idx < bcount) {
          int32_t b = wp[idx], e = wp[idx + 1];
          if (b < 0 || e < b || e > a.nnz) e = b = 0;  // malformed row pointers: an empty row
          const int32_t r = bfirst + idx;
          if (e - b > a.split) {
            for (int32_t j = gl * VEC; j < a.w; j += G * VEC)
#pragma unroll
              for (int v = 0; v < VEC; ++v) a.C[static_cast<size_t>(r) * a.w + j + v] = 0.0f;
            queue_long_row<VEC>(a, r, e - b, gl == 0);
          } else {
            row = r;
            pb = p = b;
            pe = e;
            pn0 = 0;
          }
        }
      }
      if (!hold) {
        const int given = bnext + __popc(want);
        bnext = given < bcount ? given : bcount;
      }
      if (exhausted && __ballot_sync(FULL, row >= 0) == 0u) break;
    }
    if (row >= 0 && p < pe) {
      const int cnt = pe - p < U ? pe - p : U;
      fma_step<G, VEC, PAN, MASK>(a, p, cnt, pn0 * (G * VEC) + gl * VEC, acc);
      p += cnt;
      // a short tail (a row of nine nonzeros is a full step and one more) goes along in the
      // same turn of the loop: the turn, with its hand-out of rows, costs more than the tail
      if (pe - p > 0 && pe - p <= U / 2) {
        fma_step<G, VEC, PAN, MASK, U / 2>(a, p, pe - p, pn0 * (G * VEC) + gl * VEC, acc);
        p = pe;
      }
    }
  }
}

// Second launch: the pieces (a.piece nonzeros each) of the queued long rows, spread over
// all lane groups; piece number -> queue entry by binary search on the entries' first
// piece numbers (ascending by construction).  Partial rows are added with atomics.
// Twice as many gathers in flight as the first launch has: a piece is a plain run of them, and
// what bounds it is the latency of memory (R-MAT scale 22, width 128: 1.21 ms with eight rows of B at
// a time, 0.94 with sixteen; 0.96 with eight in four blocks per SM.  The first launch, which has
// its walk in registers beside, slows down by a quarter either way).
template <int G, int VEC, int PAN, bool MASK>
__global__ void __launch_bounds__(M_THREADS, M_BLOCKS_PER_SM) spmm_long_kernel(SpmmArgs a) {
  constexpr int PER_WARP = 32 / G;
  constexpr int U = 2 * Step<PAN>::U;
  constexpr int LONG_PAIRS = 256;  // pairs staged per warp
  __shared__ int2 spair[G == 32 ? M_WARPS : 1][G == 32 ? LONG_PAIRS : 1];
  [[maybe_unused]] int2 *const sp = spair[G == 32 ? threadIdx.x >> 5 : 0];
  const int lane = threadIdx.x & 31;
  const int sub = lane / G, gl = lane % G;
  const int32_t group = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * PER_WARP + sub;
  const int32_t groups = ((gridDim.x * blockDim.x) >> 5) * PER_WARP;
  const int32_t queued = static_cast<int32_t>(a.ctrl[CTRL_PACKED + 1]);
  const int32_t total = static_cast<int32_t>(a.ctrl[CTRL_PACKED]);
  const int panels = (a.w + G * VEC - 1) / (G * VEC);
  for (int32_t id = group; id < total; id += groups) {
    int32_t lo = 0, hi = queued;  // long_rows[lo].y <= id < long_rows[hi].y
    while (hi - lo > 1) {
      const int32_t mid = (lo + hi) >> 1;
      if (a.long_rows[mid].y <= id)
        lo = mid;
      else
        hi = mid;
    }
    const int2 q = a.long_rows[lo];
    const int32_t b = a.ptr[q.x], e = a.ptr[q.x + 1];
    const int32_t pb = b + (id - q.y) * a.piece;
    const int32_t pe = pb + a.piece < e ? pb + a.piece : e;
    for (int pn0 = 0; pn0 < panels; pn0 += PAN) {
      const int32_t col0 = pn0 * (G * VEC) + gl * VEC;
      float acc[PAN][VEC];
#pragma unroll
      for (int pn = 0; pn < PAN; ++pn)
#pragma unroll
        for (int v = 0; v < VEC; ++v) acc[pn][v] = 0.0f;
      if constexpr (G == 32) {  // the pairs through shared memory, as in whole_unit
        const char *bcol = reinterpret_cast<const char *>(a.B + col0);
        for (int32_t p = pb; p < pe; p += LONG_PAIRS) {
          const int32_t part = pe - p < LONG_PAIRS ? pe - p : LONG_PAIRS;
          __syncwarp();
          for (int32_t k = lane; k < part; k += 32)
            sp[k] = make_int2(__ldcs(a.ind + p + k), __float_as_int(__ldcs(a.val + p + k)));
          __syncwarp();
          int32_t k = 0;
          for (; part - k >= U; k += U) short_slots<G, VEC, PAN, MASK, U>(sp + k, bcol, a.w * 4, col0, acc);
          staged_row<G, VEC, PAN, MASK>(sp + k, part - k, bcol, a.w * 4, col0, acc);
        }
      } else {
        for (int32_t p = pb; p < pe; p += U)
          fma_step<G, VEC, PAN, MASK, U>(a, p, pe - p < U ? pe - p : U, col0, acc);
      }
#pragma unroll
      for (int pn = 0; pn < PAN; ++pn)
        if (panel_on<G, VEC, MASK>(col0, pn, a.w))
          store_c<VEC>(a.C + static_cast<size_t>(q.x) * a.w + col0 + pn * G * VEC, acc[pn], true);
    }
  }
}

template <int G, int VEC, int PAN, bool MASK, bool WHOLE, int EVEN, int BLOCKS>
bool launch_shape(Context &ctx, const SpmmArgs &a, const SpmmPlan &p) {
  spmm_rows_kernel<G, VEC, PAN, MASK, WHOLE, EVEN, BLOCKS><<<p.rows_grid, M_THREADS, 0, ctx.stream>>>(a);
  CSG_CUDA(cudaGetLastError());
  // (a piece goes to a whole warp wherever a row may)
  constexpr int LG = WHOLE ? 32 : G;
  spmm_long_kernel<LG, G * VEC / LG, PAN, MASK><<<p.long_grid, M_THREADS, 0, ctx.stream>>>(a);
  CSG_CUDA(cudaGetLastError());
  count_launches(2);
  return true;
}

bool dispatch_spmm(Context &ctx, SpmmArgs a) {
  const uintptr_t both = reinterpret_cast<uintptr_t>(a.B) | reinterpret_cast<uintptr_t>(a.C);
  const int align = both % 16 == 0 ? 16 : both % 8 == 0 ? 8 : 4;
  const SpmmPlan p = spmm_plan(a.n, a.nnz, a.w, align, ctx.num_sms, a.queue_cap);
  a.unit = p.unit;
  a.split = p.split;
  a.piece = p.piece;
#define CSG_LAUNCH(G, VEC, PAN, MASK, WHOLE, EVEN, BLOCKS)         \
  if (p.shape == SpmmShape{G, VEC, PAN, MASK, WHOLE, EVEN, BLOCKS}) \
    return launch_shape<G, VEC, PAN, MASK != 0, WHOLE != 0, EVEN, BLOCKS>(ctx, a, p);
  CSG_SPMM_SHAPES(CSG_LAUNCH)
#undef CSG_LAUNCH
  set_error("spmm: no kernel of the planned shape (width %d)", a.w);
  return false;
}

}  // namespace

bool launch_spmm(Context &ctx, int32_t n, int32_t nnz, int32_t w, const int32_t *d_ptr,
                 const int32_t *d_ind, const float *d_val, const float *d_B, float *d_C) {
  CSG_REQUIRE(w >= 1, "spmm: dense width must be >= 1");
  SpmmArgs a;
  a.n = n;
  a.w = w;
  a.nnz = nnz;
  a.ptr = d_ptr;
  a.ind = d_ind;
  a.val = d_val;
  a.B = d_B;
  a.C = d_C;
  // scratch: counters and the queue of long rows (at most nnz / SPLIT_MIN of them)
  Arena ar;
  const size_t o_ctrl = ar.take(sizeof(uint32_t) * CTRL_SCRATCH_WORDS);
  a.queue_cap = nnz / SPLIT_MIN + 1;
  const size_t o_rows = ar.take(sizeof(int2) * static_cast<size_t>(a.queue_cap));
  if (!ensure_workspace(ctx, ar.off)) return false;
  a.ctrl = reinterpret_cast<uint32_t *>(ctx.ws + o_ctrl);
  a.long_rows = reinterpret_cast<int2 *>(ctx.ws + o_rows);
  CSG_CUDA(cudaMemsetAsync(a.ctrl, 0, sizeof(uint32_t) * CTRL_SCRATCH_WORDS, ctx.stream));
  return dispatch_spmm(ctx, a);
}

}  // namespace csg

// ---------------------------------------------------------------------------------
// SpMM without any allocation.
//
// Some hosts of this library must not see a cudaMalloc from it: applications that
// have handed all device memory to an allocator of their own (a tensor framework's
// caching pool run with a fixed memory share, a database buffer pool), where a
// driver allocation inside a library call can fail outright or push the process
// over its budget; and request paths that ban driver allocations because
// cudaMalloc / cudaFree stall every stream of the device.  For them the queue of
// long rows -- the only scratch the SpMM kernels need -- lives in a fixed array
// that is part of the loaded library image, so every GPU that loads the library
// holds these 512 KiB until the process exits.
//
// The array is shared by every call in the process and keeps what the last call
// left in it; the call clears the counters that must start at zero.  Two calls
// whose kernels can overlap on the same GPU (different streams) would race on it.
namespace csg {
namespace {

constexpr int STATIC_MAX_LONG_ROWS = 65536;  // queue capacity (entries of 8 bytes)
constexpr int STATIC_QUEUE_OFFSET = CTRL_SCRATCH_WORDS;  // words; counters own the first 256 bytes
static __device__ __align__(256) uint32_t g_spmm_static_scratch[STATIC_QUEUE_OFFSET +
                                                                2 * STATIC_MAX_LONG_ROWS];

// In host code the symbol above is only a stand-in, not a device address: the real
// address is asked for once per device, with that device current.
constexpr int MAX_DEVICES = 64;
std::mutex g_static_mutex;
uint32_t *g_static_addr[MAX_DEVICES] = {};

bool static_scratch_address(int device, uint32_t **out) {
  std::lock_guard<std::mutex> lock(g_static_mutex);
  CSG_REQUIRE(device >= 0 && device < MAX_DEVICES, "spmm_static: device %d out of range", device);
  if (!g_static_addr[device]) {
    void *p = nullptr;
    CSG_CUDA(cudaGetSymbolAddress(&p, g_spmm_static_scratch));
    g_static_addr[device] = static_cast<uint32_t *>(p);
  }
  *out = g_static_addr[device];
  return true;
}

bool run_spmm_static(int32_t n, int32_t nnz, int32_t w, const int32_t *d_ptr, const int32_t *d_ind,
                     const float *d_val, const float *d_B, float *d_C, cudaStream_t stream) {
  CSG_REQUIRE(n >= 1 && nnz >= 0 && w >= 1, "spmm_static: bad sizes n=%d nnz=%d w=%d", n, nnz, w);
  CSG_REQUIRE(d_ptr && d_B && d_C && (nnz == 0 || (d_ind && d_val)), "spmm_static: null array");
  // at most nnz / SPLIT rows can be longer than SPLIT; all of them must fit the queue
  CSG_REQUIRE(static_cast<int64_t>(nnz) / SPLIT + 1 <= STATIC_MAX_LONG_ROWS,
              "spmm_static: nnz = %d exceeds the fixed scratch (at most %lld nonzeros); use sporder_spmm",
              nnz, static_cast<long long>(STATIC_MAX_LONG_ROWS - 1) * SPLIT + SPLIT - 1);
  Context tmp;  // stack object only: stream and SM count for the launch geometry
  CSG_CUDA(cudaGetDevice(&tmp.device));
  CSG_CUDA(cudaDeviceGetAttribute(&tmp.num_sms, cudaDevAttrMultiProcessorCount, tmp.device));
  tmp.stream = stream;
  uint32_t *scratch = nullptr;
  if (!static_scratch_address(tmp.device, &scratch)) return false;
  SpmmArgs a;
  a.n = n;
  a.w = w;
  a.nnz = nnz;
  a.ptr = d_ptr;
  a.ind = d_ind;
  a.val = d_val;
  a.B = d_B;
  a.C = d_C;
  a.queue_cap = STATIC_MAX_LONG_ROWS;
  a.ctrl = scratch;
  a.long_rows = reinterpret_cast<int2 *>(scratch + STATIC_QUEUE_OFFSET);
  // the counters keep the previous call's values: clear them (the queue is overwritten)
  CSG_CUDA(cudaMemsetAsync(a.ctrl, 0, sizeof(uint32_t) * CTRL_SCRATCH_WORDS, stream));
  return dispatch_spmm(tmp, a);
}

}  // namespace
}  // namespace csg

extern "C" int32_t sporder_spmm_static(int32_t n, int32_t nnz, int32_t w, const int32_t *d_ptr,
                                       const int32_t *d_ind, const float *d_val, const float *d_B,
                                       float *d_C, void *stream) {
  csg::clear_error();
  return csg::run_spmm_static(n, nnz, w, d_ptr, d_ind, d_val, d_B, d_C,
                              static_cast<cudaStream_t>(stream))
             ? 0
             : -1;
}
