// C ABI of the library (include/sporder_b200.h): context, parameter resolution,
// the csg pipeline driver and the thin wrappers around reorder and SpMM.
#include "../../include/sporder_b200.h"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstring>

#include "common.cuh"

namespace csg {

// ---- error channel ---------------------------------------------------------
namespace {
thread_local char g_err[512];
thread_local bool g_has_err = false;
std::atomic<uint64_t> g_launches{0};
}  // namespace

void set_error(const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  g_has_err = true;
}
bool has_error() { return g_has_err; }
void clear_error() { g_has_err = false; }
void count_launches(int k) { g_launches.fetch_add(static_cast<uint64_t>(k), std::memory_order_relaxed); }

bool ensure_workspace(Context &ctx, size_t bytes) {
  if (bytes <= ctx.ws_bytes) return true;
  CSG_CUDA(cudaStreamSynchronize(ctx.stream));
  if (ctx.ws) CSG_CUDA(cudaFree(ctx.ws));
  ctx.ws = nullptr;
  ctx.ws_bytes = 0;
  const size_t want = bytes + (bytes >> 3);  // head room so that similar sizes reuse it
  cudaError_t e = cudaMalloc(&ctx.ws, want);
  if (e != cudaSuccess) {
    cudaGetLastError();
    e = cudaMalloc(&ctx.ws, bytes);
    if (e != cudaSuccess) {
      cudaGetLastError();
      set_error("device workspace of %zu bytes: %s", bytes, cudaGetErrorString(e));
      return false;
    }
    ctx.ws_bytes = bytes;
    return true;
  }
  ctx.ws_bytes = want;
  return true;
}

bool wait_outcome(Context &ctx, cudaStream_t st, int word, uint32_t ticket) {
  volatile uint32_t *const h = outcome_words(ctx, word);
  const auto start = std::chrono::steady_clock::now();
  for (int spins = 0; h[0] != ticket; ++spins) {
    // something went wrong on the device, or it is busy with other work: wait for the stream
    if ((spins & 1023) == 1023 && std::chrono::steady_clock::now() - start > std::chrono::milliseconds(200)) {
      CSG_CUDA(cudaStreamSynchronize(st));
      CSG_REQUIRE(h[0] == ticket, "internal: a kernel did not report its outcome");
    }
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  return true;
}

bool read_lists(Context &ctx, CsgScratch &s, int phase) {
  const int word = phase == PHASE_PRIO ? OUTCOME_WORD_PRIO : OUTCOME_WORD;
  if (!wait_outcome(ctx, phase == PHASE_PRIO ? ctx.side_stream : ctx.stream, word, s.ticket)) return false;
  const volatile uint32_t *const h = outcome_words(ctx, word);
  s.chain_rows = h[1];
  s.chain_need = static_cast<uint64_t>(h[4]) << 32 | h[3];
  s.no_heavy_rows = s.chain_rows == 0;
  return true;
}

namespace {
// ctx.chains[part] of `bytes` or more.  The one it replaces may be in use by the call's other stream, so it stays until the
// call ends - unless its memory is needed.
bool grow_chains(Context &ctx, int part, size_t bytes) {
  if (bytes <= ctx.chains_bytes[part]) return true;
  if (ctx.chains[part]) {
    if (ctx.outgrown[part]) cudaFree(ctx.outgrown[part]);
    ctx.outgrown[part] = ctx.chains[part];
    ctx.chains[part] = nullptr;
    ctx.chains_bytes[part] = 0;
  }
  for (const size_t want : {bytes + (bytes >> 3), bytes}) {  // (head room, so that similar calls reuse it)
    if (cudaMalloc(&ctx.chains[part], want) == cudaSuccess) {
      ctx.chains_bytes[part] = want;
      return true;
    }
    cudaGetLastError();
    ctx.chains[part] = nullptr;
    for (char *&old : ctx.outgrown) {  // (cudaFree waits for the kernels that may use it)
      if (old) cudaFree(old);
      old = nullptr;
    }
  }
  return false;
}
}  // namespace

// Streams of all listed rows if s.stream_cap and the device's memory allow; else the heaviest rows that fit get a chain
// and the kernel of the light rows computes the others, so results never depend on the size.
bool plan_chains(Context &ctx, int32_t nnz, CsgScratch &s, int phase) {
  const int part = phase == PHASE_PRIO ? 1 : 0;
  uint64_t cap = s.chain_need < s.stream_cap ? s.chain_need : s.stream_cap;
  if (cap < 1) cap = 1;
  size_t rows = s.chain_rows < s.heavy_max ? s.chain_rows : s.heavy_max;
  for (;; cap /= 2) {
    const size_t parts = static_cast<size_t>(nnz) / SKETCH_PART_COLS + rows + 1;  // column slices of these rows
    Arena ar;
    const size_t o_stream = ar.take(8 * cap), o_off = ar.take(4 * (rows + 1)), o_state = ar.take(4 * rows * 2 * s.slots);
    const size_t o_base = ar.take(4 * (rows + 2)), o_part = ar.take(4 * (parts + 1));
    if (!grow_chains(ctx, part, ar.off)) {
      rows = std::min<size_t>(rows, cap / 2 / HEAVY_WORK + 1 + CHAIN_ROWS);
      if (cap > 1) continue;
      set_error("device workspace of %zu bytes for the longest rows: %s", ar.off, cudaGetErrorString(cudaErrorMemoryAllocation));
      return false;
    }
    char *const base = ctx.chains[part];
    s.hstream = reinterpret_cast<int2 *>(base + o_stream);
    s.heavy_off = reinterpret_cast<uint32_t *>(base + o_off);
    s.heavy_state = reinterpret_cast<int32_t *>(base + o_state);
    s.part_base = reinterpret_cast<uint32_t *>(base + o_base);
    s.part_off = reinterpret_cast<uint32_t *>(base + o_part);
    s.stream_cap = static_cast<uint32_t>(cap);
    s.heavy_max = static_cast<uint32_t>(rows);
    return true;
  }
}

// sporder/src/sporder.cpp:147-161 and the checks of
// sporder/src/common/chunk_similarity_top_k.cu:143-147
bool resolve_params(int32_t n, int32_t nnz, int32_t k, float ovs, int32_t chunk, CsgParams *out) {
  CSG_REQUIRE(n >= 1, "n must be >= 1 (got %d)", n);
  CSG_REQUIRE(nnz >= 0, "nnz must be >= 0 (got %d)", nnz);
  if (k <= 0) {
    int32_t a = nnz / n;
    if (a < 16) a = 16;
    if (a > 256) a = 256;
    k = a;
  }
  if (ovs <= 0.0f) ovs = 4.0f;
  if (chunk <= 0) chunk = 1024;
  const int32_t m = static_cast<int32_t>(static_cast<float>(k) * ovs);
  out->k = k;
  out->ovs = ovs;
  out->chunk = chunk;
  out->m_used = ((m + 31) / 32) * 32;
  CSG_REQUIRE(ovs >= 1.0f, "expect oversampling >= 1 (got %g)", static_cast<double>(ovs));
  CSG_REQUIRE(m <= 512, "expect k * oversampling <= 512 (got %d)", m);
  const int32_t mm = m < 1 ? 1 : m;
  out->M = ((mm + 31) / 32) * 32;
  return true;
}

namespace {

struct ChainStatsHost {
  unsigned long long total_degree;
  double total_weight;
  double link_weight_sum;
  int32_t zero_degree_rows;
  int32_t restarts;
  int32_t links;
  int32_t pad;
  double in_chunk_weight;
};

size_t greedy_bitmap_words(int32_t n, int32_t chunk) {
  const int32_t span = chunk < n ? chunk : n;
  const size_t words = (static_cast<size_t>(span) + 31) / 32;
  if (4 /*warps*/ * 2 * words * sizeof(uint32_t) <= 48 * 1024) return 0;
  const size_t chunks = (static_cast<size_t>(n) + chunk - 1) / chunk;
  return chunks * 2 * words;
}

constexpr int32_t AHEAD_MIN_NNZ = 1 << 24;  // smaller calls do not pay for a second pipeline's launches

// Stream elements the chains of a call may take: never more than the rows could stream at all
// (nnz * chunk span), than 2 GiB or than the caller's limit.
uint64_t stream_capacity(const Context &ctx, size_t nnz, size_t span) {
  uint64_t cap = static_cast<uint64_t>(nnz) * span;
  if (cap > STREAM_CAP_MAX) cap = STREAM_CAP_MAX;
  if (ctx.stream_limit && cap > ctx.stream_limit) cap = ctx.stream_limit;
  return cap < 1 ? 1 : cap;
}

// most rows with a chain on streams of `cap` elements
uint32_t chain_rows_max(uint64_t cap, int32_t n) {
  const uint64_t rows = cap / HEAVY_WORK + 1 + CHAIN_ROWS;
  return static_cast<uint32_t>(rows < static_cast<uint64_t>(n) ? rows : n);
}

// Lays out the scratch of one csg call in the context workspace.  `transpose_only` leaves
// out everything behind the chunk-local transpose (the pillar count needs no more).
// With `prio` the call runs one chunk ahead of the rest (run_csg): that part gets control
// words, work lists and tile tables of its own.
bool plan_scratch(Context &ctx, int32_t n, int32_t nnz, const CsgParams &p, uint64_t *user_table,
                  CsgScratch *s, int32_t greedy_chunk = 0, bool transpose_only = false,
                  CsgScratch *prio = nullptr) {
  Arena ar;
  const size_t z = static_cast<size_t>(nnz > 0 ? nnz : 1);
  const size_t o_keyA = ar.take(4 * z), o_keyB = ar.take(4 * z);
  const size_t o_payA = ar.take(4 * z), o_payB = ar.take(4 * z);
  const size_t o_cand = ar.take(8 * z), o_seg = ar.take(8 * z), o_rank = ar.take(4 * z);
  const size_t o_work = ar.take(4 * static_cast<size_t>(n));
  const size_t o_rseg = ar.take(4 * static_cast<size_t>(n)), o_rcols = ar.take(4 * static_cast<size_t>(n));
  const size_t o_list = ar.take(4 * static_cast<size_t>(n));
  const size_t o_ctrl = ar.take(4 * CTRL_WORDS);
  // (the greedy stage may run with another chunk size than the sketch: chunk_greedy)
  size_t bw = transpose_only ? 0 : greedy_bitmap_words(n, p.chunk);
  if (greedy_chunk > 0 && greedy_bitmap_words(n, greedy_chunk) > bw) bw = greedy_bitmap_words(n, greedy_chunk);
  const size_t o_bm = ar.take(4 * (bw ? bw : 1));
  // heavy chunks hold more than 6144 nonzeros or 2048 rows each and are cut into tiles of 4096
  const size_t chunks = (static_cast<size_t>(n) + p.chunk - 1) / p.chunk;
  size_t heavy_max = p.chunk > 2048 ? chunks : z / 6144 + 1;
  if (heavy_max > chunks) heavy_max = chunks;
  const size_t o_nc = ar.take(4 * chunks);
  const size_t tiles_max = z / 4096 + heavy_max + 1;
  const size_t o_hc = ar.take(4 * heavy_max), o_htb = ar.take(4 * (heavy_max + 1));
  const size_t o_th = ar.take(4 * 256 * tiles_max), o_db = ar.take(4 * 256 * heavy_max);
  const size_t span = static_cast<size_t>(p.chunk < n ? p.chunk : n);
  const size_t o_table = (user_table || transpose_only) ? 0 : ar.take(8 * static_cast<size_t>(n) * p.k);
  // the part that runs ahead: one chunk's worth of lists, tile tables for up to all nonzeros
  // (nothing bounds a chunk's share of them)
  size_t o_p_list = 0, o_p_ctrl = 0, o_p_hc = 0, o_p_htb = 0, o_p_th = 0, o_p_db = 0;
  if (prio) {
    o_p_list = ar.take(4 * span);
    o_p_ctrl = ar.take(4 * CTRL_WORDS);
    o_p_hc = ar.take(4 * 2);
    o_p_htb = ar.take(4 * 4);
    o_p_th = ar.take(4 * 256 * (z / 4096 + 2));
    o_p_db = ar.take(4 * 256);
  }
  if (!ensure_workspace(ctx, ar.off)) return false;
  s->keyA = reinterpret_cast<uint32_t *>(ctx.ws + o_keyA);
  s->keyB = reinterpret_cast<uint32_t *>(ctx.ws + o_keyB);
  s->payA = reinterpret_cast<uint32_t *>(ctx.ws + o_payA);
  s->payB = reinterpret_cast<uint32_t *>(ctx.ws + o_payB);
  s->cand = reinterpret_cast<int2 *>(ctx.ws + o_cand);
  s->seg = reinterpret_cast<int2 *>(ctx.ws + o_seg);
  s->seg_rank = reinterpret_cast<int32_t *>(ctx.ws + o_rank);
  s->row_work = reinterpret_cast<uint32_t *>(ctx.ws + o_work);
  s->row_seg = reinterpret_cast<int32_t *>(ctx.ws + o_rseg);
  s->row_cols = reinterpret_cast<int32_t *>(ctx.ws + o_rcols);
  s->next_chunk = reinterpret_cast<int32_t *>(ctx.ws + o_nc);
  s->row_list = reinterpret_cast<int32_t *>(ctx.ws + o_list);
  s->ctrl = reinterpret_cast<uint32_t *>(ctx.ws + o_ctrl);
  s->table = user_table ? user_table : reinterpret_cast<uint64_t *>(ctx.ws + o_table);
  const uint64_t cap = stream_capacity(ctx, z, span);
  s->stream_cap = static_cast<uint32_t>(cap);
  s->heavy_max = chain_rows_max(cap, n);
  s->slots = p.M;
  s->heavy_chunk = reinterpret_cast<int32_t *>(ctx.ws + o_hc);
  s->heavy_tile_base = reinterpret_cast<int32_t *>(ctx.ws + o_htb);
  s->tile_hist = reinterpret_cast<uint32_t *>(ctx.ws + o_th);
  s->digit_base = reinterpret_cast<uint32_t *>(ctx.ws + o_db);
  s->gbitmaps = bw ? reinterpret_cast<uint32_t *>(ctx.ws + o_bm) : nullptr;
  if (prio) {
    *prio = *s;  // the arrays indexed by nonzero, row or table entry are common to both parts
    prio->row_list = reinterpret_cast<int32_t *>(ctx.ws + o_p_list);
    prio->ctrl = reinterpret_cast<uint32_t *>(ctx.ws + o_p_ctrl);
    prio->heavy_chunk = reinterpret_cast<int32_t *>(ctx.ws + o_p_hc);
    prio->heavy_tile_base = reinterpret_cast<int32_t *>(ctx.ws + o_p_htb);
    prio->tile_hist = reinterpret_cast<uint32_t *>(ctx.ws + o_p_th);
    prio->digit_base = reinterpret_cast<uint32_t *>(ctx.ws + o_p_db);
    // (the rest keeps a quarter of what the streams may take in any case)
    prio->stream_cap = static_cast<uint32_t>(cap - cap / 4);
    prio->heavy_max = static_cast<uint32_t>(span);
  }
  return true;
}

// End of a call that ran the transpose (and possibly the sketch): the control words come
// back with the call's one synchronisation.  Malformed input and a refused stream slice are
// errors.
bool finish_call(Context &ctx, const CsgScratch &s, const CsgScratch *prio = nullptr) {
  uint32_t *h = reinterpret_cast<uint32_t *>(ctx.h_pinned);
  CSG_CUDA(cudaMemcpyAsync(h, s.ctrl, 16 * sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx.stream));
  if (prio)  // (the side stream's work has been joined into ctx.stream by now)
    CSG_CUDA(cudaMemcpyAsync(h + 16, prio->ctrl, 16 * sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx.stream));
  CSG_CUDA(cudaStreamSynchronize(ctx.stream));
  CSG_CUDA(cudaGetLastError());
  for (char *&old : ctx.outgrown) {
    if (old) CSG_CUDA(cudaFree(old));
    old = nullptr;
  }
  if (prio) {  // the words of the part ahead: errors count like the others'
    const uint32_t *hp = h + 16;
    h[CTRL_BAD_INPUT] |= hp[CTRL_BAD_INPUT];
    h[CTRL_STREAM_OVERRUN] |= hp[CTRL_STREAM_OVERRUN];
    if (h[CTRL_CHECK] == 0 && hp[CTRL_CHECK] != 0)
      for (int i = 0; i < 3; ++i) h[CTRL_CHECK + i] = hp[CTRL_CHECK + i];
  }
  CSG_REQUIRE(h[CTRL_BAD_INPUT] == 0,
              "malformed CSR: row pointers must be non-decreasing inside [0, nnz] (results unspecified)");
  if (h[CTRL_CHECK] != 0) {  // only a build with -DSPORDER_CHECKED writes this word
    static const char *const site[] = {"?", "cand[] index of a group", "position in a stream ring",
                                       "stream offset of a heavy row", "stream key outside its chunk",
                                       "heavy-row state item", "row of the top-k table", "row list entry",
                                       "order[] position", "scatter position of a radix pass",
                                       "group position written by the transpose", "part table entry"};
    const uint32_t k = h[CTRL_CHECK] < sizeof(site) / sizeof(site[0]) ? h[CTRL_CHECK] : 0;
    const long long idx = static_cast<long long>((static_cast<uint64_t>(h[CTRL_CHECK + 2]) << 32) | h[CTRL_CHECK + 1]);
    set_error("checked build: index out of bounds (%s: %lld); results unspecified", site[k], idx);
    return false;
  }
  ctx.chain_rows = h[CTRL_HEAVY_ROWS] + (prio ? h[16 + CTRL_HEAVY_ROWS] : 0u);
  CSG_REQUIRE(h[CTRL_STREAM_OVERRUN] == 0,
              "internal: a heavy row's stream slice did not fit its place in the stream buffer");
  return true;
}

// The pipeline of sporder/src/csg/chunk_similarity_greedy.cu:100-138 with the
// stages of this library: chunk-local transpose -> sketch/top-k -> greedy.
bool run_csg(Context &ctx, int32_t n, int32_t ncols, int32_t row_base, int32_t nnz,
             const int32_t *d_ptr, const int32_t *d_ind,
             int32_t k, float ovs, int32_t chunk, int32_t *d_new_order, uint64_t *d_table,
             uint64_t table_capacity, sporder_csg_timing_t *timing, sporder_csg_stats_t *stats,
             int32_t *k_used) {
  const auto wall0 = std::chrono::steady_clock::now();
  CsgParams p;
  if (!resolve_params(n, nnz, k, ovs, chunk, &p)) return false;
  if (k_used) *k_used = p.k;
  if (stats) {
    std::memset(stats, 0, sizeof(*stats));
    stats->k_used = p.k;
    stats->m_used = p.m_used;
    stats->chunk_size_used = p.chunk;
  }
  CSG_REQUIRE(d_ptr && (d_ind || nnz == 0), "null CSR arrays");
  CSG_REQUIRE(ncols >= n && row_base >= 0 && static_cast<int64_t>(row_base) + n <= ncols,
              "row block [%d, %d + %d) does not lie inside a matrix of %d rows", row_base, row_base, n, ncols);
  CSG_REQUIRE(row_base % p.chunk == 0,
              "row_base %d is not a multiple of the chunk size %d: the block would not hold whole chunks",
              row_base, p.chunk);
  CSG_REQUIRE(!d_table || table_capacity >= static_cast<uint64_t>(n) * p.k,
              "table buffer holds %llu entries, need n * k = %llu",
              static_cast<unsigned long long>(table_capacity),
              static_cast<unsigned long long>(static_cast<uint64_t>(n) * p.k));
  CSG_CUDA(cudaSetDevice(ctx.device));
  // Large calls run one chunk ahead.  On power-law inputs the rows with the longest candidate
  // streams - the dependent chains that decide how long the call takes - sit in the chunk
  // with the most nonzeros, and all their chains need is that chunk's own transposition.  So
  // that chunk is transposed first, on a second stream, and its heavy rows' chains start
  // there while the context's stream transposes everything else; the two meet before the
  // greedy stage.  Results do not depend on the split (the same kernels on the same rows).
  // By default for calls of 2^24 nonzeros in 64 chunks or more, whose chunk ahead must hold 2^17 nonzeros:
  // smaller calls do not pay for the second pipeline's fifteen launches.  With 96 and 128 slots in tall chunks, and
  // with 128 where rows are long, the chains of the two parts slow each other.  Time ahead over time not, R-MAT and
  // its symmetrised form of 19 to 65 M nonzeros, chunks of 512 to 1024: 32 slots 0.89 to 0.96; 64 slots 0.87 to 0.96; 96
  // slots 0.81 to 0.95 at 10 to 31 nonzeros a row; 128 slots 0.84 to 0.96 up to 27, 1.02 to 1.07 from there on, 0.90 to
  // 0.95 in chunks of 512; 160 and 256 slots (a warp per row) 0.97 to 0.99; in chunks of 2048, 32 slots 0.82 to 0.88; in
  // chunks of 4096, 32 slots 0.87 to 0.97, 96 slots 1.07, 128 slots 1.28, 64 slots 0.88 to
  // 1.15.  A caller's own threshold (sporder_context_set_ahead_threshold) applies to any call of two chunks.
  const int64_t chunks = (static_cast<int64_t>(n) + p.chunk - 1) / p.chunk;
  bool ahead = ctx.side_stream != nullptr && p.chunk <= 4096;
  int32_t ahead_chunk_nnz = 1 << 17;
  if (ctx.ahead_min_nnz == 0) {
    const bool slowed =
        (p.chunk > 2048 && (p.M == 96 || p.M == 128)) || (p.chunk > 512 && p.M == 128 && nnz >= 27ll * n);
    ahead = ahead && nnz >= AHEAD_MIN_NNZ && chunks >= 64 && !slowed;
  } else {
    ahead = ahead && ctx.ahead_min_nnz > 0 && nnz >= ctx.ahead_min_nnz && chunks >= 2;
    ahead_chunk_nnz = 0;
  }
  CsgScratch s, sp;
  if (!plan_scratch(ctx, n, nnz, p, d_table, &s, 0, false, ahead ? &sp : nullptr)) return false;
  cudaStream_t st = ctx.stream;
  const bool zero_table = d_table != nullptr || stats != nullptr;

  if (timing) CSG_CUDA(cudaEventRecord(ctx.ev[0], st));
  // (a matrix without such a chunk goes on like any smaller call: mesh of 2 M rows, 64 slots 0.434 ms with both parts'
  // launches, 0.277 so; asking costs it 0.014)
  if (ahead && !launch_priority_pick(ctx, n, nnz, p.chunk, d_ptr, s, sp, ahead_chunk_nnz, &ahead)) return false;
  s.one_stream = sp.one_stream = !ahead;
  if (!ahead) {
    if (!launch_transpose(ctx, n, ncols, nnz, p.chunk, d_ptr, d_ind, s)) return false;
    if (timing) CSG_CUDA(cudaEventRecord(ctx.ev[1], st));
    if (!launch_sketch(ctx, n, nnz, p, d_ptr, s, row_base, zero_table)) return false;
  } else {
    auto two_parts = [&]() -> bool {
      if (zero_table)
        CSG_CUDA(cudaMemsetAsync(s.table, 0, sizeof(uint64_t) * static_cast<size_t>(n) * p.k, st));
      CSG_CUDA(cudaEventRecord(ctx.ev[5], st));
      CSG_CUDA(cudaStreamWaitEvent(ctx.side_stream, ctx.ev[5], 0));
      // the chunk ahead: queued first, so that the host's launches of the rest do not delay it; its chains as soon as
      // its lists say how much room their streams take
      if (!launch_transpose(ctx, n, ncols, nnz, p.chunk, d_ptr, d_ind, sp, PHASE_PRIO, s.ctrl)) return false;
      if (!launch_transpose(ctx, n, ncols, nnz, p.chunk, d_ptr, d_ind, s, PHASE_REST, sp.ctrl)) return false;
      if (!read_lists(ctx, sp, PHASE_PRIO)) return false;
      if (!sp.no_heavy_rows) {
        if (!launch_sketch(ctx, n, nnz, p, d_ptr, sp, row_base, false, PHASE_PRIO)) return false;
        s.stream_cap -= sp.stream_cap < s.stream_cap ? sp.stream_cap : s.stream_cap - 1;
        s.heavy_max = chain_rows_max(s.stream_cap, n);
      } else {
        CSG_CUDA(cudaEventRecord(ctx.ev[8], ctx.side_stream));
      }
      CSG_CUDA(cudaEventRecord(ctx.ev[7], ctx.side_stream));
      if (!launch_lists(ctx, n, p.chunk, s, sp.ctrl) || !read_lists(ctx, s, PHASE_REST)) return false;
      if (timing) CSG_CUDA(cudaEventRecord(ctx.ev[1], st));
      CSG_CUDA(cudaStreamWaitEvent(st, ctx.ev[8], 0));
      if (!launch_sketch(ctx, n, nnz, p, d_ptr, s, row_base, false, PHASE_REST)) return false;
      CSG_CUDA(cudaStreamWaitEvent(st, ctx.ev[7], 0));
      return true;
    };
    if (!two_parts()) {
      // a launch failed with the second stream forked and not joined: nothing of this call
      // may still be running when the next one reuses the workspace
      cudaStreamSynchronize(ctx.side_stream);
      cudaStreamSynchronize(st);
      return false;
    }
  }
  if (timing) CSG_CUDA(cudaEventRecord(ctx.ev[2], st));
  if (stats && !launch_table_stats(ctx, n, p.k, s.table, s.ctrl)) return false;
  if (timing) CSG_CUDA(cudaEventRecord(ctx.ev[3], st));
  if (d_new_order) {
    if (!launch_greedy(ctx, n, p, s, d_new_order, stats != nullptr, row_base)) return false;
  }
  if (timing) CSG_CUDA(cudaEventRecord(ctx.ev[4], st));
  ChainStatsHost hs;
  if (stats)
    CSG_CUDA(cudaMemcpyAsync(&hs, s.ctrl + CTRL_STATS, sizeof(hs), cudaMemcpyDeviceToHost, st));
  if (!finish_call(ctx, s, ahead ? &sp : nullptr)) return false;
  if (stats) {  // sporder/src/csg/stats_collector.cu:53-62
    stats->avg_degree = static_cast<double>(hs.total_degree) / n;
    stats->avg_edge_weight =
        hs.total_degree > 0 ? hs.total_weight / static_cast<double>(hs.total_degree) : 0.0;
    stats->zero_degree_rows = hs.zero_degree_rows;
    stats->chain_restarts = hs.restarts;
    stats->avg_followed_weight = hs.links > 0 ? hs.link_weight_sum / hs.links : 0.0;
  }
  if (timing) {
    CSG_CUDA(cudaEventElapsedTime(&timing->csr2csc_ms, ctx.ev[0], ctx.ev[1]));
    CSG_CUDA(cudaEventElapsedTime(&timing->similarity_ms, ctx.ev[1], ctx.ev[2]));
    CSG_CUDA(cudaEventElapsedTime(&timing->chunk_greedy_ms, ctx.ev[3], ctx.ev[4]));
    timing->wall_ms =
        std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - wall0).count();
  }
  return true;
}


// packed table -> separate arrays; an empty entry (0) reads as index -1, weight 0
// (sporder/src/similarity_graph.cu:13-23)
__global__ void __launch_bounds__(256) unpack_table_kernel(size_t count, const uint64_t *__restrict__ table,
                                                           int32_t *__restrict__ indices,
                                                           float *__restrict__ weights) {
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const uint64_t e = table[i];
    indices[i] = static_cast<int32_t>(static_cast<uint32_t>(e)) - 1;
    weights[i] = __uint_as_float(static_cast<uint32_t>(e >> 32));
  }
}

// The public top-k similarity graph (sporder/src/similarity_graph.cu:26-107,
// sporder/src/sporder.cpp:69-91): the same candidate stream, sketch and top-k selection as
// csg with the whole matrix as the one chunk (sporder/src/common/similarity_top_k.cu:10-51),
// other defaults (k = min(32, max(16, 2 nnz / n)), oversampling 2), results unpacked.
bool run_similarity_graph(Context &ctx, int32_t n, int32_t nnz, const int32_t *d_ptr, const int32_t *d_ind,
                          int32_t k, float ovs, int32_t *d_indices, float *d_weights,
                          sporder_sim_timing_t *timing, sporder_sim_stats_t *stats, int32_t *k_used) {
  const auto wall0 = std::chrono::steady_clock::now();
  CSG_REQUIRE(n >= 1, "n must be >= 1 (got %d)", n);
  CSG_REQUIRE(nnz >= 0, "nnz must be >= 0 (got %d)", nnz);
  if (k <= 0) {
    int32_t a = 2 * (nnz / n);
    if (a < 16) a = 16;
    if (a > 32) a = 32;
    k = a;
  }
  if (ovs <= 0.0f) ovs = 2.0f;
  CsgParams p;
  if (!resolve_params(n, nnz, k, ovs, n, &p)) return false;
  if (k_used) *k_used = p.k;
  if (stats) {
    std::memset(stats, 0, sizeof(*stats));
    stats->k_used = p.k;
    stats->m_used = p.m_used;
  }
  CSG_REQUIRE(d_ptr && (d_ind || nnz == 0), "null CSR arrays");
  CSG_REQUIRE(d_indices && d_weights, "null output arrays");
  CSG_CUDA(cudaSetDevice(ctx.device));
  CsgScratch s;
  if (!plan_scratch(ctx, n, nnz, p, nullptr, &s)) return false;
  cudaStream_t st = ctx.stream;
  if (timing) CSG_CUDA(cudaEventRecord(ctx.ev[0], st));
  if (!launch_transpose(ctx, n, n, nnz, p.chunk, d_ptr, d_ind, s)) return false;
  if (timing) CSG_CUDA(cudaEventRecord(ctx.ev[1], st));
  if (!launch_sketch(ctx, n, nnz, p, d_ptr, s, 0, true)) return false;
  if (timing) CSG_CUDA(cudaEventRecord(ctx.ev[2], st));
  if (stats && !launch_table_stats(ctx, n, p.k, s.table, s.ctrl)) return false;
  if (timing) CSG_CUDA(cudaEventRecord(ctx.ev[3], st));
  const size_t count = static_cast<size_t>(n) * p.k;
  size_t grid = (count + 255) / 256;
  if (grid > static_cast<size_t>(ctx.num_sms) * 16) grid = static_cast<size_t>(ctx.num_sms) * 16;
  unpack_table_kernel<<<static_cast<unsigned>(grid), 256, 0, st>>>(count, s.table, d_indices, d_weights);
  CSG_CUDA(cudaGetLastError());
  count_launches(1);
  if (timing) CSG_CUDA(cudaEventRecord(ctx.ev[4], st));
  ChainStatsHost hs;
  if (stats)
    CSG_CUDA(cudaMemcpyAsync(&hs, s.ctrl + CTRL_STATS, sizeof(hs), cudaMemcpyDeviceToHost, st));
  if (!finish_call(ctx, s)) return false;
  if (stats) {  // sporder/src/similarity_graph.cu:99-104
    stats->avg_degree = static_cast<double>(hs.total_degree) / n;
    stats->avg_edge_weight =
        hs.total_degree > 0 ? hs.total_weight / static_cast<double>(hs.total_degree) : 0.0;
    stats->zero_degree_rows = hs.zero_degree_rows;
  }
  if (timing) {
    CSG_CUDA(cudaEventElapsedTime(&timing->csr2csc_ms, ctx.ev[0], ctx.ev[1]));
    CSG_CUDA(cudaEventElapsedTime(&timing->similarity_ms, ctx.ev[1], ctx.ev[2]));
    CSG_CUDA(cudaEventElapsedTime(&timing->unpack_ms, ctx.ev[3], ctx.ev[4]));
    timing->wall_ms =
        std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - wall0).count();
  }
  return true;
}

// Chunked greedy on the global graph (sporder/src/cg/chunk_greedy.cu:118-163,
// sporder/src/sporder.cpp:112-138): the top-k graph of run_similarity_graph with the csg
// defaults (k = min(256, max(16, nnz / n)), oversampling 4), then the greedy chains inside
// chunks of chunk_size rows, candidates outside the chunk skipped.
bool run_chunk_greedy(Context &ctx, int32_t n, int32_t nnz, const int32_t *d_ptr, const int32_t *d_ind,
                      int32_t k, float ovs, int32_t chunk, int32_t *d_new_order,
                      sporder_cg_timing_t *timing, sporder_cg_stats_t *stats) {
  const auto wall0 = std::chrono::steady_clock::now();
  CsgParams pg;  // greedy: the caller's chunk; also resolves k and oversampling
  if (!resolve_params(n, nnz, k, ovs, chunk, &pg)) return false;
  CsgParams ps = pg;  // sketch: the whole matrix is the chunk
  ps.chunk = n;
  if (stats) {
    std::memset(stats, 0, sizeof(*stats));
    stats->k_used = pg.k;
    stats->m_used = pg.m_used;
    stats->chunk_size_used = pg.chunk;
  }
  CSG_REQUIRE(d_ptr && (d_ind || nnz == 0), "null CSR arrays");
  CSG_REQUIRE(d_new_order, "null d_new_order");
  CSG_CUDA(cudaSetDevice(ctx.device));
  CsgScratch s;
  if (!plan_scratch(ctx, n, nnz, ps, nullptr, &s, pg.chunk)) return false;
  cudaStream_t st = ctx.stream;
  if (timing) CSG_CUDA(cudaEventRecord(ctx.ev[0], st));
  if (!launch_transpose(ctx, n, n, nnz, ps.chunk, d_ptr, d_ind, s)) return false;
  if (timing) CSG_CUDA(cudaEventRecord(ctx.ev[1], st));
  if (!launch_sketch(ctx, n, nnz, ps, d_ptr, s, 0, stats != nullptr)) return false;
  if (timing) CSG_CUDA(cudaEventRecord(ctx.ev[2], st));
  if (stats) {
    if (!launch_table_stats(ctx, n, pg.k, s.table, s.ctrl)) return false;
    if (!launch_in_chunk_weight(ctx, n, pg.k, pg.chunk, s.table, s.ctrl)) return false;
  }
  if (timing) CSG_CUDA(cudaEventRecord(ctx.ev[3], st));
  if (!launch_greedy(ctx, n, pg, s, d_new_order, stats != nullptr, 0)) return false;
  if (timing) CSG_CUDA(cudaEventRecord(ctx.ev[4], st));
  ChainStatsHost hs;
  if (stats)
    CSG_CUDA(cudaMemcpyAsync(&hs, s.ctrl + CTRL_STATS, sizeof(hs), cudaMemcpyDeviceToHost, st));
  if (!finish_call(ctx, s)) return false;
  if (stats) {  // sporder/src/cg/stats_collector.cu:52-73
    stats->avg_degree = static_cast<double>(hs.total_degree) / n;
    stats->avg_edge_weight =
        hs.total_degree > 0 ? hs.total_weight / static_cast<double>(hs.total_degree) : 0.0;
    stats->zero_degree_rows = hs.zero_degree_rows;
    stats->chain_restarts = hs.restarts;
    stats->avg_followed_weight = hs.links > 0 ? hs.link_weight_sum / hs.links : 0.0;
    double cut = hs.total_weight > 0.0 ? 1.0 - hs.in_chunk_weight / hs.total_weight : 0.0;
    stats->cut_weight_fraction = cut < 0.0 ? 0.0 : (cut > 1.0 ? 1.0 : cut);
  }
  if (timing) {
    CSG_CUDA(cudaEventElapsedTime(&timing->csr2csc_ms, ctx.ev[0], ctx.ev[1]));
    CSG_CUDA(cudaEventElapsedTime(&timing->similarity_ms, ctx.ev[1], ctx.ev[2]));
    CSG_CUDA(cudaEventElapsedTime(&timing->chunk_greedy_ms, ctx.ev[3], ctx.ev[4]));
    timing->wall_ms =
        std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - wall0).count();
  }
  return true;
}

// Pillar count (sporder/src/count_pillars.cu:38-85): windows of up to 12 rows by searching
// the window's earlier rows, taller windows as the column groups of the chunk-local
// transpose with the window as the chunk.  Measured on the 65 M-nonzero R-MAT matrix the
// search costs 3 ms at height 1, 7 ms at 4 and 21 ms at 16, the transpose 26 ms at 8, 16 ms
// at 16 and 6 ms at 1024 (the reference's global key sort: 21-22 ms at every height).
constexpr int32_t PILLAR_SEARCH_ROWS = 12;

bool run_count_pillars(Context &ctx, int32_t n, int32_t nnz, const int32_t *d_ptr, const int32_t *d_ind,
                       int32_t height, int32_t *count) {
  CSG_REQUIRE(n >= 1, "n must be >= 1 (got %d)", n);
  CSG_REQUIRE(nnz >= 0, "nnz must be >= 0 (got %d)", nnz);
  CSG_REQUIRE(height >= 1, "height must be >= 1 (got %d)", height);
  CSG_REQUIRE(count, "null count");
  *count = 0;
  if (nnz == 0) return true;
  CSG_REQUIRE(d_ptr && d_ind, "null CSR arrays");
  CSG_CUDA(cudaSetDevice(ctx.device));
  unsigned long long *d_count = nullptr;
  uint32_t *d_bad = nullptr;
  if (height <= PILLAR_SEARCH_ROWS) {
    if (!ensure_workspace(ctx, 512)) return false;
    d_count = reinterpret_cast<unsigned long long *>(ctx.ws);
    d_bad = reinterpret_cast<uint32_t *>(ctx.ws + 256);
    CSG_CUDA(cudaMemsetAsync(ctx.ws, 0, 512, ctx.stream));
    if (!launch_pillars_search(ctx, n, nnz, height, d_ptr, d_ind, d_count, d_bad)) return false;
  } else {
    CsgParams p;
    if (!resolve_params(n, nnz, 1, 1.0f, height, &p)) return false;  // k = 1: smallest table the layout allows
    CsgScratch s;
    if (!plan_scratch(ctx, n, nnz, p, nullptr, &s, 0, true)) return false;
    // the counter takes the place of the (here unused) candidates
    d_count = reinterpret_cast<unsigned long long *>(s.cand);
    d_bad = s.ctrl + CTRL_BAD_INPUT;
    CSG_CUDA(cudaMemsetAsync(d_count, 0, sizeof(unsigned long long), ctx.stream));
    if (!launch_transpose(ctx, n, n, nnz, p.chunk, d_ptr, d_ind, s, PHASE_ALL, nullptr, d_count)) return false;
  }
  unsigned long long *h = reinterpret_cast<unsigned long long *>(ctx.h_pinned + 16);
  CSG_CUDA(cudaMemcpyAsync(h, d_count, sizeof(unsigned long long), cudaMemcpyDeviceToHost, ctx.stream));
  CSG_CUDA(cudaMemcpyAsync(ctx.h_pinned, d_bad, sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx.stream));
  CSG_CUDA(cudaStreamSynchronize(ctx.stream));
  CSG_REQUIRE(ctx.h_pinned[0] == 0,
              "malformed CSR: row pointers must be non-decreasing inside [0, nnz] (results unspecified)");
  *count = static_cast<int32_t>(*h);  // at most nnz
  return true;
}

}  // namespace
}  // namespace csg

struct sporder_context_struct {
  csg::Context c;
};

extern "C" {

sporder_context_t sporder_context_create(void) {
  csg::clear_error();
  auto *h = new sporder_context_struct;
  csg::Context &c = h->c;
  auto fail = [&](cudaError_t e, const char *what) {
    csg::set_error("context: %s -> %s", what, cudaGetErrorString(e));
    delete h;
    return static_cast<sporder_context_t>(nullptr);
  };
  cudaError_t e;
  if ((e = cudaGetDevice(&c.device)) != cudaSuccess) return fail(e, "cudaGetDevice");
  if ((e = cudaStreamCreateWithFlags(&c.own_stream, cudaStreamNonBlocking)) != cudaSuccess)
    return fail(e, "cudaStreamCreate");
  c.stream = c.own_stream;
  {  // the stream of the part of a large call that runs ahead: highest priority, so that its
     // small kernels are placed before the blocks of the grids on the main stream
    int least = 0, greatest = 0;
    if ((e = cudaDeviceGetStreamPriorityRange(&least, &greatest)) != cudaSuccess) return fail(e, "stream priorities");
    if ((e = cudaStreamCreateWithPriority(&c.side_stream, cudaStreamNonBlocking, greatest)) != cudaSuccess)
      return fail(e, "cudaStreamCreateWithPriority");
  }
  cudaDeviceGetAttribute(&c.num_sms, cudaDevAttrMultiProcessorCount, c.device);
  cudaDeviceGetAttribute(&c.smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c.device);
  for (auto &ev : c.ev)
    if ((e = cudaEventCreate(&ev)) != cudaSuccess) return fail(e, "cudaEventCreate");
  if ((e = cudaMallocHost(&c.h_pinned, 64 * sizeof(int))) != cudaSuccess)
    return fail(e, "cudaMallocHost");
  std::memset(c.h_pinned, 0, 64 * sizeof(int));
  return h;
}

void sporder_context_destroy(sporder_context_t h) {
  if (!h) return;
  csg::Context &c = h->c;
  cudaSetDevice(c.device);
  cudaStreamSynchronize(c.stream);
  if (c.side_stream) cudaStreamSynchronize(c.side_stream);
  if (c.ws) cudaFree(c.ws);
  for (int part = 0; part < 2; ++part) {
    if (c.chains[part]) cudaFree(c.chains[part]);
    if (c.outgrown[part]) cudaFree(c.outgrown[part]);
  }
  if (c.stage) cudaFree(c.stage);
  for (auto &ev : c.ev)
    if (ev) cudaEventDestroy(ev);
  if (c.h_pinned) cudaFreeHost(c.h_pinned);
  if (c.own_stream) cudaStreamDestroy(c.own_stream);
  if (c.side_stream) cudaStreamDestroy(c.side_stream);
  delete h;
}

void sporder_context_set_stream(sporder_context_t h, void *stream) {
  if (!h) return;
  cudaStream_t next = stream ? static_cast<cudaStream_t>(stream) : h->c.own_stream;  // see header
  // The workspace and its control words serve one stream at a time: work still queued on the
  // previous stream (sporder_spmm_async) must be over before another stream may reuse them.
  if (next != h->c.stream) cudaStreamSynchronize(h->c.stream);
  h->c.stream = next;
}

void sporder_context_set_ahead_threshold(sporder_context_t h, int64_t min_nnz) {
  if (h) h->c.ahead_min_nnz = min_nnz;
}

void sporder_context_set_stream_limit(sporder_context_t h, uint64_t max_elements) {
  if (h) h->c.stream_limit = max_elements;
}

void sporder_context_set_chain_threshold(sporder_context_t h, uint32_t min_candidates) {
  if (h) h->c.chain_min_work = min_candidates;
}

uint64_t sporder_context_chain_rows(sporder_context_t h) { return h ? h->c.chain_rows : 0; }

uint64_t sporder_context_workspace_bytes(sporder_context_t h) {
  return h ? h->c.ws_bytes + h->c.chains_bytes[0] + h->c.chains_bytes[1] : 0;
}

const char *sporder_last_error(void) { return csg::g_has_err ? csg::g_err : nullptr; }

uint64_t sporder_kernel_launches(void) { return csg::g_launches.load(); }

void sporder_chunk_similarity_greedy(sporder_context_t ctx, int32_t n, int32_t nnz,
                                     const int32_t *d_ptr, const int32_t *d_ind, bool is_symmetric,
                                     int32_t k, float oversampling, int32_t chunk_size,
                                     int32_t *d_new_order, sporder_csg_timing_t *timing,
                                     sporder_csg_stats_t *stats) {
  csg::clear_error();
  if (!ctx) {
    csg::set_error("null context");
    return;
  }
  if (!d_new_order) {
    csg::set_error("null d_new_order");
    return;
  }
  csg::run_csg(ctx->c, n, n, 0, nnz, d_ptr, d_ind, k, oversampling, chunk_size, d_new_order, nullptr, 0,
               timing, stats, nullptr);
}

int32_t sporder_csg_with_table(sporder_context_t ctx, int32_t n, int32_t nnz, const int32_t *d_ptr,
                               const int32_t *d_ind, bool is_symmetric, int32_t k,
                               float oversampling, int32_t chunk_size, int32_t *d_new_order,
                               uint64_t *d_table, uint64_t d_table_capacity,
                               sporder_csg_timing_t *timing, sporder_csg_stats_t *stats) {
  csg::clear_error();
  if (!ctx) {
    csg::set_error("null context");
    return -1;
  }
  int32_t k_used = -1;
  if (!csg::run_csg(ctx->c, n, n, 0, nnz, d_ptr, d_ind, k, oversampling, chunk_size, d_new_order, d_table,
                    d_table_capacity, timing, stats, &k_used))
    return -1;
  return k_used;
}

int32_t sporder_csg_shard(sporder_context_t ctx, int32_t n_rows, int32_t n_cols, int32_t row_base,
                          int32_t nnz, const int32_t *d_ptr, const int32_t *d_ind, int32_t k,
                          float oversampling, int32_t chunk_size, int32_t *d_new_order,
                          uint64_t *d_table, uint64_t d_table_capacity,
                          sporder_csg_timing_t *timing, sporder_csg_stats_t *stats) {
  csg::clear_error();
  if (!ctx) {
    csg::set_error("null context");
    return -1;
  }
  int32_t k_used = -1;
  if (!csg::run_csg(ctx->c, n_rows, n_cols, row_base, nnz, d_ptr, d_ind, k, oversampling,
                    chunk_size, d_new_order, d_table, d_table_capacity, timing, stats, &k_used))
    return -1;
  return k_used;
}

int32_t sporder_chunk_similarity_greedy_host(sporder_context_t ctx, int32_t n, int32_t nnz,
                                             const int32_t *h_ptr, const int32_t *h_ind,
                                             bool is_symmetric, int32_t k, float oversampling,
                                             int32_t chunk_size, int32_t *h_new_order,
                                             sporder_csg_timing_t *timing,
                                             sporder_csg_stats_t *stats) {
  csg::clear_error();
  if (!ctx || !h_ptr || !h_new_order || n < 1 || nnz < 0) {
    csg::set_error("csg_host: bad arguments");
    return -1;
  }
  csg::Context &c = ctx->c;
  auto run = [&]() -> bool {
    CSG_CUDA(cudaSetDevice(c.device));
    // Device copies of the inputs and the result live in a buffer of the context that only
    // grows: a stream-ordered allocation per call went back to the driver at every
    // synchronisation and cost more than the reorder itself.
    const size_t b_ptr = (sizeof(int32_t) * (static_cast<size_t>(n) + 1) + 255) & ~size_t(255);
    const size_t b_ind = (sizeof(int32_t) * static_cast<size_t>(nnz > 0 ? nnz : 1) + 255) & ~size_t(255);
    const size_t b_ord = sizeof(int32_t) * static_cast<size_t>(n);
    if (b_ptr + b_ind + b_ord > c.stage_bytes) {
      CSG_CUDA(cudaStreamSynchronize(c.stream));
      if (c.stage) CSG_CUDA(cudaFree(c.stage));
      c.stage = nullptr;
      c.stage_bytes = 0;
      CSG_CUDA(cudaMalloc(&c.stage, b_ptr + b_ind + b_ord));
      c.stage_bytes = b_ptr + b_ind + b_ord;
    }
    int32_t *d_ptr = reinterpret_cast<int32_t *>(c.stage);
    int32_t *d_ind = reinterpret_cast<int32_t *>(c.stage + b_ptr);
    int32_t *d_order = reinterpret_cast<int32_t *>(c.stage + b_ptr + b_ind);
    CSG_CUDA(cudaMemcpyAsync(d_ptr, h_ptr, sizeof(int32_t) * (static_cast<size_t>(n) + 1),
                             cudaMemcpyHostToDevice, c.stream));
    if (nnz > 0)
      CSG_CUDA(cudaMemcpyAsync(d_ind, h_ind, sizeof(int32_t) * static_cast<size_t>(nnz),
                               cudaMemcpyHostToDevice, c.stream));
    const bool ok = csg::run_csg(c, n, n, 0, nnz, d_ptr, d_ind, k, oversampling, chunk_size, d_order,
                                 nullptr, 0, timing, stats, nullptr);
    if (ok)
      CSG_CUDA(cudaMemcpyAsync(h_new_order, d_order, sizeof(int32_t) * static_cast<size_t>(n),
                               cudaMemcpyDeviceToHost, c.stream));
    CSG_CUDA(cudaStreamSynchronize(c.stream));
    return ok;
  };
  return run() ? 0 : -1;
}

void sporder_chunk_greedy(sporder_context_t ctx, int32_t n, int32_t nnz, const int32_t *d_ptr,
                          const int32_t *d_ind, bool is_symmetric, int32_t k, float oversampling,
                          int32_t chunk_size, int32_t *d_new_order, sporder_cg_timing_t *timing,
                          sporder_cg_stats_t *stats) {
  csg::clear_error();
  if (!ctx) {
    csg::set_error("null context");
    return;
  }
  csg::run_chunk_greedy(ctx->c, n, nnz, d_ptr, d_ind, k, oversampling, chunk_size, d_new_order, timing,
                        stats);
}

int32_t sporder_similarity_graph(sporder_context_t ctx, int32_t n, int32_t nnz, const int32_t *d_ptr,
                                 const int32_t *d_ind, bool is_symmetric, int32_t k, float oversampling,
                                 int32_t *d_indices, float *d_weights, sporder_sim_timing_t *timing,
                                 sporder_sim_stats_t *stats) {
  csg::clear_error();
  if (!ctx) {
    csg::set_error("null context");
    return -1;
  }
  int32_t k_used = -1;
  if (!csg::run_similarity_graph(ctx->c, n, nnz, d_ptr, d_ind, k, oversampling, d_indices, d_weights,
                                 timing, stats, &k_used))
    return -1;
  return k_used;
}

void sporder_count_pillars(sporder_context_t ctx, int32_t n, int32_t nnz, const int32_t *d_ptr,
                           const int32_t *d_ind, int32_t height, int32_t *count) {
  csg::clear_error();
  if (!ctx) {
    csg::set_error("null context");
    return;
  }
  csg::run_count_pillars(ctx->c, n, nnz, d_ptr, d_ind, height, count);
}

void sporder_reorder(sporder_context_t ctx, int32_t n, int32_t nnz, const int32_t *d_ptr_old,
                     const int32_t *d_ind_old, const float *d_val_old, const int32_t *d_new_order,
                     sporder_reorder_mode_t mode, int32_t *d_ptr_new, int32_t *d_ind_new,
                     float *d_val_new) {
  csg::clear_error();
  if (!ctx) {
    csg::set_error("null context");
    return;
  }
  if (mode != SPORDER_REORDER_ROWS && mode != SPORDER_REORDER_SYMMETRIC) {
    csg::set_error("invalid reorder mode");
    return;
  }
  if (n < 1 || nnz < 0 || !d_ptr_old || !d_new_order || !d_ptr_new || (nnz > 0 && (!d_ind_old || !d_ind_new))) {
    csg::set_error("reorder: bad arguments");
    return;
  }
  csg::Context &c = ctx->c;
  auto run = [&]() -> bool {
    CSG_CUDA(cudaSetDevice(c.device));
    if (!csg::launch_reorder(c, n, nnz, d_ptr_old, d_ind_old, d_val_old, d_new_order,
                             static_cast<int>(mode), d_ptr_new, d_ind_new, d_val_new))
      return false;
    CSG_CUDA(cudaStreamSynchronize(c.stream));
    CSG_CUDA(cudaGetLastError());
    return true;
  };
  run();
}

static int32_t spmm_impl(sporder_context_t ctx, int32_t n, int32_t nnz, int32_t w,
                         const int32_t *d_ptr, const int32_t *d_ind, const float *d_val,
                         const float *d_B, float *d_C, bool sync) {
  csg::clear_error();
  if (!ctx || n < 1 || nnz < 0 || !d_ptr || !d_B || !d_C || (nnz > 0 && (!d_ind || !d_val))) {
    csg::set_error("spmm: bad arguments");
    return -1;
  }
  csg::Context &c = ctx->c;
  auto run = [&]() -> bool {
    CSG_CUDA(cudaSetDevice(c.device));
    if (!csg::launch_spmm(c, n, nnz, w, d_ptr, d_ind, d_val, d_B, d_C)) return false;
    if (sync) {
      CSG_CUDA(cudaStreamSynchronize(c.stream));
      CSG_CUDA(cudaGetLastError());
    }
    return true;
  };
  return run() ? 0 : -1;
}

int32_t sporder_spmm(sporder_context_t ctx, int32_t n, int32_t nnz, int32_t w, const int32_t *d_ptr,
                     const int32_t *d_ind, const float *d_val, const float *d_B, float *d_C) {
  return spmm_impl(ctx, n, nnz, w, d_ptr, d_ind, d_val, d_B, d_C, true);
}

int32_t sporder_spmm_async(sporder_context_t ctx, int32_t n, int32_t nnz, int32_t w,
                           const int32_t *d_ptr, const int32_t *d_ind, const float *d_val,
                           const float *d_B, float *d_C) {
  return spmm_impl(ctx, n, nnz, w, d_ptr, d_ind, d_val, d_B, d_C, false);
}

int32_t sporder_row_sums(sporder_context_t ctx, int32_t n, int32_t nnz, const int32_t *d_ptr, const float *d_val,
                         float *d_out) {
  csg::clear_error();
  if (!ctx || n < 1 || nnz < 0 || !d_ptr || !d_out || (nnz > 0 && !d_val)) {
    csg::set_error("row_sums: bad arguments");
    return -1;
  }
  return csg::launch_row_sums(ctx->c, n, nnz, d_ptr, d_val, d_out) ? 0 : -1;
}

int32_t sporder_linear(sporder_context_t ctx, int32_t n, int32_t in_dim, int32_t out_dim, const float *d_x,
                       const float *d_W, const float *d_b, float *d_Y) {
  csg::clear_error();
  if (!ctx || !d_x || !d_W || !d_b || !d_Y) {
    csg::set_error("linear: bad arguments");
    return -1;
  }
  return csg::launch_linear(ctx->c, n, in_dim, out_dim, d_x, d_W, d_b, d_Y) ? 0 : -1;
}

int32_t sporder_gcn_forward_padded(sporder_context_t ctx, int32_t n, int32_t hidden, int32_t classes, int32_t columns,
                                   const float *d_Z, const float *d_W2, float *d_U) {
  csg::clear_error();
  if (!ctx || !d_Z || !d_W2 || !d_U) {
    csg::set_error("gcn_forward: bad arguments");
    return -1;
  }
  return csg::launch_gcn_forward(ctx->c, n, hidden, classes, columns, d_Z, d_W2, d_U) ? 0 : -1;
}

int32_t sporder_gcn_forward(sporder_context_t ctx, int32_t n, int32_t hidden, int32_t classes, const float *d_Z,
                            const float *d_W2, float *d_U) {
  return sporder_gcn_forward_padded(ctx, n, hidden, classes, classes, d_Z, d_W2, d_U);
}

int32_t sporder_gcn_backward_padded(sporder_context_t ctx, int32_t n, int32_t in_dim, int32_t hidden, int32_t classes,
                                    int32_t columns, const float *d_G, const float *d_Z, const float *d_P,
                                    const float *d_s, const float *d_W2, float *d_dW1, float *d_db1, float *d_dW2) {
  csg::clear_error();
  if (!ctx || !d_G || !d_Z || !d_P || !d_s || !d_W2 || !d_dW1 || !d_db1 || !d_dW2) {
    csg::set_error("gcn_backward: bad arguments");
    return -1;
  }
  return csg::launch_gcn_backward(ctx->c, n, in_dim, hidden, classes, columns, d_G, d_Z, d_P, d_s, d_W2, d_dW1, d_db1,
                                  d_dW2) ? 0 : -1;
}

int32_t sporder_gcn_backward(sporder_context_t ctx, int32_t n, int32_t in_dim, int32_t hidden, int32_t classes,
                             const float *d_G, const float *d_Z, const float *d_P, const float *d_s,
                             const float *d_W2, float *d_dW1, float *d_db1, float *d_dW2) {
  return sporder_gcn_backward_padded(ctx, n, in_dim, hidden, classes, classes, d_G, d_Z, d_P, d_s, d_W2, d_dW1, d_db1,
                                     d_dW2);
}

int32_t sporder_gcn_hidden_gradient(sporder_context_t ctx, int32_t n, int32_t hidden, int32_t classes, int32_t columns,
                                    const float *d_G, const float *d_Z, const float *d_W2, float *d_D, float *d_dW2) {
  csg::clear_error();
  if (!ctx || !d_G || !d_Z || !d_W2 || !d_D || !d_dW2) {
    csg::set_error("gcn_hidden_gradient: bad arguments");
    return -1;
  }
  return csg::launch_gcn_hidden_gradient(ctx->c, n, hidden, classes, columns, d_G, d_Z, d_W2, d_D, d_dW2) ? 0 : -1;
}

int32_t sporder_pad_columns(sporder_context_t ctx, int32_t n, int32_t from, int32_t to, const float *d_src, float *d_dst) {
  csg::clear_error();
  if (!ctx || !d_src || !d_dst) {
    csg::set_error("pad_columns: bad arguments");
    return -1;
  }
  return csg::launch_pad_columns(ctx->c, n, from, to, d_src, d_dst) ? 0 : -1;
}

int32_t sporder_gcn_input_gradients(sporder_context_t ctx, int32_t n, int32_t in_dim, int32_t hidden, const float *d_E,
                                    const float *d_x, float *d_dW1, float *d_db1) {
  csg::clear_error();
  if (!ctx || !d_E || !d_x || !d_dW1 || !d_db1) {
    csg::set_error("gcn_input_gradients: bad arguments");
    return -1;
  }
  return csg::launch_gcn_input_gradients(ctx->c, n, in_dim, hidden, d_E, d_x, d_dW1, d_db1) ? 0 : -1;
}

}  // extern "C"
