// Shared declarations of the B200 csg library: context, error channel,
// workspace arena and the launch functions of each stage.
#pragma once
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>

namespace csg {

// ---- error channel -------------------------------------------------------
// The reference aborts the process on invalid arguments and CUDA errors
// (sporder/src/common/error_checking.h:20-29).  On a shared GPU pool this
// library records the message per thread and returns instead.
void set_error(const char *fmt, ...);
bool has_error();
void clear_error();
void count_launches(int k);  // feeds sporder_kernel_launches()

#define CSG_CUDA(call)                                                                  \
  do {                                                                                  \
    cudaError_t e__ = (call);                                                           \
    if (e__ != cudaSuccess) {                                                           \
      ::csg::set_error("%s:%d: %s -> %s", __FILE__, __LINE__, #call,                    \
                       cudaGetErrorString(e__));                                        \
      return false;                                                                     \
    }                                                                                   \
  } while (0)

#define CSG_REQUIRE(cond, ...)                                                          \
  do {                                                                                  \
    if (!(cond)) {                                                                      \
      ::csg::set_error(__VA_ARGS__);                                                    \
      return false;                                                                     \
    }                                                                                   \
  } while (0)

// ---- context ---------------------------------------------------------------
// Counterpart of sporder::context (sporder/src/common/context.h:67-197): one
// stream, the device it was created on, and a grow-only device workspace so a
// warm call allocates nothing.
struct Context {
  int device = 0;
  cudaStream_t stream = nullptr;  // stream every launch of this context uses
  cudaStream_t own_stream = nullptr;
  int num_sms = 0;
  int smem_optin = 0;  // max dynamic shared memory per block (opt-in)
  char *ws = nullptr;  // device workspace
  size_t ws_bytes = 0;
  cudaEvent_t ev[10] = {};  // [0..4] stage times; [5..8] fork, joins and order of a call that runs one chunk ahead
  int *h_pinned = nullptr;  // small pinned host buffer for counters (64 ints)
  uint32_t outcome_ticket = 0;  // the newest one handed to a kernel (see OUTCOME_WORD)
  char *stage = nullptr;    // device copies of host inputs (host-buffer entry point), kept between calls
  size_t stage_bytes = 0;
  // Buffers for the chains of the heaviest rows (sketch.cu): their materialised candidate streams, sketches and lists
  // of parts; [1] for the part of a call that runs ahead.  Grown to what the call's own rows need, which the host learns
  // between the transposition and the sketch (plan_chains), so a call without such rows holds none.
  char *chains[2] = {};
  size_t chains_bytes[2] = {};
  char *outgrown[2] = {};  // buffers a call replaced while kernels may run: freed when it ends
  // Second stream (higher priority) for the part of a large call that runs ahead of the rest:
  // the transposition and the chains of the chunk that holds the most nonzeros (see run_csg).
  cudaStream_t side_stream = nullptr;
  // nonzeros from which a call runs one chunk ahead: 0 = the built-in threshold, negative =
  // never, positive = the caller's threshold (sporder_context_set_ahead_threshold)
  int64_t ahead_min_nnz = 0;
  uint64_t stream_limit = 0;       // caller's upper bound (sporder_context_set_stream_limit), 0 = none
  uint32_t chain_min_work = 0;     // rows from so many candidates on get a chain, 0 = as their costs say
  uint64_t chain_rows = 0;         // rows that got one in the last call
};

// In h_pinned, written by the device: a ticket, then what a kernel found out that decides about the
// launches behind it; the second place is that of the part that runs ahead.  wait_outcome returns once the ticket is there.
constexpr int OUTCOME_WORD = 48, OUTCOME_WORD_PRIO = 56;
inline volatile uint32_t *outcome_words(Context &ctx, int word) {
  return reinterpret_cast<volatile uint32_t *>(ctx.h_pinned) + word;
}
bool wait_outcome(Context &ctx, cudaStream_t st, int word, uint32_t ticket);

bool ensure_workspace(Context &ctx, size_t bytes);

// Bump allocator over the context workspace (256-byte aligned blocks).
struct Arena {
  size_t off = 0;
  size_t take(size_t bytes) {
    size_t o = off;
    off += (bytes + 255) & ~size_t(255);
    return o;
  }
};

// ---- resolved csg parameters (sporder/src/sporder.cpp:147-161) ---------------
struct CsgParams {
  int32_t k;
  float ovs;
  int32_t chunk;
  int32_t m_used;  // value the stats struct reports
  int32_t M;       // sketch capacity actually used (multiple of 32, <= 512)
};
bool resolve_params(int32_t n, int32_t nnz, int32_t k, float ovs, int32_t chunk, CsgParams *out);

// ---- device scratch of one csg call -------------------------------------------
struct CsgScratch {
  // chunk-local transpose (see transpose.cu)
  uint32_t *keyA, *keyB, *payA, *payB;  // ping-pong buffers of the global sort path
  int2 *cand;                           // (row, row length) grouped by (chunk, column), rows ascending
  int2 *seg;                            // per row and shared column: (first index into cand, group length)
  int32_t *seg_rank;                    // ... and the place of the row itself inside that group
  int32_t *row_seg, *row_cols;          // per row: its first entry of seg, and how many
  uint32_t *row_work;                   // candidates each row will see
  // work list of rows with candidates, heaviest bucket first
  int32_t *row_list;
  uint32_t *ctrl;  // [0]=chunk ticket [1]=row ticket [2]=rows listed [3..] see CTRL_* below
  uint64_t *table;  // n*k packed top-k entries
  uint32_t *gbitmaps;  // greedy bitmaps when they do not fit shared memory, else nullptr
  // materialised candidate streams of the heaviest rows (see sketch.cu): what they may take, what the lists asked for,
  // and from plan_chains on the buffers and what they hold
  uint32_t stream_cap, heavy_max;
  uint32_t chain_rows = 0;
  uint64_t chain_need = 0;
  int2 *hstream = nullptr;
  uint32_t *heavy_off = nullptr;
  int32_t *heavy_state = nullptr;
  uint32_t *part_base = nullptr, *part_off = nullptr;
  int32_t slots;  // of a row's sketch
  uint32_t ticket = 0;  // of the lists' outcome
  bool no_heavy_rows = false;  // known on the host already: nothing for the chain kernel
  bool one_stream = true;      // the call runs on one stream: its kernels may be programmatic dependent launches
  // compact_kernel's second list, tiled sort of heavy chunks (see transpose.cu)
  int32_t *next_chunk, *heavy_chunk, *heavy_tile_base;
  uint32_t *tile_hist, *digit_base;
};
enum {
  CTRL_CHUNK_TICKET = 0,
  CTRL_ROW_TICKET = 1,
  CTRL_ROWS_LISTED = 2,
  CTRL_BAD_INPUT = 3,      // set by a kernel that met row pointers outside [0, nnz]
  CTRL_HEAVY_COUNT = 4,    // chunks sorted by the tiled path
  CTRL_HEAVY_TILES = 5,    // their tiles
  CTRL_HEAVY_ROWS = 6,     // rows at the head of row_list that the heavy sketch kernel takes
  CTRL_HEAVY_TICKET = 7,   // and the word after it: a second ticket
  CTRL_HEAVY_PARTS = 9,    // column slices of the heavy rows
  CTRL_STREAM_OVERRUN = 12,  // set by heavy_expand_kernel when a slice would pass the stream buffer
  CTRL_CHECK = 13,         // checked build: site of the first index out of bounds, then the index (64-bit)
  CTRL_MID_END = 16,       // end of the rows in row_list that are not run by a lane (those past CTRL_HEAVY_ROWS: by a warp)
  CTRL_LANE_TICKET = 17,   // next row for the kernel that runs a row per lane
  CTRL_NEXT_COUNT = 18,    // chunks compact_kernel's small form left to the large one, and that one's ticket
  CTRL_NEXT_TICKET = 19,
  CTRL_PRIO = 50,          // chunk whose heavy rows run ahead of the rest (PRIO_NONE: no such chunk)
  CTRL_PRIO_WORK = 51,     // shortest candidate stream among the rows the chunk ahead lists
  CTRL_STATS = 56,         // see greedy.cu (8-byte aligned)
  CTRL_BUCKET_COUNT = 128,  // WORK_BUCKETS entries each: rows,
  CTRL_BUCKET_WORK = 256,   // their candidates (64-bit),
  CTRL_BUCKET_BASE = 512,   // first place in the list, places taken
  CTRL_BUCKET_FILL = 640,
  CTRL_WORDS = 768
};

// Rows are listed by the length of their candidate stream, in quarter octaves (bucket 4 e + f
// holds the lengths in [2^e (1 + f/4), 2^e (1 + (f+1)/4)), longest bucket first): 32 consecutive
// rows of the list, one per lane of a warp (sketch.cu), then differ by a quarter at most.
constexpr int WORK_BUCKETS = 128;

constexpr uint32_t PRIO_NONE = 0xFFFFFFFFu;
// phases of a call that runs one chunk ahead: everything (no such split), the chunk ahead, the rest
enum CallPhase { PHASE_ALL = 0, PHASE_PRIO = 1, PHASE_REST = 2 };
// SMs the chains of the chunk ahead may hold (the other chains get the remaining ones)
inline int prio_chain_blocks(int num_sms) { return num_sms / 4 > 0 ? num_sms / 4 : 1; }

constexpr uint64_t STREAM_CAP_MAX = uint64_t(1) << 28;  // largest stream buffer: 2^28 elements = 2 GiB
constexpr int SKETCH_PART_COLS = 128;   // columns of a heavy row whose stream one warp writes out
// Rows that stream at least HEAVY_WORK candidates are "heavy": a group of warps of the chain kernel each.
// Shorter rows of CHAIN_WORK_MIN candidates or more join them, longest first, up to CHAIN_ROWS rows: as many as the
// times of ChainCosts say (bucket_scan_kernel), in sketches without such times while there are FEW_CHAIN_ROWS.
constexpr uint32_t HEAVY_WORK = 1u << 16;
constexpr uint32_t CHAIN_ROWS = 4096;
constexpr uint32_t FEW_CHAIN_ROWS = 296;
constexpr uint32_t CHAIN_WORK_MIN = 64;
constexpr int32_t LANE_TABLE_ROWS = 1024;  // largest chunk whose keys the row-per-lane kernel finds in a byte table
// Larger chunks: rows of at least this many candidates and in the longest octaves go to a warp each, more octaves
// up to this many rows (bucket_scan_kernel)
constexpr uint32_t WARP_WORK_MIN = 1024;
constexpr int32_t WARP_FEW_ROWS = 32768;

// stage launchers; all enqueue on ctx.stream and return false after set_error()
bool launch_transpose(Context &ctx, int32_t n, int32_t ncols, int32_t nnz, int32_t chunk, const int32_t *d_ptr,
                      const int32_t *d_ind, CsgScratch &s, int phase = PHASE_ALL, uint32_t *ctrl_other = nullptr,
                      unsigned long long *d_count = nullptr);
// work lists of the rows with candidates (part of launch_transpose but in a call that runs one chunk ahead)
bool launch_lists(Context &ctx, int32_t n, int32_t chunk, CsgScratch &s, const uint32_t *ctrl_ahead);
// waits for what the lists say about the call's longest rows: s.chain_rows, s.chain_need, s.no_heavy_rows
bool read_lists(Context &ctx, CsgScratch &s, int phase);
// rows a block of the chain kernel (one to an SM) works on side by side; 0 beyond the slots that are resolved in rounds
int chain_groups(const Context &ctx, int slots, int64_t span);
// buffers for the chains of the listed rows, no larger than they need; fewer chains where memory is short
bool plan_chains(Context &ctx, int32_t nnz, CsgScratch &s, int phase);
// start of a call that runs one chunk ahead: clears the counters of both parts and names the chunk, if there is one (on)
bool launch_priority_pick(Context &ctx, int32_t n, int32_t nnz, int32_t chunk, const int32_t *d_ptr,
                          CsgScratch &s, CsgScratch &prio, int32_t min_chunk_nnz, bool *on);
bool launch_sketch(Context &ctx, int32_t n, int32_t nnz, const CsgParams &p, const int32_t *d_ptr,
                   CsgScratch &s, int32_t row_base, bool zero_table, int phase = PHASE_ALL);
bool launch_greedy(Context &ctx, int32_t n, const CsgParams &p, CsgScratch &s,
                   int32_t *d_new_order, bool with_stats, int32_t row_base);
bool launch_pillars_search(Context &ctx, int32_t n, int32_t nnz, int32_t height, const int32_t *d_ptr,
                           const int32_t *d_ind, unsigned long long *d_count, uint32_t *d_bad);
bool launch_in_chunk_weight(Context &ctx, int32_t n, int32_t k, int32_t chunk, const uint64_t *table,
                            uint32_t *ctrl);
bool launch_table_stats(Context &ctx, int32_t n, int32_t k, const uint64_t *table, uint32_t *ctrl);

bool launch_reorder(Context &ctx, int32_t n, int32_t nnz, const int32_t *d_ptr_old,
                    const int32_t *d_ind_old, const float *d_val_old, const int32_t *d_new_order,
                    int mode, int32_t *d_ptr_new, int32_t *d_ind_new, float *d_val_new);

bool launch_spmm(Context &ctx, int32_t n, int32_t nnz, int32_t w, const int32_t *d_ptr,
                 const int32_t *d_ind, const float *d_val, const float *d_B, float *d_C);

bool launch_gcn_forward(Context &ctx, int32_t n, int32_t hid, int32_t cls, int32_t ld, const float *Z, const float *W2,
                        float *U);
bool launch_gcn_backward(Context &ctx, int32_t n, int32_t in, int32_t hid, int32_t cls, int32_t ld, const float *G,
                         const float *Z, const float *P, const float *s, const float *W2, float *dW1, float *db1, float *dW2);
bool launch_gcn_hidden_gradient(Context &ctx, int32_t n, int32_t hid, int32_t cls, int32_t ld, const float *G,
                                const float *Z, const float *W2, float *D, float *dW2);
bool launch_pad_columns(Context &ctx, int32_t n, int32_t from, int32_t to, const float *src, float *dst);
bool launch_gcn_input_gradients(Context &ctx, int32_t n, int32_t in, int32_t hid, const float *E, const float *x,
                                float *dW1, float *db1);
bool launch_linear(Context &ctx, int32_t n, int32_t in, int32_t hid, const float *x, const float *W, const float *b, float *Y);
bool launch_row_sums(Context &ctx, int32_t n, int32_t nnz, const int32_t *d_ptr, const float *d_val, float *d_out);

// ---- small device helpers -------------------------------------------------------
#ifdef __CUDACC__
constexpr unsigned FULL = 0xFFFFFFFFu;
__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

// Programmatic dependent launches: the blocks of a kernel may be placed while the kernel in front of it in its stream
// still runs, once all of that one's blocks run or are through.  Such a kernel waits before it touches anything an
// earlier one of the call writes; each of them waits, so that the end of one means the end of all before it.
// Nothing an earlier kernel of the call writes may be read through a pointer to const that is __restrict__, or by
// __ldg: both promise that the memory stays the same for as long as the kernel runs, the time before the wait included,
// and the load may go through the read-only path or in front of the wait.  The caller's own arrays may.
__device__ __forceinline__ void wait_for_kernels_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_kernel_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---- checked build ----------------------------------------------------------------------
// Compiled with -DSPORDER_CHECKED (python -m chunkedgreedy_b200.build --checked) every index
// that a kernel derives from data another kernel wrote - positions in the transposed chunk,
// stream offsets, table slots, list entries - is tested before use; the first one out of
// bounds is recorded (site, index) and the access is skipped, so the kernel runs on with
// harmless values and the host reports the site instead of the GPU faulting.  This stands in
// for compute-sanitizer on machines where that tool may not be run.  In the normal build the
// test is a constant `true` and costs nothing.
enum CheckSite : uint32_t {
  CHK_CAND = 1,      // cand[] index from a group descriptor
  CHK_RING = 2,      // position in a warp's stream ring
  CHK_STREAM = 3,    // hstream[] offset of a heavy row
  CHK_KEY = 4,       // stream key outside its chunk (key -> slot table)
  CHK_STATE = 5,     // heavy_state[] / heavy_off[] item
  CHK_TABLE = 6,     // row of the top-k table
  CHK_LIST = 7,      // row_list[] entry
  CHK_ORDER = 8,     // order[] position in the greedy stage
  CHK_SORT = 9,      // scatter position of a radix pass
  CHK_GROUP = 10,    // group start / position written by the transpose
  CHK_PART = 11,     // part_off[] / part_base[] entry
};
#ifdef SPORDER_CHECKED
__device__ __forceinline__ bool index_ok(uint32_t *ctrl, uint32_t site, long long idx, long long bound) {
  if (idx >= 0 && idx < bound) return true;
  if (atomicCAS(&ctrl[CTRL_CHECK], 0u, site) == 0u) {
    ctrl[CTRL_CHECK + 1] = static_cast<uint32_t>(static_cast<unsigned long long>(idx));
    ctrl[CTRL_CHECK + 2] = static_cast<uint32_t>(static_cast<unsigned long long>(idx) >> 32);
  }
  return false;
}
#else
__device__ __forceinline__ bool index_ok(uint32_t *, uint32_t, long long, long long) { return true; }
#endif

// counter += v, sticking at 0xFFFFFFFF instead of wrapping.  Whoever sees the sum wrap puts
// the ceiling back; the last operation on a counter that ever wrapped is such a repair, so
// once all adders are done the counter reads 0xFFFFFFFF ("more than fits").
__device__ __forceinline__ void saturating_add(uint32_t *counter, uint32_t v) {
  const uint32_t old = atomicAdd(counter, v);
  if (old + v < old) atomicMax(counter, 0xFFFFFFFFu);
}

// Lanes of the warp whose 8-bit digit equals this lane's (d in [0, 255]; lanes that pass
// d = 256 take no part and get their own bit).  Eight ballots and eight selects: match.any, the
// instruction made for this, measures some 380 cycles per call on this part with a lone warp,
// this sequence about 80.
__device__ __forceinline__ unsigned match_digit(uint32_t d) {
  unsigned peers = __ballot_sync(FULL, d < 256u);
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const unsigned has = __ballot_sync(FULL, (d >> b) & 1u);
    peers &= ((d >> b) & 1u) ? has : ~has;
  }
  return d < 256u ? peers : 1u << (threadIdx.x & 31);
}

// bucket of a row that streams t >= 1 candidates
__device__ __forceinline__ int work_bucket(uint32_t t) {
  const int e = 31 - __clz(t);
  return 4 * e + static_cast<int>((e >= 2 ? t >> (e - 2) : t << (2 - e)) & 3u);
}

// least length that falls into bucket b (from 8 candidates on)
__device__ __forceinline__ float bucket_floor(int b) {
  return static_cast<float>(1ull << (b >> 2)) * (1.0f + 0.25f * static_cast<float>(b & 3));
}

// packed entry of the top-k table; wire format of the reference
// (sporder/src/common/weighted_index.h:15-27): high word = fp32 bits of the
// weight, low word = index + 1, all-zero = empty.
__device__ __forceinline__ uint64_t pack_entry(int32_t idx, float w) {
  return (static_cast<uint64_t>(__float_as_uint(w)) << 32) | static_cast<uint32_t>(idx + 1);
}
__device__ __forceinline__ int32_t entry_index(uint64_t e) {
  return static_cast<int32_t>(static_cast<uint32_t>(e)) - 1;
}
__device__ __forceinline__ uint32_t entry_weight_bits(uint64_t e) {
  return static_cast<uint32_t>(e >> 32);
}
#endif

#ifdef __CUDACC__
// launch of a kernel that calls wait_for_kernels_before(), as a programmatic dependent one or like any other
template <typename... Params, typename... Args>
cudaError_t launch_behind(bool dependent, void (*kernel)(Params...), int grid, int threads, int smem, cudaStream_t st,
                          Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = dependent ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}
#endif

}  // namespace csg
