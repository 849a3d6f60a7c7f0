/*
 * sporder_b200.h -- C ABI of the B200 (sm_100a) Chunked Greedy library.
 *
 * The first four entry points are the ones the reference's Python binding and C
 * callers bind for the csg path; names, argument order, argument meaning and
 * struct layouts are those of the reference header, so a program linked against
 * the reference's libsporder can load this library instead for that path.
 * Everything below them is new surface without a reference counterpart.
 *
 * Conventions (same as sporder/include/sporder.h:13-41 unless stated):
 *   - calls are synchronous: results are ready when the call returns;
 *   - d_ pointers are device memory on the context's device, h_ pointers are host
 *     memory, all other pointers are host memory;
 *   - CSR patterns are square, zero-based, column indices sorted and unique
 *     inside a row;
 *   - permutations are new2old: new row p holds old row d_new_order[p];
 *   - DIFFERENCE: the reference aborts the process on invalid arguments and CUDA
 *     errors (sporder/src/common/error_checking.h:20-29).  This library never
 *     aborts: the call returns early, outputs are unspecified, and
 *     sporder_last_error() returns the message (NULL when the last call on this
 *     thread succeeded).
 *   - `is_symmetric` is the reference's promise that the pattern equals its
 *     transpose (sporder/src/common/csr2csc.h:49-59, where the CSR arrays are then
 *     read as the CSC).  The library accepts it and does not depend on it: results
 *     and times are the same with and without, and a false promise has no effect.
 *     Row shards (sporder_csg_shard) have no such parameter.
 */
#ifndef SPORDER_B200_H
#define SPORDER_B200_H

#include <stdbool.h>
#include <stdint.h>

#define SPORDER_API __attribute__((visibility("default")))

#ifdef __cplusplus
extern "C" {
#endif

/* replaces sporder/include/sporder.h:43-52 */
typedef struct sporder_context_struct *sporder_context_t;
SPORDER_API sporder_context_t sporder_context_create(void);
SPORDER_API void sporder_context_destroy(sporder_context_t h);

/* replaces sporder/include/sporder.h:203-211 (same layout) */
typedef struct {
  double wall_ms;
  float csr2csc_ms;      /* here: the chunk-local transpose */
  float similarity_ms;   /* sketch + top-k */
  float chunk_greedy_ms; /* greedy chaining */
} sporder_csg_timing_t;

/* replaces sporder/include/sporder.h:213-222 (same layout) */
typedef struct {
  int32_t k_used;
  int32_t m_used;
  double avg_degree;
  double avg_edge_weight;
  int32_t zero_degree_rows;
  int32_t chunk_size_used;
  int32_t chain_restarts;
  double avg_followed_weight;
} sporder_csg_stats_t;

/* replaces sporder/include/sporder.h:224-228.
 * k <= 0 -> min(256, max(16, nnz / n)); oversampling <= 0 -> 4.0;
 * chunk_size <= 0 -> 1024 (sporder/src/sporder.cpp:147-155).
 * Errors (instead of the reference's abort): oversampling in (0,1),
 * int(k * oversampling) > 512, n < 1. */
SPORDER_API void sporder_chunk_similarity_greedy(
    sporder_context_t ctx, int32_t n, int32_t nnz, const int32_t *d_ptr, const int32_t *d_ind,
    bool is_symmetric, int32_t k, float oversampling, int32_t chunk_size, int32_t *d_new_order,
    sporder_csg_timing_t *timing, sporder_csg_stats_t *stats);

/* replaces sporder/include/sporder.h:128-133 (same layout) */
typedef struct {
  double wall_ms;
  float csr2csc_ms;
  float similarity_ms;
  float chunk_greedy_ms;
} sporder_cg_timing_t;

/* replaces sporder/include/sporder.h:154-167 (same layout) */
typedef struct {
  int32_t k_used;
  int32_t m_used;
  double avg_degree;
  double avg_edge_weight;
  int32_t zero_degree_rows;
  int32_t chunk_size_used;
  int32_t chain_restarts;
  double avg_followed_weight;
  double cut_weight_fraction; /* edge weight crossing chunk boundaries over total edge weight */
} sporder_cg_stats_t;

/* replaces sporder/include/sporder.h:176-182 (sporder/src/cg/chunk_greedy.cu:118-163): the
 * top-k graph of the WHOLE matrix (as sporder_similarity_graph, with the defaults
 * k <= 0 -> min(256, max(16, nnz / n)), oversampling <= 0 -> 4.0, chunk_size <= 0 -> 1024 of
 * sporder/src/sporder.cpp:118-126), then greedy chains inside chunks of chunk_size rows;
 * neighbours outside a row's chunk are skipped.  new2old permutation, as csg. */
SPORDER_API void sporder_chunk_greedy(sporder_context_t ctx, int32_t n, int32_t nnz,
                                      const int32_t *d_ptr, const int32_t *d_ind, bool is_symmetric,
                                      int32_t k, float oversampling, int32_t chunk_size,
                                      int32_t *d_new_order, sporder_cg_timing_t *timing,
                                      sporder_cg_stats_t *stats);

/* replaces sporder/include/sporder.h:312-317 (same layout) */
typedef struct {
  double wall_ms;
  float csr2csc_ms;    /* here: the transpose with the matrix as one chunk */
  float similarity_ms; /* sketch + top-k */
  float unpack_ms;
} sporder_sim_timing_t;

/* replaces sporder/include/sporder.h:322-328 (same layout) */
typedef struct {
  int32_t k_used;
  int32_t m_used;
  double avg_degree;
  double avg_edge_weight;
  int32_t zero_degree_rows;
} sporder_sim_stats_t;

/* replaces sporder/include/sporder.h:330-335 (sporder/src/similarity_graph.cu:26-107):
 * for each row up to k rows with the largest sketched Dice similarity, as
 * d_indices[r * k + j] / d_weights[r * k + j], unused entries index -1, weight 0.
 * k <= 0 -> min(32, max(16, 2 * (nnz / n))); oversampling <= 0 -> 2.0
 * (sporder/src/sporder.cpp:75-80).  The outputs must hold n * k entries for the k in
 * use; the return value is that k (the reference returns nothing), -1 on error.
 * is_symmetric: see sporder_chunk_similarity_greedy. */
SPORDER_API int32_t sporder_similarity_graph(sporder_context_t ctx, int32_t n, int32_t nnz,
                                             const int32_t *d_ptr, const int32_t *d_ind,
                                             bool is_symmetric, int32_t k, float oversampling,
                                             int32_t *d_indices, float *d_weights,
                                             sporder_sim_timing_t *timing,
                                             sporder_sim_stats_t *stats);

/* replaces sporder/include/sporder.h:276-279 (sporder/src/count_pillars.cu:38-85):
 * *count = number of distinct (row / height, column) pairs of the pattern, the
 * reordering quality metric of the reference (fewer is better).  height >= 1.
 * Rows must hold their columns in ascending order for height <= 12 (the CSR contract of
 * this library and of the reference); taller windows accept any order.  count is a host
 * pointer; the call synchronises the context's stream.  On error *count is 0 and
 * sporder_last_error() says why (the reference aborts). */
SPORDER_API void sporder_count_pillars(sporder_context_t ctx, int32_t n, int32_t nnz,
                                       const int32_t *d_ptr, const int32_t *d_ind, int32_t height,
                                       int32_t *count);

/* replaces sporder/include/sporder.h:230-233 */
typedef enum {
  SPORDER_REORDER_ROWS = 0,
  SPORDER_REORDER_SYMMETRIC = 1,
} sporder_reorder_mode_t;

/* replaces sporder/include/sporder.h:253-258 */
SPORDER_API void sporder_reorder(sporder_context_t ctx, int32_t n, int32_t nnz,
                                 const int32_t *d_ptr_old, const int32_t *d_ind_old,
                                 const float *d_val_old, const int32_t *d_new_order,
                                 sporder_reorder_mode_t mode, int32_t *d_ptr_new,
                                 int32_t *d_ind_new, float *d_val_new);

/* ---- new surface (no counterpart in the reference) ------------------------- */

/* Message of the last failed call on this thread, or NULL. */
SPORDER_API const char *sporder_last_error(void);

/* Run the context's work on `stream` (a cudaStream_t) instead of the context's
 * private stream; NULL restores the private stream.  To name the legacy default
 * stream pass cudaStreamLegacy ((cudaStream_t)0x1), not 0.  Calls stay synchronous.
 * A context serves one stream at a time: switching to another stream first waits for
 * the work the context queued on the previous one (sporder_spmm_async). */
SPORDER_API void sporder_context_set_stream(sporder_context_t ctx, void *stream);

/* Upper bound, in stream elements of 8 bytes, on the buffer that holds the materialised
 * candidate streams of the heaviest rows (rows that stream tens of thousands of candidates are
 * computed fastest from such a copy).  0 = no bound beyond the built-in 2^28 elements (2 GiB).
 * A call makes the buffer as large as its own rows need, once it knows them, and the context keeps
 * it; a call without such rows holds none.  Rows that do not fit, because of a bound or for want
 * of memory, are computed by the kernel of the lighter rows; results are the same for every bound. */
SPORDER_API void sporder_context_set_stream_limit(sporder_context_t ctx, uint64_t max_elements);

/* Calls of sporder_chunk_similarity_greedy (and its variants with a table, on host buffers or
 * on a row shard) with many nonzeros run the chunk that holds the most of them ahead of the
 * rest, on a second stream of the context: that chunk's transposition first, then the
 * chains of its heaviest rows, while everything else is still being transposed.  min_nnz
 * = 0: the built-in rule (2^24 nonzeros and 64 chunks or more, and by slots of the sketch where it
 * gains); > 0: every call of at least
 * min_nnz nonzeros and two chunks; < 0: never.  Results are the same either way.  No
 * reference counterpart. */
SPORDER_API void sporder_context_set_ahead_threshold(sporder_context_t ctx, int64_t min_nnz);

/* Which rows the kernel of the longest candidate streams takes, a group of warps each.  0: as
 * many as its measured costs and those of the kernel beside it say; otherwise the rows with
 * min_candidates candidates or more (no fewer than 64, rounded down to a quarter octave), as far
 * as there is room for their streams.  Results are the same either way. */
SPORDER_API void sporder_context_set_chain_threshold(sporder_context_t ctx, uint32_t min_candidates);

/* Rows that kernel took in the context's last csg or similarity graph call. */
SPORDER_API uint64_t sporder_context_chain_rows(sporder_context_t ctx);

/* Bytes of device workspace the context currently holds (grow-only cache). */
SPORDER_API uint64_t sporder_context_workspace_bytes(sporder_context_t ctx);

/* csg that also returns the top-k table: d_table receives n * k_used packed
 * entries (high 32 bits = fp32 bits of the weight, low 32 bits = index + 1,
 * 0 = empty; the reference's internal format, sporder/src/common/weighted_index.h:15-27).
 * d_table_capacity is the number of entries d_table can hold; d_new_order may be
 * NULL to skip the greedy stage.  Returns k_used, or -1 on error. */
SPORDER_API int32_t sporder_csg_with_table(sporder_context_t ctx, int32_t n, int32_t nnz,
                                           const int32_t *d_ptr, const int32_t *d_ind,
                                           bool is_symmetric, int32_t k, float oversampling,
                                           int32_t chunk_size, int32_t *d_new_order,
                                           uint64_t *d_table, uint64_t d_table_capacity,
                                           sporder_csg_timing_t *timing,
                                           sporder_csg_stats_t *stats);

/* csg of one row shard: rows [row_base, row_base + n_rows) of a matrix with n_cols
 * columns, given as a CSR block whose d_ptr is rebased to start at 0 and whose
 * column ids are the matrix's own.  row_base must be a multiple of chunk_size so
 * that the shard holds whole chunks; then its chunks see exactly the candidates
 * they see in the full matrix and the results (d_new_order[i], table indices) are
 * the full matrix's, already offset by row_base.  k and chunk_size should be
 * passed resolved (k <= 0 would resolve from the shard's own nnz / n_rows).
 * d_new_order and d_table may be NULL.  Returns k_used, or -1 on error. */
SPORDER_API int32_t sporder_csg_shard(sporder_context_t ctx, int32_t n_rows, int32_t n_cols,
                                      int32_t row_base, int32_t nnz, const int32_t *d_ptr,
                                      const int32_t *d_ind, int32_t k, float oversampling,
                                      int32_t chunk_size, int32_t *d_new_order,
                                      uint64_t *d_table, uint64_t d_table_capacity,
                                      sporder_csg_timing_t *timing, sporder_csg_stats_t *stats);

/* csg on host buffers: copies ptr/ind to the device, reorders, copies the
 * permutation back.  Returns 0, or -1 on error. */
SPORDER_API int32_t sporder_chunk_similarity_greedy_host(
    sporder_context_t ctx, int32_t n, int32_t nnz, const int32_t *h_ptr, const int32_t *h_ind,
    bool is_symmetric, int32_t k, float oversampling, int32_t chunk_size, int32_t *h_new_order,
    sporder_csg_timing_t *timing, sporder_csg_stats_t *stats);

/* fp32 CSR SpMM: C[n x w] = A * B with B, C row-major (ld = w).  n is the number of rows
 * of A (and of C); B must hold a row for every column id in d_ind, so A may be a row block
 * of a wider matrix (the row-partitioned multi-GPU product).  The reference
 * times third-party kernels (bench/spmm/spmm_bench/base.py:48-59) and cuSPARSE
 * (sporder/src/bench_cusparse_spmm.cu:64-90) here; it has no SpMM of its own.
 * Returns 0, or -1 on error. */
SPORDER_API int32_t sporder_spmm(sporder_context_t ctx, int32_t n, int32_t nnz, int32_t w,
                                 const int32_t *d_ptr, const int32_t *d_ind, const float *d_val,
                                 const float *d_B, float *d_C);

/* Same without the final stream synchronisation (for callers that time a train
 * of launches with events on the context's stream).  Returns 0 or -1. */
SPORDER_API int32_t sporder_spmm_async(sporder_context_t ctx, int32_t n, int32_t nnz, int32_t w,
                                       const int32_t *d_ptr, const int32_t *d_ind,
                                       const float *d_val, const float *d_B, float *d_C);

/* SpMM for callers that must not trigger a device allocation (no counterpart in the
 * reference).  Same product as sporder_spmm, but it takes no context and calls no
 * cudaMalloc / cudaFree or allocating routine: the queue of long rows sits in a fixed
 * array of 512 KiB plus 256 bytes of counters inside the library image (held by every
 * GPU that loads the library until the process exits).  Meant for hosts that gave all device memory to their own
 * pool, or that ban driver allocations on their request path because those stall the
 * whole device.
 *   - limit: nnz < 65536 * 1024 (67,108,864); larger inputs are rejected with an error;
 *   - the work is queued on `stream` (a cudaStream_t; NULL = default stream) and the
 *     call returns without waiting for it;
 *   - the first call on each device looks up the array's device address; make that
 *     first call before any stream capture;
 *   - all calls share the array: calls whose kernels may overlap on one GPU race.
 * Returns 0, or -1 on error (see sporder_last_error). */
SPORDER_API int32_t sporder_spmm_static(int32_t n, int32_t nnz, int32_t w, const int32_t *d_ptr,
                                        const int32_t *d_ind, const float *d_val,
                                        const float *d_B, float *d_C, void *stream);

/* d_out[r] = sum of row r's values (A times the vector of ones).  Queued on the context's
 * stream without waiting, as the two calls below.  Returns 0 or -1. */
SPORDER_API int32_t sporder_row_sums(sporder_context_t ctx, int32_t n, int32_t nnz,
                                     const int32_t *d_ptr, const float *d_val, float *d_out);

/* Y = x W^T + b, fp32, row-major: x n x in_dim, W out_dim x in_dim, both dimensions in multiples
 * of 4 up to 128, x and Y 16-byte aligned.  Inputs are summed in order, the bias added last.
 * Queued without waiting.  Returns 0 or -1. */
SPORDER_API int32_t sporder_linear(sporder_context_t ctx, int32_t n, int32_t in_dim,
                                   int32_t out_dim, const float *d_x, const float *d_W,
                                   const float *d_b, float *d_Y);

/* Dense parts of a two-layer GCN, fp32, row-major.  With Z the first sparse product
 * (n x hidden), P = A x (n x in_dim) and s = A 1 (n):
 *   forward:  U = relu(Z) W2^T (n x classes);
 *   backward, for G = dL/dU: with D = (G W2) masked by Z > 0,
 *             dW1 = D^T P, db1 = D^T s, dW2 = G^T relu(Z) (overwritten, not added to).
 * in_dim and hidden in multiples of 4 up to 128, classes up to 48, P and Z 16-byte aligned.
 * The sums of the backward pass are taken in the same order on every call.  Return 0 or -1. */
SPORDER_API int32_t sporder_gcn_forward(sporder_context_t ctx, int32_t n, int32_t hidden,
                                        int32_t classes, const float *d_Z, const float *d_W2,
                                        float *d_U);
SPORDER_API int32_t sporder_gcn_backward(sporder_context_t ctx, int32_t n, int32_t in_dim,
                                         int32_t hidden, int32_t classes, const float *d_G,
                                         const float *d_Z, const float *d_P, const float *d_s,
                                         const float *d_W2, float *d_dW1, float *d_db1,
                                         float *d_dW2);

/* The same with U and G in rows of `columns` floats (classes <= columns <= 48): forward writes
 * zeros behind the classes, backward does not read there.  sporder_pad_columns brings a matrix of
 * `from` columns into that form.  (A sparse product of a ragged width costs more than the next
 * full one.) */
SPORDER_API int32_t sporder_gcn_forward_padded(sporder_context_t ctx, int32_t n, int32_t hidden,
                                               int32_t classes, int32_t columns, const float *d_Z,
                                               const float *d_W2, float *d_U);
SPORDER_API int32_t sporder_gcn_backward_padded(sporder_context_t ctx, int32_t n, int32_t in_dim,
                                                int32_t hidden, int32_t classes, int32_t columns,
                                                const float *d_G, const float *d_Z,
                                                const float *d_P, const float *d_s,
                                                const float *d_W2, float *d_dW1, float *d_db1,
                                                float *d_dW2);
SPORDER_API int32_t sporder_pad_columns(sporder_context_t ctx, int32_t n, int32_t from, int32_t to,
                                        const float *d_src, float *d_dst);

/* The same gradients in two halves around a sparse product at the hidden width, for layers whose
 * inputs are wider (the operator is symmetric, E = A D):
 *   hidden_gradient: D as above (n x hidden) and dW2;
 *   input_gradients: dW1 = E^T x, db1 = column sums of E, x n x in_dim.
 * Limits as above, Z, D, E and x 16-byte aligned.  Return 0 or -1. */
SPORDER_API int32_t sporder_gcn_hidden_gradient(sporder_context_t ctx, int32_t n, int32_t hidden,
                                                int32_t classes, int32_t columns,
                                                const float *d_G, const float *d_Z,
                                                const float *d_W2, float *d_D, float *d_dW2);
SPORDER_API int32_t sporder_gcn_input_gradients(sporder_context_t ctx, int32_t n, int32_t in_dim,
                                                int32_t hidden, const float *d_E,
                                                const float *d_x, float *d_dW1, float *d_db1);

/* Number of kernels this library has launched in this process (all contexts). */
SPORDER_API uint64_t sporder_kernel_launches(void);

#ifdef __cplusplus
}
#endif
#endif /* SPORDER_B200_H */
