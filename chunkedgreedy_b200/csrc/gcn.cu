// Dense parts of a two-layer GCN around the library's SpMM, fp32.
//
// The caller's model is Linear(in, hidden) -> A -> ReLU -> A -> Linear(hidden, classes)
// (experiments/e2e_gcn.py:126-137).  With Z the first sparse product, P = A x and s = A 1 (the row
// sums), and the second sparse product taken behind the second linear layer (it is narrower there):
//   forward   U = relu(Z) W2^T
//   backward  (G = dL/dU)  D = (G W2) * (Z > 0),  dW1 = D^T P,  db1 = D^T s,  dW2 = G^T relu(Z);
// or, where the hidden layer is narrower than the inputs, with E = A D in place of P (A is symmetric):
//             dW1 = E^T x,  db1 = E^T 1.
// One kernel forward, one backward, where D never exists in memory, or two around E = A D.  The
// backward pass is bound by fp32 multiply-adds (2 n in hidden of them, against three passes over n
// rows of 128 floats): blocks are persistent, one per SM, operands staged with cp.async a tile ahead,
// 8 x 8 results per thread.  On 1.05 M rows,
// 128 -> 128 -> 16, on a B200: 1.09 ms (53 % of the fp32 pipes; two warps per scheduler, and the
// phases of a tile do not overlap); one torch kernel per operation took 2.4 ms.
#include "../../include/sporder_b200.h"
#include "common.cuh"

namespace csg {

namespace {

constexpr int D_THREADS = 256;
constexpr int F_ROWS = 128;  // rows per tile, forward
constexpr int B_ROWS = 32;   // ... and backward
constexpr int MAX_CLASSES = 48;

struct DenseArgs {
  int32_t n, in, hid, cls, ld;  // ld: floats per row of U and G, those behind the classes zero
  const float *P, *s, *W2, *Z;
  float *U, *D;
  const float *G;
  float *part;        // backward: a block's sums
  float *dW1, *db1, *dW2;
};

// 16 (4) bytes global -> shared without registers; zeros when off
__device__ __forceinline__ void copy16(float *dst, const float *src, bool on) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy4(float *dst, const float *src, bool on) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(on ? 4 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// ROWS rows of `cols` floats (a multiple of 4) from row r0 of src into dst, COLS_T + 4 apart, zeros
// behind the last column and the last row
template <int ROWS, int COLS_T, int THREADS>
__device__ __forceinline__ void stage_rows(float *dst, const float *src, int64_t r0, int32_t n, int32_t cols) {
  constexpr int PER_ROW = COLS_T / 4;
  for (int i = threadIdx.x; i < ROWS * PER_ROW; i += THREADS) {
    const int r = i / PER_ROW, c = (i % PER_ROW) * 4;
    const bool on = r0 + r < n && c < cols;
    copy16(dst + r * (COLS_T + 4) + c, src + (on ? (r0 + r) * cols + c : 0), on);
  }
}

// acc.x += a.x * b.x, acc.y += a.y * b.y in one instruction
__device__ __forceinline__ void fma2(float2 &acc, float2 a, float2 b) {
  unsigned long long &c = reinterpret_cast<unsigned long long &>(acc);
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(c)
      : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)));
}

// ---- Y = x W^T + b --------------------------------------------------------------------------
// Every result is one chain of multiply-adds over the inputs in order, then the bias: the order,
// and so the rounding, of a plain fp32 matrix product with the bias added behind it.  Two columns
// to an instruction.  1.05 M rows, 128 -> 128: 0.71 ms (34.4 GF at 74 TF/s of fp32 pipes: 0.46; the
// library product 0.72, and the bias 0.36 more as a kernel of its own).
template <int IN_T, int HID_T>
struct LinearShared {
  static constexpr int XS = IN_T + 4;
  static constexpr int W = 0, B = W + IN_T * HID_T, TILES = B + HID_T, FLOATS = TILES + 2 * F_ROWS * XS;
};
template <int IN_T, int HID_T>
__global__ void __launch_bounds__(D_THREADS, 1) linear_kernel(int32_t n, int32_t in, int32_t hid, const float *x,
                                                              const float *W, const float *bias, float *Y) {
  using L = LinearShared<IN_T, HID_T>;
  constexpr int NP = HID_T / 32;  // pairs of columns per thread: j, j + 1 with j = 32 i + 2 tx
  extern __shared__ __align__(16) float dense_smem[];
  float *const w = dense_smem + L::W, *const b = dense_smem + L::B;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  for (int i = tid; i < IN_T * HID_T; i += D_THREADS) {
    const int k = i / HID_T, j = i % HID_T;
    w[i] = k < in && j < hid ? W[static_cast<size_t>(j) * in + k] : 0.0f;
  }
  for (int i = tid; i < HID_T; i += D_THREADS) b[i] = i < hid ? bias[i] : 0.0f;
  const int64_t tiles = (static_cast<int64_t>(n) + F_ROWS - 1) / F_ROWS;
  auto stage = [&](int64_t t, int buf) {
    if (t < tiles) stage_rows<F_ROWS, IN_T, D_THREADS>(dense_smem + L::TILES + buf * F_ROWS * L::XS, x, t * F_ROWS, n, in);
    copies_commit();
  };
  stage(blockIdx.x, 0);
  int buf = 0;
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x, buf ^= 1) {
    stage(t + gridDim.x, buf ^ 1);
    copies_wait<1>();
    __syncthreads();
    const float *const tile = dense_smem + L::TILES + buf * F_ROWS * L::XS + ty * L::XS;
    float2 acc[8][NP];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < NP; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
#pragma unroll 2
    for (int k = 0; k < IN_T; k += 4) {
      float4 p[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) p[i] = *reinterpret_cast<const float4 *>(tile + 16 * i * L::XS + k);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        float2 q[NP];
#pragma unroll
        for (int j = 0; j < NP; ++j) q[j] = *reinterpret_cast<const float2 *>(w + (k + kk) * HID_T + 32 * j + 2 * tx);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float v = kk == 0 ? p[i].x : kk == 1 ? p[i].y : kk == 2 ? p[i].z : p[i].w;
#pragma unroll
          for (int j = 0; j < NP; ++j) fma2(acc[i][j], make_float2(v, v), q[j]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int64_t r = t * F_ROWS + ty + 16 * i;
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        const int c = 32 * j + 2 * tx;
        if (r < n && c < hid)
          *reinterpret_cast<float2 *>(Y + r * hid + c) = make_float2(acc[i][j].x + b[c], acc[i][j].y + b[c + 1]);
      }
    }
    __syncthreads();
  }
  copies_wait<0>();
}

template <int HID_T>
struct ForwardShared {
  static constexpr int HS = HID_T + 4;
  static constexpr int W2 = 0, TILES = MAX_CLASSES * HS, FLOATS = TILES + 2 * F_ROWS * HS;
};

// Two threads per row, every other group of four classes each.  Bound by shared memory: a row of
// Z and the weights are read from there once per group.
template <int HID_T>
__global__ void __launch_bounds__(D_THREADS, 1) gcn_forward_kernel(DenseArgs a) {
  using L = ForwardShared<HID_T>;
  extern __shared__ __align__(16) float dense_smem[];
  float *const w2 = dense_smem + L::W2;
  const int tid = threadIdx.x;
  for (int i = tid; i < MAX_CLASSES * L::HS; i += D_THREADS) {
    const int c = i / L::HS, j = i % L::HS;
    w2[i] = c < a.cls && j < a.hid ? a.W2[static_cast<size_t>(c) * a.hid + j] : 0.0f;
  }
  const int64_t tiles = (static_cast<int64_t>(a.n) + F_ROWS - 1) / F_ROWS;
  auto stage = [&](int64_t t, int buf) {
    if (t < tiles) stage_rows<F_ROWS, HID_T, D_THREADS>(dense_smem + L::TILES + buf * F_ROWS * L::HS, a.Z, t * F_ROWS, a.n, a.hid);
    copies_commit();
  };
  stage(blockIdx.x, 0);
  int buf = 0;
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x, buf ^= 1) {
    stage(t + gridDim.x, buf ^ 1);
    copies_wait<1>();
    __syncthreads();
    const float *const z = dense_smem + L::TILES + buf * F_ROWS * L::HS + (tid >> 1) * L::HS;
    const int64_t r = t * F_ROWS + (tid >> 1);
    for (int c0 = (tid & 1) * 4; c0 < a.ld; c0 += 8) {
      float u[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 8
      for (int k = 0; k < HID_T; k += 4) {
        float4 h = *reinterpret_cast<const float4 *>(z + k);
        h = make_float4(fmaxf(h.x, 0.0f), fmaxf(h.y, 0.0f), fmaxf(h.z, 0.0f), fmaxf(h.w, 0.0f));
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float4 w = *reinterpret_cast<const float4 *>(w2 + (c0 + c) * L::HS + k);
          u[c] = fmaf(h.x, w.x, fmaf(h.y, w.y, fmaf(h.z, w.z, fmaf(h.w, w.w, u[c]))));
        }
      }
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (c0 + c < a.ld && r < a.n) a.U[r * a.ld + c0 + c] = u[c];
    }
    __syncthreads();  // the tile's place is free for the copies of the round after next
  }
  copies_wait<0>();
}

template <int IN_T, int HID_T, int CLS_T>
struct BackwardShared {
  static constexpr int PS = IN_T + 4, HS = HID_T + 4;
  static constexpr int D = 0, BUF = D + B_ROWS * HS;
  static constexpr int P = 0, H = P + B_ROWS * PS, G = H + B_ROWS * HS, S = G + B_ROWS * CLS_T, BUF_FLOATS = S + B_ROWS;
  static constexpr int FLOATS = BUF + 2 * BUF_FLOATS;
};
// a block's sums in `part`: dW1 (HID_T x IN_T), dW2 (CLS_T x HID_T), then db1 from each of the
// D_THREADS / HID_T groups of threads
template <int IN_T, int HID_T, int CLS_T>
struct PartLayout {
  static constexpr int W2 = HID_T * IN_T, B1 = W2 + CLS_T * HID_T, FLOATS = B1 + D_THREADS;
};

// B_ROWS rows of G from row r0 into dst, CLS_T apart, zeros behind the last row
template <int CLS_T>
__device__ __forceinline__ void stage_classes(float *dst, const DenseArgs &a, int64_t r0) {
  for (int i = threadIdx.x; i < B_ROWS * a.cls; i += D_THREADS) {
    const int r = i / a.cls, c = i % a.cls;
    const bool on = r0 + r < a.n;
    copy4(dst + r * CLS_T + c, a.G + (on ? (r0 + r) * a.ld + c : 0), on);
  }
}

// (G W2) of one row and hidden unit, masked: w2 is the unit's column of W2, z its row's value of Z
template <int CLS_T>
__device__ __forceinline__ float hidden_gradient(const float *g, const float (&w2)[CLS_T], float z) {
  float x[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int c = 0; c < CLS_T; c += 4) {
    const float4 q = *reinterpret_cast<const float4 *>(g + c);
    x[0] = fmaf(q.x, w2[c], x[0]);
    x[1] = fmaf(q.y, w2[c + 1], x[1]);
    x[2] = fmaf(q.z, w2[c + 2], x[2]);
    x[3] = fmaf(q.w, w2[c + 3], x[3]);
  }
  return z > 0.0f ? (x[0] + x[1]) + (x[2] + x[3]) : 0.0f;
}

// acc2 += g * hv for PER classes
template <int PER>
__device__ __forceinline__ void add_classes(float (&acc2)[PER], const float *g, float hv) {
  constexpr int VC = PER % 4 == 0 ? 4 : 2;
#pragma unroll
  for (int c = 0; c < PER; c += VC) {
    float gv[VC];
    if constexpr (VC == 4) *reinterpret_cast<float4 *>(gv) = *reinterpret_cast<const float4 *>(g + c);
    else *reinterpret_cast<float2 *>(gv) = *reinterpret_cast<const float2 *>(g + c);
#pragma unroll
    for (int x = 0; x < VC; ++x) acc2[c + x] = fmaf(gv[x], hv, acc2[c + x]);
  }
}

// CLS_T == 0: a.Z holds E, which takes the place of D; neither G nor s nor W2 is there, dW2 is not asked for
template <int IN_T, int HID_T, int CLS_T>
__global__ void __launch_bounds__(D_THREADS, 1) gcn_backward_kernel(DenseArgs a) {
  using L = BackwardShared<IN_T, HID_T, CLS_T>;
  using O = PartLayout<IN_T, HID_T, CLS_T>;
  constexpr int NJ = HID_T / 16, VJ = NJ < 4 ? NJ : 4, QJ = NJ / VJ;  // hidden units per thread, QJ runs of VJ
  constexpr int NI = IN_T / 16, VI = 4, QI = NI / VI;   // inputs per thread, in fours
  constexpr bool GIVEN = CLS_T == 0;
  constexpr int GROUPS = D_THREADS / HID_T, PER = CLS_T / GROUPS;  // dW2: PER classes of one hidden unit per thread
  extern __shared__ __align__(16) float dense_smem[];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int hj = tid % HID_T, group = tid / HID_T;
  float w2[GIVEN ? 1 : CLS_T];  // this thread's hidden unit's column of W2
#pragma unroll
  for (int c = 0; c < CLS_T; ++c)
    w2[c] = c < a.cls && hj < a.hid ? a.W2[static_cast<size_t>(c) * a.hid + hj] : 0.0f;
  float2 acc[NJ][NI / 2];
  float acc2[GIVEN ? 1 : PER], accb = 0.0f;
  [[maybe_unused]] float lost = 0.0f;
#pragma unroll
  for (int j = 0; j < NJ; ++j)
#pragma unroll
    for (int i = 0; i < NI / 2; ++i) acc[j][i] = make_float2(0.0f, 0.0f);
  // (E is read where it lies, so there are registers for a tile's sums apart from the sums of all tiles: these
  // largely cancel, and a chain over all rows of a block loses more)
  [[maybe_unused]] float2 all[GIVEN ? NJ : 1][GIVEN ? NI / 2 : 1] = {};
#pragma unroll
  for (int c = 0; c < PER; ++c) acc2[c] = 0.0f;
  for (int i = tid; i < 2 * L::BUF_FLOATS; i += D_THREADS) dense_smem[L::BUF + i] = 0.0f;  // classes behind the last
  __syncthreads();
  const int64_t tiles = (static_cast<int64_t>(a.n) + B_ROWS - 1) / B_ROWS;
  auto stage = [&](int64_t t, int buf) {
    if (t < tiles) {
      float *const b = dense_smem + L::BUF + buf * L::BUF_FLOATS;
      const int64_t r0 = t * B_ROWS;
      stage_rows<B_ROWS, IN_T, D_THREADS>(b + L::P, a.P, r0, a.n, a.in);
      stage_rows<B_ROWS, HID_T, D_THREADS>(b + L::H, a.Z, r0, a.n, a.hid);
      if constexpr (!GIVEN) {
        stage_classes<CLS_T>(b + L::G, a, r0);
        for (int i = tid; i < B_ROWS; i += D_THREADS) copy4(b + L::S + i, a.s + (r0 + i < a.n ? r0 + i : 0), r0 + i < a.n);
      }
    }
    copies_commit();
  };
  stage(blockIdx.x, 0);
  int buf = 0;
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x, buf ^= 1) {
    stage(t + gridDim.x, buf ^ 1);
    copies_wait<1>();
    __syncthreads();
    const float *const b = dense_smem + L::BUF + buf * L::BUF_FLOATS;
    const float *const p = b + L::P, *const h = b + L::H, *const g = b + L::G, *const s = b + L::S;
    const float *d = h;
    if constexpr (GIVEN) {
      // (the sum over all rows largely cancels: the tile's rows first, then compensated)
      float tile = 0.0f;
      for (int r = group; r < B_ROWS; r += GROUPS) tile += h[r * L::HS + hj];
      const float y = tile - lost, sum = accb + y;
      lost = (sum - accb) - y;
      accb = sum;
    } else {
      float *const own = dense_smem + L::D;
#pragma unroll 4
      for (int r = group; r < B_ROWS; r += GROUPS) {
        const float y = hidden_gradient<CLS_T>(g + r * CLS_T, w2, h[r * L::HS + hj]);
        own[r * L::HS + hj] = y;
        accb = fmaf(y, s[r], accb);
      }
      d = own;
      __syncthreads();
    }
#pragma unroll 4
    for (int r = 0; r < B_ROWS; ++r) {
      float dj[NJ];
      float2 pi[NI / 2];
#pragma unroll
      for (int q = 0; q < QJ; ++q) {
        const float *src = d + r * L::HS + q * (HID_T / QJ) + ty * VJ;
        if constexpr (VJ == 4) *reinterpret_cast<float4 *>(dj + q * VJ) = *reinterpret_cast<const float4 *>(src);
        else *reinterpret_cast<float2 *>(dj + q * VJ) = *reinterpret_cast<const float2 *>(src);
      }
#pragma unroll
      for (int q = 0; q < QI; ++q)
        *reinterpret_cast<float4 *>(pi + 2 * q) = *reinterpret_cast<const float4 *>(p + r * L::PS + q * (IN_T / QI) + tx * VI);
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int i = 0; i < NI / 2; ++i) fma2(acc[j][i], make_float2(dj[j], dj[j]), pi[i]);
      if constexpr (!GIVEN) add_classes<PER>(acc2, g + r * CLS_T + group * PER, fmaxf(h[r * L::HS + hj], 0.0f));
    }
    if constexpr (GIVEN) {
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int i = 0; i < NI / 2; ++i) {
          all[j][i] = make_float2(all[j][i].x + acc[j][i].x, all[j][i].y + acc[j][i].y);
          acc[j][i] = make_float2(0.0f, 0.0f);
        }
    }
    __syncthreads();
  }
  copies_wait<0>();
  if constexpr (GIVEN) {
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int i = 0; i < NI / 2; ++i) acc[j][i] = all[j][i];
  }
  float *const out = a.part + static_cast<size_t>(blockIdx.x) * O::FLOATS;
#pragma unroll
  for (int j = 0; j < NJ; ++j)
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int row = (j / VJ) * (HID_T / QJ) + ty * VJ + j % VJ, col = (i / VI) * (IN_T / QI) + tx * VI + i % VI;
      out[row * IN_T + col] = i & 1 ? acc[j][i / 2].y : acc[j][i / 2].x;
    }
#pragma unroll
  for (int c = 0; c < PER; ++c) out[O::W2 + (group * PER + c) * HID_T + hj] = acc2[c];
  out[O::B1 + tid] = accb;
}

// D written out, and dW2 = G^T relu(Z): the first half where the operator goes over D.  Bound by its three
// passes (Z and G in, D out); two blocks per SM keep their copies in flight.
template <int HID_T, int CLS_T>
struct HiddenShared {
  static constexpr int HS = HID_T + 4;
  static constexpr int H = 0, G = H + B_ROWS * HS, BUF_FLOATS = G + B_ROWS * CLS_T, FLOATS = 2 * BUF_FLOATS;
};
template <int HID_T, int CLS_T>
__global__ void __launch_bounds__(D_THREADS, 2) gcn_hidden_kernel(DenseArgs a) {
  using L = HiddenShared<HID_T, CLS_T>;
  using O = PartLayout<0, HID_T, CLS_T>;
  constexpr int GROUPS = D_THREADS / HID_T, PER = CLS_T / GROUPS;
  extern __shared__ __align__(16) float dense_smem[];
  const int tid = threadIdx.x, hj = tid % HID_T, group = tid / HID_T;
  float w2[CLS_T], acc2[PER];
#pragma unroll
  for (int c = 0; c < CLS_T; ++c)
    w2[c] = c < a.cls && hj < a.hid ? a.W2[static_cast<size_t>(c) * a.hid + hj] : 0.0f;
#pragma unroll
  for (int c = 0; c < PER; ++c) acc2[c] = 0.0f;
  for (int i = tid; i < L::FLOATS; i += D_THREADS) dense_smem[i] = 0.0f;  // classes behind the last
  __syncthreads();
  const int64_t tiles = (static_cast<int64_t>(a.n) + B_ROWS - 1) / B_ROWS;
  auto stage = [&](int64_t t, int buf) {
    if (t < tiles) {
      float *const b = dense_smem + buf * L::BUF_FLOATS;
      stage_rows<B_ROWS, HID_T, D_THREADS>(b + L::H, a.Z, t * B_ROWS, a.n, a.hid);
      stage_classes<CLS_T>(b + L::G, a, t * B_ROWS);
    }
    copies_commit();
  };
  stage(blockIdx.x, 0);
  int buf = 0;
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x, buf ^= 1) {
    stage(t + gridDim.x, buf ^ 1);
    copies_wait<1>();
    __syncthreads();
    const float *const h = dense_smem + buf * L::BUF_FLOATS + L::H, *const g = dense_smem + buf * L::BUF_FLOATS + L::G;
#pragma unroll 4
    for (int r = group; r < B_ROWS; r += GROUPS) {
      const float y = hidden_gradient<CLS_T>(g + r * CLS_T, w2, h[r * L::HS + hj]);
      if (t * B_ROWS + r < a.n && hj < a.hid) a.D[(t * B_ROWS + r) * a.hid + hj] = y;
    }
#pragma unroll 4
    for (int r = 0; r < B_ROWS; ++r) add_classes<PER>(acc2, g + r * CLS_T + group * PER, fmaxf(h[r * L::HS + hj], 0.0f));
    __syncthreads();
  }
  copies_wait<0>();
  float *const out = a.part + static_cast<size_t>(blockIdx.x) * O::FLOATS;
#pragma unroll
  for (int c = 0; c < PER; ++c) out[O::W2 + (group * PER + c) * HID_T + hj] = acc2[c];
}

// The blocks' sums, always in the same order, in 64 bits (some hundred terms that largely cancel).
// Bound by the latency of its reads: 128 -> 128 -> 16 in small blocks, sixteen reads in flight 18 us,
// 28.5 in blocks of 256 with four.
constexpr int SUMS_THREADS = 64;
template <int IN_T, int HID_T, int CLS_T>
__global__ void __launch_bounds__(SUMS_THREADS) gcn_sums_kernel(DenseArgs a, int blocks) {
  using O = PartLayout<IN_T, HID_T, CLS_T>;
  const int w1 = a.hid * a.in, w2 = a.cls * a.hid, total = w1 + w2 + (a.db1 ? a.hid : 0);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    int at, times = 1;
    float *to;
    if (i < w1) {
      at = i / a.in * IN_T + i % a.in;
      to = a.dW1 + i;
    } else if (i < w1 + w2) {
      const int x = i - w1;
      at = O::W2 + x / a.hid * HID_T + x % a.hid;
      to = a.dW2 + x;
    } else {
      at = O::B1 + i - w1 - w2;
      to = a.db1 + (i - w1 - w2);
      times = D_THREADS / HID_T;
    }
    double sum[4] = {0.0, 0.0, 0.0, 0.0};
    for (int g = 0; g < times; ++g) {
      const float *src = a.part + at + g * HID_T;
      int b = 0;
      for (; b + 16 <= blocks; b += 16) {
        float v[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) v[u] = src[static_cast<size_t>(b + u) * O::FLOATS];
#pragma unroll
        for (int u = 0; u < 16; ++u) sum[u & 3] += v[u];
      }
      for (; b + 4 <= blocks; b += 4)
#pragma unroll
        for (int u = 0; u < 4; ++u) sum[u] += src[static_cast<size_t>(b + u) * O::FLOATS];
      for (; b < blocks; ++b) sum[0] += src[static_cast<size_t>(b) * O::FLOATS];
    }
    *to = static_cast<float>((sum[0] + sum[1]) + (sum[2] + sum[3]));
  }
}

// A 1.  Eight lanes a row; rows of more than SUM_SPLIT entries are queued in pieces for a second
// kernel, where a warp adds a piece at a time (one row of a power-law graph holds 10^5 entries).
constexpr int SUM_SPLIT = 512, SUM_PIECE = 2048;
__global__ void __launch_bounds__(256) row_sums_kernel(int32_t n, int32_t nnz, const int32_t *__restrict__ ptr,
                                                       const float *__restrict__ val, float *__restrict__ out,
                                                       uint32_t *queued, int2 *queue) {
  constexpr int G = 8;
  const int gl = threadIdx.x % G;
  const int64_t groups = static_cast<int64_t>(gridDim.x) * blockDim.x / G;
  const int64_t rounds = (static_cast<int64_t>(n) + groups - 1) / groups;
  int64_t r = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / G;
  for (int64_t i = 0; i < rounds; ++i, r += groups) {
    int32_t b = 0, e = 0;
    if (r < n) {
      b = ptr[r];
      e = ptr[r + 1];
      if (b < 0 || e < b || e > nnz) e = b = 0;  // malformed row pointers: an empty row
    }
    float v = 0.0f;
    if (e - b > SUM_SPLIT) {
      if (gl == 0) {
        const int32_t pieces = (e - b + SUM_PIECE - 1) / SUM_PIECE;
        uint32_t at = atomicAdd(queued, static_cast<uint32_t>(pieces));
        for (int32_t p = b; p < e; p += SUM_PIECE) queue[at++] = make_int2(static_cast<int32_t>(r), p);
      }
    } else {
      for (int32_t p = b + gl; p < e; p += G) v += val[p];
    }
#pragma unroll
    for (int off = G / 2; off > 0; off >>= 1) v += __shfl_xor_sync(FULL, v, off);
    if (gl == 0 && r < n) out[r] = v;
  }
}

__global__ void __launch_bounds__(256) row_pieces_kernel(const int32_t *__restrict__ ptr, const float *__restrict__ val,
                                                         float *__restrict__ out, const uint32_t *queued,
                                                         const int2 *queue) {
  const int lane = threadIdx.x & 31;
  const uint32_t total = *queued, warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < total; i += warps) {
    const int2 q = queue[i];
    const int32_t end = min(ptr[q.x + 1], q.y + SUM_PIECE);
    float x[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    for (int32_t p = q.y + lane; p < end; p += 256)
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (p + 32 * u < end) x[u] += val[p + 32 * u];
    float v = ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(FULL, v, off);
    if (lane == 0) atomicAdd(out + q.x, v);
  }
}

// dst: n rows of `to` floats, the first `from` of them src's, zeros behind
__global__ void __launch_bounds__(256) pad_columns_kernel(int32_t n, int32_t from, int32_t to, const float *__restrict__ src,
                                                          float *__restrict__ dst) {
  const int64_t total = static_cast<int64_t>(n) * to, step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += step) {
    const int64_t r = i / to;
    const int32_t c = static_cast<int32_t>(i - r * to);
    dst[i] = c < from ? src[r * from + c] : 0.0f;
  }
}

template <typename Kernel>
bool dense_smem_limit(Kernel kernel, size_t bytes) {
  CSG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)));
  return true;
}

template <int HID_T>
bool forward_variant(Context &ctx, const DenseArgs &a) {
  const size_t smem = sizeof(float) * ForwardShared<HID_T>::FLOATS;
  if (!dense_smem_limit(gcn_forward_kernel<HID_T>, smem)) return false;
  const int64_t tiles = (static_cast<int64_t>(a.n) + F_ROWS - 1) / F_ROWS;
  const int grid = static_cast<int>(tiles < ctx.num_sms ? tiles : ctx.num_sms);
  gcn_forward_kernel<HID_T><<<grid, D_THREADS, smem, ctx.stream>>>(a);
  CSG_CUDA(cudaGetLastError());
  count_launches(1);
  return true;
}

template <int IN_T, int HID_T, int CLS_T>
bool backward_variant(Context &ctx, DenseArgs a) {
  const size_t smem = sizeof(float) * BackwardShared<IN_T, HID_T, CLS_T>::FLOATS;
  if (!dense_smem_limit(gcn_backward_kernel<IN_T, HID_T, CLS_T>, smem)) return false;
  const int64_t tiles = (static_cast<int64_t>(a.n) + B_ROWS - 1) / B_ROWS;
  const int grid = static_cast<int>(tiles < ctx.num_sms ? tiles : ctx.num_sms);
  if (!ensure_workspace(ctx, sizeof(float) * PartLayout<IN_T, HID_T, CLS_T>::FLOATS * static_cast<size_t>(grid))) return false;
  a.part = reinterpret_cast<float *>(ctx.ws);
  gcn_backward_kernel<IN_T, HID_T, CLS_T><<<grid, D_THREADS, smem, ctx.stream>>>(a);
  CSG_CUDA(cudaGetLastError());
  const int total = a.hid * a.in + a.cls * a.hid + a.hid;
  gcn_sums_kernel<IN_T, HID_T, CLS_T><<<(total + SUMS_THREADS - 1) / SUMS_THREADS, SUMS_THREADS, 0, ctx.stream>>>(a, grid);
  CSG_CUDA(cudaGetLastError());
  count_launches(2);
  return true;
}

template <int HID_T, int CLS_T>
bool hidden_variant(Context &ctx, DenseArgs a) {
  const size_t smem = sizeof(float) * HiddenShared<HID_T, CLS_T>::FLOATS;
  if (!dense_smem_limit(gcn_hidden_kernel<HID_T, CLS_T>, smem)) return false;
  const int64_t tiles = (static_cast<int64_t>(a.n) + B_ROWS - 1) / B_ROWS;
  const int grid = static_cast<int>(tiles < 2 * ctx.num_sms ? tiles : 2 * ctx.num_sms);
  if (!ensure_workspace(ctx, sizeof(float) * PartLayout<0, HID_T, CLS_T>::FLOATS * static_cast<size_t>(grid))) return false;
  a.part = reinterpret_cast<float *>(ctx.ws);
  gcn_hidden_kernel<HID_T, CLS_T><<<grid, D_THREADS, smem, ctx.stream>>>(a);
  CSG_CUDA(cudaGetLastError());
  gcn_sums_kernel<0, HID_T, CLS_T><<<(a.cls * a.hid + SUMS_THREADS - 1) / SUMS_THREADS, SUMS_THREADS, 0, ctx.stream>>>(a, grid);
  CSG_CUDA(cudaGetLastError());
  count_launches(2);
  return true;
}

template <int IN_T, int HID_T>
bool linear_variant(Context &ctx, int32_t n, int32_t in, int32_t hid, const float *x, const float *W, const float *b, float *Y) {
  const size_t smem = sizeof(float) * LinearShared<IN_T, HID_T>::FLOATS;
  if (!dense_smem_limit(linear_kernel<IN_T, HID_T>, smem)) return false;
  const int64_t tiles = (static_cast<int64_t>(n) + F_ROWS - 1) / F_ROWS;
  const int grid = static_cast<int>(tiles < ctx.num_sms ? tiles : ctx.num_sms);
  linear_kernel<IN_T, HID_T><<<grid, D_THREADS, smem, ctx.stream>>>(n, in, hid, x, W, b, Y);
  CSG_CUDA(cudaGetLastError());
  count_launches(1);
  return true;
}

// Limits: the weights and two tiles of `linear_kernel` (200 KB for 128 x 128) and the sums that the backward
// kernels hold in registers (64 per thread) fill an SM; wider layers take library products.
bool check_dense(const DenseArgs &a) {
  CSG_REQUIRE(a.n >= 1 && a.in >= 4 && a.in <= 128 && a.in % 4 == 0 && a.hid >= 4 && a.hid <= 128 && a.hid % 4 == 0 &&
                  a.cls >= 1 && a.cls <= a.ld && a.ld <= MAX_CLASSES,
              "gcn: expect in and hidden in multiples of 4 up to 128 and up to %d classes (got %d, %d, %d in %d columns)",
              MAX_CLASSES, a.in, a.hid, a.cls, a.ld);
  const uintptr_t all = reinterpret_cast<uintptr_t>(a.P) | reinterpret_cast<uintptr_t>(a.Z);
  CSG_REQUIRE(all % 16 == 0, "gcn: dense operands must be 16-byte aligned");
  return true;
}

bool run_forward(Context &ctx, const DenseArgs &a) {
  if (!check_dense(a)) return false;
  CSG_CUDA(cudaSetDevice(ctx.device));
  return a.hid <= 32 ? forward_variant<32>(ctx, a) : a.hid <= 64 ? forward_variant<64>(ctx, a) : forward_variant<128>(ctx, a);
}

template <int CLS_T>
bool run_backward_classes(Context &ctx, const DenseArgs &a) {
  if (a.in <= 64)
    return a.hid <= 32   ? backward_variant<64, 32, CLS_T>(ctx, a)
           : a.hid <= 64 ? backward_variant<64, 64, CLS_T>(ctx, a)
                         : backward_variant<64, 128, CLS_T>(ctx, a);
  return a.hid <= 32   ? backward_variant<128, 32, CLS_T>(ctx, a)
         : a.hid <= 64 ? backward_variant<128, 64, CLS_T>(ctx, a)
                       : backward_variant<128, 128, CLS_T>(ctx, a);
}

bool run_backward(Context &ctx, const DenseArgs &a) {
  if (!check_dense(a)) return false;
  CSG_CUDA(cudaSetDevice(ctx.device));
  return a.cls <= 16   ? run_backward_classes<16>(ctx, a)
         : a.cls <= 32 ? run_backward_classes<32>(ctx, a)
                       : run_backward_classes<MAX_CLASSES>(ctx, a);
}

template <int CLS_T>
bool run_hidden_classes(Context &ctx, const DenseArgs &a) {
  return a.hid <= 32   ? hidden_variant<32, CLS_T>(ctx, a)
         : a.hid <= 64 ? hidden_variant<64, CLS_T>(ctx, a)
                       : hidden_variant<128, CLS_T>(ctx, a);
}

bool run_hidden(Context &ctx, DenseArgs a) {
  if (!check_dense(a)) return false;
  CSG_CUDA(cudaSetDevice(ctx.device));
  a.in = 0;  // (no input gradients among the sums)
  return a.cls <= 16 ? run_hidden_classes<16>(ctx, a) : a.cls <= 32 ? run_hidden_classes<32>(ctx, a) : run_hidden_classes<MAX_CLASSES>(ctx, a);
}

bool run_inputs(Context &ctx, DenseArgs a) {
  if (!check_dense(a)) return false;
  CSG_CUDA(cudaSetDevice(ctx.device));
  a.cls = 0;
  return run_backward_classes<0>(ctx, a);
}

bool run_row_sums(Context &ctx, int32_t n, int32_t nnz, const int32_t *ptr, const float *val, float *out) {
  CSG_CUDA(cudaSetDevice(ctx.device));
  int64_t grid = (static_cast<int64_t>(n) + 31) / 32;
  if (grid > ctx.num_sms * 8) grid = ctx.num_sms * 8;
  // at most nnz / SUM_SPLIT pieces: a piece shorter than that is the end of a row with a full one
  if (!ensure_workspace(ctx, 256 + sizeof(int2) * (static_cast<size_t>(nnz) / SUM_SPLIT + 1))) return false;
  uint32_t *const queued = reinterpret_cast<uint32_t *>(ctx.ws);
  int2 *const queue = reinterpret_cast<int2 *>(ctx.ws + 256);
  CSG_CUDA(cudaMemsetAsync(queued, 0, sizeof(uint32_t), ctx.stream));
  row_sums_kernel<<<static_cast<int>(grid), 256, 0, ctx.stream>>>(n, nnz, ptr, val, out, queued, queue);
  CSG_CUDA(cudaGetLastError());
  row_pieces_kernel<<<ctx.num_sms, 256, 0, ctx.stream>>>(ptr, val, out, queued, queue);
  CSG_CUDA(cudaGetLastError());
  count_launches(2);
  return true;
}

}  // namespace

bool launch_gcn_forward(Context &ctx, int32_t n, int32_t hid, int32_t cls, int32_t ld, const float *Z, const float *W2,
                        float *U) {
  DenseArgs a = {};
  a.n = n, a.in = 4, a.hid = hid, a.cls = cls, a.ld = ld, a.Z = Z, a.W2 = W2, a.U = U;
  return run_forward(ctx, a);
}
bool launch_gcn_backward(Context &ctx, int32_t n, int32_t in, int32_t hid, int32_t cls, int32_t ld, const float *G,
                         const float *Z, const float *P, const float *s, const float *W2, float *dW1, float *db1, float *dW2) {
  DenseArgs a = {};
  a.n = n, a.in = in, a.hid = hid, a.cls = cls, a.ld = ld, a.G = G, a.Z = Z, a.P = P, a.s = s, a.W2 = W2;
  a.dW1 = dW1, a.db1 = db1, a.dW2 = dW2;
  return run_backward(ctx, a);
}
bool launch_gcn_hidden_gradient(Context &ctx, int32_t n, int32_t hid, int32_t cls, int32_t ld, const float *G,
                                const float *Z, const float *W2, float *D, float *dW2) {
  DenseArgs a = {};
  a.n = n, a.in = 4, a.hid = hid, a.cls = cls, a.ld = ld, a.G = G, a.Z = Z, a.W2 = W2, a.D = D, a.dW2 = dW2;
  return run_hidden(ctx, a);
}
bool launch_gcn_input_gradients(Context &ctx, int32_t n, int32_t in, int32_t hid, const float *E, const float *x,
                                float *dW1, float *db1) {
  DenseArgs a = {};
  a.n = n, a.in = in, a.hid = hid, a.cls = a.ld = 1, a.Z = E, a.P = x, a.dW1 = dW1, a.db1 = db1;
  return run_inputs(ctx, a);
}
bool launch_pad_columns(Context &ctx, int32_t n, int32_t from, int32_t to, const float *src, float *dst) {
  CSG_REQUIRE(n >= 1 && from >= 1 && to >= from, "pad_columns: bad sizes n=%d from=%d to=%d", n, from, to);
  CSG_CUDA(cudaSetDevice(ctx.device));
  const int64_t blocks = (static_cast<int64_t>(n) * to + 255) / 256;
  pad_columns_kernel<<<static_cast<int>(blocks < ctx.num_sms * 8 ? blocks : ctx.num_sms * 8), 256, 0, ctx.stream>>>(n, from, to, src, dst);
  CSG_CUDA(cudaGetLastError());
  count_launches(1);
  return true;
}
bool launch_linear(Context &ctx, int32_t n, int32_t in, int32_t hid, const float *x, const float *W, const float *b, float *Y) {
  CSG_REQUIRE(n >= 1 && in >= 4 && in <= 128 && in % 4 == 0 && hid >= 4 && hid <= 128 && hid % 4 == 0,
              "linear: expect inputs and outputs in multiples of 4 up to 128 (got %d, %d)", in, hid);
  CSG_REQUIRE((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(Y)) % 16 == 0, "linear: x and Y must be 16-byte aligned");
  CSG_CUDA(cudaSetDevice(ctx.device));
  if (in <= 64)
    return hid <= 32   ? linear_variant<64, 32>(ctx, n, in, hid, x, W, b, Y)
           : hid <= 64 ? linear_variant<64, 64>(ctx, n, in, hid, x, W, b, Y)
                       : linear_variant<64, 128>(ctx, n, in, hid, x, W, b, Y);
  return hid <= 32   ? linear_variant<128, 32>(ctx, n, in, hid, x, W, b, Y)
         : hid <= 64 ? linear_variant<128, 64>(ctx, n, in, hid, x, W, b, Y)
                     : linear_variant<128, 128>(ctx, n, in, hid, x, W, b, Y);
}
bool launch_row_sums(Context &ctx, int32_t n, int32_t nnz, const int32_t *d_ptr, const float *d_val, float *d_out) {
  return run_row_sums(ctx, n, nnz, d_ptr, d_val, d_out);
}

}  // namespace csg
