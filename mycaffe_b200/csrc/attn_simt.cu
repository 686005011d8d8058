// Exact-fp32 scaled-dot-product attention on CUDA cores: forward, and a recompute-based
// backward.  Handles with MCA_FLAG_EXACT_FP32 run it, and fp32 handles where there is no split-operand tensor-core kernel
// (attn_tc.cu, attn_tc_bwd.cu): other head sizes than 16, 32, 64 and 128, and the backward of 128.  It reproduces the
// reference's arithmetic (attn.cu:518-661 of CudaDnnDLL) -- scale applied to the finished dot
// product, masked logits overwritten with the finite value -1e29, max-subtracted softmax --
// without ever materialising the (B,H,T,T) score tensors the reference allocates in
// attnHandle::Set (attn.cu:436-452).  It accepts every mask form of the reference and any head
// size up to 128.
//
// Tiling.  What bounds these kernels is the fp32 FMA pipe, and what keeps a kernel from it is feeding the pipe: every
// product reads both operands from shared memory, and a 16-byte load of a warp takes two cycles of the shared-memory pipe
// whatever it reads -- four unless each address is shared by lanes that differ in one of the low two lane bits (measured).
// One CTA of 256 threads keeps R rows resident (R = 128, or 64 where 128-row tiles would not give every SM one: queries in
// the forward and dQ kernels, keys in the dK/dV kernel) and walks the other side 64 rows at a time.
//   * A . B^T over the head (scores, dP): a thread owns an 8 x 4 piece (4 x 8 in the forward, where a warp keeps whole
//     rows) of the R x 64 tile and reads 16-byte vectors along the head: 12 loads for 128 multiply-adds.
//   * X B over the 64 walked rows (P V, P^T dY, dS K, dS^T Q): X is written to shared memory transposed, a thread owns
//     8 rows x DP / 16 columns of the result: 4 loads for 64 multiply-adds at 128-wide heads, issued as packed pairs
//     (fma.rn.f32x2: exact fp32 at half the issue slots).
// Lane bit 0 selects a column and lane bit 1 a row, so that the operands of both sides load in two cycles.
// Tiles have no padding: the 16-byte vectors of a row are XOR-permuted by the row's low three bits, which keeps all of
// these reads and the transposed write free of bank conflicts and lets 128-wide heads fit (224 KB in the dK/dV kernel).
// The tiles arrive by cp.async under the products that do not need them.
// Backward of B = 2, H = 16, T = 1500, D = 128, causal: 2.71 ms with 64 x 64 tiles and 4 x 4 pieces, 1.92 ms with this (57 % of the
// fp32 pipe: two warps per scheduler do not hide every load), 1.35 with dS formed once; B = 1, H = 12, T = 1516, D = 80 forward and backward: 1.75 -> 0.78 ms.
#include <algorithm>

#include "classify.cuh"
#include "common.cuh"
#include "kernels.h"

namespace {

constexpr int SX = 64;         // rows of the walked side per step
constexpr int NT = 256;        // threads per CTA

// Head sizes are padded to DP; a shared row holds LD floats (whole groups of eight 16-byte vectors).
template <int DP> struct Row {
  static constexpr int LD = (DP + 31) / 32 * 32;
  static constexpr int V4 = DP / 4;
};
// Where float4 c4 of row r lives.
template <int DP> __device__ __forceinline__ int at(int r, int c4) { return r * Row<DP>::LD + ((c4 ^ (r & 7)) << 2); }
// Where element r of walked row j lives in the transposed tile X (SX x R).
template <int R> __device__ __forceinline__ int xat(int j, int r) { return j * R + (((r >> 2) ^ (j & 7)) << 2) + (r & 3); }

// Lane -> (row, column) of a 4 x 8 lane grid, and the grid of the products X B over all threads (16 row groups x 16 column
// groups: a warp is 4 x 8 of it).
__device__ __forceinline__ int lane_row(int lane) { return ((lane >> 1) & 1) | ((lane >> 4) << 1); }
__device__ __forceinline__ int lane_col(int lane) { return (lane & 1) | (((lane >> 2) & 3) << 1); }

// A thread's share of a product X B: R / 16 rows x DP / 16 columns.  Column group cg owns four columns of every whole 64,
// then two of a remaining 32 and one of a remaining 16.
template <int DP, int R> struct Out {
  static constexpr int RPT = R / 16;
  static constexpr int N4 = DP / 64;                // 16-byte chunks
  static constexpr int N2 = (DP % 64) / 32;         // 8-byte chunk
  static constexpr int N1 = (DP % 32) / 16;         // 4-byte chunk
  static constexpr int OFF2 = N4 * 64, OFF1 = OFF2 + N2 * 32;
  static constexpr int NP = N4 * 2 + N2;            // accumulator pairs per row, then N1 single ones
};
template <int DP, int R> struct Acc {
  float2 p[Out<DP, R>::RPT][Out<DP, R>::NP > 0 ? Out<DP, R>::NP : 1];
  float s[Out<DP, R>::RPT];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < Out<DP, R>::RPT; ++i) {
      s[i] = 0.f;
#pragma unroll
      for (int c = 0; c < Out<DP, R>::NP; ++c) p[i][c] = make_float2(0.f, 0.f);
    }
  }
  __device__ __forceinline__ void scale(int i, float f) {
    s[i] *= f;
#pragma unroll
    for (int c = 0; c < Out<DP, R>::NP; ++c) { p[i][c].x *= f; p[i][c].y *= f; }
  }
};

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(d)
      : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)), "l"(*reinterpret_cast<uint64_t*>(&c)));
  return *reinterpret_cast<float2*>(&d);
}

// Rows [row0, row0 + ROWS) of a (T,D) matrix with row stride ld -> a shared tile; rows >= T and columns >= D are zero.
// With 16-byte aligned rows the copies are asynchronous (the caller commits and waits).
template <int DP, int ROWS>
__device__ __forceinline__ void load_rows(float* __restrict__ s, const float* __restrict__ g, int64_t ld, int row0, int T, int D,
                                          bool vec_ok, int tid) {
  constexpr int V4 = Row<DP>::V4;
  if (vec_ok) {
    for (int idx = tid; idx < ROWS * V4; idx += NT) {
      const int r = idx / V4, c4 = idx - r * V4;
      const bool in = row0 + r < T && c4 * 4 < D;
      const float* src = in ? g + (int64_t)(row0 + r) * ld + c4 * 4 : g;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(s + at<DP>(r, c4))), "l"(src),
                   "r"(in ? 16 : 0)
                   : "memory");
    }
  } else {
    for (int idx = tid; idx < ROWS * DP; idx += NT) {
      const int r = idx / DP, c = idx - r * DP;
      s[at<DP>(r, c >> 2) + (c & 3)] = (row0 + r < T && c < D) ? __ldg(g + (int64_t)(row0 + r) * ld + c) : 0.f;
    }
  }
}

// s[a][b] = sum_d A[ra + RS a][d] * B[cb + CS b][d]; the even and the odd d are summed apart, as the halves of a pair
template <int DP, int NA, int RS, int NB, int CS>
__device__ __forceinline__ void product_nt(const float* __restrict__ As, const float* __restrict__ Bs, int ra, int cb, float (&s)[NA][NB]) {
  float2 acc[NA][NB];
#pragma unroll
  for (int a = 0; a < NA; ++a)
#pragma unroll
    for (int b = 0; b < NB; ++b) acc[a][b] = make_float2(0.f, 0.f);
#pragma unroll 2
  for (int c4 = 0; c4 < Row<DP>::V4; ++c4) {
    float4 av[NA], bv[NB];
#pragma unroll
    for (int a = 0; a < NA; ++a) av[a] = *reinterpret_cast<const float4*>(As + at<DP>(ra + RS * a, c4));
#pragma unroll
    for (int b = 0; b < NB; ++b) bv[b] = *reinterpret_cast<const float4*>(Bs + at<DP>(cb + CS * b, c4));
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        acc[a][b] = fma2(make_float2(av[a].x, av[a].y), make_float2(bv[b].x, bv[b].y), acc[a][b]);
        acc[a][b] = fma2(make_float2(av[a].z, av[a].w), make_float2(bv[b].z, bv[b].w), acc[a][b]);
      }
  }
#pragma unroll
  for (int a = 0; a < NA; ++a)
#pragma unroll
    for (int b = 0; b < NB; ++b) s[a][b] = acc[a][b].x + acc[a][b].y;
}

// Row j of B, the columns of group cg.
template <int DP, int R>
__device__ __forceinline__ void load_columns(const float* __restrict__ Bs, int j, int cg, float2* bp, float& b1) {
  using O = Out<DP, R>;
  b1 = 0.f;
#pragma unroll
  for (int c = 0; c < O::N4; ++c) {
    const float4 b = *reinterpret_cast<const float4*>(Bs + at<DP>(j, 16 * c + cg));
    bp[2 * c] = make_float2(b.x, b.y); bp[2 * c + 1] = make_float2(b.z, b.w);
  }
  if constexpr (O::N2 > 0) bp[2 * O::N4] = *reinterpret_cast<const float2*>(Bs + at<DP>(j, (O::OFF2 + 2 * cg) >> 2) + ((2 * cg) & 3));
  if constexpr (O::N1 > 0) b1 = Bs[at<DP>(j, (O::OFF1 + cg) >> 2) + (cg & 3)];
}

// acc[i] += sum_j X[j][r0 + i] * B[j][columns of group cg]
template <int DP, int R>
__device__ __forceinline__ void product_nn(const float* __restrict__ X, const float* __restrict__ Bs, int r0, int cg, Acc<DP, R>& acc) {
  using O = Out<DP, R>;
#pragma unroll 2
  for (int j = 0; j < SX; ++j) {
    float2 bp[O::NP > 0 ? O::NP : 1];
    float b1;
    load_columns<DP, R>(Bs, j, cg, bp, b1);
    float x[O::RPT];
#pragma unroll
    for (int h = 0; h < O::RPT / 4; ++h) {
      const float4 t = *reinterpret_cast<const float4*>(X + xat<R>(j, r0 + 4 * h));
      x[4 * h] = t.x; x[4 * h + 1] = t.y; x[4 * h + 2] = t.z; x[4 * h + 3] = t.w;
    }
#pragma unroll
    for (int i = 0; i < O::RPT; ++i) {
      const float2 xx = make_float2(x[i], x[i]);
#pragma unroll
      for (int c = 0; c < O::NP; ++c) acc.p[i][c] = fma2(xx, bp[c], acc.p[i][c]);
      if constexpr (O::N1 > 0) acc.s[i] = fmaf(x[i], b1, acc.s[i]);
    }
  }
}

// This thread's piece -> rows row0, row0 + RS, ... of a (T,D) view.
template <int DP, int R, int RS = 1>
__device__ __forceinline__ void store_piece(float* __restrict__ g, int64_t ld, int row0, int cg, int T, int D, bool vec_ok,
                                            const Acc<DP, R>& acc) {
  using O = Out<DP, R>;
#pragma unroll
  for (int i = 0; i < O::RPT; ++i) {
    if (row0 + RS * i >= T) continue;
    float* dst = g + (int64_t)(row0 + RS * i) * ld;
#pragma unroll
    for (int c = 0; c < O::N4; ++c) {
      const int col = 64 * c + 4 * cg;
      const float v[4] = {acc.p[i][2 * c].x, acc.p[i][2 * c].y, acc.p[i][2 * c + 1].x, acc.p[i][2 * c + 1].y};
      if (vec_ok && col < D) *reinterpret_cast<float4*>(dst + col) = make_float4(v[0], v[1], v[2], v[3]);
      else {
#pragma unroll
        for (int k = 0; k < 4; ++k) if (col + k < D) dst[col + k] = v[k];
      }
    }
    if constexpr (O::N2 > 0) {
      const int col = O::OFF2 + 2 * cg;
      if (vec_ok && col < D) *reinterpret_cast<float2*>(dst + col) = acc.p[i][2 * O::N4];
      else {
        if (col < D) dst[col] = acc.p[i][2 * O::N4].x;
        if (col + 1 < D) dst[col + 1] = acc.p[i][2 * O::N4].y;
      }
    }
    if constexpr (O::N1 > 0) {
      const int col = O::OFF1 + cg;
      if (col < D) dst[col] = acc.s[i];
    }
  }
}

// Logit after scale and mask, the reference's order (attn.cu:567-583).  Keys beyond T do not
// exist: they get -inf so that they contribute exactly zero probability.
__device__ __forceinline__ float masked_logit(float dot, float scale, int i, int j, int b, int T, int mode,
                                              const float* __restrict__ mask) {
  if (j >= T) return -INFINITY;
  float s = dot * scale;
  if (mode == MCA_MASK_CAUSAL) { if (j > i) s = MCA_MASKED_LOGIT; }
  else if (mode == MCA_MASK_TT) { if (i < T && __ldg(mask + (int64_t)i * T + j) == 0.f) s = MCA_MASKED_LOGIT; }
  else if (mode == MCA_MASK_BATCH) { if (__ldg(mask + (int64_t)b * T + j) == 0.f) s = MCA_MASKED_LOGIT; }
  return s;
}

// A (T,T) mask that a preceding classification launch found to be exactly tril(ones) is
// treated as analytic causal (tiles above the diagonal are skipped).
__device__ __forceinline__ int effective_mode(int mode, const int* __restrict__ causal_flag) {
  if (mode == MCA_MASK_TT && causal_flag != nullptr && *causal_flag != 0) return MCA_MASK_CAUSAL;
  return mode;
}

__device__ __forceinline__ void load_commit() { mca_cp_async_commit(); }

// (batch, head) of the CTA is blockIdx.x and the tile blockIdx.y, so that CTAs start tile by tile over all heads: with a
// causal mask the long tiles first.
template <int DP, int R>
constexpr size_t fwd_smem_bytes() { return sizeof(float) * ((R + 2 * SX) * Row<DP>::LD + SX * R + 2 * R); }

template <int DP, int R>
__global__ void __launch_bounds__(NT) sdpa_fwd_f32_kernel(const float* __restrict__ Q, const float* __restrict__ K,
                                                         const float* __restrict__ V,
                                                         const float* __restrict__ mask, int mask_mode,
                                                         const int* __restrict__ causal_flag, int H, int T, int D,
                                                         float scale, float* __restrict__ Y,
                                                         float* __restrict__ row_max, float* __restrict__ row_sum,
                                                         float* __restrict__ y_copy, int vec_ok, int vec_out,
                                                         const McaStrides sin, const McaStrides sout) {
  extern __shared__ __align__(16) float smem[];
  constexpr int LD = Row<DP>::LD, NA = R / 32, RPT = Out<DP, R>::RPT;
  float* Qs = smem;
  float* Ks = Qs + R * LD;
  float* Vs = Ks + SX * LD;
  float* X = Vs + SX * LD;        // P transposed: [key][query]
  float* s_corr = X + SX * R;     // this step's rescale of each row; the reciprocal row sums at the end
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ra = warp * (R / 8) + lane_row(lane), cb = lane_col(lane);         // scores: rows ra + 4 a, keys cb + 8 b: a warp has whole rows
  const int cg = (warp & 1) * 8 + lane_col(lane), r0 = ((warp >> 1) * 4 + lane_row(lane)) * RPT;   // P V: rows r0 .., column group cg
  const int bh = blockIdx.x, b = bh / H;
  const int q0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * R;
  const int mode = effective_mode(mask_mode, causal_flag);
  const int64_t in_base = (int64_t)b * sin.b + (int64_t)(bh - b * H) * sin.h;
  const float* Kg = K + in_base;
  const float* Vg = V + in_base;

  load_rows<DP, R>(Qs, Q + in_base, sin.t, q0, T, D, vec_ok, tid);
  load_rows<DP, SX>(Ks, Kg, sin.t, 0, T, D, vec_ok, tid);
  load_commit();
  load_rows<DP, SX>(Vs, Vg, sin.t, 0, T, D, vec_ok, tid);
  load_commit();
  float m[NA], l[NA];
  Acc<DP, R> acc;
  acc.clear();
#pragma unroll
  for (int a = 0; a < NA; ++a) { m[a] = -INFINITY; l[a] = 0.f; }
  const int kv_end = (mode == MCA_MASK_CAUSAL) ? min(T, q0 + R) : T;
  for (int k0 = 0; k0 < kv_end; k0 += SX) {
    mca_cp_async_wait<1>();   // K of this step (and Q); V may still be on its way
    __syncthreads();
    float s[NA][8];
    product_nt<DP, NA, 4, 8, 8>(Qs, Ks, ra, cb, s);
#pragma unroll
    for (int a = 0; a < NA; ++a) {
      const int r = ra + 4 * a, i = q0 + r;
      float mx = -INFINITY;
#pragma unroll
      for (int bb = 0; bb < 8; ++bb) {
        s[a][bb] = masked_logit(s[a][bb], scale, i, k0 + cb + 8 * bb, b, T, mode, mask);
        mx = fmaxf(mx, s[a][bb]);
      }
      for (const int o : {1, 4, 8}) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));   // the lanes of a row (lane_col)
      const float m_new = fmaxf(m[a], mx);
      const float corr = __expf(m[a] - m_new);  // exp(-inf) = 0 on the first step
      float rs = 0.f;
#pragma unroll
      for (int bb = 0; bb < 8; ++bb) {
        const float p = expf(s[a][bb] - m_new);
        rs += p;
        X[xat<R>(cb + 8 * bb, r)] = p;
      }
      for (const int o : {1, 4, 8}) rs += __shfl_xor_sync(0xffffffffu, rs, o);
      l[a] = l[a] * corr + rs;
      m[a] = m_new;
      if (cb == 0) s_corr[r] = corr;
    }
    mca_cp_async_wait<0>();   // V of this step
    __syncthreads();          // P, the rescale factors and V are in place; K has been read
    if (k0 + SX < kv_end) load_rows<DP, SX>(Ks, Kg, sin.t, k0 + SX, T, D, vec_ok, tid);
    load_commit();
#pragma unroll
    for (int i = 0; i < RPT; ++i) acc.scale(i, s_corr[r0 + i]);
    product_nn<DP, R>(X, Vs, r0, cg, acc);
    __syncthreads();
    if (k0 + SX < kv_end) load_rows<DP, SX>(Vs, Vg, sin.t, k0 + SX, T, D, vec_ok, tid);
    load_commit();
  }
#pragma unroll
  for (int a = 0; a < NA; ++a) {
    const int r = ra + 4 * a, i = q0 + r;
    if (cb == 0) {
      s_corr[r] = 1.f / l[a];
      if (i < T && row_max) { row_max[(int64_t)bh * T + i] = m[a]; row_sum[(int64_t)bh * T + i] = l[a]; }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < RPT; ++i) acc.scale(i, s_corr[r0 + i]);
  store_piece<DP, R>(Y + (int64_t)b * sout.b + (int64_t)(bh - b * H) * sout.h, sout.t, q0 + r0, cg, T, D, vec_out != 0, acc);
  if (y_copy) store_piece<DP, R>(y_copy + (int64_t)bh * T * D, D, q0 + r0, cg, T, D, vec_out != 0, acc);
}

// delta[i] = sum_c dY[i][c] * Y[i][c]  (the rowsum(dP o P) term of the softmax backward).
__global__ void sdpa_bwd_delta_kernel(const float* __restrict__ dY, const float* __restrict__ Ysaved, int64_t rows,
                                      int H, int T, int D, const McaStrides sdy, float* __restrict__ delta) {
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  const int64_t bh = row / T;
  const int64_t b = bh / H;
  const float* dyr = dY + b * sdy.b + (bh - b * H) * sdy.h + (row - bh * T) * sdy.t;   // Ysaved is the handle's own contiguous copy
  float acc = 0.f;
  for (int c = lane; c < D; c += 32) acc = fmaf(dyr[c], Ysaved[row * D + c], acc);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) delta[row] = acc;
}

template <int DP, int R>
constexpr size_t bwd_smem_bytes() { return sizeof(float) * (2 * (R + SX) * Row<DP>::LD + SX * R + 3 * SX); }

// dS of (SX queries) x (R keys), as the dK/dV kernel leaves it for the dQ kernel: its tile X as it lies in shared memory, by head,
// query block and key block.
template <int R> __host__ __device__ __forceinline__ int64_t ds_tile(int bh, int qb, int kb, int T) {
  const int nq = (T + SX - 1) / SX, nk = (T + R - 1) / R;
  return (((int64_t)bh * nq + qb) * nk + kb) * (SX * R);
}

// dK, dV for one tile of R keys: walks the query tiles, recomputes P from the saved row
// statistics, and accumulates dV += P^T dY, dK += dS^T Q (attn.cu:380-397, 637-657).
template <int DP, int R>
__global__ void __launch_bounds__(NT) sdpa_bwd_dkdv_f32_kernel(
    const float* __restrict__ Q, const float* __restrict__ K, const float* __restrict__ V,
    const float* __restrict__ dY, const float* __restrict__ mask, int mask_mode, const int* __restrict__ causal_flag,
    const float* __restrict__ row_max, const float* __restrict__ row_sum, const float* __restrict__ delta, int H,
    int T, int D, float scale, float* __restrict__ dK, float* __restrict__ dV, float* __restrict__ dS, int vec_ok, int vec_out,
    const McaStrides sin, const McaStrides sout) {
  extern __shared__ __align__(16) float smem[];
  constexpr int LD = Row<DP>::LD, NA = R / 16, RPT = Out<DP, R>::RPT;
  float* Ks = smem;
  float* Vs = Ks + R * LD;
  float* Qs = Vs + R * LD;
  float* dOs = Qs + SX * LD;
  float* X = dOs + SX * LD;      // P^T, then dS^T, transposed: [query][key]
  float* s_m = X + SX * R;       // the step's query statistics: row maximum, 1 / row sum, delta
  float *s_il = s_m + SX, *s_de = s_il + SX;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ra = (warp >> 1) * 4 + lane_row(lane), cb = (warp & 1) * 8 + lane_col(lane);   // scores: keys ra + 16 a, queries cb + 16 b
  const int cg = (warp & 1) * 8 + lane_col(lane), r0 = ((warp >> 1) * 4 + lane_row(lane)) * RPT;
  const int bh = blockIdx.x, b = bh / H;
  const int k0 = blockIdx.y * R;
  const int mode = effective_mode(mask_mode, causal_flag);
  const int64_t base = (int64_t)b * sin.b + (int64_t)(bh - b * H) * sin.h;
  const float* Qg = Q + base;
  const float* dYg = dY + (int64_t)b * sout.b + (int64_t)(bh - b * H) * sout.h;
  const int q_begin = (mode == MCA_MASK_CAUSAL) ? k0 : 0;  // k0 is a multiple of 64
  mca_pdl_launch_dependents();   // an ordinary launch: all before it is complete, so the dQ kernel may use the SMs this one leaves
  load_rows<DP, R>(Ks, K + base, sin.t, k0, T, D, vec_ok, tid);
  load_rows<DP, R>(Vs, V + base, sin.t, k0, T, D, vec_ok, tid);
  load_rows<DP, SX>(Qs, Qg, sin.t, q_begin, T, D, vec_ok, tid);
  load_rows<DP, SX>(dOs, dYg, sout.t, q_begin, T, D, vec_ok, tid);
  load_commit();
  Acc<DP, R> dk, dv;
  dk.clear(); dv.clear();
  for (int q0 = q_begin; q0 < T; q0 += SX) {
    if (tid < SX) {
      const int i = q0 + tid;
      const bool in = i < T;         // queries beyond T: probability 0
      s_m[tid] = in ? row_max[(int64_t)bh * T + i] : 0.f;
      s_il[tid] = in ? 1.f / row_sum[(int64_t)bh * T + i] : 0.f;
      s_de[tid] = in ? delta[(int64_t)bh * T + i] : 0.f;
    }
    mca_cp_async_wait<0>();
    __syncthreads();
    {
      float s[NA][4];
      product_nt<DP, NA, 16, 4, 16>(Ks, Qs, ra, cb, s);     // s[a][b]: key ra + 16 a, query cb + 16 b
#pragma unroll
      for (int bb = 0; bb < 4; ++bb) {
        const int c = cb + 16 * bb;
        const float mi = s_m[c], il = s_il[c];
#pragma unroll
        for (int a = 0; a < NA; ++a) {
          const float sv = masked_logit(s[a][bb], scale, q0 + c, k0 + ra + 16 * a, b, T, mode, mask);
          X[xat<R>(c, ra + 16 * a)] = q0 + c < T ? expf(sv - mi) * il : 0.f;
        }
      }
    }
    __syncthreads();
    product_nn<DP, R>(X, dOs, r0, cg, dv);
    {
      float dp[NA][4];
      product_nt<DP, NA, 16, 4, 16>(Vs, dOs, ra, cb, dp);
      __syncthreads();                // P^T and dY have been read
      if (q0 + SX < T) load_rows<DP, SX>(dOs, dYg, sout.t, q0 + SX, T, D, vec_ok, tid);
      load_commit();
#pragma unroll
      for (int bb = 0; bb < 4; ++bb) {   // P^T -> dS^T in place, each thread its own elements
        const float de = s_de[cb + 16 * bb];
#pragma unroll
        for (int a = 0; a < NA; ++a) {
          float* x = X + xat<R>(cb + 16 * bb, ra + 16 * a);
          *x = *x * (dp[a][bb] - de) * scale;
        }
      }
      if (dS != nullptr) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    if (dS != nullptr && tid == 0) {   // the whole tile as it lies, in one copy under the product
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n\tcp.async.bulk.commit_group;" ::"l"(
                       dS + ds_tile<R>(bh, q0 / SX, k0 / R, T)),
                   "r"((uint32_t)__cvta_generic_to_shared(X)), "n"(SX * R * 4)
                   : "memory");
    }
    product_nn<DP, R>(X, Qs, r0, cg, dk);
    if (dS != nullptr && tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // X may be overwritten
    __syncthreads();
    if (q0 + SX < T) load_rows<DP, SX>(Qs, Qg, sin.t, q0 + SX, T, D, vec_ok, tid);
    load_commit();
  }
  store_piece<DP, R>(dK + base, sin.t, k0 + r0, cg, T, D, vec_out != 0, dk);
  store_piece<DP, R>(dV + base, sin.t, k0 + r0, cg, T, D, vec_out != 0, dv);
  if (dS != nullptr && tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// dQ for 64 queries from the dS the dK/dV kernel left: one product instead of three, so 5 of the backward's 7 are formed.  The FMA
// pipe is the bound (70 % active; the dK/dV kernel, with two warps per scheduler, keeps it at 61 %).  Steps of 32 keys in a ring of
// three, so that two CTAs share an SM and four warps a scheduler; 64 queries a CTA whatever R is, so that the last ones are
// short; a thread's rows are 16 apart, so that the rows a warp reads at a time lie in different banks.
// B = 2, H = 16, T = 1500, D = 128, causal, forward and backward: 2048 us with dS formed twice, 1486 with this (dK/dV 1146 and dQ
// 238 us when each runs alone).
constexpr int DS_KEYS = 32, DS_STAGES = 3;
template <int DP> constexpr size_t dq_ds_smem_bytes() { return sizeof(float) * DS_STAGES * (SX * DS_KEYS + DS_KEYS * Row<DP>::LD); }
template <int DP, int RK>
__global__ void __launch_bounds__(NT, 2) sdpa_bwd_dq_ds_f32_kernel(const float* __restrict__ K, const float* dS, int mask_mode,
                                                                   const int* __restrict__ causal_flag, int H, int T, int D,
                                                                   float* __restrict__ dQ, int vec_ok, int vec_out, const McaStrides sin) {
  extern __shared__ __align__(16) float smem[];
  constexpr int R = SX;
  using O = Out<DP, R>;
  constexpr int A = R * DS_KEYS, STAGE = A + DS_KEYS * Row<DP>::LD;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cg = (warp & 1) * 8 + lane_col(lane), rg = (warp >> 1) * 4 + lane_row(lane);   // rows rg + 16 i
  const int bh = blockIdx.x, b = bh / H;
  const int q0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * R;
  const int mode = effective_mode(mask_mode, causal_flag);
  const int64_t base = (int64_t)b * sin.b + (int64_t)(bh - b * H) * sin.h;
  const int kv_end = (mode == MCA_MASK_CAUSAL) ? min(T, q0 + R) : T;
  // This thread copies 16-byte vector lc of rows lr, lr + 32, ... of the step's dS (R rows of 32 keys).
  constexpr int VPR = DS_KEYS / 4, RPP = NT / VPR;
  const int lr = tid / VPR, lc = tid % VPR;
  const float* src0 = dS + ds_tile<RK>(bh, q0 / SX, 0, T) + lr * RK;
  auto load = [&](int k0, float* st) {
    const float* src = src0 + (int64_t)(k0 / RK) * (SX * RK) + ((((k0 % RK) / 4 + lc) ^ (lr & 7)) << 2);
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(st + at<DS_KEYS>(lr, lc));
#pragma unroll
    for (int i = 0; i < R / RPP; ++i)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * RPP * DS_KEYS * 4), "l"(src + i * RPP * RK) : "memory");
    load_rows<DP, DS_KEYS>(st + A, K + base, sin.t, k0, T, D, vec_ok, tid);
  };
  mca_pdl_wait();   // dS is the kernel before's
#pragma unroll
  for (int i = 0; i < DS_STAGES - 1; ++i) {
    if (i * DS_KEYS < kv_end) load(i * DS_KEYS, smem + i * STAGE);
    load_commit();
  }
  Acc<DP, R> dq;
  dq.clear();
  for (int k0 = 0, s = 0; k0 < kv_end; k0 += DS_KEYS, s = s + 1 == DS_STAGES ? 0 : s + 1) {
    mca_cp_async_wait<DS_STAGES - 2>();
    __syncthreads();                  // the step's tiles are in place, and the stage before them has been read
    const int next = s == 0 ? DS_STAGES - 1 : s - 1;
    if (k0 + (DS_STAGES - 1) * DS_KEYS < kv_end) load(k0 + (DS_STAGES - 1) * DS_KEYS, smem + next * STAGE);
    load_commit();
    const float *As = smem + s * STAGE, *Bs = As + A;
#pragma unroll 2
    for (int j4 = 0; j4 < DS_KEYS / 4; ++j4) {
      float4 x[O::RPT];
#pragma unroll
      for (int i = 0; i < O::RPT; ++i) x[i] = *reinterpret_cast<const float4*>(As + at<DS_KEYS>(rg + 16 * i, j4));
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        const int j = 4 * j4 + jj;
        float2 bp[O::NP > 0 ? O::NP : 1];
        float b1;
        load_columns<DP, R>(Bs, j, cg, bp, b1);
#pragma unroll
        for (int i = 0; i < O::RPT; ++i) {
          const float xi = jj == 0 ? x[i].x : jj == 1 ? x[i].y : jj == 2 ? x[i].z : x[i].w;
          const float2 xx = make_float2(xi, xi);
#pragma unroll
          for (int c = 0; c < O::NP; ++c) dq.p[i][c] = fma2(xx, bp[c], dq.p[i][c]);
          if constexpr (O::N1 > 0) dq.s[i] = fmaf(xi, b1, dq.s[i]);
        }
      }
    }
  }
  store_piece<DP, R, 16>(dQ + base, sin.t, q0 + rg, cg, T, D, vec_out != 0, dq);
}

// dQ for one tile of R queries: dQ = dS K with dS recomputed per key tile.  For when there is no room for dS, and for problems
// small enough that this kernel runs beside the dK/dV kernel.
template <int DP, int R>
__global__ void __launch_bounds__(NT) sdpa_bwd_dq_f32_kernel(
    const float* __restrict__ Q, const float* __restrict__ K, const float* __restrict__ V,
    const float* __restrict__ dY, const float* __restrict__ mask, int mask_mode, const int* __restrict__ causal_flag,
    const float* __restrict__ row_max, const float* __restrict__ row_sum, const float* __restrict__ delta, int H,
    int T, int D, float scale, float* __restrict__ dQ, int vec_ok, int vec_out, const McaStrides sin, const McaStrides sout) {
  extern __shared__ __align__(16) float smem[];
  constexpr int LD = Row<DP>::LD, NA = R / 16, RPT = Out<DP, R>::RPT;
  float* Qs = smem;
  float* dOs = Qs + R * LD;
  float* Ks = dOs + R * LD;
  float* Vs = Ks + SX * LD;
  float* X = Vs + SX * LD;       // dS transposed: [key][query]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ra = (warp >> 1) * 4 + lane_row(lane), cb = (warp & 1) * 8 + lane_col(lane);   // scores: queries ra + 16 a, keys cb + 16 b
  const int cg = (warp & 1) * 8 + lane_col(lane), r0 = ((warp >> 1) * 4 + lane_row(lane)) * RPT;
  const int bh = blockIdx.x, b = bh / H;
  const int q0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * R;
  const int mode = effective_mode(mask_mode, causal_flag);
  const int64_t base = (int64_t)b * sin.b + (int64_t)(bh - b * H) * sin.h;
  const float* Kg = K + base;
  const float* Vg = V + base;
  load_rows<DP, R>(Qs, Q + base, sin.t, q0, T, D, vec_ok, tid);
  load_rows<DP, R>(dOs, dY + (int64_t)b * sout.b + (int64_t)(bh - b * H) * sout.h, sout.t, q0, T, D, vec_ok, tid);
  load_rows<DP, SX>(Ks, Kg, sin.t, 0, T, D, vec_ok, tid);
  load_rows<DP, SX>(Vs, Vg, sin.t, 0, T, D, vec_ok, tid);
  load_commit();
  float mi[NA], inv_l[NA], di[NA];
  Acc<DP, R> dq;
#pragma unroll
  for (int a = 0; a < NA; ++a) {
    const int i = q0 + ra + 16 * a;
    mi[a] = 0.f; inv_l[a] = 0.f; di[a] = 0.f;
    if (i < T) { mi[a] = row_max[(int64_t)bh * T + i]; inv_l[a] = 1.f / row_sum[(int64_t)bh * T + i]; di[a] = delta[(int64_t)bh * T + i]; }
  }
  dq.clear();
  const int kv_end = (mode == MCA_MASK_CAUSAL) ? min(T, q0 + R) : T;
  for (int k0 = 0; k0 < kv_end; k0 += SX) {
    mca_cp_async_wait<0>();
    __syncthreads();
    float s[NA][4], dp[NA][4];
    product_nt<DP, NA, 16, 4, 16>(Qs, Ks, ra, cb, s);
#pragma unroll
    for (int a = 0; a < NA; ++a) {
      const int i = q0 + ra + 16 * a;
#pragma unroll
      for (int bb = 0; bb < 4; ++bb) {
        const float sv = masked_logit(s[a][bb], scale, i, k0 + cb + 16 * bb, b, T, mode, mask);
        s[a][bb] = i < T ? expf(sv - mi[a]) * inv_l[a] : 0.f;
      }
    }
    product_nt<DP, NA, 16, 4, 16>(dOs, Vs, ra, cb, dp);
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
      for (int bb = 0; bb < 4; ++bb) X[xat<R>(cb + 16 * bb, ra + 16 * a)] = s[a][bb] * (dp[a][bb] - di[a]) * scale;
    __syncthreads();                  // dS is in place; V has been read
    if (k0 + SX < kv_end) load_rows<DP, SX>(Vs, Vg, sin.t, k0 + SX, T, D, vec_ok, tid);
    load_commit();
    product_nn<DP, R>(X, Ks, r0, cg, dq);
    __syncthreads();
    if (k0 + SX < kv_end) load_rows<DP, SX>(Ks, Kg, sin.t, k0 + SX, T, D, vec_ok, tid);
    load_commit();
  }
  store_piece<DP, R>(dQ + base, sin.t, q0 + r0, cg, T, D, vec_out != 0, dq);
  mca_pdl_wait();   // launched under the dK/dV kernel's tail and reading nothing it writes: only complete after it
}

// Sets *flag to 1 iff mask (T,T) is exactly lower-triangular ones (fillMask,
// CausalSelfAttentionLayer.cs:276-291).  *flag must hold 1 on entry.
__global__ void classify_causal_kernel(const float* __restrict__ mask, int T, int* __restrict__ flag) {
  const int64_t n = (int64_t)T * T;
  bool ok = true;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(idx / T), j = (int)(idx % T);
    const float want = (j <= i) ? 1.f : 0.f;
    if (mask[idx] != want) ok = false;
  }
  if (!ok) *flag = 0;
}
__global__ void set_int_kernel(int* p, int v) { *p = v; }

// The same answer from one launch (mca_classify_rows).
__global__ void __launch_bounds__(256) classify_causal_rows_kernel(const McaClassifyJob job) {
  mca_classify_rows(job, (int)blockIdx.x, (int)gridDim.x);
}

// The padded head size: what lies between two of these costs its zeros in every product (48 as 64 a third more work, 80 as
// 128 three fifths more), so the sizes models use have their own.
int pick_dp(int D) {
  for (const int dp : {16, 32, 48, 64, 80, 96, 128})
    if (D <= dp) return dp;
  return 0;
}

// Rows per CTA: 128, or 64 where that is estimated to end sooner -- few or short heads, whose 128-row tiles would leave SMs
// idle, or a last tile that is nearly empty.  A step of a 64-row tile is taken for 0.65 of a 128-row one (its products load
// more per multiply-add); the kernel ends no sooner than its longest CTA nor than the work spread over 148 SMs.
// Either tile throughout, forward and backward, us with 128 and with 64 rows: B=2 H=16 T=1536 D=128 key mask 4119 and 4727,
// causal 1499 and 1570; B=1 H=16 T=1024 D=128 causal 570 and 478; B=1 H=8 T=700 D=128 403 and 258; B=2 H=16 T=1536 D=80 1533 and
// 1414 (heads below 128 would bear a smaller factor).
bool small_tiles(int B, int H, int T, bool causal) {
  auto cost = [&](int R, double step) {
    int64_t steps = 0;
    int longest = 0;
    for (int t = 0; t * R < T; ++t) {
      const int n = mca_ceil_div(causal ? std::min(T, (t + 1) * R) : T, SX);
      steps += n;
      longest = std::max(longest, n);
    }
    return step * std::max((double)longest, (double)steps * B * H / 148.0);
  };
  return cost(64, 0.65) < cost(128, 1.0);
}

// dS passes through memory where the work, not the longest CTA, decides when the dK/dV kernel ends: where SMs would be idle,
// the other dQ kernel runs on them beside the dK/dV kernel, and this one could not (the work per SM over the longest CTA's:
// 0.55, H = 9, T = 1088, D = 128: 406 -> 500 us; 0.8, B = 2, H = 7, T = 967, D = 96: 702 -> 547).
bool passes_ds(int R, int B, int H, int T, bool causal) {
  const int64_t tiles = mca_ceil_div(T, R), steps = causal ? tiles * (tiles + 1) / 2 : tiles * tiles;
  return 3 * steps * B * H > 2 * 148 * tiles;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

int mca_classify_causal_mask_ws(const McaClassifyJob* job, void* stream) {
  if (!job->mask || !job->flag || !job->scratch) return ERROR_PARAM_NULL;
  if (job->T <= 0) return ERROR_PARAM_OUT_OF_RANGE;
  classify_causal_rows_kernel<<<std::min(1184, (job->T + 7) / 8), 256, 0, (cudaStream_t)stream>>>(*job);
  return mca_launch_status();
}

int mca_classify_causal_mask(const float* mask, int T, int* flag, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  set_int_kernel<<<1, 1, 0, st>>>(flag, 1);
  const int64_t n = (int64_t)T * T;
  const int blocks = (int)((n + 1023) / 1024 > 1184 ? 1184 : (n + 1023) / 1024);
  classify_causal_kernel<<<blocks, 256, 0, st>>>(mask, T, flag);
  return mca_launch_status();
}

template <int DP, int R>
static int launch_fwd_tile(const float* q, const float* k, const float* v, const float* mask, int mode, const int* flag,
                           int B, int H, int T, int D, float* y, float* rmax, float* rsum, float* ycopy, int layout,
                           cudaStream_t st) {
  constexpr size_t smem = fwd_smem_bytes<DP, R>();
  static std::atomic<uint64_t> done{0};
  int e = mca_smem_once(done, sdpa_fwd_f32_kernel<DP, R>, smem);
  if (e) return e;
  const McaStrides sin = mca_in_strides(layout, H, T, D), sout = mca_out_strides(layout, H, T, D);
  const int vec_ok = (D % 4 == 0) && aligned16(q) && aligned16(k) && aligned16(v);  // every stride is a multiple of D
  const int vec_out = (D % 4 == 0) && aligned16(y) && aligned16(ycopy);
  dim3 grid(B * H, mca_ceil_div(T, R));
  sdpa_fwd_f32_kernel<DP, R><<<grid, NT, smem, st>>>(q, k, v, mask, mode, flag, H, T, D, 1.0f / sqrtf((float)D), y, rmax,
                                                    rsum, ycopy, vec_ok, vec_out, sin, sout);
  return mca_launch_status();
}
template <int DP>
static int launch_fwd(const float* q, const float* k, const float* v, const float* mask, int mode, const int* flag,
                      int B, int H, int T, int D, float* y, float* rmax, float* rsum, float* ycopy, int layout,
                      cudaStream_t st) {
  if (small_tiles(B, H, T, mode == MCA_MASK_CAUSAL || mode == MCA_MASK_TT)) return launch_fwd_tile<DP, 64>(q, k, v, mask, mode, flag, B, H, T, D, y, rmax, rsum, ycopy, layout, st);
  return launch_fwd_tile<DP, 128>(q, k, v, mask, mode, flag, B, H, T, D, y, rmax, rsum, ycopy, layout, st);
}

int mca_sdpa_forward_f32(const float* q, const float* k, const float* v, const float* mask, int mask_mode,
                         const int* causal_flag, int B, int H, int T, int D, float* y, float* row_max,
                         float* row_sum, float* y_copy, void* stream) {
  return mca_sdpa_forward_f32_layout(q, k, v, mask, mask_mode, causal_flag, B, H, T, D, y, row_max, row_sum, y_copy,
                                     MCA_LAYOUT_BHTD, stream);
}

int mca_sdpa_forward_f32_layout(const float* q, const float* k, const float* v, const float* mask, int mask_mode,
                                const int* causal_flag, int B, int H, int T, int D, float* y, float* row_max,
                                float* row_sum, float* y_copy, int layout, void* stream) {
  if (!q || !k || !v || !y) return ERROR_PARAM_NULL;
  if (layout != MCA_LAYOUT_BHTD && layout != MCA_LAYOUT_PACKED) return ERROR_PARAM_OUT_OF_RANGE;
  if (B <= 0 || H <= 0 || T <= 0 || D <= 0 || (int64_t)B * H > 65535) return ERROR_PARAM_OUT_OF_RANGE;
  if ((mask_mode == MCA_MASK_TT || mask_mode == MCA_MASK_BATCH) && !mask) return ERROR_PARAM_NULL;
  if ((row_max == nullptr) != (row_sum == nullptr)) return ERROR_PARAM_NULL;
  cudaStream_t st = (cudaStream_t)stream;
  switch (pick_dp(D)) {
    case 16: return launch_fwd<16>(q, k, v, mask, mask_mode, causal_flag, B, H, T, D, y, row_max, row_sum, y_copy, layout, st);
    case 32: return launch_fwd<32>(q, k, v, mask, mask_mode, causal_flag, B, H, T, D, y, row_max, row_sum, y_copy, layout, st);
    case 48: return launch_fwd<48>(q, k, v, mask, mask_mode, causal_flag, B, H, T, D, y, row_max, row_sum, y_copy, layout, st);
    case 64: return launch_fwd<64>(q, k, v, mask, mask_mode, causal_flag, B, H, T, D, y, row_max, row_sum, y_copy, layout, st);
    case 80: return launch_fwd<80>(q, k, v, mask, mask_mode, causal_flag, B, H, T, D, y, row_max, row_sum, y_copy, layout, st);
    case 96: return launch_fwd<96>(q, k, v, mask, mask_mode, causal_flag, B, H, T, D, y, row_max, row_sum, y_copy, layout, st);
    case 128: return launch_fwd<128>(q, k, v, mask, mask_mode, causal_flag, B, H, T, D, y, row_max, row_sum, y_copy, layout, st);
  }
  return ERROR_ATTN_UNSUPPORTED_SHAPE;
}

template <int DP, int R>
static int launch_bwd_tile(const float* q, const float* k, const float* v, const float* dy, const float* mask, int mode,
                           const int* flag, const float* rmax, const float* rsum, const float* delta, int B, int H, int T,
                           int D, float* dq, float* dk, float* dv, float* ds, int64_t ds_floats, int layout, cudaStream_t st) {
  const McaStrides sin = mca_in_strides(layout, H, T, D), sout = mca_out_strides(layout, H, T, D);
  constexpr size_t smem = bwd_smem_bytes<DP, R>();
  static_assert(smem <= 227 * 1024, "one CTA per SM");
  static std::atomic<uint64_t> done_kv{0}, done_dq{0};
  int e;
  if ((e = mca_smem_once(done_kv, sdpa_bwd_dkdv_f32_kernel<DP, R>, smem)) || (e = mca_smem_once(done_dq, sdpa_bwd_dq_f32_kernel<DP, R>, smem)))
    return e;
  const int vec_ok = (D % 4 == 0) && aligned16(q) && aligned16(k) && aligned16(v) && aligned16(dy);
  const int vec_out = (D % 4 == 0) && aligned16(dq) && aligned16(dk) && aligned16(dv);
  const float scale = 1.0f / sqrtf((float)D);
  dim3 grid(B * H, mca_ceil_div(T, R));
  if (ds_floats < ds_tile<R>(B * H, 0, 0, T) || !passes_ds(R, B, H, T, mode == MCA_MASK_CAUSAL || mode == MCA_MASK_TT)) ds = nullptr;
  sdpa_bwd_dkdv_f32_kernel<DP, R><<<grid, NT, smem, st>>>(q, k, v, dy, mask, mode, flag, rmax, rsum, delta, H, T, D,
                                                         scale, dk, dv, ds, vec_ok, vec_out, sin, sout);
  e = mca_launch_status();
  if (e) return e;
  if (ds != nullptr) {
    constexpr size_t smem_ds = dq_ds_smem_bytes<DP>();
    static_assert(2 * (smem_ds + 1024) <= 228 * 1024, "two CTAs per SM");
    static std::atomic<uint64_t> done_ds{0};
    if ((e = mca_smem_once(done_ds, sdpa_bwd_dq_ds_f32_kernel<DP, R>, smem_ds))) return e;
    return mca_launch_pdl(sdpa_bwd_dq_ds_f32_kernel<DP, R>, dim3(B * H, mca_ceil_div(T, SX)), dim3(NT), smem_ds, st, k, ds, mode, flag, H, T, D, dq, vec_ok, vec_out, sin);
  }
  return mca_launch_pdl(sdpa_bwd_dq_f32_kernel<DP, R>, grid, dim3(NT), smem, st, q, k, v, dy, mask, mode, flag, rmax, rsum, delta, H,
                        T, D, scale, dq, vec_ok, vec_out, sin, sout);
}
template <int DP>
static int launch_bwd(const float* q, const float* k, const float* v, const float* dy, const float* mask, int mode,
                      const int* flag, const float* rmax, const float* rsum, const float* delta, int B, int H, int T,
                      int D, float* dq, float* dk, float* dv, float* ds, int64_t ds_floats, int layout, cudaStream_t st) {
  if (small_tiles(B, H, T, mode == MCA_MASK_CAUSAL || mode == MCA_MASK_TT))
    return launch_bwd_tile<DP, 64>(q, k, v, dy, mask, mode, flag, rmax, rsum, delta, B, H, T, D, dq, dk, dv, ds, ds_floats, layout, st);
  return launch_bwd_tile<DP, 128>(q, k, v, dy, mask, mode, flag, rmax, rsum, delta, B, H, T, D, dq, dk, dv, ds, ds_floats, layout, st);
}

int mca_sdpa_backward_f32(const float* q, const float* k, const float* v, const float* dy, const float* y_saved,
                          const float* mask, int mask_mode, const int* causal_flag, const float* row_max,
                          const float* row_sum, float* delta_scratch, int B, int H, int T, int D, float* dq,
                          float* dk, float* dv, void* stream) {
  return mca_sdpa_backward_f32_layout(q, k, v, dy, y_saved, mask, mask_mode, causal_flag, row_max, row_sum, delta_scratch,
                                      B, H, T, D, dq, dk, dv, MCA_LAYOUT_BHTD, stream);
}

int mca_sdpa_backward_f32_layout(const float* q, const float* k, const float* v, const float* dy, const float* y_saved,
                                 const float* mask, int mask_mode, const int* causal_flag, const float* row_max,
                                 const float* row_sum, float* delta_scratch, int B, int H, int T, int D, float* dq,
                                 float* dk, float* dv, int layout, void* stream) {
  return mca_sdpa_backward_f32_ws(q, k, v, dy, y_saved, mask, mask_mode, causal_flag, row_max, row_sum, delta_scratch, B, H, T, D, dq, dk,
                                  dv, nullptr, 0, layout, stream);
}

int64_t mca_sdpa_backward_f32_ws_bytes(int B, int H, int T) {
  int64_t floats = 0;   // of the mask forms that have a use for it
  for (const bool causal : {false, true}) {
    const int R = small_tiles(B, H, T, causal) ? 64 : 128;
    if (passes_ds(R, B, H, T, causal)) floats = std::max(floats, R == 64 ? ds_tile<64>(B * H, 0, 0, T) : ds_tile<128>(B * H, 0, 0, T));
  }
  return floats * 4;
}

int mca_sdpa_backward_f32_ws(const float* q, const float* k, const float* v, const float* dy, const float* y_saved, const float* mask,
                             int mask_mode, const int* causal_flag, const float* row_max, const float* row_sum, float* delta_scratch,
                             int B, int H, int T, int D, float* dq, float* dk, float* dv, float* ds, int64_t ds_floats, int layout,
                             void* stream) {
  if (layout != MCA_LAYOUT_BHTD && layout != MCA_LAYOUT_PACKED) return ERROR_PARAM_OUT_OF_RANGE;
  if (!q || !k || !v || !dy || !y_saved || !row_max || !row_sum || !delta_scratch || !dq || !dk || !dv)
    return ERROR_PARAM_NULL;
  if (B <= 0 || H <= 0 || T <= 0 || D <= 0 || (int64_t)B * H > 65535) return ERROR_PARAM_OUT_OF_RANGE;
  if ((mask_mode == MCA_MASK_TT || mask_mode == MCA_MASK_BATCH) && !mask) return ERROR_PARAM_NULL;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t rows = (int64_t)B * H * T;
  sdpa_bwd_delta_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(dy, y_saved, rows, H, T, D,
                                                                    mca_out_strides(layout, H, T, D), delta_scratch);
  int e = mca_launch_status();
  if (e) return e;
  switch (pick_dp(D)) {
    case 16: return launch_bwd<16>(q, k, v, dy, mask, mask_mode, causal_flag, row_max, row_sum, delta_scratch, B, H, T, D, dq, dk, dv, ds, ds_floats, layout, st);
    case 32: return launch_bwd<32>(q, k, v, dy, mask, mask_mode, causal_flag, row_max, row_sum, delta_scratch, B, H, T, D, dq, dk, dv, ds, ds_floats, layout, st);
    case 48: return launch_bwd<48>(q, k, v, dy, mask, mask_mode, causal_flag, row_max, row_sum, delta_scratch, B, H, T, D, dq, dk, dv, ds, ds_floats, layout, st);
    case 64: return launch_bwd<64>(q, k, v, dy, mask, mask_mode, causal_flag, row_max, row_sum, delta_scratch, B, H, T, D, dq, dk, dv, ds, ds_floats, layout, st);
    case 80: return launch_bwd<80>(q, k, v, dy, mask, mask_mode, causal_flag, row_max, row_sum, delta_scratch, B, H, T, D, dq, dk, dv, ds, ds_floats, layout, st);
    case 96: return launch_bwd<96>(q, k, v, dy, mask, mask_mode, causal_flag, row_max, row_sum, delta_scratch, B, H, T, D, dq, dk, dv, ds, ds_floats, layout, st);
    case 128: return launch_bwd<128>(q, k, v, dy, mask, mask_mode, causal_flag, row_max, row_sum, delta_scratch, B, H, T, D, dq, dk, dv, ds, ds_floats, layout, st);
  }
  return ERROR_ATTN_UNSUPPORTED_SHAPE;
}
