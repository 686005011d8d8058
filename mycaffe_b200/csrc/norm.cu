// Row normalisations that sit either side of the attention block in every transformer layer,
// each as ONE pass over the tensor (read x once, write y once), bound by HBM bandwidth:
//   * LayerNorm forward / backward -- replaces LayerNormData<T>::Forward / Backward
//     (CudaDnnDLL/Cuda Files/layernorm.cu:291-333, :340-384), which issue 10 and 9 elementwise or
//     reduction kernels over seven full-size scratch tensors; their row means are computed by one
//     thread per row walking the row serially (channel_mean_kernel, math.cu:6817-6831).
//   * RMSNorm layer forward / backward -- replaces the 8 (forward) and 14 (backward) CudaDnn calls of
//     RMSNormLayer<T>.forward / backward (MyCaffe.layers.gpt/layers.gpt/RMSNormLayer.cs:156-179, :190-231).
// A row is held in the registers of a group of G threads (a warp for short rows, a whole CTA for
// long ones); sums are reduced with shuffles (and one pass through shared memory for G > 32) in a
// fixed order, so results do not depend on timing.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace {

constexpr int NORM_MAX_PARTIALS = 296;   // CTAs of the RMSNorm backward (two per SM): one dW partial each

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sums of N values over the G threads that share a row.  G == 32: the warp.  G > 32: the CTA (G == blockDim.x), through one of two
// buffers in turn, so that one barrier is enough.
template <int G, int N>
__device__ __forceinline__ void group_sum(float (&v)[N], float (*sred)[2][32], int& turn) {
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = warp_sum(v[k]);
  if (G == 32) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float (*buf)[32] = sred[turn];
  turn ^= 1;
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < N; ++k) buf[k][warp] = v[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; ++k) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < G / 32; ++w) t += buf[k][w];
    v[k] = t;
  }
}

// a / b from r, the reciprocal of b as a division gives it: the quotient a r put right by its own remainder, which a fused
// multiply-add forms exactly (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34, 1990: correctly rounded but for a b whose significand is all ones).  A division per element was a third of these kernels'
// instructions.  The remainder is q b - a, not a - q b: a zero one then leaves the sign of a zero quotient as it is.
// For b within 2^-60 .. 2^24 and a zero or |a| within 2^-100 .. 2^60 (or up to sqrt(inner) b): nothing overflows, the quotient is
// normal (>= 2^-125) and the remainder, a multiple of the product of two last places (>= 2^-148), is held exactly.  Of smaller
// numerators it is rounded, and at 2^-124 one quotient in twenty is not the division's.
constexpr float DIV_A_MIN = 7.888609052210118e-31f, DIV_A_MAX = 1.152921504606847e18f;   // 2^-100, 2^60
constexpr float DIV_B_MIN = 8.673617379884035e-19f, DIV_B_MAX = 16777216.f;              // 2^-60, 2^24
// Orders magnitudes, zero above them all (two integer instructions an element for the smallest that is not zero).
__device__ __forceinline__ unsigned above_zero(float a) { return 2u * __float_as_uint(a) - 1u; }
__device__ __forceinline__ float div_by(float a, float b, float r) {
  const float q = a * r;
  return fmaf(fmaf(q, b, -a), -r, q);
}

// The part of a row one thread holds: MAXV pieces of VEC floats, piece i at element (i*G + g)*VEC.
template <int G, int MAXV, int VEC>
struct RowPart {
  float v[MAXV][VEC];
  __device__ __forceinline__ void load(const float* row, int inner, int g) {
#pragma unroll
    for (int i = 0; i < MAXV; ++i) {
      const int e = (i * G + g) * VEC;
      if (e < inner) {
        if (VEC == 4) {
          const float4 t = *reinterpret_cast<const float4*>(row + e);
          v[i][0] = t.x; v[i][1 % VEC] = t.y; v[i][2 % VEC] = t.z; v[i][3 % VEC] = t.w;
        } else {
          v[i][0] = row[e];
        }
      } else {
#pragma unroll
        for (int j = 0; j < VEC; ++j) v[i][j] = 0.f;
      }
    }
  }
  __device__ __forceinline__ void store(float* row, int inner, int g) const {
#pragma unroll
    for (int i = 0; i < MAXV; ++i) {
      const int e = (i * G + g) * VEC;
      if (e < inner) {
        if (VEC == 4) *reinterpret_cast<float4*>(row + e) = make_float4(v[i][0], v[i][1 % VEC], v[i][2 % VEC], v[i][3 % VEC]);
        else row[e] = v[i][0];
      }
    }
  }
  template <typename F> __device__ __forceinline__ void each(F f) {
#pragma unroll
    for (int i = 0; i < MAXV; ++i)
#pragma unroll
      for (int j = 0; j < VEC; ++j) f(v[i][j], i, j);
  }
  // least: the smallest above_zero of the elements
  __device__ __forceinline__ void divide(float b, unsigned least) {
    if (b >= DIV_B_MIN && b <= DIV_B_MAX && least >= above_zero(DIV_A_MIN)) {
      const float r = 1.f / b;
      each([&](float& e, int, int) { e = div_by(e, b, r); });
    } else {
      each([&](float& e, int, int) { e = e / b; });
    }
  }
};

// which: 0 LayerNorm forward, 1 LayerNorm backward, 2 RMSNorm forward, 3 RMSNorm backward
struct NormParams {
  const float* a;      // LN fwd: x.  LN bwd: y.  RMS fwd: x.  RMS bwd: x
  const float* b;      // LN bwd: dy.  RMS bwd: dy
  const float* w;      // RMS: weights or null
  const float* stat;   // LN bwd: stdev (rows).  RMS bwd: 1/rms (rows)
  float* out;          // y or dx
  float* stat_out;     // LN fwd: stdev.  RMS fwd: 1/rms (may be null)
  float* dw_partial;   // RMS bwd: (gridDim.x, inner) or null
  int64_t rows;
  int inner;
  float eps;
};

template <int WHICH, int G, int MAXV, int VEC, int CTAS = G == 32 ? 2 : 1>   // CTAS: per SM, at least
__global__ void __launch_bounds__(G == 32 ? 256 : G, CTAS) norm_rows_kernel(const NormParams p) {
  __shared__ float sred[2][2][32];
  extern __shared__ float dw_smem[];   // RMS bwd with G == 32: (inner) floats, the CTA's dW partial
  constexpr int GROUPS = G == 32 ? 8 : 1;   // rows in flight per CTA
  using Part = RowPart<G, MAXV, VEC>;
  const int g = threadIdx.x % G, grp = threadIdx.x / G;
  const int inner = p.inner;
  const float inv_n = 1.0f / (float)inner;
  int turn = 0;
  Part dw;
  if (WHICH == 3) dw.each([](float& e, int, int) { e = 0.f; });
  // every group walks the same number of rows so that the CTA-wide barriers of G > 32 stay uniform
  for (int64_t row0 = (int64_t)blockIdx.x * GROUPS; row0 < p.rows; row0 += (int64_t)gridDim.x * GROUPS) {
    const int64_t row = row0 + grp;
    const bool live = row < p.rows;
    const int64_t off = (live ? row : 0) * inner;
    Part x;
    x.load(p.a + off, inner, g);
    if (WHICH == 0) {
      // mean, centred squares, stdev = sqrt(var + eps), y = (x - mean) / stdev   (layernorm.cu:296-330)
      float s[1] = {0.f}, q[1] = {0.f};
      x.each([&](float& e, int, int) { s[0] += e; });
      group_sum<G>(s, sred, turn);
      const float mean = s[0] * inv_n;
      unsigned least = ~0u;
#pragma unroll
      for (int i = 0; i < MAXV; ++i) {
        const bool in = (i * G + g) * VEC < inner;
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
          x.v[i][j] = in ? x.v[i][j] - mean : 0.f;
          least = min(least, above_zero(x.v[i][j]));
          q[0] = fmaf(x.v[i][j], x.v[i][j], q[0]);
        }
      }
      group_sum<G>(q, sred, turn);
      const float sd = sqrtf(q[0] * inv_n + p.eps);
      x.divide(sd, least);             // |x - mean| <= sqrt(inner) stdev
      if (live) {
        x.store(p.out + off, inner, g);
        if (g == 0) p.stat_out[row] = sd;
      }
    } else if (WHICH == 1) {
      // dx = (dy - (y * mean(y*dy) + mean(dy))) / stdev   (layernorm.cu:345-381).  The reference adds eps
      // to the first `rows` ELEMENTS of its row-broadcast stdev tensor before the division
      // (add_scalar over outer*channels items of a count-sized buffer, :377): reproduced here.
      Part dy;
      dy.load(p.b + off, inner, g);
      const float sd = p.stat[live ? row : 0];
      float s[2] = {0.f, 0.f};
#pragma unroll
      for (int i = 0; i < MAXV; ++i)
#pragma unroll
        for (int j = 0; j < VEC; ++j) { s[0] = fmaf(x.v[i][j], dy.v[i][j], s[0]); s[1] += dy.v[i][j]; }
      group_sum<G>(s, sred, turn);
      const float m1 = s[0] * inv_n, m2 = s[1] * inv_n;
      float most = 0.f;
      unsigned least = ~0u;
      x.each([&](float& e, int i, int j) {
        e = dy.v[i][j] - (e * m1 + m2);
        most = fmaxf(most, fabsf(e));
        least = min(least, above_zero(e));
      });
      if (off < p.rows || !(most < DIV_A_MAX)) {
        x.each([&](float& e, int i, int j) {
          const float denom = off + (i * G + g) * VEC + j < p.rows ? sd + p.eps : sd;
          e = e / denom;
        });
      } else {
        x.divide(sd, least);
      }
      if (live) x.store(p.out + off, inner, g);
    } else if (WHICH == 2) {
      // rms = sqrt(mean(x^2) + eps); y = w * (x * (1 / rms))   (RMSNormLayer.cs:158-173)
      float q[1] = {0.f};
      x.each([&](float& e, int, int) { q[0] = fmaf(e, e, q[0]); });
      group_sum<G>(q, sred, turn);
      const float rms = sqrtf(q[0] * inv_n + p.eps);
      const float inv = rms == 0.f ? 0.f : 1.0f / rms;   // invert_kernel maps 0 to 0, math.cu:6018-6024
      if (p.w != nullptr) {
        Part w;
        w.load(p.w, inner, g);
        x.each([&](float& e, int i, int j) { e = w.v[i][j] * (e * inv); });
      } else {
        x.each([&](float& e, int, int) { e = e * inv; });
      }
      if (live) {
        x.store(p.out + off, inner, g);
        if (g == 0 && p.stat_out != nullptr) p.stat_out[row] = inv;
      }
    } else {
      // g = dy * w; dW += dy * (x * inv); dx = g * inv - x * sum(g * x) * inv^3 / n   (RMSNormLayer.cs:194-229:
      // dinv = sum(g x), drms = -dinv / rms^2, dmean = drms / (2 rms), dx += 2 x dmean / n)
      Part dy;
      dy.load(p.b + off, inner, g);
      const float inv = live ? p.stat[row] : 0.f;
      if (p.w != nullptr) {
        Part w;
        w.load(p.w, inner, g);
        dy.each([&](float& e, int i, int j) {
          dw.v[i][j] = fmaf(e, x.v[i][j] * inv, dw.v[i][j]);
          e *= w.v[i][j];
        });
      }
      float s[1] = {0.f};
      dy.each([&](float& e, int i, int j) { s[0] = fmaf(e, x.v[i][j], s[0]); });
      group_sum<G>(s, sred, turn);
      const float dinv = s[0];
      const float drms = -dinv * (inv * inv);
      const float dmean = drms * (0.5f * inv);
      const float c = 2.0f * dmean * inv_n;
      x.each([&](float& e, int i, int j) { e = fmaf(e, c, dy.v[i][j] * inv); });
      if (live) x.store(p.out + off, inner, g);
    }
  }
  if (WHICH == 3 && p.dw_partial != nullptr) {
    float* dst = p.dw_partial + (int64_t)blockIdx.x * inner;
    if (G == 32) {   // the CTA's eight row groups add their partials in group order
      for (int e = threadIdx.x; e < inner; e += blockDim.x) dw_smem[e] = 0.f;
      __syncthreads();
      for (int turn = 0; turn < GROUPS; ++turn) {
        if (grp == turn) {
#pragma unroll
          for (int i = 0; i < MAXV; ++i)
#pragma unroll
            for (int j = 0; j < VEC; ++j) {
              const int e = (i * G + g) * VEC + j;
              if (e < inner) dw_smem[e] += dw.v[i][j];
            }
        }
        __syncthreads();
      }
      for (int e = threadIdx.x; e < inner; e += blockDim.x) dst[e] = dw_smem[e];
    } else {
      dw.store(dst, inner, g);
    }
  }
}

// dW[e] = sum over the CTAs' partials: eight warps of a CTA take every eighth of them for 32 columns, and their sums are added in
// order (one thread a column walked all 296 of them, one behind the other).
constexpr int DW_WARPS = 8;
__global__ void __launch_bounds__(DW_WARPS * 32) norm_dw_reduce_kernel(const float* __restrict__ partial, int n_partials, int inner, float* __restrict__ dw) {
  __shared__ float part[DW_WARPS][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, e = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (e < inner) {
#pragma unroll 8
    for (int c = warp; c < n_partials; c += DW_WARPS) s += partial[(int64_t)c * inner + e];
  }
  part[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && e < inner) {
#pragma unroll
    for (int w = 1; w < DW_WARPS; ++w) s += part[w][lane];
    dw[e] = s;
  }
}

struct Shape { int G, MAXV, VEC; };

// the narrowest group that holds a row, and as few pieces a thread as there is an instantiation for: every second number of 16-byte
// pieces of a warp, two or four of 256 threads, four of 1024; of single floats 8 or 16, 4 or 16, and 16 (a LayerNorm of 768 as eight
// pieces instead of six: a quarter of the arithmetic on zeros, and 96 registers in the backward, two CTAs an SM, instead of 79, three); vector
// loads need inner % 4 == 0 and 16-byte aligned tensors
bool pick(int inner, bool aligned, Shape* s) {
  auto pieces = [&](int G, int VEC) { return (inner + G * VEC - 1) / (G * VEC); };
  if (aligned && inner % 4 == 0) {
    if (inner <= 32 * 8 * 4) { *s = {32, (pieces(32, 4) + 1) / 2 * 2, 4}; return true; }
    if (inner <= 256 * 4 * 4) { *s = {256, pieces(256, 4) <= 2 ? 2 : 4, 4}; return true; }
    if (inner <= 1024 * 4 * 4) { *s = {1024, 4, 4}; return true; }
    return false;
  }
  if (inner <= 32 * 16) { *s = {32, pieces(32, 1) <= 8 ? 8 : 16, 1}; return true; }
  if (inner <= 256 * 16) { *s = {256, pieces(256, 1) <= 4 ? 4 : 16, 1}; return true; }
  if (inner <= 1024 * 16) { *s = {1024, 16, 1}; return true; }
  return false;
}

template <int WHICH, int G, int MAXV, int VEC>
int launch_norm(NormParams p, int grid_cap, cudaStream_t st) {
  constexpr int GROUPS = G == 32 ? 8 : 1;
  constexpr int THREADS = G == 32 ? 256 : G;
  const int64_t want = (p.rows + GROUPS - 1) / GROUPS;
  const int grid = (int)std::min<int64_t>(want, grid_cap);
  const size_t smem = (WHICH == 3 && G == 32 && p.dw_partial) ? sizeof(float) * (size_t)p.inner : 0;
  // The RMSNorm backward of eight pieces holds four tensors' rows: two CTAs per SM take registers away from it that a grid with one
  // to an SM has no use for giving up (forward and backward, us: 200 x 800 16.8 / 15.8, 1000 x 900 19.8 / 18.0; 2500 x 900 23.8 / 25.9).
  if constexpr (WHICH == 3 && G == 32 && MAXV * VEC == 32) {
    if (grid <= NORM_MAX_PARTIALS / 2) {
      norm_rows_kernel<WHICH, G, MAXV, VEC, 1><<<grid, THREADS, smem, st>>>(p);
      return mca_launch_status();
    }
  }
  norm_rows_kernel<WHICH, G, MAXV, VEC><<<grid, THREADS, smem, st>>>(p);
  return mca_launch_status();
}

template <int WHICH>
int dispatch_norm(const NormParams& p, bool aligned, int grid_cap, cudaStream_t st) {
  Shape s;
  if (!pick(p.inner, aligned, &s)) return ERROR_ATTN_UNSUPPORTED_SHAPE;
  if (s.VEC == 4) {
    if (s.G == 32) {
      switch (s.MAXV) {
        case 2: return launch_norm<WHICH, 32, 2, 4>(p, grid_cap, st);
        case 4: return launch_norm<WHICH, 32, 4, 4>(p, grid_cap, st);
        case 6: return launch_norm<WHICH, 32, 6, 4>(p, grid_cap, st);
        default: return launch_norm<WHICH, 32, 8, 4>(p, grid_cap, st);
      }
    }
    if (s.G == 256) return s.MAXV == 2 ? launch_norm<WHICH, 256, 2, 4>(p, grid_cap, st) : launch_norm<WHICH, 256, 4, 4>(p, grid_cap, st);
    return launch_norm<WHICH, 1024, 4, 4>(p, grid_cap, st);
  }
  if (s.G == 32) return s.MAXV == 8 ? launch_norm<WHICH, 32, 8, 1>(p, grid_cap, st) : launch_norm<WHICH, 32, 16, 1>(p, grid_cap, st);
  if (s.G == 256) return s.MAXV == 4 ? launch_norm<WHICH, 256, 4, 1>(p, grid_cap, st) : launch_norm<WHICH, 256, 16, 1>(p, grid_cap, st);
  return launch_norm<WHICH, 1024, 16, 1>(p, grid_cap, st);
}

bool a16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
constexpr int NORM_GRID_CAP = 148 * 16;

}  // namespace

int mca_layernorm_forward_f32(const float* x, float* y, float* stdev, int64_t rows, int inner, float eps, void* stream) {
  if (!x || !y || !stdev) return ERROR_PARAM_NULL;
  if (rows <= 0 || inner <= 0) return ERROR_PARAM_OUT_OF_RANGE;
  NormParams p = {};
  p.a = x; p.out = y; p.stat_out = stdev; p.rows = rows; p.inner = inner; p.eps = eps;
  return dispatch_norm<0>(p, a16(x) && a16(y), NORM_GRID_CAP, (cudaStream_t)stream);
}

int mca_layernorm_backward_f32(const float* y, const float* dy, const float* stdev, float* dx, int64_t rows, int inner,
                               float eps, void* stream) {
  if (!y || !dy || !stdev || !dx) return ERROR_PARAM_NULL;
  if (rows <= 0 || inner <= 0) return ERROR_PARAM_OUT_OF_RANGE;
  NormParams p = {};
  p.a = y; p.b = dy; p.stat = stdev; p.out = dx; p.rows = rows; p.inner = inner; p.eps = eps;
  return dispatch_norm<1>(p, a16(y) && a16(dy) && a16(dx), NORM_GRID_CAP, (cudaStream_t)stream);
}

int mca_rmsnorm_forward_f32(const float* x, const float* w, float* y, float* inv_rms, int64_t rows, int inner, float eps,
                            void* stream) {
  if (!x || !y) return ERROR_PARAM_NULL;
  if (rows <= 0 || inner <= 0) return ERROR_PARAM_OUT_OF_RANGE;
  NormParams p = {};
  p.a = x; p.w = w; p.out = y; p.stat_out = inv_rms; p.rows = rows; p.inner = inner; p.eps = eps;
  return dispatch_norm<2>(p, a16(x) && a16(y) && a16(w), NORM_GRID_CAP, (cudaStream_t)stream);
}

int64_t mca_rmsnorm_backward_scratch_floats(int inner) { return (int64_t)NORM_MAX_PARTIALS * inner; }

int mca_rmsnorm_backward_f32(const float* x, const float* w, const float* dy, const float* inv_rms, float* dx, float* dw,
                             float* scratch, int64_t scratch_floats, int64_t rows, int inner, void* stream) {
  if (!x || !dy || !inv_rms || !dx) return ERROR_PARAM_NULL;
  if (rows <= 0 || inner <= 0) return ERROR_PARAM_OUT_OF_RANGE;
  if (dw != nullptr && (w == nullptr || scratch == nullptr)) return ERROR_PARAM_NULL;
  if (dw != nullptr && scratch_floats < mca_rmsnorm_backward_scratch_floats(inner)) return ERROR_ATTN_SCRATCH_TOO_SMALL;
  NormParams p = {};
  p.a = x; p.b = dy; p.w = w; p.stat = inv_rms; p.out = dx; p.dw_partial = dw ? scratch : nullptr;
  p.rows = rows; p.inner = inner;
  Shape s;
  const bool aligned = a16(x) && a16(dy) && a16(dx) && a16(w) && a16(scratch);
  if (!pick(inner, aligned, &s)) return ERROR_ATTN_UNSUPPORTED_SHAPE;
  const int groups = s.G == 32 ? 8 : 1;
  const int grid = (int)std::min<int64_t>((rows + groups - 1) / groups, NORM_MAX_PARTIALS);
  int e = dispatch_norm<3>(p, aligned, NORM_MAX_PARTIALS, (cudaStream_t)stream);
  if (e || dw == nullptr) return e;
  norm_dw_reduce_kernel<<<mca_ceil_div(inner, 32), DW_WARPS * 32, 0, (cudaStream_t)stream>>>(scratch, grid, inner, dw);
  return mca_launch_status();
}
