// Attention forward of a short fp32 call that keeps nothing for a Backward (inference), in one launch and exact fp32: the same
// mathematics as the reference's attnHandle<T>::Forward (CudaDnnDLL/Cuda Files/attn.cu:518-602), masks read as the caller has them
// (apply_mask / apply_mask_batch, math.cu:2994-3057: a masked logit becomes -1e29, so a fully masked row is uniform).
//
// Bound by latency: such a call has microseconds of launches, not of work.  The tensor-core path takes two dependent launches (operand
// split, forward: 6.6 + 6.9 us for 4 heads of 128 x 16, each a chain of TMA, barrier and tensor latencies) and a third to pack a key mask;
// this kernel is one round trip to memory, the products from shared memory, and the stores.  The keys are one tile, which K (16-byte
// pieces swizzled by row: a lane reads its own rows) and V fill by cp.async.  A warp owns RW query rows, so that few heads still spread over
// the chip: a lane has every 32nd key for the scores, and for P V four columns over every KG-th group of U keys.
#include "kernels.h"
#include "common.cuh"
#include "small_rules.h"

namespace {

using small_rules::KEYS;
using small_rules::WARPS;
constexpr int THREADS = WARPS * 32, KPL = KEYS / 32;

template <int D> struct Tile {
  static constexpr int CG = D / 4, KG = 32 / CG;             // 16-byte column groups of a row, key groups of a warp
  static constexpr int FLOATS = 2 * KEYS * D;                // K and V
  // piece i of key j is stored at piece swz(i, j): eight consecutive rows put one piece in eight bank groups
  static __device__ __forceinline__ int swz(int i, int j) { return i ^ (D == 16 ? (j >> 1) & 3 : j & 7); }
};
template <int D, int RW> constexpr size_t smem_bytes() { return sizeof(float) * (Tile<D>::FLOATS + WARPS * RW * (D + KEYS)); }

struct SmallParams {
  const float *q, *k, *v, *mask;
  float* y;
  McaStrides in, out;
  int mode, H, T;
  float scale_log2;   // (1/sqrt(D)) log2(e)
};

template <int D, int RW>
__global__ void __launch_bounds__(THREADS) sdpa_fwd_small_kernel(const SmallParams p) {
  using TL = Tile<D>;
  constexpr int CG = TL::CG, KG = TL::KG;
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int bh = blockIdx.y, b = bh / p.H, h = bh - b * p.H, T = p.T;
  const int row0 = (blockIdx.x * WARPS + w) * RW;            // this warp's first query
  const bool causal = p.mode == MCA_MASK_CAUSAL;
  const int keys = causal ? min(T, (int)(blockIdx.x + 1) * WARPS * RW) : T, keys_pad = min(KEYS, (keys + 31) & ~31);
  const float *K = p.k + b * p.in.b + h * p.in.h, *V = p.v + b * p.in.b + h * p.in.h;
  float *Kt = smem, *Vt = smem + KEYS * D;
  float* Qs = smem + TL::FLOATS + w * RW * (D + KEYS);       // this warp's rows of Q, then of P
  float* Ps = Qs + RW * D;
  // What follows is not let go before this kernel ends: the next call's CTAs, launched at the top, took the SMs that were free, two and
  // three to one (calls that do not wait, us, so / with the signal / split operands: 24 heads of 128 x 32 6.0 / 11.0 / 8.4, 20 of 128 x 32 under a key mask
  // 6.2 / 12.9 / 11.3, 16 of 128 x 64 6.5 / 8.9 / 8.4, 28 8.8 / 12.6 / 8.7).
  mca_pdl_wait();                                            // q, k, v may be the kernel before's
  for (int idx = tid; idx < keys_pad * CG; idx += THREADS) {
    const int j = idx / CG, c = idx % CG;
    if (j < keys) mca_cp_async16((uint32_t)__cvta_generic_to_shared(Kt + j * D + TL::swz(c, j) * 4), K + (int64_t)j * p.in.t + c * 4);
    else *reinterpret_cast<float4*>(Kt + j * D + TL::swz(c, j) * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  mca_cp_async_commit();
  for (int idx = tid; idx < keys_pad * CG; idx += THREADS) {
    const int j = idx / CG, c = idx % CG;
    if (j < keys) mca_cp_async16((uint32_t)__cvta_generic_to_shared(Vt + j * D + c * 4), V + (int64_t)j * p.in.t + c * 4);
    else *reinterpret_cast<float4*>(Vt + j * D + c * 4) = make_float4(0.f, 0.f, 0.f, 0.f);   // probability 0 times a number
  }
  mca_cp_async_commit();
  for (int idx = lane; idx < RW * CG; idx += 32) {
    const int r = idx / CG, c = idx % CG;
    *reinterpret_cast<float4*>(Qs + r * D + c * 4) =
        mca_ld_f4(p.q + b * p.in.b + h * p.in.h + (int64_t)min(row0 + r, T - 1) * p.in.t + c * 4);
  }
  // keep-flags of this lane's keys for the warp's rows, requested beside the tile
  float keep[RW][KPL];
  if (p.mask != nullptr) {
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
      for (int c = 0; c < KPL; ++c) {
        const int64_t key = min(lane + 32 * c, T - 1), row = p.mode == MCA_MASK_BATCH ? b : min(row0 + r, T - 1);
        keep[r][c] = mca_ld_f1(p.mask + row * T + key);
      }
  }
  mca_cp_async_wait<1>();
  __syncthreads();
  float s[RW][KPL];
#pragma unroll
  for (int r = 0; r < RW; ++r)
#pragma unroll
    for (int c = 0; c < KPL; ++c) s[r][c] = 0.f;
#pragma unroll 4
  for (int i = 0; i < CG; ++i) {
    float4 qv[RW];
#pragma unroll
    for (int r = 0; r < RW; ++r) qv[r] = *reinterpret_cast<const float4*>(Qs + r * D + i * 4);
#pragma unroll
    for (int c = 0; c < KPL; ++c)
      if (32 * c < keys_pad) {
        const float4 kv = *reinterpret_cast<const float4*>(Kt + (lane + 32 * c) * D + TL::swz(i, lane) * 4);
#pragma unroll
        for (int r = 0; r < RW; ++r)
          s[r][c] = fmaf(qv[r].w, kv.w, fmaf(qv[r].z, kv.z, fmaf(qv[r].y, kv.y, fmaf(qv[r].x, kv.x, s[r][c]))));
      }
  }
  float inv[RW];
#pragma unroll
  for (int r = 0; r < RW; ++r) {
    const int last = causal ? min(row0 + r, T - 1) : T - 1;       // the last key that exists for this row
    float mx = -INFINITY, sum = 0.f;
#pragma unroll
    for (int c = 0; c < KPL; ++c) {
      s[r][c] *= p.scale_log2;
      if (p.mask != nullptr && keep[r][c] == 0.f) s[r][c] = MCA_MASKED_LOGIT;
      if (lane + 32 * c <= last) mx = fmaxf(mx, s[r][c]);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
#pragma unroll
    for (int c = 0; c < KPL; ++c) {
      const float e = lane + 32 * c <= last ? exp2f(s[r][c] - mx) : 0.f;
      sum += e;
      if (32 * c < keys_pad) Ps[r * KEYS + lane + 32 * c] = e;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
    inv[r] = 1.0f / sum;
  }
  mca_cp_async_wait<0>();
  __syncthreads();
  const int cg = lane % CG, kg = lane / CG;
  float4 o[RW];
#pragma unroll
  for (int r = 0; r < RW; ++r) o[r] = make_float4(0.f, 0.f, 0.f, 0.f);
  // U keys a read of P; where a quarter of the warp spans several rows of V they have to be neighbours
  constexpr int U = D == 64 ? 4 : 1;
#pragma unroll(U == 4 ? 2 : 8)
  for (int j = kg * U; j < keys_pad; j += KG * U) {
    float4 vv[U];
    float pr[RW][U];
#pragma unroll
    for (int u = 0; u < U; ++u) vv[u] = *reinterpret_cast<const float4*>(Vt + (j + u) * D + cg * 4);
#pragma unroll
    for (int r = 0; r < RW; ++r) {
      if constexpr (U == 4) *reinterpret_cast<float4*>(pr[r]) = *reinterpret_cast<const float4*>(Ps + r * KEYS + j);
      else pr[r][0] = Ps[r * KEYS + j];
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        o[r].x = fmaf(pr[r][u], vv[u].x, o[r].x); o[r].y = fmaf(pr[r][u], vv[u].y, o[r].y);
        o[r].z = fmaf(pr[r][u], vv[u].z, o[r].z); o[r].w = fmaf(pr[r][u], vv[u].w, o[r].w);
      }
  }
#pragma unroll
  for (int r = 0; r < RW; ++r) {
    float4 a = o[r];
#pragma unroll
    for (int d = CG; d < 32; d <<= 1) {
      a.x += __shfl_xor_sync(0xffffffffu, a.x, d); a.y += __shfl_xor_sync(0xffffffffu, a.y, d);
      a.z += __shfl_xor_sync(0xffffffffu, a.z, d); a.w += __shfl_xor_sync(0xffffffffu, a.w, d);
    }
    if (kg == 0 && row0 + r < T)
      *reinterpret_cast<float4*>(p.y + b * p.out.b + h * p.out.h + (int64_t)(row0 + r) * p.out.t + cg * 4) =
          make_float4(a.x * inv[r], a.y * inv[r], a.z * inv[r], a.w * inv[r]);
  }
}

template <int D, int RW> int launch(const SmallParams& p, int B, cudaStream_t st) {
  static std::atomic<uint64_t> done{0};
  constexpr size_t smem = smem_bytes<D, RW>();
  if (const int e = mca_smem_once(done, sdpa_fwd_small_kernel<D, RW>, smem)) return e;
  return mca_launch_pdl(sdpa_fwd_small_kernel<D, RW>, dim3(mca_ceil_div(p.T, WARPS * RW), B * p.H), dim3(THREADS), smem, st, p);
}
template <int D> int pick(const SmallParams& p, int B, cudaStream_t st) {
  // as few rows a warp as give every CTA an SM of its own: two CTAs on one read K and V from shared memory twice
  const int64_t heads = (int64_t)B * p.H;
  if (heads * mca_ceil_div(p.T, WARPS) <= 148) return launch<D, 1>(p, B, st);
  if (heads * mca_ceil_div(p.T, WARPS * 2) <= 148) return launch<D, 2>(p, B, st);
  return launch<D, 4>(p, B, st);
}

}  // namespace

int mca_sdpa_forward_small(const float* q, const float* k, const float* v, const float* mask, int mode, int B, int H, int T, int D, float* y,
                           int layout, void* stream) {
  SmallParams p;
  p.q = q; p.k = k; p.v = v; p.y = y;
  p.mask = mode == MCA_MASK_TT || mode == MCA_MASK_BATCH ? mask : nullptr;
  p.mode = mode; p.H = H; p.T = T;
  p.in = mca_in_strides(layout, H, T, D);
  p.out = mca_out_strides(layout, H, T, D);
  p.scale_log2 = 1.4426950408889634f / sqrtf((float)D);
  cudaStream_t st = (cudaStream_t)stream;
  return D == 64 ? pick<64>(p, B, st) : D == 32 ? pick<32>(p, B, st) : pick<16>(p, B, st);
}
