// Pre-pass of the split-operand tensor-core kernels for fp32 callers: every (batch, head) of an fp32 tensor is scaled by a
// power of two (chosen from its largest magnitude) and written as rows [hi (64 fp16, HD used) | lo (64 fp16, HD used)] -- for
// 128-wide heads (forward only) [hi (128) | lo (128)] -- with
// hi = fp16(x), lo = fp16(x - hi): 22 mantissa bits per element, both halves inside the normal range of fp16 for
// every element that matters.
//
// Workspace (one per attention handle or caller):
//   float4 scale[BH]     the scales of q, k, v and dY of each (batch, head)
//   from the next multiple of 1024 bytes: four tensors of rows x 128 fp16 (256 for 128-wide heads): q, k, v, dY
//
// It is bound by memory: 4 bytes read and 4 written per element.  A cluster of up to eight CTAs (sixteen for few heads) takes
// one (batch, head) of one tensor: a CTA keeps its rows in registers (32 floats a thread; what a very long head has beyond
// that is read again, from L2 if it fits), finds their largest magnitude, the CTAs exchange those through distributed
// shared memory, and the rows are converted where they are.  One launch and one read from HBM, where a scale per tensor took a clear, a
// grid-wide reduction and a second kernel that read everything again: B = 8, H = 12, T = 1024, D = 64,
// the pre-passes of forward and backward 71 -> 54 us together (36 + 18 alone), and three launches fewer.
// The same launch classifies the caller's (T,T) mask when it is given one (its CTAs come before those of the tensors).
#pragma once
#include <cuda_fp16.h>

#include <algorithm>

#include "classify.cuh"
#include "common.cuh"

namespace split {

constexpr int TENSOR_Q = 0, TENSOR_K = 1, TENSOR_V = 2, TENSOR_DY = 3;

struct Workspace {
  float4* scale;
  __half* tensor[4];
};

// fp16 values per row of a split tensor: two halves of 64 (head sizes up to 64) or of 128
__host__ __device__ constexpr int row_halves(int HD) { return HD > 64 ? 256 : 128; }

inline int64_t scale_bytes(int64_t BH) { return (BH * 16 + 1023) / 1024 * 1024; }
inline int64_t workspace_bytes(int64_t BH, int T, int HD = 64) { return scale_bytes(BH) + 4 * BH * T * row_halves(HD) * 2; }

inline Workspace carve(void* base, int64_t BH, int T, int HD = 64) {
  Workspace w;
  w.scale = static_cast<float4*>(base);
  __half* t = reinterpret_cast<__half*>(static_cast<char*>(base) + scale_bytes(BH));
  for (int i = 0; i < 4; ++i) w.tensor[i] = t + (size_t)i * BH * T * row_halves(HD);
  return w;
}

struct Job {
  const float* src[3];   // up to three fp32 tensors with the same element strides
  __half* dst[3];
  int slot[3];           // which tensor each one is (TENSOR_*)
};

// 16-byte load that asks L2 to keep, or to give up first, the line.
__device__ __forceinline__ uint64_t l2_policy_keep() {
  uint64_t pol;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ uint64_t l2_policy_drop() {
  uint64_t pol;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ float4 ld_f4_hint(const float* ptr, uint64_t pol) {
  float4 v;
  asm volatile("ld.global.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(ptr), "l"(pol));
  return v;
}
__device__ __forceinline__ float amax4(const float4& v) { return fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))); }

// The power of two that brings max |x| into [2^12, 2^13): the largest fp16 is 65504 and the low half of an element
// is about 2^-11 of it, so both halves of everything within 2^-14 of the maximum are normal fp16 numbers.  It lies in
// [2^-115, 2^126], so that it and its reciprocal are normal (a subnormal maximum stays below 2^12; its halves carry every
// bit it has, the split dS of such a V fewer).  Products of several scales are not: the kernels multiply by them through
// pow2_factors, or one after the other where every partial product is bounded, as said there.
__device__ __forceinline__ float pow2_scale(float a) {
  if (!(a > 0.f) || !(a < 3.0e38f)) return 1.0f;
  int e;
  frexpf(a, &e);                    // a = f * 2^e, f in [0.5, 1)
  return ldexpf(1.0f, min(13 - e, 126));
}
__device__ __forceinline__ int scale_exp(float scale) { return (__float_as_int(scale) >> 23) - 127; }
__device__ __forceinline__ float pow2(int e) { return __int_as_float((max(-126, min(127, e)) + 127) << 23); }
// 2^e as two factors, applied one after the other: exact wherever the result is a normal number, without an infinity or a
// zero on the way (beyond 2^254 and 2^-252 the result is one anyway).
__device__ __forceinline__ float2 pow2_factors(int e) { return make_float2(pow2(e / 2), pow2(e - e / 2)); }
// Factor of the logits S' = Q'K'^T back to their own units (times `scale`).  |S'| < 2^33: below 2^-100 every logit is zero to
// the exponential anyway, and the bound keeps the masked logit (a constant over this factor) finite.
__device__ __forceinline__ float logit_scale(float scale, const float4& sc) {
  return scale * pow2(max(-100, min(120, -(scale_exp(sc.x) + scale_exp(sc.y)))));
}
// dY' V'^T products (below 2^32) are taken down by this before dS is split, and delta is left by the pre-pass in the units of dY'
// times this: delta x (the scale of v) is then below 2^13, whatever the magnitudes of dY and v.
constexpr float DS_SHIFT = 1.0f / 524288.0f;
constexpr int DS_SHIFT_LOG2 = -19;

constexpr int THREADS = 256, KEEP = 4;   // eight-element pieces a thread keeps in registers

// with ydot / delta given: also delta[row] = sum_c x[row][c] * ydot[row][c] (ydot contiguous rows) x scale x DS_SHIFT, the
// softmax backward's row term in the units the backward kernels need, from the elements this kernel holds anyway.
// grid: (CTAs of a cluster, BH, cls_layers of CTAs that classify a (T,T) mask or pack a key mask + tensors); the classification comes
// first, so that its answer is on the host before the tensors are done
template <int HD>
__global__ void __launch_bounds__(THREADS) split_kernel(const Job job, const McaStrides st, int H, int T,
                                                        float* __restrict__ scale, const float* __restrict__ ydot,
                                                        float* __restrict__ delta, const McaClassifyJob cls, const McaPackJob pack, int cls_layers) {
  mca_pdl_wait();   // the tensors are earlier kernels' output
  const int tid = threadIdx.x, which = (int)blockIdx.z - cls_layers;
  if (which < 0) {
    mca_pdl_launch_dependents();   // what the others wait for below is no concern of these
    const int cta = (int)((blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x), ctas = cls_layers * (int)(gridDim.x * gridDim.y);
    if (pack.mask != nullptr) mca_pack_rows(pack, cta, ctas);
    else mca_classify_rows(cls, cta, ctas);
    return;
  }
  constexpr int V8 = HD / 8;
  const int bh = blockIdx.y, b = bh / H;
  const int per = (T + gridDim.x - 1) / gridDim.x;                  // rows of a CTA
  const int row0 = blockIdx.x * per, rows = max(0, min(per, T - row0));
  const int n8 = rows * V8, rounds = (n8 + THREADS - 1) / THREADS;
  const float* src = job.src[which] + (int64_t)b * st.b + (int64_t)(bh - b * H) * st.h + (int64_t)row0 * st.t;
  const uint64_t keep = l2_policy_keep(), drop = l2_policy_drop();
  const int c8 = (tid % V8) * 8;                                    // THREADS is a multiple of V8: a thread keeps its columns
  auto piece = [&](int i) { return src + (int64_t)((tid + i * THREADS) / V8) * st.t + c8; };
  float4 x[KEEP][2];
  float m = 0.f;
#pragma unroll
  for (int i = 0; i < KEEP; ++i) {
    if (tid + i * THREADS < n8) {
      x[i][0] = ld_f4_hint(piece(i), drop);
      x[i][1] = ld_f4_hint(piece(i) + 4, drop);
    } else {
      x[i][0] = x[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
#pragma unroll
  for (int i = 0; i < KEEP; ++i) m = fmaxf(m, fmaxf(amax4(x[i][0]), amax4(x[i][1])));
#pragma unroll 2
  for (int i = KEEP; i < rounds; ++i)
    if (tid + i * THREADS < n8) m = fmaxf(m, fmaxf(amax4(ld_f4_hint(piece(i), keep)), amax4(ld_f4_hint(piece(i) + 4, keep))));
  // largest magnitude of the CTA, then of the cluster
  __shared__ float s_m[THREADS / 32];
  __shared__ float s_cta;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((tid & 31) == 0) s_m[tid >> 5] = m;
  __syncthreads();
  m = s_m[0];
#pragma unroll
  for (int w = 1; w < THREADS / 32; ++w) m = fmaxf(m, s_m[w]);
  const int ctas = gridDim.x;                                       // one cluster spans the x extent of the grid
  if (ctas > 1) {
    if (tid == 0) s_cta = m;
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const uint32_t mine = (uint32_t)__cvta_generic_to_shared(&s_cta);
    for (int r = 0; r < ctas; ++r) {
      uint32_t peer;
      float v;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(mine), "r"(r));
      asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(peer) : "memory");
      m = fmaxf(m, v);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // its peers may still be reading this CTA's word
  }
  // Only now may the kernel behind this one be launched: its CTAs, launched at this kernel's top, took whatever SMs the kernel before had
  // left, two to one of them where the grid has one for each (layers forward and backward, us: 12 heads of 1024 x 64 86 -> 82, 24 of 512
  // 67.5 -> 64.0, 24 of 200 under a key mask 54.5 -> 52.9).
  mca_pdl_launch_dependents();
  const int slot = job.slot[which];
  const float sc = pow2_scale(m), sc_delta = sc * DS_SHIFT;
  if (blockIdx.x == 0 && tid == 0) scale[bh * 4 + slot] = sc;
  constexpr int RH = row_halves(HD);
  const int64_t out_row0 = (int64_t)bh * T + row0;
  auto convert = [&](int i, const float4& v0, const float4& v1) {
    const int idx = tid + i * THREADS, row = idx / V8;
    const bool in = idx < n8;
    if (delta != nullptr) {   // uniform: the HD / 8 consecutive lanes of a row are in or out together
      float acc = 0.f;
      if (in) {
        const float* yd = ydot + (out_row0 + row) * HD + c8;
        const float4 y0 = mca_ld_f4(yd), y1 = mca_ld_f4(yd + 4);
        const float d[8] = {v0.x * sc_delta, v0.y * sc_delta, v0.z * sc_delta, v0.w * sc_delta,
                            v1.x * sc_delta, v1.y * sc_delta, v1.z * sc_delta, v1.w * sc_delta};
        acc = fmaf(d[0], y0.x, fmaf(d[1], y0.y, fmaf(d[2], y0.z, d[3] * y0.w)));
        acc += fmaf(d[4], y1.x, fmaf(d[5], y1.y, fmaf(d[6], y1.z, d[7] * y1.w)));
      }
#pragma unroll
      for (int o = V8 / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (in && c8 == 0) delta[out_row0 + row] = acc;
    }
    if (!in) return;
    const float e[8] = {v0.x * sc, v0.y * sc, v0.z * sc, v0.w * sc, v1.x * sc, v1.y * sc, v1.z * sc, v1.w * sc};
    __align__(16) __half hi[8];
    __align__(16) __half lo[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      hi[j] = __float2half_rn(e[j]);
      lo[j] = __float2half_rn(e[j] - __half2float(hi[j]));
    }
    __half* o = job.dst[which] + (out_row0 + row) * RH + c8;
    *reinterpret_cast<uint4*>(o) = *reinterpret_cast<const uint4*>(hi);
    *reinterpret_cast<uint4*>(o + RH / 2) = *reinterpret_cast<const uint4*>(lo);
  };
#pragma unroll
  for (int i = 0; i < KEEP; ++i)
    if (i < rounds) convert(i, x[i][0], x[i][1]);
#pragma unroll 2
  for (int i = KEEP; i < rounds; ++i) {
    const bool in = tid + i * THREADS < n8;
    const float4 v0 = in ? ld_f4_hint(piece(i), drop) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 v1 = in ? ld_f4_hint(piece(i) + 4, drop) : make_float4(0.f, 0.f, 0.f, 0.f);
    convert(i, v0, v1);
  }
  if (ctas > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Split `count` tensors (q, k, v for the forward; dY for the backward) into the workspace.
template <int HD>
inline int run(const Job& job, int count, const McaStrides& st, int B, int H, int T, const Workspace& w, cudaStream_t stream,
               const float* ydot = nullptr, float* delta = nullptr, const McaClassifyJob* cls = nullptr, const McaPackJob* pack = nullptr) {
  // CTAs of a cluster: as many as leave each at most what its threads keep in registers, up to the portable eight -- or sixteen
  // where a few long heads would not give every SM one (forward of
  // four heads of 8192 rows 208 -> 198 us, of one of 16384 378 -> 360)
  const int64_t pieces = (int64_t)T * (HD / 8);
  const int most = B * H * count * 8 < 148 ? 16 : 8;
  int ctas = 1;
  while (ctas < most && pieces > (int64_t)ctas * KEEP * THREADS) ctas *= 2;
  if (ctas > 8) {
    static std::atomic<uint64_t> done{0};
    const int e = mca_attribute_once(done, split_kernel<HD>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e) return e;
  }
  // The mask is T x T whatever the heads are: as many layers as give every eight rows of it a CTA, up to 1184 CTAs (with
  // one layer a single head of 16384 rows had eight CTAs read a gigabyte: 6.04 ms, 0.53 with this)
  const int layers = cls != nullptr ? mca_ceil_div(std::min(1184, mca_ceil_div(T, 8)), ctas * B * H) : pack != nullptr ? 1 : 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas, B * H, count + layers);
  cfg.blockDim = dim3(THREADS);
  cfg.stream = stream;
  return mca_launch_pdl_cluster(split_kernel<HD>, cfg, ctas, job, st, H, T, reinterpret_cast<float*>(w.scale), ydot, delta,
                                cls != nullptr ? *cls : McaClassifyJob{}, pack != nullptr ? *pack : McaPackJob{}, layers);
}

}  // namespace split
