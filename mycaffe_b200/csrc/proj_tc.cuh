// Decode projections for more than eight sequences: one pass over the weights, on the tensor cores.
//
// The streaming kernel of gemv.cu shares a pass over the weights between at most eight sequences; sixteen to
// sixty-four sequences (the batched decode configurations) would take two to eight passes.  Here the product
// Y[b, r] = sum_k W[r, k] X[b, k] is a tcgen05 contraction with the weights as the M = 128 operand and the sequences
// as N, so every weight byte leaves HBM once whatever the batch, and the kernel is bound by that stream.
// Replaces the per-sequence cublasSgemv calls of the reference's decode step (CudaExtension.llm32.llama2/Files/
// primitives.cu:322-340) with the arithmetic of its CPU twin (llama2_cpu.cpp:189-202,224-237) kept to fp32 accuracy:
//   * fp32 weights: a tile of 128 rows x 64 k arrives by TMA as fp32; eight warps rewrite it in place as two fp16
//     tiles hi = 16 w cut to fp16's mantissa, lo = fp16(16 w - hi) in the 128-byte-swizzled K-major layout the MMA reads
//     (in place: a tile costs 32 KB of shared memory, not 64, and what a tile costs in shared-memory traffic -- the TMA
//     write, the converters' read and write, the MMAs' operand reads -- is what bounds the kernel); the activations are
//     split the same way by a small pre-pass (after RMSNorm and a per-sequence power-of-two scale), and the product is
//     the three MMAs hi.hi + hi.lo + lo.hi into one fp32 accumulator in TMEM (the dropped lo.lo term is 2^-22);
//   * bf16 weights: the TMA tile is the MMA operand itself, the activations are two bf16 pieces (16 mantissa bits; the
//     weights themselves carry 8), two MMAs per k16.
// The (tile of 128 rows) x (64-wide k chunk) units of all tiles, in that order, are dealt to the CTAs in equal contiguous
// ranges: every SM streams the same number of bytes whatever the matrix (whole tiles, or tiles cut into a fixed number of
// slices, left the last of two waves a seventh to a half empty: the feed-forward pair of a 7B-shaped layer, bf16,
// 16 sequences, 87 -> 65 us with what is said at the epilogue, the issuing warp and the pre-pass).
// A CTA whose range covers part of a tile leaves fp32 partial sums in a scratch array, and the one that arrives last (a
// ticket per tile and quarter of its rows) adds all of the tile's parts in their order, so the result does not depend on
// timing.  The gated pair W1/W3 of the feed-forward block is one tile with two accumulators and silu(a) * b in the epilogue.
// Roles of a CTA (one CTA per SM, persistent over its range): eight warps convert (fp32 weights only), eight are the epilogue
// (two for each quarter of the TMEM lanes, alternating by eight columns: what is left to do when the last chunk has been
// multiplied is a chain of memory round trips, so it is spread wide), one is the TMA producer of the weights, one the MMA
// issuer and TMEM owner, one the TMA producer of the
// activation pieces.  The weight ring (five 32 KB slots for fp32, eight 16 KB slots for bf16) and the activation ring
// have their own barriers.  Every wait is bounded.
// The activation pieces, per-sequence scales, partial sums and tickets live in arrays that are part of the library
// image (about 24 MB per device): nothing is allocated, but two of these products must not overlap on one device.
#pragma once
#define MCA_TU_FAIL_FAMILY MCA_FAIL_PROJ
#include <algorithm>

#include "tc_common.cuh"

namespace proj {
using namespace tc;

constexpr int ROWS = 128;          // weight rows per tile (MMA M)
constexpr int KC = 64;             // k per stage: one 128-byte row of 16-bit operands
constexpr int MAX_B = 64;          // sequences (MMA N, rounded up to 16)
constexpr int MAX_N = 16384;       // longest contraction
constexpr int MAX_CTAS = 148;      // one per SM; each has room for two partial tiles, at either end of its range
constexpr int MAX_TILES = 2048;
constexpr int PIECES = 2;          // 16-bit pieces of an activation
constexpr int MAX_SX = 16;         // stages of the activation ring, at most
constexpr int CONV_WARPS = 8, EPI_WARPS = 8;
// warps of a CTA: converters (fp32 weights only), epilogue, weight TMA, MMA, activation TMA
template <bool CONVERT> struct Roles {
  static constexpr int EPI0 = CONVERT ? CONV_WARPS : 0, TMA = EPI0 + EPI_WARPS, MMA = TMA + 1, TMA_X = MMA + 1;
  static constexpr int THREADS = (TMA_X + 1) * 32;
};
constexpr float W_SCALE = 16.f;    // fp32 weights are split after this exact scaling (keeps the low halves normal)
constexpr uint32_t TMEM_ALLOC = 512, ACC_COLS = 256;   // two accumulators of up to two results x two pieces x 64 sequences

__device__ __align__(1024) uint16_t g_x_pieces[2 * MAX_B * MAX_N];
__device__ float g_x_scale[MAX_B];
__device__ float g_partials[(size_t)MAX_CTAS * 2 * ROWS * 2 * MAX_B];
__device__ unsigned int g_tickets[MAX_TILES * EPI_WARPS];
__device__ int g_status[4];

template <typename WT> struct Plan;
template <> struct Plan<float> {
  static constexpr bool CONVERT = true;
#ifndef MCA_PROJ_SW
#define MCA_PROJ_SW 5
#endif
  static constexpr int SW = MCA_PROJ_SW, FMT = 0;                       // weight ring depth; fp16 operands
  static constexpr uint32_t W_BYTES = ROWS * KC * 4;                    // a slot: the fp32 tile, then hi | lo in its place
  static constexpr uint32_t X_RING = 3 * PIECES * MAX_B * 128;          // the activation ring: as many stages as fit
  static constexpr uint32_t OP_BYTES = ROWS * KC * 2;                   // one fp16 operand tile (half a slot)
  static constexpr uint32_t OFF_W = 0, OFF_X = OFF_W + SW * W_BYTES, OFF_OP = OFF_X + X_RING;
  static constexpr uint32_t OFF_BAR = OFF_OP;
};
template <> struct Plan<__nv_bfloat16> {
  static constexpr bool CONVERT = false;
  static constexpr int SW = 8, FMT = 1;                                // bf16 operands
  static constexpr uint32_t W_BYTES = ROWS * KC * 2;
  static constexpr uint32_t X_RING = 6 * PIECES * MAX_B * 128;
  static constexpr uint32_t OP_BYTES = 0;
  static constexpr uint32_t OFF_W = 0, OFF_X = OFF_W + SW * W_BYTES, OFF_OP = OFF_X + X_RING;
  static constexpr uint32_t OFF_BAR = OFF_OP;
};
// barriers: wfull[SW] wempty[SW] xfull[MAX_SX] xempty[MAX_SX] convdone[SW] accfull[2] accfree[2], then the TMEM address
constexpr uint32_t BAR_BYTES = 512;
template <typename WT> constexpr size_t smem_bytes() { return Plan<WT>::OFF_BAR + BAR_BYTES + MAX_B * 4 + 1024; }
static_assert(smem_bytes<float>() <= 227 * 1024 && smem_bytes<__nv_bfloat16>() <= 227 * 1024, "one CTA per SM");

struct Params {
  float* out[3];
  int rows[3];
  int tile0[4];        // first tile of each matrix (not gated); tile0[n_mats] = tiles
  int n_mats, B, Bp, n, accumulate, swiglu, tiles, kchunks;
};

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// Barrier 1 over the converter warps, returning the AND of their predicates.
__device__ __forceinline__ bool conv_bar_and(bool pred) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)pred), "n"(CONV_WARPS * 32)
      : "memory");
  return r != 0;
}

constexpr int X_THREADS = 512;
__device__ __forceinline__ float block_sum(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int w = 0; w < X_THREADS / 32; ++w) t += red[w];
  return t;
}
__device__ __forceinline__ float block_max(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int w = 0; w < X_THREADS / 32; ++w) t = fmaxf(t, red[w]);
  return t;
}

// Activations of sequence b -> 16-bit pieces (row p * Bp + b of a (pieces * Bp, n) array): RMSNorm as the CPU twin
// orders it, o[j] = w[j] * (s * x[j]) with s = 1 / sqrt(sum(x^2) / n + eps) (llama2_cpu.cpp:189-202), then
//   BF16 = false: v / 2^e with 2^e chosen so that the row's largest magnitude lands in [2^13, 2^14), as fp16 hi + lo;
//   BF16 = true:  v as two bf16 pieces, hi = bf16(v), lo = bf16(v - hi): 16 mantissa bits, two hundred times finer than
//                 the bf16 weights they multiply.
// Rows from B up to Bp are written as zeros.  One CTA per row, the row in its threads' registers (NV float4 each): this kernel
// is a latency in front of every contraction (its x is the kernel before's last result), so the row is read once, with all
// loads in flight and the norm's weights requested before that kernel has finished, and no shared memory is taken that an
// SM still holding a contraction's CTA could not give (5.8 us of exposed time at n = 4096, 16 sequences -> 2.2).
template <bool BF16, bool NORM, int NV>
__global__ void __launch_bounds__(X_THREADS) x_pieces_kernel(const float* __restrict__ x, const float* __restrict__ norm_w, float eps,
                                                             int n, int B, int Bp, uint16_t* __restrict__ pieces,
                                                             float* __restrict__ xscale) {
  __shared__ float red[2][X_THREADS / 32];
  const int b = blockIdx.x, tid = threadIdx.x;
  mca_pdl_launch_dependents();                          // the contraction kernel may start fetching weights
  const bool live = b < B;
  float4 g[NORM ? NV : 1], v[NV];
  if (NORM && live) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int k = (tid + i * X_THREADS) * 4;
      g[i] = k < n ? __ldg(reinterpret_cast<const float4*>(norm_w + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  mca_pdl_wait();                                       // launched ahead of the kernels before it: their results (x, and the
                                                        // previous contraction's last reads of the pieces) come first
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int k = (tid + i * X_THREADS) * 4;
    v[i] = live && k < n ? mca_ld_f4(x + (size_t)b * n + k) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (NORM && live) {
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      ss = fmaf(v[i].x, v[i].x, ss); ss = fmaf(v[i].y, v[i].y, ss); ss = fmaf(v[i].z, v[i].z, ss); ss = fmaf(v[i].w, v[i].w, ss);
    }
    ss = block_sum(ss, red[0]);
    const float s = 1.0f / sqrtf(ss / (float)n + eps);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const float4 gi = g[NORM ? i : 0];
      v[i].x = gi.x * (s * v[i].x); v[i].y = gi.y * (s * v[i].y); v[i].z = gi.z * (s * v[i].z); v[i].w = gi.w * (s * v[i].w);
    }
  }
  float down = 1.f;
  if constexpr (!BF16) {
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v[i].x), fabsf(v[i].y)), fmaxf(fabsf(v[i].z), fabsf(v[i].w))));
    amax = block_max(amax, red[1]);
    int e = 0;
    if (amax > 0.f && amax < INFINITY) { frexpf(amax, &e); e -= 14; }
    down = ldexpf(1.f, -e);
    if (tid == 0 && live) xscale[b] = ldexpf(1.f, e) / W_SCALE;
  } else {
    if (tid == 0 && live) xscale[b] = 1.f;
  }
  uint16_t* dst = pieces + (size_t)b * n;
  uint16_t* dst_lo = dst + (size_t)Bp * n;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int k = (tid + i * X_THREADS) * 4;
    if (k >= n) continue;
    const float e4[4] = {v[i].x * down, v[i].y * down, v[i].z * down, v[i].w * down};
    uint32_t h[2], l[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      if constexpr (BF16) {
        const __nv_bfloat16 h0 = __float2bfloat16_rn(e4[2 * j]), h1 = __float2bfloat16_rn(e4[2 * j + 1]);
        h[j] = (uint32_t)__bfloat16_as_ushort(h0) | ((uint32_t)__bfloat16_as_ushort(h1) << 16);
        l[j] = pack_bf16(e4[2 * j] - __bfloat162float(h0), e4[2 * j + 1] - __bfloat162float(h1));
      } else {
        const __half h0 = __float2half_rn(e4[2 * j]), h1 = __float2half_rn(e4[2 * j + 1]);
        h[j] = (uint32_t)__half_as_ushort(h0) | ((uint32_t)__half_as_ushort(h1) << 16);
        l[j] = pack_f16(e4[2 * j] - __half2float(h0), e4[2 * j + 1] - __half2float(h1));
      }
    }
    *reinterpret_cast<uint2*>(dst + k) = make_uint2(h[0], h[1]);
    *reinterpret_cast<uint2*>(dst_lo + k) = make_uint2(l[0], l[1]);
  }
}

// The register limit leaves room on the SM for a CTA of the pre-pass (512 threads of up to 32, or 40, registers): where it did
// not, the SMs that held the pre-pass fetched no weights ahead and finished late.
template <typename WT>
__global__ void __maxnreg__(Plan<WT>::CONVERT ? 72 : 112) proj_tc_kernel(const __grid_constant__ CUtensorMap mw0,
                                                             const __grid_constant__ CUtensorMap mw1,
                                                             const __grid_constant__ CUtensorMap mw2,
                                                             const __grid_constant__ CUtensorMap mx, const Params p) {
  using PL = Plan<WT>;
  constexpr int SW = PL::SW;
  using RO = Roles<PL::CONVERT>;
  constexpr int WARP_EPI0 = RO::EPI0, WARP_TMA = RO::TMA, WARP_MMA = RO::MMA, WARP_TMA_X = RO::TMA_X;
  // The activation ring: a stage is the two pieces of every sequence for one k chunk, read from L2.  A chunk costs the
  // tensor pipe a third of a microsecond and L2 answers after one, so with few sequences, whose stages are small, many are kept
  // in flight (three of them, whatever their size, held 16 sequences to 40 % of the memory bandwidth).
  const uint32_t x_piece_bytes = (uint32_t)p.Bp * 128u, x_stage_bytes = PIECES * x_piece_bytes;
  const int SX = min((int)MAX_SX, (int)(PL::X_RING / x_stage_bytes));
  extern __shared__ unsigned char pj_smem_raw[];
  const uint32_t raw = smem_u32(pj_smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* gen = pj_smem_raw + (base - raw);
  const uint32_t bar0 = base + PL::OFF_BAR;
  auto wfull = [&](int s) { return bar0 + 8u * s; };
  auto wempty = [&](int s) { return bar0 + 8u * (SW + s); };
  auto xfull = [&](int s) { return bar0 + 8u * (2 * SW + s); };
  auto xempty = [&](int s) { return bar0 + 8u * (2 * SW + MAX_SX + s); };
  constexpr int NB0 = 2 * SW + 2 * MAX_SX;
  auto convdone = [&](int c) { return bar0 + 8u * (NB0 + c); };        // [SW]: slot c holds the converted tiles
  auto accfull = [&](int a) { return bar0 + 8u * (NB0 + SW + a); };
  auto accfree = [&](int a) { return bar0 + 8u * (NB0 + SW + 2 + a); };
  static_assert(8 * (NB0 + SW + 4) + 8 <= BAR_BYTES, "barriers fit their block");
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + PL::OFF_BAR + 8 * (NB0 + SW + 4));
  float* cs = reinterpret_cast<float*>(gen + PL::OFF_BAR + BAR_BYTES);   // per-sequence output scales
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int* status = g_status;

  if (tid == 0) {
    for (int s = 0; s < SW; ++s) {
      mbar_init(wfull(s), 1);
      mbar_init(wempty(s), 1);                              // the MMA has read the slot
      mbar_init(convdone(s), CONV_WARPS);
    }
    for (int s = 0; s < MAX_SX; ++s) {
      mbar_init(xfull(s), 1);
      mbar_init(xempty(s), 1);
    }
    for (int c = 0; c < 2; ++c) {
      mbar_init(accfull(c), 1);
      mbar_init(accfree(c), EPI_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == WARP_MMA) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), TMEM_ALLOC);
    tmem_relinquish();
  }
  if (warp == WARP_TMA && lane == 0) {
    prefetch_tensormap(&mw0);
    if (p.n_mats > 1) prefetch_tensormap(&mw1);
    if (p.n_mats > 2) prefetch_tensormap(&mw2);
    prefetch_tensormap(&mx);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  mca_pdl_launch_dependents();   // a dependent launch may take the SMs as this kernel's CTAs leave them
  const int nacc = p.swiglu ? 2 : 1;
  // this CTA's units [lo, hi) of the (tile, k chunk) order: segments (tile u, chunks [k0, k1))
  const int64_t total = (int64_t)p.tiles * p.kchunks;
  auto range_lo = [&](int c) { return (int)(((int64_t)c * total) / (int)gridDim.x); };
  auto owner = [&](int64_t unit) { return (int)(((unit + 1) * (int)gridDim.x - 1) / total); };
  const int lo = range_lo(blockIdx.x), hi = range_lo(blockIdx.x + 1);
  struct Segment { int u, k0, k1; };
  auto segment = [&](int pos) {
    Segment g;
    g.u = pos / p.kchunks;
    g.k0 = pos - g.u * p.kchunks;
    g.k1 = min(p.kchunks, g.k0 + hi - pos);
    return g;
  };
  bool ok = true;

  if (warp == WARP_TMA) {
    // ------------------------------------------------------------------ weight producer
    // The weights depend on nothing this stream computes: their tiles are requested from the first instruction on, also
    // while the pre-pass that this launch may have overtaken is still running.  A slot is free again as soon as the
    // converters have read it (fp32) or the MMA has (bf16).
    if (lane == 0) {
      int g = 0;
      for (int pos = lo; pos < hi && ok;) {
        const Segment sg = segment(pos);
        pos += sg.k1 - sg.k0;
        int m = 0, row0 = sg.u * ROWS;
        if (!p.swiglu) {
          if (p.n_mats > 1 && sg.u >= p.tile0[1]) m = 1;
          if (p.n_mats > 2 && sg.u >= p.tile0[2]) m = 2;
          row0 = (sg.u - p.tile0[m]) * ROWS;
        }
        for (int kc = sg.k0; kc < sg.k1 && ok; ++kc) {
          for (int mi = 0; mi < nacc; ++mi, ++g) {
            const int mm = p.swiglu ? mi : m;
            const CUtensorMap* mw = mm == 0 ? &mw0 : (mm == 1 ? &mw1 : &mw2);
            const int s = g % SW;
            ok = mbar_wait(wempty(s), (uint32_t)(((g / SW) & 1) ^ 1), status, 1, g);
            if (!ok) break;
            mbar_expect_tx(wfull(s), PL::W_BYTES);
            tma_load_2d(base + PL::OFF_W + s * PL::W_BYTES, mw, wfull(s), kc * KC, row0);
          }
        }
      }
    }
  } else if (warp == WARP_TMA_X) {
    // ------------------------------------------------------------------ activation producer
    if (lane == 0) {
      mca_pdl_wait();                                     // the pieces are the pre-pass's output
      int g = 0, s = 0;
      uint32_t ph = 0;
      for (int pos = lo; pos < hi && ok;) {
        const Segment sg = segment(pos);
        pos += sg.k1 - sg.k0;
        for (int kc = sg.k0; kc < sg.k1; ++kc, ++g) {
          ok = mbar_wait(xempty(s), ph ^ 1u, status, 8, g);
          if (!ok) break;
          mbar_expect_tx(xfull(s), x_stage_bytes);
          // both pieces are consecutive rows of the array: one box
          tma_load_2d(base + PL::OFF_X + s * x_stage_bytes, &mx, xfull(s), kc * KC, 0);
          if (++s == SX) { s = 0; ph ^= 1u; }
        }
      }
    }
  } else if (warp == WARP_MMA) {
    // ------------------------------------------------------------------ MMA issuer
    // The warp runs this role in lock step and one elected lane issues: descriptors are warp-uniform values, made once and
    // stepped by additions on their address field.  What a chunk costs the issuing thread is what bounds the kernel before
    // the memory does.
    {
      const uint32_t leader = elect_one() ? 1u : 0u;
      const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
      // hi and lo pieces of all sequences are one operand of 2 Bp columns: an instruction costs about the same up to 128
      // columns, so W . [x_hi | x_lo] is one instruction per 16 k, and the epilogue adds the two halves of its result
      const uint32_t idesc2 = make_idesc_fmt(ROWS, 2 * p.Bp, 0, 0, PL::FMT), idesc = make_idesc_fmt(ROWS, p.Bp, 0, 0, PL::FMT);
      const uint64_t desc_w = make_desc(base + PL::OFF_W, 16, 1024), desc_x = make_desc(base + PL::OFF_X, 16, 1024);
      const uint32_t x_step = x_stage_bytes >> 4;
      int sw = 0, sx = 0, it = 0, g = 0;
      uint32_t wph = 0, xph = 0;
      for (int pos = lo; pos < hi && ok; ++it) {
        const Segment sg = segment(pos);
        const int n = sg.k1 - sg.k0;
        pos += n;
        const int a = it & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(accfree(a), (uint32_t)(((it >> 1) & 1) ^ 1), status, 2, it));
        if (!ok) break;
        tc_fence_after();
        const uint32_t d0 = tmem_u + (uint32_t)a * ACC_COLS;
        for (int kc = 0; kc < n && ok; ++kc) {
          ok = __all_sync(0xffffffffu, mbar_wait(xfull(sx), xph, status, 9, g));
          if (!ok) break;
          const uint64_t dx = desc_x + (uint64_t)((uint32_t)sx * x_step);
          for (int mi = 0; mi < nacc; ++mi, ++g) {       // the gated pair shares the chunk's activations
            // fp32 weights: the slot holds the converted hi | lo tiles once all converter warps have arrived
            ok = __all_sync(0xffffffffu, mbar_wait(PL::CONVERT ? convdone(sw) : wfull(sw), wph, status, 3, g));
            if (!ok) break;
            tc_fence_after();
            const uint32_t d_tmem = d0 + (uint32_t)(mi * 2 * p.Bp);
            const uint64_t dw = desc_w + (uint64_t)((uint32_t)sw * (PL::W_BYTES >> 4));
#pragma unroll
            for (int kk = 0; kk < KC / 16; ++kk) {
              umma_ss_if<false>(leader, d_tmem, dw + 2 * kk, dx + 2 * kk, idesc2, (kc | kk) != 0 ? 1u : 0u);   // W_hi . [x_hi | x_lo]
              if constexpr (PL::CONVERT)
                umma_ss_if<false>(leader, d_tmem, dw + (PL::OP_BYTES >> 4) + 2 * kk, dx + 2 * kk, idesc, 1u);  // W_lo . x_hi
            }
            umma_commit_if(leader, wempty(sw));
            if (++sw == SW) { sw = 0; wph ^= 1u; }
          }
          if (!ok) break;
          umma_commit_if(leader, xempty(sx));
          if (++sx == SX) { sx = 0; xph ^= 1u; }
        }
        if (ok) umma_commit_if(leader, accfull(a));
      }
    }
  } else if (warp < WARP_EPI0) {
    // ------------------------------------------------------------------ converters (fp32 weights)
    if constexpr (PL::CONVERT) {
      int g = 0;
      {
        const int steps = nacc * (hi - lo);
        for (int t = 0; t < steps; ++t, ++g) {
          const int s = g % SW;
          const bool mine = __all_sync(0xffffffffu, mbar_wait(wfull(s), (uint32_t)((g / SW) & 1), status, 5, g));
          // The tile is rewritten in place: hi over the first half of the slot, lo over the second.  A lane takes the
          // sixteen rows of its warp into registers (k = 2 lane, 2 lane + 1: 8-byte reads, no bank conflicts); nobody
          // writes before all eight warps have read.  The barrier also carries the vote on the wait's outcome, so that
          // either every converter warp goes on or none does.
          float2 v[ROWS / CONV_WARPS];
          const float* wst = reinterpret_cast<const float*>(gen + PL::OFF_W + s * PL::W_BYTES);
          if (mine) {
#pragma unroll
            for (int rr = 0; rr < ROWS / CONV_WARPS; ++rr)
              v[rr] = *reinterpret_cast<const float2*>(wst + (warp * (ROWS / CONV_WARPS) + rr) * KC + 2 * lane);
          }
          ok = conv_bar_and(mine);
          if (!ok) break;
          unsigned char* ohi = gen + PL::OFF_W + s * PL::W_BYTES;
          unsigned char* olo = ohi + PL::OP_BYTES;
#pragma unroll
          for (int rr = 0; rr < ROWS / CONV_WARPS; ++rr) {
            const int r = warp * (ROWS / CONV_WARPS) + rr;
            // hi = the scaled weight cut to fp16's mantissa (exact in fp16), lo = the rest (exact in fp32, rounded once)
            const float a0 = v[rr].x * W_SCALE, a1 = v[rr].y * W_SCALE;
            const float h0 = __uint_as_float(__float_as_uint(a0) & 0xffffe000u), h1 = __uint_as_float(__float_as_uint(a1) & 0xffffe000u);
            uint32_t h, l;
            asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(h1), "f"(h0));
            asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(l) : "f"(a1 - h1), "f"(a0 - h0));
            const uint32_t off = (uint32_t)(r >> 3) * 1024u + (uint32_t)(r & 7) * 128u + (uint32_t)(((lane >> 2) ^ (r & 7)) << 4) +
                                 (uint32_t)(lane & 3) * 4u;
            *reinterpret_cast<uint32_t*>(ohi + off) = h;
            *reinterpret_cast<uint32_t*>(olo + off) = l;
          }
          fence_proxy_async();          // the MMA reads these tiles through the asynchronous proxy
          __syncwarp();
          if (lane == 0) mbar_arrive(convdone(s));
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue warps
    const int e = warp - WARP_EPI0, quarter = warp & 3;   // TMEM lanes 32 quarter .. 32 quarter + 31
    const int r = quarter * 32 + lane;                    // row of the tile
    const int col_first = (e >> 2) * 8;                   // this warp's columns: col_first + 16 i .. + 7
    // per-sequence output scales, written by the pre-pass this launch may have overtaken: every warp writes the same copy
    mca_pdl_wait();
    cs[lane] = lane < p.B ? __ldcg(g_x_scale + lane) : 0.f;
    cs[lane + 32] = lane + 32 < p.B ? __ldcg(g_x_scale + lane + 32) : 0.f;
    __syncwarp();
    int it = 0;
    for (int pos = lo; pos < hi && ok; ++it) {
      const Segment sg = segment(pos);
      const int u = sg.u;
      pos += sg.k1 - sg.k0;
      const int a = it & 1;
      int m = 0, row0 = u * ROWS;
      if (!p.swiglu) {
        if (p.n_mats > 1 && u >= p.tile0[1]) m = 1;
        if (p.n_mats > 2 && u >= p.tile0[2]) m = 2;
        row0 = (u - p.tile0[m]) * ROWS;
      }
      float* outm = m == 0 ? p.out[0] : (m == 1 ? p.out[1] : p.out[2]);
      const int rows_m = m == 0 ? p.rows[0] : (m == 1 ? p.rows[1] : p.rows[2]);
      const int row = row0 + r;
      const bool whole = sg.k0 == 0 && sg.k1 == p.kchunks;
      // the parts of this tile: CTAs c_first .. c_last, all but the first of which begin inside it
      const int c_first = owner((int64_t)u * p.kchunks), c_last = owner((int64_t)(u + 1) * p.kchunks - 1);
      const int first_slot = 2 * c_first + (range_lo(c_first) / p.kchunks == u ? 0 : 1);
      constexpr size_t SLOT = (size_t)2 * MAX_B * ROWS;   // floats of a part: (column, row)
      auto slot_of = [&](int c) { return c == c_first ? first_slot : 2 * c; };
      const uint32_t t_acc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)a * ACC_COLS;
      // the residuals of eight output elements of this thread's row, requested before anything is waited for
      auto residuals = [&](int c0, float (&res)[8]) {
        const float* src = outm + (size_t)c0 * rows_m + row;
#pragma unroll
        for (int i = 0; i < 8; ++i) res[i] = (p.accumulate && row < rows_m && c0 + i < p.B) ? __ldcg(src + (size_t)i * rows_m) : 0.f;
      };
      float res[8];
      residuals(col_first, res);                          // the first eight's before the products are waited for
      ok = __all_sync(0xffffffffu, mbar_wait(accfull(a), (uint32_t)((it >> 1) & 1), status, 7, it));
      if (!ok) break;
      tc_fence_after();
      // eight output elements: the products scaled back, gated if asked, added to the residual
      auto finish8 = [&](int c0, const float (&va)[8], const float (&vb)[8], const float (&res)[8]) {
        if (row >= rows_m) return;
        float* dst = outm + (size_t)c0 * rows_m + row;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (c0 + i < p.B) {
            const float sc = cs[c0 + i];
            float y = va[i] * sc;
            if (p.swiglu) {
              y *= (1.0f / (1.0f + expf(-y)));          // silu, llama2_cpu.cpp:360-365
              y *= vb[i] * sc;
            }
            dst[(size_t)i * rows_m] = y + res[i];
          }
        }
      };
      // eight columns of a result: the x_hi half plus the x_lo half
      auto load_acc = [&](uint32_t t, int col, float (&v)[8]) {
        uint32_t h[8], l[8];
        tmem_ld8(t + col, h);
        tmem_ld8(t + col + p.Bp, l);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(h[i]) + __uint_as_float(l[i]);
      };
      if (whole) {
        for (int c0 = col_first; c0 < p.Bp; c0 += 16) {
          float fa[8], fb[8];
          if (c0 != col_first) residuals(c0, res);
          load_acc(t_acc, c0, fa);
          if (p.swiglu) load_acc(t_acc, 2 * p.Bp + c0, fb);
          else {
#pragma unroll
            for (int i = 0; i < 8; ++i) fb[i] = 0.f;
          }
          finish8(c0, fa, fb, res);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(accfree(a));
        continue;
      }
      float* part = g_partials + (size_t)slot_of(blockIdx.x) * SLOT + r;
      for (int c0 = col_first; c0 < p.Bp; c0 += 16) {
        for (int mi = 0; mi < nacc; ++mi) {
          float v[8];
          load_acc(t_acc, mi * 2 * p.Bp + c0, v);       // the second result starts behind both halves of the first
#pragma unroll
          for (int i = 0; i < 8; ++i) __stcg(part + (size_t)(mi * MAX_B + c0 + i) * ROWS, v[i]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(accfree(a));
      // a ticket per tile and epilogue warp: the one that arrives last adds up all parts
      __syncwarp();
      int last = 0;
      if (lane == 0) {
        // releases the warp's partial sums and acquires the other CTAs' at once.  A fence on either side of the ticket, and the residuals
        // asked for only here instead of ahead of the last products, made the end of every product 1.5 us longer (a step of 16 sequences,
        // four 7B-shaped layers, bf16: 759 -> 724 us; 64 sequences, two layers 491 -> 478; fp32, 16: 528 -> 521).
        unsigned int old;
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(&g_tickets[u * EPI_WARPS + e]) : "memory");
        last = old == (unsigned int)(c_last - c_first);
        if (last) g_tickets[u * EPI_WARPS + e] = 0;    // ready for the next launch
      }
      last = __shfl_sync(0xffffffffu, last, 0);
      if (!last) continue;
      __syncwarp();   // what lane 0 has acquired is the other lanes' too: a shuffle orders no memory
      // all of a round's loads in flight together; the sums are taken in the parts' order whoever arrived last
      const float* p0 = g_partials + r;
      for (int c0 = col_first; c0 < p.Bp; c0 += 16) {
        float va[8], vb[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) va[i] = vb[i] = 0.f;
        if (c0 != col_first) residuals(c0, res);
        if (p.swiglu) {
          constexpr int Q = PL::CONVERT ? 2 : 4;
          for (int s0 = c_first; s0 <= c_last; s0 += Q) {
            float t[Q][2][8];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
              const float* src = p0 + (size_t)slot_of(min(s0 + q, c_last)) * SLOT + (size_t)c0 * ROWS;
#pragma unroll
              for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                for (int i = 0; i < 8; ++i) t[q][mi][i] = s0 + q <= c_last ? __ldcg(src + (size_t)(mi * MAX_B + i) * ROWS) : 0.f;
            }
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
              for (int i = 0; i < 8; ++i) { va[i] += t[q][0][i]; vb[i] += t[q][1][i]; }
          }
        } else {
          constexpr int Q = PL::CONVERT ? 4 : 8;
          for (int s0 = c_first; s0 <= c_last; s0 += Q) {
            float t[Q][8];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
              const float* src = p0 + (size_t)slot_of(min(s0 + q, c_last)) * SLOT + (size_t)c0 * ROWS;
#pragma unroll
              for (int i = 0; i < 8; ++i) t[q][i] = s0 + q <= c_last ? __ldcg(src + (size_t)i * ROWS) : 0.f;
            }
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
              for (int i = 0; i < 8; ++i) va[i] += t[q][i];
          }
        }
        finish8(c0, va, vb, res);
      }
    }
  }
  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (warp == WARP_MMA) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_ALLOC);
  }
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
inline int make_map_2d(CUtensorMap* map, const void* basep, CUtensorMapDataType type, int elt, int64_t rows, int64_t cols,
                       int box_cols, int box_rows, CUtensorMapSwizzle swizzle) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return ERROR_ATTN_UNSUPPORTED_SHAPE;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)cols * elt};
  const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, type, 2, const_cast<void*>(basep), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : ERROR_ATTN_UNSUPPORTED_SHAPE;
}

inline bool& enabled() { static bool on = true; return on; }

// CTAs for `units` (row tile, k chunk) units on `sms` SMs: one per SM, with at least four units each.
inline int pick_ctas(int64_t units, int sms) { return (int)std::max<int64_t>(1, std::min<int64_t>(std::min(sms, MAX_CTAS), units / 4)); }

}  // namespace proj
