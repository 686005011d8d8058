// Fused attention backward on the tensor cores (sm_100a, bf16): the counterpart of the forward
// kernel in attn_tc.cu for training.
//
// Same mathematics as the reference's attnHandle<T>::Backward (CudaDnnDLL/Cuda Files/
// attn.cu:608-661 with blob<T>::matmulgrad attn.cu:380-397):
//   dP = dY V^T,  dV = P^T dY,  dS = P o (dP - rowsum(dP o P)),  dS *= 1/sqrt(D),
//   dQ = dS K,    dK = dS^T Q
// The reference reads the (B,H,T,T) probabilities its Forward saved; here P is recomputed tile
// by tile from the log-sum-exp kept by the forward kernel, and rowsum(dP o P) is taken as
// delta = rowsum(dY o Y), so no T x T tensor exists.
//
// Two kernels (no atomics, deterministic):
//   * dq kernel: one CTA per 128-row query tile walks the key tiles:  S = Q K^T and dP = dY V^T
//     (tcgen05.mma, both operands in shared memory), dS computed by sixteen (or eight) warps straight from
//     TMEM and written back as a bf16 A operand, dQ += dS K accumulated in TMEM.
//   * dkdv kernel: one CTA per 128-row key tile walks the query tiles with the transposed
//     products S^T = K Q^T and dP^T = V dY^T, so that P^T and dS^T come out in the layout the
//     A operand of dV += P^T dY and dK += dS^T Q needs.
// Where it gains (ds_rules) the dkdv kernel leaves its dS tiles in a workspace and dQ = dS K is one product over them.
// Q/K/V/dY tiles arrive by TMA (no multicast) through rings; every mbarrier wait is
// bounded as in the forward kernel.
//
// SPLIT = true is the variant for fp32 callers: every operand is carried as two fp16 halves (rows [hi | lo] written by
// the pre-pass in split_prepass.cuh, each head of each tensor scaled by a power of two), every product is the three kind::f16
// products hi.hi + hi.lo + lo.hi into one fp32 TMEM tile, P^T / dS / dS^T are split the same way by the element-wise
// warps, and the gradients are written in fp32.  Head sizes up to 64: a split tile is as large as a 128-wide bf16 one.
#include <type_traits>

#include "ds_rules.h"
#include "kernels.h"
#include "launch_rules.h"
#include "tc_common.cuh"
#include "split_prepass.cuh"

namespace {

using namespace tc;

// dS between the dK/dV kernel and the dQ kernel that is one product over it (DS): one 128 x 128 tile per (query tile, key tile)
// of a head, the lower triangle alone under the causal mask.  A tile is the image of the tensor core's unswizzled MN-major A
// operand: four blocks of 32 keys, each (hi, then in split mode lo) sixteen groups of 8 queries x 32 keys x 16 bytes.  A key's eight
// queries are what a thread that reads dS^T from TMEM has in four registers, so a warp writes 512 consecutive bytes an instruction without
// a shuffle, and the dQ kernel reads a tile by plain bulk copies.
constexpr int DS_GROUP_BYTES = 32 * 16, DS_BLOCK_BYTES = 16 * DS_GROUP_BYTES;
static_assert(launch_rules::TILE == BLK);
static_assert(ds_rules::TILE == BLK && ds_rules::tile_bytes(false) == 4 * DS_BLOCK_BYTES && ds_rules::tile_bytes(true) == 8 * DS_BLOCK_BYTES);
template <bool SPLIT> __device__ __forceinline__ int64_t ds_tile_offset(int64_t head, int qt, int kt, int T, int causal) {
  const int nt = (T + BLK - 1) / BLK;
  return (head * ds_rules::head_tiles(T, causal) + (causal ? (int64_t)qt * (qt + 1) / 2 : (int64_t)qt * nt) + kt) * ds_rules::tile_bytes(SPLIT);
}

// What a CTA looks like.  It keeps two 128-row tiles (Q and dY, or K and V) and streams the other two tensors BN rows a step.
//   WIDE    128 rows a step, sixteen element-wise warps (four threads per row, 32 columns each), all of TMEM, one CTA per SM.
//   NARROW  64 rows a step, eight element-wise warps (two threads per row, 32 columns each), half of TMEM and under half of the
//           shared memory: two CTAs share an SM, and one's set-up, first loads, pipeline fill and gradient stores run beside
//           the other's steps.  At T = 1024 a causal CTA walks four and a half key tiles on average, and those fixed parts were
//           half of its life: B=8 H=12 T=1024 D=64 bf16, dK/dV 59 -> 52 us, dQ 49 -> 40, the whole layer 142 -> 118; T = 9200 and
//           more gain 4 % (two steps in flight).  For bf16 heads of 64; 128-wide heads and split operands have no room for two.
// ROW: elements of 2 bytes per operand row (a split row is two 128-byte sub-tiles [hi | lo]).
template <int ROW, bool NARROW> struct BwdPlan {
  static constexpr int BN = NARROW ? 64 : 128;
  static constexpr int EW_WARPS = NARROW ? 8 : 16;         // element-wise warps
  static constexpr int WARP_TMA = EW_WARPS, WARP_MMA = EW_WARPS + 1, THREADS = (EW_WARPS + 2) * 32;
  static constexpr int CTAS_PER_SM = NARROW ? 2 : 1;
  static constexpr uint32_t TMEM_COLS = NARROW ? 256 : 512;
  static constexpr int SUB = ROW / 64;
  static constexpr uint32_t SUB_BYTES = BLK * 128;         // a resident tile's sub-tile; of a streamed one:
  static constexpr uint32_t RING_SUB_BYTES = BN * 128;
  static constexpr uint32_t TILE_BYTES = SUB * SUB_BYTES, RING_TILE_BYTES = SUB * RING_SUB_BYTES;
  static constexpr uint32_t OFF_RES0 = 0, OFF_RES1 = TILE_BYTES;
  // dQ kernel: K lives until the step's dQ product, so its ring is one stage deeper than V's (K(j+2) could
  // otherwise only be requested when dQ(j) has finished, one step before it is needed, and every step
  // would wait out the load latency).  The dK/dV kernel has Q where the dQ kernel has K, and dY where it has V.
  static constexpr int K_STAGES = NARROW ? 4 : 3, V_STAGES = NARROW ? 3 : 2;
  static constexpr uint32_t OFF_KRING = 2 * TILE_BYTES;
  static constexpr uint32_t OFF_VRING = OFF_KRING + K_STAGES * RING_TILE_BYTES;
  static constexpr uint32_t OFF_BAR = OFF_VRING + V_STAGES * RING_TILE_BYTES;
  static constexpr uint32_t BYTES_DQ = OFF_BAR + 256 + 1024;
  // dK/dV kernel: behind the barriers the staged per-query terms ([2][BN] floats twice) and the
  // abort flag, all in dynamic shared memory (no static allocation, so the dynamic base keeps its alignment).
  // At 128-wide heads this leaves 752 bytes for aligning the base to 1024; the kernel checks that it fits.
  static constexpr uint32_t OFF_STAGE_KV = OFF_BAR + 256;
  static constexpr uint32_t OFF_FLAG_KV = OFF_STAGE_KV + 2 * 2 * BN * 4;
  static constexpr uint32_t NEED_KV = OFF_FLAG_KV + 16;
  static constexpr uint32_t BYTES_KV = (NEED_KV + 1024 <= 227u * 1024u) ? NEED_KV + 1024 : 227u * 1024u;
  static_assert(CTAS_PER_SM == 1 || CTAS_PER_SM * ((BYTES_KV > BYTES_DQ ? BYTES_KV : BYTES_DQ) + 1024 + 128) <= 228 * 1024,
                "shared memory of the CTAs of one SM");
};

// fp16 halves of a value the tensor core must see at fp32 accuracy: hi = v with the mantissa cut to fp16 width (the
// conversion is then exact for normal numbers), lo = v - hi.
__device__ __forceinline__ void split_pack(float v0, float v1, uint32_t& hi, uint32_t& lo) {
  const float h0 = __uint_as_float(__float_as_uint(v0) & 0xffffe000u), h1 = __uint_as_float(__float_as_uint(v1) & 0xffffe000u);
  hi = pack_f16(h0, h1);
  lo = pack_f16(v0 - h0, v1 - h1);
}
// Split mode keeps dS 2^-19 smaller than dP' = dY' V'^T (both operands scaled to below 2^13, so |dP'| < 2^32 at 64-wide
// heads) and P^T 2^10 larger than P <= 1: both then sit in the middle of the fp16 range.
using split::DS_SHIFT, split::DS_SHIFT_LOG2;
constexpr float PT_SHIFT = 1024.0f;
constexpr int PT_SHIFT_LOG2 = 10;

struct BwdParams {
  const float4* scales;   // split mode: the pre-pass's scales (q, k, v, dY) of each (batch, head)
  const float* lse;    // (BH, T) log2-domain log-sum-exp of the scaled logits, from the forward kernel
  const float* delta;  // (BH, T) rowsum(dY o Y); split mode: times the head's scale of dY and DS_SHIFT
  void* out0;          // dq kernel: dQ;  dkdv kernel: dK
  void* out1;          // dkdv kernel: dV
  int* status;
  int T, causal, H;
  int bh0;             // first (batch, head) of this launch
  uint8_t* ds;         // DS: the dS tiles of this launch's heads (see ds_tile_offset)
  int group;           // (batch, head) pairs whose CTAs are interleaved longest-first (their tensors fit in L2 together)
  float scale_log2;    // (1/sqrt(HD)) * log2(e)
  float scale;         // 1/sqrt(HD)
  McaStrides os;       // element strides of the gradient views dQ, dK, dV
  // MASKED: keep-bits of the caller's mask as the forward kernel reads them (word of query row r, key tile j, quarter
  // c: mask_bits[b * batch_stride + r * row_stride + 4 j + c]) and, for a (T,T) mask, their transpose (word of key k,
  // query tile i, quarter c: mask_bits_t[k * row_stride + 4 i + c]); a (B,T) key mask has row stride 0 and no transpose.
  // A masked entry has probability 0, or 1 / T in a row whose every key is masked (the forward marks those rows
  // with lse = +inf).
  const uint32_t* mask_bits;
  const uint32_t* mask_bits_t;
  int64_t mask_batch_stride, mask_row_stride;
  float inv_T;
};


// The gradient tiles leave through shared memory.  In the TMEM layout a thread owns a quarter of one row, so direct
// stores are 32 sixteen-byte pieces from 32 rows per instruction (9-12 % of the backward at T = 1024 was these
// stores).  Instead the element-wise warps write their pieces into a resident operand tile that every product
// has finished with (Q or K for the first result, dY or V for the second), meet at a named barrier, and each warp
// stores its share of whole rows.  Every element-wise warp reaches the barrier, also after a failed wait.
template <int EW_WARPS> __device__ __forceinline__ void ew_bar_sync() { asm volatile("bar.sync 1, %0;" ::"n"(EW_WARPS * 32) : "memory"); }
// 16-byte piece `piece` of row `row` of a staged 128-row tile with PR pieces per row (XOR-swizzled by row)
template <int PR> __device__ __forceinline__ uint4* staged_piece(uint8_t* tile, int row, int piece) {
  return reinterpret_cast<uint4*>(tile) + row * PR + (piece ^ (row & (PR - 1)));
}
// this thread's OC columns of its row, as 16-byte pieces of bf16, or of fp32 times scale x (the split operands' power of two)
template <int PR, int OC, bool F32>
__device__ __forceinline__ void stage_columns(uint8_t* tile, int row, int qtr, uint32_t t_addr, float scale, float2 pow2) {
  constexpr int CH = OC < 16 ? OC : 16;
  const float first = scale * pow2.x;
#pragma unroll
  for (int c = 0; c < OC / CH; ++c) {
    uint32_t o[CH];
    if constexpr (CH == 16) tmem_ld16(t_addr + c * 16, o);
    else if constexpr (CH == 8) tmem_ld8(t_addr, o);
    else tmem_ld4(t_addr, o);
    tmem_wait_ld();
    if constexpr (F32) {
      auto v = [&](int i) { return __float_as_uint(__uint_as_float(o[i]) * first * pow2.y); };
#pragma unroll
      for (int i = 0; i < CH; i += 4)
        *staged_piece<PR>(tile, row, (qtr * OC + c * CH + i) / 4) = make_uint4(v(i), v(i + 1), v(i + 2), v(i + 3));
    } else {
      auto v = [&](int i) { return pack_bf16(__uint_as_float(o[i]), __uint_as_float(o[i + 1])); };
#pragma unroll
      for (int i = 0; i < CH; i += 8)
        *staged_piece<PR>(tile, row, (qtr * OC + c * CH + i) / 8) = make_uint4(v(i), v(i + 2), v(i + 4), v(i + 6));
    }
  }
}
// warp w of the element-wise warps stores rows RPW w .. RPW (w + 1) - 1 of a staged tile; off0: element offset of the tile's row 0
template <int PR, int ESZ, int RPW>
__device__ __forceinline__ void store_staged_rows(uint8_t* tile, int w, int lane, void* out, int64_t off0, int64_t row_stride,
                                                  int rows_valid) {
  constexpr int RPI = 32 / PR;   // rows per store instruction
#pragma unroll
  for (int kk = 0; kk < RPW / RPI; ++kk) {
    const int row = RPW * w + kk * RPI + lane / PR, piece = lane % PR;
    if (row < rows_valid)
      *reinterpret_cast<uint4*>(static_cast<char*>(out) + (off0 + (int64_t)row * row_stride) * ESZ + piece * 16) =
          *staged_piece<PR>(tile, row, piece);
  }
}

// ---------------------------------------------------------------------------------------------
// dQ kernel.  TMEM columns: S [0,BN)  dP [BN,2 BN)  dS (16-bit, packed) [2 BN, 5/2 BN) and, in split mode, its lo half
// [5/2 BN, 3 BN)  dQ behind them
// ---------------------------------------------------------------------------------------------
enum DqBar : int {
  DQ_Q_FULL = 0,
  DQ_K_FULL = 1,    // [K_STAGES, at most 4]
  DQ_K_EMPTY = 5,
  DQ_V_FULL = 9,    // [V_STAGES, at most 3]
  DQ_V_EMPTY = 12,
  DQ_SDP_FULL = 15, // S and dP of the step written by the MMA
  DQ_SDP_FREE = 16, // element-wise warps have S and dP in registers
  DQ_DS_READY = 17, // dS written to TMEM
  DQ_DQ_DONE = 18,  // dQ += dS K of the step finished (dS may be overwritten)
  DQ_DRAIN = 19,
  DQ_DO_FULL = 20,
  DQ_BAR_COUNT = 21
};

template <int HD, bool SPLIT, bool MASKED, bool NARROW>
__global__ void __launch_bounds__((BwdPlan<SPLIT ? 128 : HD, NARROW>::THREADS), (BwdPlan<SPLIT ? 128 : HD, NARROW>::CTAS_PER_SM))
sdpa_bwd_dq_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                      const BwdParams p) {
  using PL = BwdPlan<SPLIT ? 128 : HD, NARROW>;
  constexpr int BN = PL::BN, EW_WARPS = PL::EW_WARPS, WARP_TMA = PL::WARP_TMA, WARP_MMA = PL::WARP_MMA;
  constexpr uint32_t TMEM_COLS = PL::TMEM_COLS;
  constexpr int FMT = SPLIT ? 0 : 1;       // operand format of the instruction descriptor: fp16 or bf16
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar0 = smem_base + PL::OFF_BAR;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + PL::OFF_BAR + DQ_BAR_COUNT * 8);
  auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // launch order -> work item: longest causal work first inside groups of p.group heads (see the forward kernel)
  const int lin = (int)(blockIdx.y * gridDim.x + blockIdx.x);
  const int grp = lin / (p.group * (int)gridDim.x);
  const int in_grp = lin - grp * p.group * (int)gridDim.x;
  const int grp_heads = min(p.group, (int)gridDim.y - grp * p.group);
  const int rank = in_grp / grp_heads;
  const int bh = p.bh0 + grp * p.group + (in_grp - rank * grp_heads), T = p.T;
  const int bi = bh / p.H, hi = bh - bi * p.H;   // batch item and head
  const int qt = (int)gridDim.x - 1 - rank;
  const int q0 = qt * BLK;
  const int n = ((p.causal ? min(q0 + BLK, T) : T) + BN - 1) / BN;   // key steps

  // set-up, each part by another warp so that their latencies overlap (status word, barriers, descriptors, TMEM)
  __shared__ int s_abort;
  mca_pdl_launch_dependents();
  if (tid == 32) s_abort = *reinterpret_cast<volatile int*>(p.status);
  if (warp == WARP_TMA && lane == 0) {
    prefetch_tensormap(&map_q); prefetch_tensormap(&map_k); prefetch_tensormap(&map_v); prefetch_tensormap(&map_do);
  }
  if (tid == 0) {
    for (int i = 0; i < DQ_BAR_COUNT; ++i)
      mbar_init(bar(i), (i == DQ_SDP_FREE || i == DQ_DS_READY) ? (uint32_t)EW_WARPS : 1u);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == WARP_MMA) { tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // No wait here.  The kernel before this one in a backward is the dK/dV kernel, which lets its dependents go only
  // after its own wait: when a CTA of this kernel runs, everything before that kernel (delta, the forward, the operand
  // split) is complete and visible, and that is all this kernel reads.  It writes dQ only, which the dK/dV kernel does
  // not touch, so its CTAs work in the SMs that kernel's last wave leaves free.  The wait at the end keeps the order
  // for what follows: this kernel is not complete before the dK/dV kernel is.
  if (s_abort != 0) {   // an earlier CTA already failed: leave (uniform decision) before any copy or product is issued
    if (warp == WARP_MMA) tmem_dealloc(tmem_base, TMEM_COLS);
    mca_pdl_wait();
    return;
  }
  constexpr uint32_t C_S = 0, C_DP = BN, C_DS = 2 * BN, DS_LO = BN / 2, C_DQ = C_DS + (SPLIT ? BN : BN / 2);
  static_assert(C_DQ + HD <= TMEM_COLS);
  bool ok = true;

  if (warp == WARP_TMA) {
    if (lane == 0) {
      // one resident tile; S(0) waits for Q and K(0) only, so those come first
      auto load_resident = [&](uint32_t dst, const CUtensorMap* map, int full) {
        mbar_expect_tx(bar(full), PL::TILE_BYTES);
#pragma unroll
        for (int s = 0; s < PL::SUB; ++s)
#pragma unroll
          for (int r = 0; r < BLK; r += BN)   // a copy's box is BN rows
            tma_load_4d(smem_base + dst + s * PL::SUB_BYTES + r * 128, map, bar(full), s * 64, q0 + r, hi, bi);
      };
      load_resident(PL::OFF_RES0, &map_q, DQ_Q_FULL);
      int issued_k = 0, issued_v = 0;
      for (int j = 0; j < n && ok; ++j) {
        const int ks = j % PL::K_STAGES, vs = j % PL::V_STAGES;
        const uint32_t kph = (uint32_t)((j / PL::K_STAGES) & 1), vph = (uint32_t)((j / PL::V_STAGES) & 1);
        const uint32_t k_dst = smem_base + PL::OFF_KRING + ks * PL::RING_TILE_BYTES, v_dst = smem_base + PL::OFF_VRING + vs * PL::RING_TILE_BYTES;
        ok = mbar_wait(bar(DQ_K_EMPTY + ks), kph ^ 1u, p.status, 110, j);
        if (!ok) break;
        mbar_expect_tx(bar(DQ_K_FULL + ks), PL::RING_TILE_BYTES);
#pragma unroll
        for (int s = 0; s < PL::SUB; ++s) tma_load_4d(k_dst + s * PL::RING_SUB_BYTES, &map_k, bar(DQ_K_FULL + ks), s * 64, j * BN, hi, bi);
        issued_k = j + 1;
        if (j == 0) load_resident(PL::OFF_RES1, &map_do, DQ_DO_FULL);
        ok = mbar_wait(bar(DQ_V_EMPTY + vs), vph ^ 1u, p.status, 111, j);
        if (!ok) break;
        mbar_expect_tx(bar(DQ_V_FULL + vs), PL::RING_TILE_BYTES);
#pragma unroll
        for (int s = 0; s < PL::SUB; ++s) tma_load_4d(v_dst + s * PL::RING_SUB_BYTES, &map_v, bar(DQ_V_FULL + vs), s * 64, j * BN, hi, bi);
        issued_v = j + 1;
      }
      if (!ok) {  // let copies in flight land (bounded) before the CTA's memory is released
        mbar_wait(bar(DQ_Q_FULL), 0, p.status, 112, 0);
        if (issued_k > 0) mbar_wait(bar(DQ_DO_FULL), 0, p.status, 115, 0);
        for (int j = max(0, issued_k - PL::K_STAGES); j < issued_k; ++j)
          mbar_wait(bar(DQ_K_FULL + j % PL::K_STAGES), (uint32_t)((j / PL::K_STAGES) & 1), p.status, 113, j);
        for (int j = max(0, issued_v - PL::V_STAGES); j < issued_v; ++j)
          mbar_wait(bar(DQ_V_FULL + j % PL::V_STAGES), (uint32_t)((j / PL::V_STAGES) & 1), p.status, 114, j);
      }
    }
  } else if (warp == WARP_MMA) {
    // The warp runs this role in lock step and one elected lane issues, so that addresses and
    // descriptors are warp-uniform values (fewer instructions per tcgen05.mma for the issuing thread).
    {
      const uint32_t leader = elect_one() ? 1u : 0u;
      const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
      constexpr uint32_t IDESC_NT = make_idesc_fmt(BLK, BN, 0, 0, FMT);  // both operands K-major
      constexpr uint32_t IDESC_DQ = make_idesc_fmt(BLK, HD, 0, 1, FMT);   // A from TMEM, B = K tile MN-major
      const uint32_t q_addr = smem_base + PL::OFF_RES0, do_addr = smem_base + PL::OFF_RES1;
      // D = A B^T over the head dimension, both operands K-major in shared memory; split mode: hi.hi + hi.lo + lo.hi
      auto issue_nt = [&](uint32_t d_col, uint32_t a_addr, uint32_t b_addr) {
        if constexpr (SPLIT) {
#pragma unroll
          for (int term = 0; term < 3; ++term) {
            const uint32_t oa = term == 2 ? PL::SUB_BYTES : 0u, ob = term == 1 ? PL::RING_SUB_BYTES : 0u;
#pragma unroll
            for (int kk = 0; kk < HD / 16; ++kk)
              umma_ss_if<false>(leader, tmem_u + d_col, make_desc(a_addr + oa + kk * 32, 16, 1024), make_desc(b_addr + ob + kk * 32, 16, 1024),
                                IDESC_NT, (term > 0 || kk > 0) ? 1u : 0u);
          }
        } else {
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk) {
            umma_ss_if<false>(leader, tmem_u + d_col, make_desc(a_addr + (kk / 4) * PL::SUB_BYTES + (kk % 4) * 32, 16, 1024),
                              make_desc(b_addr + (kk / 4) * PL::RING_SUB_BYTES + (kk % 4) * 32, 16, 1024), IDESC_NT, kk > 0);
          }
        }
      };
      auto issue_sdp = [&](int j) {
        const uint32_t k_addr = smem_base + PL::OFF_KRING + (j % PL::K_STAGES) * PL::RING_TILE_BYTES;
        const uint32_t v_addr = smem_base + PL::OFF_VRING + (j % PL::V_STAGES) * PL::RING_TILE_BYTES;
        issue_nt(C_S, q_addr, k_addr);
        issue_nt(C_DP, do_addr, v_addr);
      };
      ok = __all_sync(0xffffffffu, mbar_wait(bar(DQ_Q_FULL), 0, p.status, 120, 0));
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(bar(DQ_K_FULL + 0), 0, p.status, 121, 0));
      if (ok) {
        tc_fence_after();
        issue_nt(C_S, q_addr, smem_base + PL::OFF_KRING);
        ok = __all_sync(0xffffffffu, mbar_wait(bar(DQ_DO_FULL), 0, p.status, 128, 0));
      }
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(bar(DQ_V_FULL + 0), 0, p.status, 122, 0));
      if (ok) {
        tc_fence_after();
        issue_nt(C_DP, do_addr, smem_base + PL::OFF_VRING);
        umma_commit_if(leader, bar(DQ_SDP_FULL));
        umma_commit_if(leader, bar(DQ_V_EMPTY + 0));
      }
      for (int j = 0; j < n && ok; ++j) {
        const int jn = j + 1;
        if (j + 1 < n) {
          // next S / dP as soon as the element-wise warps hold the current ones in registers (their tiles, long there,
          // are waited for first)
          ok = __all_sync(0xffffffffu, mbar_wait(bar(DQ_K_FULL + jn % PL::K_STAGES), (uint32_t)((jn / PL::K_STAGES) & 1), p.status, 124, j));
          if (ok) ok = __all_sync(0xffffffffu, mbar_wait(bar(DQ_V_FULL + jn % PL::V_STAGES), (uint32_t)((jn / PL::V_STAGES) & 1), p.status, 125, j));
          if (ok) ok = __all_sync(0xffffffffu, mbar_wait(bar(DQ_SDP_FREE), (uint32_t)(j & 1), p.status, 123, j));
          if (!ok) break;
          tc_fence_after();
          issue_sdp(jn);
          umma_commit_if(leader, bar(DQ_SDP_FULL));
          umma_commit_if(leader, bar(DQ_V_EMPTY + jn % PL::V_STAGES));
        }
        ok = __all_sync(0xffffffffu, mbar_wait(bar(DQ_DS_READY), (uint32_t)(j & 1), p.status, 126, j));
        if (!ok) break;
        tc_fence_after();
        const uint32_t k_addr = smem_base + PL::OFF_KRING + (j % PL::K_STAGES) * PL::RING_TILE_BYTES;
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk) {
          umma_ts_if<false>(leader, tmem_u + C_DQ, tmem_u + C_DS + kk * 8, make_desc(k_addr + kk * 2048, PL::RING_SUB_BYTES, 1024), IDESC_DQ,
                  (j > 0 || kk > 0) ? 1u : 0u);
          if constexpr (SPLIT) {   // + dS_hi K_lo + dS_lo K_hi
            umma_ts_if<false>(leader, tmem_u + C_DQ, tmem_u + C_DS + kk * 8, make_desc(k_addr + PL::RING_SUB_BYTES + kk * 2048, PL::RING_SUB_BYTES, 1024),
                              IDESC_DQ, 1u);
            umma_ts_if<false>(leader, tmem_u + C_DQ, tmem_u + C_DS + DS_LO + kk * 8, make_desc(k_addr + kk * 2048, PL::RING_SUB_BYTES, 1024), IDESC_DQ, 1u);
          }
        }
        umma_commit_if(leader, bar(DQ_DQ_DONE));
        umma_commit_if(leader, bar(DQ_K_EMPTY + j % PL::K_STAGES));
      }
      umma_commit_if(leader, bar(DQ_DRAIN));
      mbar_wait(bar(DQ_DRAIN), 0, p.status, 127, 0);
    }
  } else {
    // ------------------------------------------------------------------ element-wise warps
    const int qtr = warp >> 2, lane_base = (warp & 3) * 32, row = lane_base + lane;
    const int qi = q0 + row;
    constexpr int OC = HD / (EW_WARPS / 4);
    const uint32_t t_row = tmem_base + ((uint32_t)lane_base << 16);
    const bool row_ok = qi < T;
    const float lse = row_ok ? p.lse[(int64_t)bh * T + qi] : 0.f;
    const float delta = row_ok ? p.delta[(int64_t)bh * T + qi] : 0.f;
    float4 sc = make_float4(1.f, 1.f, 1.f, 1.f);   // powers of two: every product and quotient of them is exact
    if constexpr (SPLIT) sc = mca_ld_f4(reinterpret_cast<const float*>(p.scales + bh));
    const float sl2 = SPLIT ? split::logit_scale(p.scale_log2, sc) : p.scale_log2;
    const float dmul = SPLIT ? DS_SHIFT : p.scale;
    const float dsub = SPLIT ? delta * sc.z : delta * p.scale;
    for (int j = 0; j < n && ok; ++j) {
      ok = __all_sync(0xffffffffu, mbar_wait(bar(DQ_SDP_FULL), (uint32_t)(j & 1), p.status, 130, j));
      if (!ok) break;
      tc_fence_after();
      uint32_t s[32], dp[32];
      tmem_ld32(t_row + C_S + qtr * 32, s);
      tmem_ld32(t_row + C_DP + qtr * 32, dp);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(DQ_SDP_FREE));
      const int k0 = j * BN + qtr * 32;
      const bool edge = (p.causal && j * BN + BN - 1 > q0) || (j * BN + BN > T);
      uint32_t mw = 0xffffffffu;          // keep-bits of this thread's 32 keys
      float p_masked = 0.f;
      if constexpr (MASKED) {
        mw = __ldg(p.mask_bits + (int64_t)bi * p.mask_batch_stride + (int64_t)min(qi, T - 1) * p.mask_row_stride + (BN / 32) * j + qtr);
        p_masked = (row_ok && lse == INFINITY) ? p.inv_T : 0.f;
      }
      // dS = P o (dP - delta) scale with P = 2^(S scale_log2 - lse); adjacent keys go through as fp32 pairs.
      // Split mode: S and dP carry the pre-pass's scales; dS is kept in the units of dP' x 2^-19 and the factor
      // scale x 2^19 / (s_dy s_v s_k) is applied once to dQ.
      const float2 sc2 = make_float2(sl2, sl2), nl2 = make_float2(-lse, -lse);
      const float2 ps2 = make_float2(dmul, dmul), nd2 = make_float2(-dsub, -dsub);
      const float2 zero2 = make_float2(0.f, 0.f);
      uint32_t pk[16];
      uint32_t pk_lo[SPLIT ? 16 : 1];
      // keys of this thread's 32 that its row sees
      const int visible = min(T, p.causal ? qi + 1 : T) - k0;
      // Only the diagonal tile (causal) and the last one (keys beyond T) test their elements, in a loop of their own: tests in
      // the other tiles' loop cost branches and selects per pair.  Rows beyond T need none: dY is zero there, and so is dS.
      auto form_ds = [&](auto edge_tag) {
        constexpr bool EDGE = decltype(edge_tag)::value;
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float2 x = ffma2(make_float2(__uint_as_float(s[i]), __uint_as_float(s[i + 1])), sc2, nl2);
          const float2 g = ffma2(make_float2(__uint_as_float(dp[i]), __uint_as_float(dp[i + 1])), ps2, nd2);
          float e0 = fast_exp2(x.x), e1 = fast_exp2(x.y);
          if constexpr (MASKED) {
            if (((mw >> i) & 1u) == 0u) e0 = p_masked;
            if (((mw >> (i + 1)) & 1u) == 0u) e1 = p_masked;
          }
          const float2 d = ffma2(make_float2(e0, e1), g, zero2);
          float d0 = d.x, d1 = d.y;
          if constexpr (EDGE) {
            if (i >= visible) d0 = 0.f;
            if (i + 1 >= visible) d1 = 0.f;
          }
          if constexpr (SPLIT) split_pack(d0, d1, pk[i / 2], pk_lo[i / 2]);
          else pk[i / 2] = pack_bf16(d0, d1);
        }
      };
      if (edge) form_ds(std::true_type{});
      else form_ds(std::false_type{});
      if (j > 0) {  // the previous dQ product must have consumed the previous dS
        ok = __all_sync(0xffffffffu, mbar_wait(bar(DQ_DQ_DONE), (uint32_t)((j - 1) & 1), p.status, 131, j));
        if (!ok) break;
        tc_fence_after();
      }
      tmem_st16(t_row + C_DS + qtr * 16, pk);
      if constexpr (SPLIT) tmem_st16(t_row + C_DS + DS_LO + qtr * 16, pk_lo);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(DQ_DS_READY));
    }
    if (ok && n > 0) ok = __all_sync(0xffffffffu, mbar_wait(bar(DQ_DQ_DONE), (uint32_t)((n - 1) & 1), p.status, 132, n));
    constexpr int ESZ = SPLIT ? 4 : 2, PR = HD * ESZ / 16;
    uint8_t* tile = smem_gen + PL::OFF_RES0;           // the Q tile: every product has finished with it
    const bool fin = ok && n > 0;
    if (fin) {
      tc_fence_after();
      const float2 mul = split::pow2_factors(-DS_SHIFT_LOG2 - split::scale_exp(sc.y) - split::scale_exp(sc.z) - split::scale_exp(sc.w));
      stage_columns<PR, OC, SPLIT>(tile, row, qtr, t_row + C_DQ + qtr * OC, p.scale, mul);
    }
    ew_bar_sync<EW_WARPS>();
    if (fin)
      store_staged_rows<PR, ESZ, BLK / EW_WARPS>(tile, warp, lane, p.out0, (int64_t)bi * p.os.b + (int64_t)hi * p.os.h + (int64_t)q0 * p.os.t, p.os.t,
                                 min(BLK, T - q0));
  }
  tc_fence_before();
  __syncthreads();
  if (warp == WARP_MMA) { tc_fence_after(); tmem_dealloc(tmem_base, TMEM_COLS); }
  mca_pdl_wait();   // see the set-up: complete only after the kernels before it
}

// ---------------------------------------------------------------------------------------------
// dK/dV kernel.  TMEM columns: S^T [0,BN)  dP^T [BN,2 BN)  dV [2 BN,2 BN+HD)  dK [3 BN,3 BN+HD);
// P^T and dS^T (bf16, packed) overwrite the first 16 columns of each 32-column quarter of S^T / dP^T; in split
// mode their fp16 hi halves do, and the lo halves take the other 16 columns of the quarter.
// ---------------------------------------------------------------------------------------------
enum KvBar : int {
  KV_K_FULL = 0,
  KV_Q_FULL = 1,     // [K_STAGES, at most 4]  Q of a step (lives until the step's dK product: one stage deeper than dY)
  KV_Q_EMPTY = 5,
  KV_DO_FULL = 9,    // [V_STAGES, at most 3]  dY of a step (last used by the step's dV product)
  KV_DO_EMPTY = 12,
  KV_ST_FULL = 15,   // S^T written by the MMA
  KV_DPT_FULL = 16,  // dP^T written by the MMA
  KV_ACC_DONE = 17,  // the last dV / dK products finished
  KV_DRAIN = 18,
  KV_V_FULL = 19,
  KV_DV_DONE = 20,   // the last dV product finished
  // the element-wise warps arrive on these:
  KV_LD_READY = 21,  // the step's per-query log-sum-exp and delta are staged in shared memory
  KV_PT_READY = 22,  // P^T written to TMEM (over S^T)
  KV_DST_READY = 23, // dS^T written to TMEM (over dP^T)
  KV_PT_HALF = 24,   // the first sixteen queries of every quarter of P^T, and
  KV_DST_HALF = 25,  // of dS^T: their part of the product starts while the rest is formed
  KV_BAR_COUNT = 26
};

// DS (WIDE CTAs): the dS tiles are also left in p.ds for sdpa_bwd_dq_ds_tc_kernel, half a step's at a time from the registers of the
// element-wise warps.  They bound the kernel, so it costs 9 % (16 heads of 7001 x 128 333 -> 364 us).  Tried and slower: all of it behind
// the step's last hand-over (366; split 64-wide heads 111 -> 117), a bulk copy from shared memory that a stage of Q gives up (400), four
// warps of their own that read dS^T back from TMEM and keep the next dP^T waiting for it (418).
template <int HD, bool SPLIT, bool MASKED, bool NARROW, bool DS>
__global__ void __launch_bounds__((BwdPlan<SPLIT ? 128 : HD, NARROW>::THREADS), (BwdPlan<SPLIT ? 128 : HD, NARROW>::CTAS_PER_SM))
sdpa_bwd_dkdv_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                        const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                        const BwdParams p) {
  using PL = BwdPlan<SPLIT ? 128 : HD, NARROW>;
  constexpr int BN = PL::BN, EW_WARPS = PL::EW_WARPS, WARP_TMA = PL::WARP_TMA, WARP_MMA = PL::WARP_MMA;
  constexpr uint32_t TMEM_COLS = PL::TMEM_COLS;
  constexpr int FMT = SPLIT ? 0 : 1;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar0 = smem_base + PL::OFF_BAR;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + PL::OFF_BAR + KV_BAR_COUNT * 8);
  auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // launch order -> work item: longest causal work first inside groups of p.group heads (see the forward kernel)
  const int lin = (int)(blockIdx.y * gridDim.x + blockIdx.x);
  const int grp = lin / (p.group * (int)gridDim.x);
  const int in_grp = lin - grp * p.group * (int)gridDim.x;
  const int grp_heads = min(p.group, (int)gridDim.y - grp * p.group);
  const int rank = in_grp / grp_heads;
  const int bh = p.bh0 + grp * p.group + (in_grp - rank * grp_heads), T = p.T;
  const int bi = bh / p.H, hi = bh - bi * p.H;   // batch item and head
  const int kt = rank;                  // key tile; tile 0 has the most causal work and comes first
  const int k0 = kt * BLK;
  const int i_begin = p.causal ? k0 / BN : 0;
  const int n = (T + BN - 1) / BN - i_begin;    // query steps to walk

  static_assert(!DS || !NARROW);
  // the aligned plan must fit in what was requested (it does unless the dynamic base is unusually placed)
  uint32_t dyn_bytes;
  asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_bytes));
  if (smem_base + PL::NEED_KV > smem_u32(smem_raw) + dyn_bytes) {
    if (tid == 0 && atomicCAS(p.status, 0, 2) == 0) { p.status[1] = 299; p.status[2] = (int)(smem_base - smem_u32(smem_raw)); raise_failure(); }
    return;
  }
  volatile int* s_abort = reinterpret_cast<volatile int*>(smem_gen + PL::OFF_FLAG_KV);
  if (tid == 32) *s_abort = *reinterpret_cast<volatile int*>(p.status);
  if (warp == WARP_TMA && lane == 0) {
    prefetch_tensormap(&map_q); prefetch_tensormap(&map_k); prefetch_tensormap(&map_v); prefetch_tensormap(&map_do);
  }
  if (tid == 0) {
    for (int i = 0; i < KV_BAR_COUNT; ++i) mbar_init(bar(i), i >= KV_LD_READY ? (uint32_t)EW_WARPS : 1u);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == WARP_MMA) { tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  mca_pdl_wait();   // launched ahead of the kernels before it: from here on their results are complete and visible
  mca_pdl_launch_dependents();   // only now: the dQ kernel behind this one starts without a wait of its own
  if (*s_abort != 0) {   // an earlier CTA already failed: leave (uniform decision) before any copy or product is issued
    if (warp == WARP_MMA) tmem_dealloc(tmem_base, TMEM_COLS);
    return;
  }
  constexpr uint32_t C_ST = 0, C_DPT = BN, C_DV = 2 * BN, C_DK = 3 * BN;
  static_assert(HD <= BN);
  bool ok = true;

  if (warp == WARP_TMA) {
    if (lane == 0) {
      // one resident tile; S^T(0) waits for K and Q(0) only, so those come first
      auto load_resident = [&](uint32_t dst, const CUtensorMap* map, int full) {
        mbar_expect_tx(bar(full), PL::TILE_BYTES);
#pragma unroll
        for (int s = 0; s < PL::SUB; ++s)
#pragma unroll
          for (int r = 0; r < BLK; r += BN)
            tma_load_4d(smem_base + dst + s * PL::SUB_BYTES + r * 128, map, bar(full), s * 64, k0 + r, hi, bi);
      };
      load_resident(PL::OFF_RES0, &map_k, KV_K_FULL);
      int issued = 0, issued_do = 0;
      for (int it = 0; it < n && ok; ++it) {
        const int qs = it % PL::K_STAGES, ds = it % PL::V_STAGES;
        const uint32_t qph = (uint32_t)((it / PL::K_STAGES) & 1), dph = (uint32_t)((it / PL::V_STAGES) & 1);
        const uint32_t q_dst = smem_base + PL::OFF_KRING + qs * PL::RING_TILE_BYTES, do_dst = smem_base + PL::OFF_VRING + ds * PL::RING_TILE_BYTES;
        ok = mbar_wait(bar(KV_Q_EMPTY + qs), qph ^ 1u, p.status, 210, it);
        if (!ok) break;
        mbar_expect_tx(bar(KV_Q_FULL + qs), PL::RING_TILE_BYTES);
#pragma unroll
        for (int s = 0; s < PL::SUB; ++s)
          tma_load_4d(q_dst + s * PL::RING_SUB_BYTES, &map_q, bar(KV_Q_FULL + qs), s * 64, (i_begin + it) * BN, hi, bi);
        issued = it + 1;
        if (it == 0) load_resident(PL::OFF_RES1, &map_v, KV_V_FULL);
        ok = mbar_wait(bar(KV_DO_EMPTY + ds), dph ^ 1u, p.status, 211, it);
        if (!ok) break;
        mbar_expect_tx(bar(KV_DO_FULL + ds), PL::RING_TILE_BYTES);
#pragma unroll
        for (int s = 0; s < PL::SUB; ++s)
          tma_load_4d(do_dst + s * PL::RING_SUB_BYTES, &map_do, bar(KV_DO_FULL + ds), s * 64, (i_begin + it) * BN, hi, bi);
        issued_do = it + 1;
      }
      if (!ok) {
        mbar_wait(bar(KV_K_FULL), 0, p.status, 212, 0);
        if (issued > 0) mbar_wait(bar(KV_V_FULL), 0, p.status, 215, 0);
        for (int it = max(0, issued - PL::K_STAGES); it < issued; ++it)
          mbar_wait(bar(KV_Q_FULL + it % PL::K_STAGES), (uint32_t)((it / PL::K_STAGES) & 1), p.status, 213, it);
        for (int it = max(0, issued_do - PL::V_STAGES); it < issued_do; ++it)
          mbar_wait(bar(KV_DO_FULL + it % PL::V_STAGES), (uint32_t)((it / PL::V_STAGES) & 1), p.status, 214, it);
      }
    }
  } else if (warp == WARP_MMA) {
    // The warp runs this role in lock step and one elected lane issues, so that addresses and
    // descriptors are warp-uniform values (fewer instructions per tcgen05.mma for the issuing thread).
    {
      const uint32_t leader = elect_one() ? 1u : 0u;
      const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
      constexpr uint32_t IDESC_NT = make_idesc_fmt(BLK, BN, 0, 0, FMT);
      constexpr uint32_t IDESC_ACC = make_idesc_fmt(BLK, HD, 0, 1, FMT);
      const uint32_t k_addr = smem_base + PL::OFF_RES0, v_addr = smem_base + PL::OFF_RES1;
      auto issue_nt = [&](uint32_t d_col, uint32_t a_addr, uint32_t b_addr) {
        if constexpr (SPLIT) {
#pragma unroll
          for (int term = 0; term < 3; ++term) {
            const uint32_t oa = term == 2 ? PL::SUB_BYTES : 0u, ob = term == 1 ? PL::RING_SUB_BYTES : 0u;
#pragma unroll
            for (int kk = 0; kk < HD / 16; ++kk)
              umma_ss_if<false>(leader, tmem_u + d_col, make_desc(a_addr + oa + kk * 32, 16, 1024), make_desc(b_addr + ob + kk * 32, 16, 1024),
                                IDESC_NT, (term > 0 || kk > 0) ? 1u : 0u);
          }
        } else {
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk) {
            umma_ss_if<false>(leader, tmem_u + d_col, make_desc(a_addr + (kk / 4) * PL::SUB_BYTES + (kk % 4) * 32, 16, 1024),
                              make_desc(b_addr + (kk / 4) * PL::RING_SUB_BYTES + (kk % 4) * 32, 16, 1024), IDESC_NT, kk > 0);
          }
        }
      };
      // acc += A^T-from-TMEM x B with B a BN x HD tile read MN-major; split mode: hi.hi + hi.lo + lo.hi
      auto issue_acc = [&](uint32_t d_col, uint32_t a_col, uint32_t b_addr, bool first_step, int half) {   // half: the even or the odd sixteens
#pragma unroll
        for (int k2 = 0; k2 < BN / 32; ++k2) {
          const int kk = 2 * k2 + half;
          const uint32_t a_hi = tmem_u + a_col + (kk / 2) * 32 + (kk % 2) * 8;
          umma_ts_if<false>(leader, tmem_u + d_col, a_hi, make_desc(b_addr + kk * 2048, PL::RING_SUB_BYTES, 1024), IDESC_ACC,
                            (!first_step || kk > 0) ? 1u : 0u);
          if constexpr (SPLIT) {
            umma_ts_if<false>(leader, tmem_u + d_col, a_hi, make_desc(b_addr + PL::RING_SUB_BYTES + kk * 2048, PL::RING_SUB_BYTES, 1024), IDESC_ACC, 1u);
            umma_ts_if<false>(leader, tmem_u + d_col, a_hi + 16, make_desc(b_addr + kk * 2048, PL::RING_SUB_BYTES, 1024), IDESC_ACC, 1u);
          }
        }
      };
      // S^T = K Q^T and dP^T = V dY^T (rows = keys, columns = queries); P^T overwrites S^T and dS^T overwrites
      // dP^T.  The two halves of a step are interleaved with the next step's first products,
      //   dV(it), S^T(it+1), dK(it), dP^T(it+1),
      // (the in-order pipe keeps every product behind the one that still reads the columns it overwrites),
      // so the element-wise warps work on P^T(it+1) while dK(it) and dP^T(it+1) run.
      auto q_stage = [&](int it) { return smem_base + PL::OFF_KRING + (it % PL::K_STAGES) * PL::RING_TILE_BYTES; };
      auto do_stage = [&](int it) { return smem_base + PL::OFF_VRING + (it % PL::V_STAGES) * PL::RING_TILE_BYTES; };
      auto wait_q = [&](int it) {
        return __all_sync(0xffffffffu, mbar_wait(bar(KV_Q_FULL + it % PL::K_STAGES), (uint32_t)((it / PL::K_STAGES) & 1), p.status, 221, it));
      };
      auto wait_do = [&](int it) {
        return __all_sync(0xffffffffu, mbar_wait(bar(KV_DO_FULL + it % PL::V_STAGES), (uint32_t)((it / PL::V_STAGES) & 1), p.status, 224, it));
      };
      auto issue_st = [&](int it) {
        issue_nt(C_ST, k_addr, q_stage(it));
        umma_commit_if(leader, bar(KV_ST_FULL));
      };
      auto issue_dpt = [&](int it) {
        issue_nt(C_DPT, v_addr, do_stage(it));
        umma_commit_if(leader, bar(KV_DPT_FULL));
      };
      ok = __all_sync(0xffffffffu, mbar_wait(bar(KV_K_FULL), 0, p.status, 220, 0));
      if (ok && n > 0) {
        ok = wait_q(0);
        if (ok) {
          tc_fence_after();
          issue_st(0);
          ok = __all_sync(0xffffffffu, mbar_wait(bar(KV_V_FULL), 0, p.status, 228, 0));
        }
        if (ok) ok = wait_do(0);
        if (ok) {
          tc_fence_after();
          issue_dpt(0);
        }
      }
      for (int it = 0; it < n && ok; ++it) {
        const uint32_t q_addr = q_stage(it), do_addr = do_stage(it);
        // dV += P^T dY: A from TMEM (16 queries = 8 packed columns per step), B MN-major
        ok = __all_sync(0xffffffffu, mbar_wait(bar(KV_PT_HALF), (uint32_t)(it & 1), p.status, 225, it));
        if (!ok) break;
        tc_fence_after();
        issue_acc(C_DV, C_ST, do_addr, it == 0, 0);
        if (it + 1 < n && !(ok = wait_q(it + 1))) break;   // long there: waited for here, off the way from P^T to S^T
        ok = __all_sync(0xffffffffu, mbar_wait(bar(KV_PT_READY), (uint32_t)(it & 1), p.status, 222, it));
        if (!ok) break;
        tc_fence_after();
        issue_acc(C_DV, C_ST, do_addr, it == 0, 1);
        if (it + 1 < n) issue_st(it + 1);
        else umma_commit_if(leader, bar(KV_DV_DONE));
        umma_commit_if(leader, bar(KV_DO_EMPTY + it % PL::V_STAGES));   // dY(it) was last read by dV
        // dK += dS^T Q
        ok = __all_sync(0xffffffffu, mbar_wait(bar(KV_DST_HALF), (uint32_t)(it & 1), p.status, 226, it));
        if (!ok) break;
        tc_fence_after();
        issue_acc(C_DK, C_DPT, q_addr, it == 0, 0);
        if (it + 1 < n && !(ok = wait_do(it + 1))) break;
        ok = __all_sync(0xffffffffu, mbar_wait(bar(KV_DST_READY), (uint32_t)(it & 1), p.status, 223, it));
        if (!ok) break;
        tc_fence_after();
        issue_acc(C_DK, C_DPT, q_addr, it == 0, 1);
        if (it + 1 < n) issue_dpt(it + 1);
        else umma_commit_if(leader, bar(KV_ACC_DONE));
        umma_commit_if(leader, bar(KV_Q_EMPTY + it % PL::K_STAGES));
      }
      umma_commit_if(leader, bar(KV_DRAIN));
      mbar_wait(bar(KV_DRAIN), 0, p.status, 227, 0);
    }
  } else {
    // ------------------------------------------------------------------ element-wise warps
    const int qtr = warp >> 2, lane_base = (warp & 3) * 32, row = lane_base + lane;
    const int kj = k0 + row;               // this thread's key
    constexpr int OC = HD / (EW_WARPS / 4);
    const uint32_t t_row = tmem_base + ((uint32_t)lane_base << 16);
    // The query-dependent terms (minus log-sum-exp, minus delta x scale) are the same for every key row: the first 2 BN
    // element-wise threads fetch one value each a step ahead and stage them in shared memory, so that the
    // inner loop reads them as broadcasts instead of 64 global loads per thread.  Rows beyond T get
    // lse = +inf, which makes their probabilities exactly zero.
    float (*s_nlse)[BN] = reinterpret_cast<float (*)[BN]>(smem_gen + PL::OFF_STAGE_KV);
    float (*s_del)[BN] = s_nlse + 2;
    // split mode: S^T and dP^T carry the pre-pass's scales; dS^T is kept in the units of dP' x 2^-19 and P^T 2^10 larger
    float4 sc = make_float4(1.f, 1.f, 1.f, 1.f);
    if constexpr (SPLIT) sc = mca_ld_f4(reinterpret_cast<const float*>(p.scales + bh));
    const float sl2 = SPLIT ? split::logit_scale(p.scale_log2, sc) : p.scale_log2;
    const float dmul = SPLIT ? DS_SHIFT : p.scale;
    const float del_mul = SPLIT ? sc.z : p.scale;
    auto fetch = [&](int it) -> float {
      const int qi = (i_begin + it) * BN + (tid & (BN - 1));
      if (tid >= 2 * BN || it >= n || qi >= T) return tid < BN ? -INFINITY : 0.f;
      return tid < BN ? -mca_ld_f1(p.lse + (int64_t)bh * T + qi) : -mca_ld_f1(p.delta + (int64_t)bh * T + qi) * del_mul;
    };
    auto stage = [&](int it, float v) {
      if (tid < BN) s_nlse[it & 1][tid] = v;
      else if (tid < 2 * BN) s_del[it & 1][tid - BN] = v;
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(KV_LD_READY));
    };
    // DS: where this thread's key and its quarter's queries of the first query tile are
    constexpr int SUBS = SPLIT ? 2 : 1;
    uint8_t* d = nullptr;
    if constexpr (DS)
      d = p.ds + ds_tile_offset<SPLIT>(bh - p.bh0, i_begin, kt, T, p.causal) + (warp & 3) * SUBS * DS_BLOCK_BYTES + qtr * 4 * DS_GROUP_BYTES + lane * 16;
    if (n > 0) stage(0, fetch(0));
    for (int it = 0; it < n && ok; ++it) {
      const int q_local = qtr * 32;                         // first of this thread's 32 queries within the tile
      const int q_base = (i_begin + it) * BN + q_local;
      const float next = fetch(it + 1);                     // in flight while this step is processed
      ok = __all_sync(0xffffffffu, mbar_wait(bar(KV_LD_READY), (uint32_t)(it & 1), p.status, 231, it));
      if (!ok) break;
      ok = __all_sync(0xffffffffu, mbar_wait(bar(KV_ST_FULL), (uint32_t)(it & 1), p.status, 230, it));
      if (!ok) break;
      tc_fence_after();
      const float* nlse_s = s_nlse[it & 1] + q_local;
      const float* del_s = s_del[it & 1] + q_local;
      const bool diag = p.causal && (i_begin + it) * BN < k0 + BLK;   // only the diagonal tile needs the causal test
      uint32_t mw = 0xffffffffu;          // keep-bits of this thread's key against its 32 queries of the step
      if constexpr (MASKED) {
        if (p.mask_bits_t != nullptr)
          mw = __ldg(p.mask_bits_t + (int64_t)min(kj, T - 1) * p.mask_row_stride + (BN / 32) * (i_begin + it) + qtr);
        else
          mw = ((__ldg(p.mask_bits + (int64_t)bi * p.mask_batch_stride + (min(kj, T - 1) >> 5)) >> (kj & 31)) & 1u) ? 0xffffffffu : 0u;
      }
      // pass 1: P^T = 2^(S^T scale - lse), kept in fp32 for pass 2, packed to bf16 over S^T (fp32 pairs)
      const float2 sc2 = make_float2(sl2, sl2), ps2 = make_float2(dmul, dmul);
      const float2 zero2 = make_float2(0.f, 0.f);
      uint32_t s[32], pk[16];
      uint32_t pk_lo[SPLIT ? 16 : 1];
      tmem_ld32(t_row + C_ST + qtr * 32, s);
      tmem_wait_ld();
      // The causal test is the diagonal tile's alone (a loop of its own, as in the dQ kernel).  A key beyond T needs none: its
      // row of P^T and dS^T reaches only its own rows of dV and dK, which are not stored.
      auto form_p = [&](auto diag_tag, const int lo, const int hi) {
        constexpr bool DIAG = decltype(diag_tag)::value;
        const int first = kj - q_base;      // queries before the key do not see it
#pragma unroll
        for (int i = lo; i < hi; i += 4) {
          const float4 nl = *reinterpret_cast<const float4*>(nlse_s + i);
          const float nls[4] = {nl.x, nl.y, nl.z, nl.w};
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            const float2 x = ffma2(make_float2(__uint_as_float(s[i + e]), __uint_as_float(s[i + e + 1])), sc2,
                                   make_float2(nls[e], nls[e + 1]));
            float v0 = fast_exp2(x.x), v1 = fast_exp2(x.y);
            if constexpr (MASKED) {
              // a masked entry: 0, or 1 / T in a fully masked row (staged -lse = -inf; rows beyond T are staged the same
              // way and stay 0)
              if (((mw >> (i + e)) & 1u) == 0u) v0 = (nls[e] == -INFINITY && q_base + i + e < T) ? p.inv_T : 0.f;
              if (((mw >> (i + e + 1)) & 1u) == 0u) v1 = (nls[e + 1] == -INFINITY && q_base + i + e + 1 < T) ? p.inv_T : 0.f;
            }
            if constexpr (DIAG) {
              if (first > i + e) v0 = 0.f;
              if (first > i + e + 1) v1 = 0.f;
            }
            s[i + e] = __float_as_uint(v0);
            s[i + e + 1] = __float_as_uint(v1);
          }
          if constexpr (SPLIT) {
            split_pack(__uint_as_float(s[i]) * PT_SHIFT, __uint_as_float(s[i + 1]) * PT_SHIFT, pk[i / 2], pk_lo[i / 2]);
            split_pack(__uint_as_float(s[i + 2]) * PT_SHIFT, __uint_as_float(s[i + 3]) * PT_SHIFT, pk[i / 2 + 1], pk_lo[i / 2 + 1]);
          } else {
            pk[i / 2] = pack_bf16(__uint_as_float(s[i]), __uint_as_float(s[i + 1]));
            pk[i / 2 + 1] = pack_bf16(__uint_as_float(s[i + 2]), __uint_as_float(s[i + 3]));
          }
        }
      };
      // sixteen of the 32 queries are stored and handed over while the others are formed
      auto store_half = [&](uint32_t col, int half) {
        tmem_st8(t_row + col + qtr * 32 + half * 8, pk + half * 8);
        if constexpr (SPLIT) tmem_st8(t_row + col + qtr * 32 + 16 + half * 8, pk_lo + half * 8);
      };
      auto hand_over = [&](int b) {
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(b));
      };
      auto pass1 = [&](auto diag_tag) {
        form_p(diag_tag, 0, 16);
        store_half(C_ST, 0);
        form_p(diag_tag, 16, 24);
        hand_over(KV_PT_HALF);
        form_p(diag_tag, 24, 32);
        store_half(C_ST, 1);
        hand_over(KV_PT_READY);
      };
      if (diag) pass1(std::true_type{});
      else pass1(std::false_type{});
      // pass 2: dS^T = P^T o (dP^T - delta) scale, packed to bf16 over dP^T
      ok = __all_sync(0xffffffffu, mbar_wait(bar(KV_DPT_FULL), (uint32_t)(it & 1), p.status, 233, it));
      if (!ok) break;
      tc_fence_after();
      uint32_t dp[32];
      tmem_ld32(t_row + C_DPT + qtr * 32, dp);
      tmem_wait_ld();
      auto form_ds = [&](const int lo, const int hi) {
#pragma unroll
        for (int i = lo; i < hi; i += 4) {
          const float4 de = *reinterpret_cast<const float4*>(del_s + i);
          const float des[4] = {de.x, de.y, de.z, de.w};
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            // (dP - delta) scale as one fused pair operation, then times P
            const float2 g = ffma2(make_float2(__uint_as_float(dp[i + e]), __uint_as_float(dp[i + e + 1])), ps2,
                                   make_float2(des[e], des[e + 1]));
            const float2 d = ffma2(make_float2(__uint_as_float(s[i + e]), __uint_as_float(s[i + e + 1])), g, zero2);
            if constexpr (SPLIT) split_pack(d.x, d.y, pk[(i + e) / 2], pk_lo[(i + e) / 2]);
            else pk[(i + e) / 2] = pack_bf16(d.x, d.y);
          }
        }
      };
      // the same registers once more, to memory.  In the diagonal tile the pairs that the causal mask hides, and everywhere the keys beyond
      // T, are zeros there whatever dP is: dQ is a sum over them, dK's rows are not.
      auto pass_on = [&](int half) {
        if constexpr (DS) {
          if (diag || k0 + BLK > T) {
            const int hidden = kj >= T ? 32 : diag ? kj - q_base : 0;   // of this thread's queries
#pragma unroll
            for (int i = 8 * half; i < 8 * half + 8; ++i) {
              const uint32_t keep = (2 * i < hidden ? 0u : 0x0000ffffu) | (2 * i + 1 < hidden ? 0u : 0xffff0000u);
              pk[i] &= keep;
              if constexpr (SPLIT) pk_lo[i] &= keep;
            }
          }
#pragma unroll
          for (int g = 2 * half; g < 2 * half + 2; ++g) {
            *reinterpret_cast<uint4*>(d + g * DS_GROUP_BYTES) = make_uint4(pk[4 * g], pk[4 * g + 1], pk[4 * g + 2], pk[4 * g + 3]);
            if constexpr (SPLIT)
              *reinterpret_cast<uint4*>(d + DS_BLOCK_BYTES + g * DS_GROUP_BYTES) = make_uint4(pk_lo[4 * g], pk_lo[4 * g + 1], pk_lo[4 * g + 2], pk_lo[4 * g + 3]);
          }
        }
      };
      form_ds(0, 16);
      store_half(C_DPT, 0);
      form_ds(16, 24);
      hand_over(KV_DST_HALF);
      pass_on(0);
      form_ds(24, 32);
      store_half(C_DPT, 1);
      if (it + 1 < n) stage(it + 1, next);
      hand_over(KV_DST_READY);
      pass_on(1);
      if constexpr (DS) d += (int64_t)(p.causal ? i_begin + it + 1 : (int)gridDim.x) * (4 * SUBS * DS_BLOCK_BYTES);   // the next query tile's
    }
    if (ok && n > 0) ok = __all_sync(0xffffffffu, mbar_wait(bar(KV_DV_DONE), 0, p.status, 234, n));
    constexpr int ESZ = SPLIT ? 4 : 2, PR = HD * ESZ / 16;
    uint8_t* tile_k = smem_gen + PL::OFF_RES0;         // the K and V tiles: every product has finished with them
    uint8_t* tile_v = smem_gen + PL::OFF_RES1;
    if (ok && n > 0) {   // dV beside the last dK product
      tc_fence_after();
      const float2 mul_v = split::pow2_factors(-PT_SHIFT_LOG2 - split::scale_exp(sc.w));
      stage_columns<PR, OC, SPLIT>(tile_v, row, qtr, t_row + C_DV + qtr * OC, 1.0f, mul_v);
      ok = __all_sync(0xffffffffu, mbar_wait(bar(KV_ACC_DONE), 0, p.status, 232, n));
    }
    const bool fin = ok && n > 0;
    if (fin) {
      tc_fence_after();
      const float2 mul_k = split::pow2_factors(-DS_SHIFT_LOG2 - split::scale_exp(sc.x) - split::scale_exp(sc.z) - split::scale_exp(sc.w));
      stage_columns<PR, OC, SPLIT>(tile_k, row, qtr, t_row + C_DK + qtr * OC, p.scale, mul_k);
    }
    ew_bar_sync<EW_WARPS>();
    if (fin) {
      const int64_t off0 = (int64_t)bi * p.os.b + (int64_t)hi * p.os.h + (int64_t)k0 * p.os.t;
      store_staged_rows<PR, ESZ, BLK / EW_WARPS>(tile_k, warp, lane, p.out0, off0, p.os.t, min(BLK, T - k0));
      store_staged_rows<PR, ESZ, BLK / EW_WARPS>(tile_v, warp, lane, p.out1, off0, p.os.t, min(BLK, T - k0));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == WARP_MMA) { tc_fence_after(); tmem_dealloc(tmem_base, TMEM_COLS); }
}

// ---------------------------------------------------------------------------------------------
// dQ from the dS the dK/dV kernel left: dQ = dS K, one product instead of three.  A CTA accumulates QT query tiles of one head in
// TMEM (columns [0, QT HD)) and streams steps of 64 keys: the halves of their dS tiles by bulk copies, the K rows by TMA.
// Bound by the bytes of dS (HBM, or L2 where it is still there), so the ring is as deep as it fits: QT = 2 for 128-wide heads,
// whose K rows are as many bytes as a dS half and are read once for both; QT = 1 and two CTAs per SM for the others, whose items are
// short: one's first loads and last stores run beside the other's steps.
// ---------------------------------------------------------------------------------------------
template <int HD, bool SPLIT> struct DqDsPlan {
  static constexpr int QT = HD == 128 ? 2 : 1, BN = 64, EW_WARPS = 8, WARP_TMA = 8, WARP_MMA = 9, THREADS = 320;
  static constexpr int CTAS_PER_SM = QT == 2 ? 1 : 2;
  static constexpr int SUB = SPLIT ? 2 : HD / 64;
  static constexpr uint32_t SUB_BYTES = BN * 128, K_BYTES = SUB * SUB_BYTES;
  static constexpr uint32_t HALF_BYTES = (SPLIT ? 4 : 2) * DS_BLOCK_BYTES;   // one query tile's dS of a step
  static constexpr uint32_t STAGE_BYTES = QT * HALF_BYTES + K_BYTES;
  static constexpr int STAGES = QT == 2 ? 4 : (SPLIT ? 2 : 4);
  static constexpr uint32_t OFF_BAR = STAGES * STAGE_BYTES, BYTES = OFF_BAR + 128 + 1024;
  static constexpr uint32_t TMEM_COLS = QT * HD < 32 ? 32 : QT * HD;
  static_assert(STAGES * STAGE_BYTES >= (uint32_t)(QT * BLK * HD * (SPLIT ? 4 : 2)), "the finished tiles are staged in the ring");
  static_assert(CTAS_PER_SM * (BYTES + 1024 + 64) <= 228 * 1024, "shared memory of the CTAs of one SM");
};

template <int HD, bool SPLIT>
__global__ void __launch_bounds__((DqDsPlan<HD, SPLIT>::THREADS), (DqDsPlan<HD, SPLIT>::CTAS_PER_SM))
sdpa_bwd_dq_ds_tc_kernel(const __grid_constant__ CUtensorMap map_k, const BwdParams p) {
  using PL = DqDsPlan<HD, SPLIT>;
  constexpr int QT = PL::QT, BN = PL::BN, EW_WARPS = PL::EW_WARPS, STAGES = PL::STAGES;
  constexpr int FMT = SPLIT ? 0 : 1;
  constexpr int FULL = 0, EMPTY = STAGES, DONE = 2 * STAGES, BAR_COUNT = 2 * STAGES + 1;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  auto bar = [&](int i) { return smem_base + PL::OFF_BAR + 8u * (uint32_t)i; };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + PL::OFF_BAR + BAR_COUNT * 8);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, T = p.T;
  // longest causal work first; the heads the dK/dV kernel wrote last, whose dS is still in L2, come first
  const int heads = (int)gridDim.y, lin = (int)(blockIdx.y * gridDim.x + blockIdx.x);
  const int n_groups = (heads + p.group - 1) / p.group, last = heads - (n_groups - 1) * p.group;   // heads of the last group
  int grp, in_grp, grp_heads;
  if (lin < last * (int)gridDim.x) { grp = n_groups - 1; in_grp = lin; grp_heads = last; }
  else {
    const int rest = lin - last * (int)gridDim.x, back = rest / (p.group * (int)gridDim.x);
    grp = n_groups - 2 - back; in_grp = rest - back * p.group * (int)gridDim.x; grp_heads = p.group;
  }
  const int rank = in_grp / grp_heads;
  const int head = grp * p.group + (in_grp - rank * grp_heads), bh = p.bh0 + head;
  const int bi = bh / p.H, hi = bh - bi * p.H;
  const int qt0 = ((int)gridDim.x - 1 - rank) * QT;
  const int steps_T = (T + BN - 1) / BN, nt = (T + BLK - 1) / BLK;
  // key steps that query tile qt0 + t sees
  auto steps_of = [&](int t) { return qt0 + t >= nt ? 0 : p.causal ? min(2 * (qt0 + t + 1), steps_T) : steps_T; };
  const int n0 = steps_of(0), n1 = QT == 2 ? steps_of(1) : 0, n = max(n0, n1);

  __shared__ int s_abort;
  mca_pdl_launch_dependents();
  if (warp == PL::WARP_TMA && lane == 0) prefetch_tensormap(&map_k);
  if (tid == 0) {
    for (int i = 0; i < BAR_COUNT; ++i) mbar_init(bar(i), 1u);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == PL::WARP_MMA) { tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), PL::TMEM_COLS); tmem_relinquish(); }
  mca_pdl_wait();   // dS is the kernel before's
  if (tid == 32) s_abort = *reinterpret_cast<volatile int*>(p.status);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (s_abort != 0) {   // uniform, before any copy or product is issued
    if (warp == PL::WARP_MMA) tmem_dealloc(tmem_base, PL::TMEM_COLS);
    return;
  }
  bool ok = true;
  if (warp == PL::WARP_TMA) {
    if (lane == 0) {
      int issued = 0;
      for (int j = 0; j < n; ++j) {
        const int s = j % STAGES;
        ok = mbar_wait(bar(EMPTY + s), (uint32_t)((j / STAGES) & 1) ^ 1u, p.status, 310, j);
        if (!ok) break;
        const uint32_t dst = smem_base + s * PL::STAGE_BYTES, full = bar(FULL + s);
        const int tiles = (j < n0 ? 1 : 0) + (j < n1 ? 1 : 0);
        mbar_expect_tx(full, PL::K_BYTES + tiles * PL::HALF_BYTES);
#pragma unroll
        for (int t = 0; t < QT; ++t)
          if (j < (t == 0 ? n0 : n1)) {
            const uint8_t* src = p.ds + ds_tile_offset<SPLIT>(head, qt0 + t, j >> 1, T, p.causal) + (j & 1) * PL::HALF_BYTES;
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             dst + t * PL::HALF_BYTES),
                         "l"(src), "r"(PL::HALF_BYTES), "r"(full)
                         : "memory");
          }
#pragma unroll
        for (int b = 0; b < PL::SUB; ++b)
          tma_load_4d(dst + QT * PL::HALF_BYTES + b * PL::SUB_BYTES, &map_k, full, b * 64, j * BN, hi, bi);
        issued = j + 1;
      }
      if (!ok)  // let copies in flight land (bounded) before the CTA's memory is released
        for (int j = max(0, issued - STAGES); j < issued; ++j)
          mbar_wait(bar(FULL + j % STAGES), (uint32_t)((j / STAGES) & 1), p.status, 311, j);
    }
  } else if (warp == PL::WARP_MMA) {
    const uint32_t leader = elect_one() ? 1u : 0u;
    const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
    constexpr uint32_t IDESC = make_idesc_fmt(BLK, HD, 1, 1, FMT);   // both operands MN-major
    for (int j = 0; j < n && ok; ++j) {
      const int s = j % STAGES;
      ok = __all_sync(0xffffffffu, mbar_wait(bar(FULL + s), (uint32_t)((j / STAGES) & 1), p.status, 320, j));
      if (!ok) break;
      tc_fence_after();
      const uint32_t a_addr = smem_base + s * PL::STAGE_BYTES, k_addr = a_addr + QT * PL::HALF_BYTES;
#pragma unroll
      for (int t = 0; t < QT; ++t)
        if (j < (t == 0 ? n0 : n1)) {
#pragma unroll
          for (int kk = 0; kk < BN / 16; ++kk) {
            const uint32_t a = a_addr + t * PL::HALF_BYTES + (kk / 2) * (PL::HALF_BYTES / 2) + (kk % 2) * 256;
            const uint64_t a_hi = make_desc_plain(a, 128, DS_GROUP_BYTES);
            const uint64_t b_hi = make_desc(k_addr + kk * 2048, PL::SUB_BYTES, 1024);
            umma_ss_if<false>(leader, tmem_u + t * HD, a_hi, b_hi, IDESC, (j > 0 || kk > 0) ? 1u : 0u);
            if constexpr (SPLIT) {   // + dS_hi K_lo + dS_lo K_hi
              umma_ss_if<false>(leader, tmem_u + t * HD, a_hi, make_desc(k_addr + PL::SUB_BYTES + kk * 2048, PL::SUB_BYTES, 1024), IDESC, 1u);
              umma_ss_if<false>(leader, tmem_u + t * HD, make_desc_plain(a + DS_BLOCK_BYTES, 128, DS_GROUP_BYTES), b_hi, IDESC, 1u);
            }
          }
        }
      umma_commit_if(leader, bar(EMPTY + s));
    }
    umma_commit_if(leader, bar(DONE));
    mbar_wait(bar(DONE), 0, p.status, 321, 0);
  } else {
    // eight warps: with QT = 2 four a tile, a thread a whole row; with QT = 1 a thread half a row
    const int t = QT == 2 ? warp >> 2 : 0, half = QT == 2 ? 0 : warp >> 2, lane_base = (warp & 3) * 32, row = lane_base + lane;
    constexpr int OC = QT == 2 ? HD : HD / 2, ESZ = SPLIT ? 4 : 2, PR = HD * ESZ / 16;
    const int q0 = (qt0 + t) * BLK;
    uint8_t* tile = smem_gen + t * (BLK * HD * ESZ);
    ok = __all_sync(0xffffffffu, mbar_wait(bar(DONE), 0, p.status, 330, n));
    ok = ok && *reinterpret_cast<volatile int*>(p.status) == 0;
    const bool fin = __all_sync(0xffffffffu, ok) && q0 < T;
    if (fin) {
      tc_fence_after();
      float4 sc = make_float4(1.f, 1.f, 1.f, 1.f);
      if constexpr (SPLIT) sc = mca_ld_f4(reinterpret_cast<const float*>(p.scales + bh));
      const float2 mul = split::pow2_factors(-DS_SHIFT_LOG2 - split::scale_exp(sc.y) - split::scale_exp(sc.z) - split::scale_exp(sc.w));
      stage_columns<PR, OC, SPLIT>(tile, row, half, tmem_base + ((uint32_t)lane_base << 16) + t * HD + half * OC, p.scale, mul);
    }
    ew_bar_sync<EW_WARPS>();
    if (fin) {
      constexpr int RPW = BLK * QT / EW_WARPS;
      store_staged_rows<PR, ESZ, RPW>(tile, QT == 2 ? (warp & 3) : warp, lane, p.out0, (int64_t)bi * p.os.b + (int64_t)hi * p.os.h + (int64_t)q0 * p.os.t,
                                      p.os.t, min(BLK, T - q0));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == PL::WARP_MMA) { tc_fence_after(); tmem_dealloc(tmem_base, PL::TMEM_COLS); }
}

// delta[row] = sum_c dY[row][c] * Y[row][c]  (bf16 inputs, fp32 result).  D / 8 lanes share a row (16-byte loads), so a
// warp covers 256 / D rows; a CTA takes DELTA_STEPS of those per warp.  The kernel stands between the forward's tail and the
// dK/dV kernel, so dY (which the forward does not write) is asked for into L2 before the wait, and all of a thread's loads
// are in flight together behind it: T = 7001, 16 heads x 128: 18 us behind the forward -> 15.
constexpr int DELTA_STEPS = 4;
__global__ void __launch_bounds__(256) bwd_delta_bf16_kernel(const __nv_bfloat16* dy, const __nv_bfloat16* y, int64_t rows, int H, int T,
                                                             int D, const McaStrides ys, float* __restrict__ delta, int late) {
  if (!late) mca_pdl_launch_dependents();
  const int lane = threadIdx.x & 31, g = D / 8, rpw = 32 / g;        // g in {8, 16}
  const int64_t row0 = ((int64_t)blockIdx.x * (256 / 32) + (threadIdx.x >> 5)) * rpw * DELTA_STEPS + lane / g;
  int64_t off[DELTA_STEPS];
#pragma unroll
  for (int i = 0; i < DELTA_STEPS; ++i) {
    const int64_t row = min(row0 + i * rpw, rows - 1);
    const unsigned bh = (unsigned)(row / T), bi = bh / (unsigned)H;
    off[i] = (int64_t)bi * ys.b + (int64_t)(bh - bi * H) * ys.h + (row - (int64_t)bh * T) * ys.t + (lane % g) * 8;
    asm volatile("prefetch.global.L2 [%0];" ::"l"(dy + off[i]));
  }
  mca_pdl_wait();   // dy and y are earlier kernels' output
  if (late) mca_pdl_launch_dependents();
  float4 a[DELTA_STEPS], b[DELTA_STEPS];
#pragma unroll
  for (int i = 0; i < DELTA_STEPS; ++i) {
    a[i] = mca_ld_f4(reinterpret_cast<const float*>(dy + off[i]));   // y and dy share the output layout
    b[i] = mca_ld_f4(reinterpret_cast<const float*>(y + off[i]));
  }
#pragma unroll
  for (int i = 0; i < DELTA_STEPS; ++i) {
    const uint32_t aw[4] = {__float_as_uint(a[i].x), __float_as_uint(a[i].y), __float_as_uint(a[i].z), __float_as_uint(a[i].w)};
    const uint32_t bw[4] = {__float_as_uint(b[i].x), __float_as_uint(b[i].y), __float_as_uint(b[i].z), __float_as_uint(b[i].w)};
    float acc = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 fa = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&aw[e]));
      const float2 fb = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&bw[e]));
      acc = fmaf(fa.x, fb.x, fmaf(fa.y, fb.y, acc));
    }
    for (int o = g / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    const int64_t row = row0 + i * rpw;
    if (row < rows && lane % g == 0) delta[row] = acc;
  }
}

// What the caller has for the dS tiles (see ds_rules); with less than the plan asks dS is formed twice.
struct DsRoom {
  uint8_t* ptr;
  int64_t bytes;
};

// Both kernels of one backward, with or without the caller's mask.  make_mk64 encodes the map of K in boxes of 64 rows, which the dQ kernel
// of passed dS alone reads.
template <int HD, bool SPLIT, bool MASKED, bool NARROW, typename MapK64>
int launch_bwd_pair(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mdo, const MapK64& make_mk64, BwdParams p,
                    void* dq, void* dk, void* dv, int B, int H, int T, const DsRoom& room, cudaStream_t st) {
  using PL = BwdPlan<SPLIT ? 128 : HD, NARROW>;
  const size_t smem_kv = PL::BYTES_KV;
  int e;
  if constexpr (ds_rules::possible(HD, SPLIT)) {
    const ds_rules::Plan plan = ds_rules::plan((int64_t)B * H, T, HD, SPLIT, p.causal);
    if (plan.parts != 0 && room.ptr != nullptr && plan.bytes <= room.bytes) {
      using PD = DqDsPlan<HD, SPLIT>;
      static std::atomic<uint64_t> done_kv{0}, done_dq{0};
      if ((e = mca_smem_once(done_kv, sdpa_bwd_dkdv_tc_kernel<HD, SPLIT, MASKED, NARROW, true>, smem_kv)) ||
          (e = mca_smem_once(done_dq, sdpa_bwd_dq_ds_tc_kernel<HD, SPLIT>, (size_t)PD::BYTES)))
        return e;
      CUtensorMap mk64;
      if ((e = make_mk64(&mk64))) return e;
      const int nt = mca_ceil_div(T, BLK), group = p.group;
      p.ds = room.ptr;
      for (int i = 0; i < plan.parts; ++i) {
        p.bh0 = ds_rules::part_begin((int64_t)B * H, plan.parts, i);
        const int heads = ds_rules::part_begin((int64_t)B * H, plan.parts, i + 1) - p.bh0;
        p.group = std::min(group, heads);
        p.out0 = dk; p.out1 = dv;
        if ((e = mca_launch_pdl(sdpa_bwd_dkdv_tc_kernel<HD, SPLIT, MASKED, NARROW, true>, dim3(nt, heads), dim3(PL::THREADS), smem_kv, st, mq, mk, mv, mdo, p)))
          return e;
        p.out0 = dq; p.out1 = nullptr;
        if ((e = mca_launch_pdl(sdpa_bwd_dq_ds_tc_kernel<HD, SPLIT>, dim3(mca_ceil_div(nt, PD::QT), heads), dim3(PD::THREADS), (size_t)PD::BYTES, st, mk64, p)))
          return e;
      }
      return 0;
    }
  }
  const size_t smem_dq = PL::BYTES_DQ;
  static std::atomic<uint64_t> done_kv{0}, done_dq{0};
  if ((e = mca_smem_once(done_kv, sdpa_bwd_dkdv_tc_kernel<HD, SPLIT, MASKED, NARROW, false>, smem_kv)) ||
      (e = mca_smem_once(done_dq, sdpa_bwd_dq_tc_kernel<HD, SPLIT, MASKED, NARROW>, smem_dq)))
    return e;
  dim3 grid(mca_ceil_div(T, BLK), B * H);
  p.ds = nullptr; p.bh0 = 0;
  p.out0 = dk; p.out1 = dv;
  e = mca_launch_pdl(sdpa_bwd_dkdv_tc_kernel<HD, SPLIT, MASKED, NARROW, false>, grid, dim3(PL::THREADS), smem_kv, st, mq, mk, mv, mdo, p);
  if (e) return e;
  p.out0 = dq; p.out1 = nullptr;
  return mca_launch_pdl(sdpa_bwd_dq_tc_kernel<HD, SPLIT, MASKED, NARROW>, grid, dim3(PL::THREADS), smem_dq, st, mq, mk, mv, mdo, p);
}

void set_mask(BwdParams& p, const McaMaskBits* mask, int T) {
  p.mask_bits = mask ? mask->bits : nullptr;
  p.mask_bits_t = mask ? mask->bits_t : nullptr;
  p.mask_batch_stride = mask ? mask->batch_stride : 0;
  p.mask_row_stride = mask ? mask->row_stride : 0;
  p.inv_T = 1.0f / (float)T;
}

template <int HD>
int launch_bwd(const void* q, const void* k, const void* v, const void* dy, const float* lse, const float* delta,
               int causal, int B, int H, int T, void* dq, void* dk, void* dv, int* status, int layout, cudaStream_t st,
               const McaMaskBits* mask, const DsRoom& room) {
  if (mask != nullptr && causal) return ERROR_ATTN_UNSUPPORTED_SHAPE;
  constexpr bool NARROW = HD <= 64;
  constexpr int BN = BwdPlan<HD, NARROW>::BN;
  CUtensorMap mq, mk, mv, mdo;
  int e;
  const McaStrides sin = mca_in_strides(layout, H, T, HD), sout = mca_out_strides(layout, H, T, HD);
  if ((e = make_map_bf16(&mq, q, B, H, T, HD, sin, BN)) || (e = make_map_bf16(&mk, k, B, H, T, HD, sin, BN)) ||
      (e = make_map_bf16(&mv, v, B, H, T, HD, sin, BN)) || (e = make_map_bf16(&mdo, dy, B, H, T, HD, sout, BN)))
    return e;
  const auto mk64 = [&](CUtensorMap* m) { return make_map_bf16(m, k, B, H, T, HD, sin, 64); };
  BwdParams p;
  p.scales = nullptr;
  p.lse = lse; p.delta = delta; p.status = status; p.T = T; p.causal = causal; p.H = H;
  {
    // Q, K, V, dY of one (batch, head): keep a group's set under about 64 MB of the 126 MB L2
    const int64_t g = (64ll << 20) / ((int64_t)4 * T * HD * 2);
    p.group = causal ? (int)std::max<int64_t>(1, std::min<int64_t>(g, (int64_t)B * H)) : 1;
  }
  p.os = sin;
  p.scale = 1.0f / sqrtf((float)HD);
  p.scale_log2 = p.scale * 1.4426950408889634f;
  set_mask(p, mask, T);
  if (mask != nullptr) return launch_bwd_pair<HD, false, true, NARROW>(mq, mk, mv, mdo, mk64, p, dq, dk, dv, B, H, T, room, st);
  return launch_bwd_pair<HD, false, false, NARROW>(mq, mk, mv, mdo, mk64, p, dq, dk, dv, B, H, T, room, st);
}

// Split-operand backward for fp32 callers.  The workspace still holds the fp16 halves of q, k, v the forward's pre-pass
// wrote; dY is split here.
template <int HD>
int launch_bwd_split(const float* dy, const float* y_copy, const float* lse, float* delta, int causal, int B, int H, int T,
                     float* dq, float* dk, float* dv, void* workspace, int* status, int layout, cudaStream_t st,
                     const McaMaskBits* mask, const DsRoom& room) {
  if (mask != nullptr && causal) return ERROR_ATTN_UNSUPPORTED_SHAPE;
  const split::Workspace w = split::carve(workspace, (int64_t)B * H, T);
  const McaStrides sin = mca_in_strides(layout, H, T, HD), sout = mca_out_strides(layout, H, T, HD);
  split::Job job;
  job.src[0] = dy; job.dst[0] = w.tensor[split::TENSOR_DY]; job.slot[0] = split::TENSOR_DY;
  job.src[1] = job.src[2] = nullptr; job.dst[1] = job.dst[2] = nullptr; job.slot[1] = job.slot[2] = 0;
  // the kernel that splits dY also forms delta = rowsum(dY o Y) from the elements it holds
  int e = split::run<HD>(job, 1, sout, B, H, T, w, st, y_copy, delta);
  if (e) return e;
  CUtensorMap mq, mk, mv, mdo;
  const McaStrides sp{(int64_t)H * T * 128, (int64_t)T * 128, 128};
  const CUtensorMap* maps[4] = {&mq, &mk, &mv, &mdo};
  for (int i = 0; i < 4; ++i)
    if ((e = make_map_4d(const_cast<CUtensorMap*>(maps[i]), w.tensor[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, B, H, T, 128, sp,
                         CU_TENSOR_MAP_SWIZZLE_128B)))
      return e;
  const auto mk64 = [&](CUtensorMap* m) {
    return make_map_4d(m, w.tensor[split::TENSOR_K], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, B, H, T, 128, sp, CU_TENSOR_MAP_SWIZZLE_128B, 64);
  };
  BwdParams p;
  p.scales = w.scale;
  p.lse = lse; p.delta = delta; p.status = status; p.T = T; p.causal = causal; p.H = H;
  {
    const int64_t g = (64ll << 20) / ((int64_t)4 * T * 256);
    p.group = causal ? (int)std::max<int64_t>(1, std::min<int64_t>(g, (int64_t)B * H)) : 1;
  }
  p.os = sin;
  p.scale = 1.0f / sqrtf((float)HD);
  p.scale_log2 = p.scale * 1.4426950408889634f;
  set_mask(p, mask, T);
  if (mask != nullptr) return launch_bwd_pair<HD, true, true, false>(mq, mk, mv, mdo, mk64, p, dq, dk, dv, B, H, T, room, st);
  return launch_bwd_pair<HD, true, false, false>(mq, mk, mv, mdo, mk64, p, dq, dk, dv, B, H, T, room, st);
}

}  // namespace

int mca_sdpa_backward_tc(const void* q, const void* k, const void* v, const void* y, const void* dy, const float* lse,
                         float* delta_scratch, int dtype, int causal, int B, int H, int T, int D, void* dq, void* dk,
                         void* dv, int* status, void* stream) {
  return mca_sdpa_backward_tc_layout(q, k, v, y, dy, lse, delta_scratch, dtype, causal, B, H, T, D, dq, dk, dv, status,
                                     MCA_LAYOUT_BHTD, stream);
}

int mca_sdpa_backward_tc_layout(const void* q, const void* k, const void* v, const void* y, const void* dy,
                                const float* lse, float* delta_scratch, int dtype, int causal, int B, int H, int T, int D,
                                void* dq, void* dk, void* dv, int* status, int layout, void* stream) {
  return mca_sdpa_backward_tc_masked(q, k, v, y, dy, lse, delta_scratch, dtype, causal, B, H, T, D, dq, dk, dv, status, layout,
                                     nullptr, nullptr, MCA_MASK_NONE, stream);
}

int mca_sdpa_backward_tc_masked(const void* q, const void* k, const void* v, const void* y, const void* dy, const float* lse,
                                float* delta_scratch, int dtype, int causal, int B, int H, int T, int D, void* dq, void* dk,
                                void* dv, int* status, int layout, const uint32_t* mask_bits, const uint32_t* mask_bits_t,
                                int mask_mode, void* stream) {
  return mca_sdpa_backward_tc_ws(q, k, v, y, dy, lse, delta_scratch, dtype, causal, B, H, T, D, dq, dk, dv, status, layout, mask_bits,
                                 mask_bits_t, mask_mode, nullptr, 0, stream);
}

int mca_sdpa_backward_tc_ws(const void* q, const void* k, const void* v, const void* y, const void* dy, const float* lse,
                            float* delta_scratch, int dtype, int causal, int B, int H, int T, int D, void* dq, void* dk, void* dv,
                            int* status, int layout, const uint32_t* mask_bits, const uint32_t* mask_bits_t, int mask_mode, void* ds,
                            int64_t ds_bytes, void* stream) {
  McaMaskBits mb;
  const McaMaskBits* mask = nullptr;
  int me = mca_mask_bits_view(mask_bits, mask_bits_t, mask_mode, T, true, &mb, &mask);
  if (me) return me;
  if (layout != MCA_LAYOUT_BHTD && layout != MCA_LAYOUT_PACKED) return ERROR_PARAM_OUT_OF_RANGE;
  if (!q || !k || !v || !y || !dy || !lse || !delta_scratch || !dq || !dk || !dv || !status) return ERROR_PARAM_NULL;
  if (B <= 0 || H <= 0 || T <= 0 || (int64_t)B * H > 65535) return ERROR_PARAM_OUT_OF_RANGE;
  if (dtype != MCA_DTYPE_BF16) return ERROR_ATTN_UNSUPPORTED_SHAPE;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dq) | reinterpret_cast<uintptr_t>(dk) |
       reinterpret_cast<uintptr_t>(dv)) & 15)
    return ERROR_PARAM_OUT_OF_RANGE;
  if (D != 64 && D != 128) return ERROR_ATTN_UNSUPPORTED_SHAPE;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t rows = (int64_t)B * H * T;
  int e;
  {
    const int64_t rows_per_block = 8 * (256 / D) * DELTA_STEPS;   // eight warps, 256 / D rows each a step
    e = mca_launch_pdl(bwd_delta_bf16_kernel, dim3((unsigned)((rows + rows_per_block - 1) / rows_per_block)), dim3(256), 0, st,
                       (const __nv_bfloat16*)dy, (const __nv_bfloat16*)y, rows, H, T, D, mca_out_strides(layout, H, T, D), delta_scratch,
                       (int)launch_rules::delta_lets_go_late((int64_t)B * H, T, D, causal != 0));
  }
  if (e) return e;
  const DsRoom room{static_cast<uint8_t*>(ds), ds_bytes};
  if (D == 128) return launch_bwd<128>(q, k, v, dy, lse, delta_scratch, causal, B, H, T, dq, dk, dv, status, layout, st, mask, room);
  return launch_bwd<64>(q, k, v, dy, lse, delta_scratch, causal, B, H, T, dq, dk, dv, status, layout, st, mask, room);
}

int mca_sdpa_backward_f32_tc(const float* dy, const float* y_copy, const float* lse, float* delta_scratch, int causal, int B,
                             int H, int T, int D, float* dq, float* dk, float* dv, void* workspace, int64_t workspace_bytes,
                             int* status, int layout, void* stream) {
  return mca_sdpa_backward_f32_tc_masked(dy, y_copy, lse, delta_scratch, causal, B, H, T, D, dq, dk, dv, workspace, workspace_bytes,
                                         status, layout, nullptr, nullptr, MCA_MASK_NONE, stream);
}

int mca_sdpa_backward_f32_tc_masked(const float* dy, const float* y_copy, const float* lse, float* delta_scratch, int causal,
                                    int B, int H, int T, int D, float* dq, float* dk, float* dv, void* workspace,
                                    int64_t workspace_bytes, int* status, int layout, const uint32_t* mask_bits,
                                    const uint32_t* mask_bits_t, int mask_mode, void* stream) {
  return mca_sdpa_backward_f32_tc_ws(dy, y_copy, lse, delta_scratch, causal, B, H, T, D, dq, dk, dv, workspace, workspace_bytes, status,
                                     layout, mask_bits, mask_bits_t, mask_mode, nullptr, 0, stream);
}

int mca_sdpa_backward_f32_tc_ws(const float* dy, const float* y_copy, const float* lse, float* delta_scratch, int causal, int B, int H,
                                int T, int D, float* dq, float* dk, float* dv, void* workspace, int64_t workspace_bytes, int* status,
                                int layout, const uint32_t* mask_bits, const uint32_t* mask_bits_t, int mask_mode, void* ds,
                                int64_t ds_bytes, void* stream) {
  McaMaskBits mb;
  const McaMaskBits* mask = nullptr;
  int me = mca_mask_bits_view(mask_bits, mask_bits_t, mask_mode, T, true, &mb, &mask);
  if (me) return me;
  if (layout != MCA_LAYOUT_BHTD && layout != MCA_LAYOUT_PACKED) return ERROR_PARAM_OUT_OF_RANGE;
  if (!dy || !y_copy || !lse || !delta_scratch || !dq || !dk || !dv || !workspace || !status) return ERROR_PARAM_NULL;
  if (B <= 0 || H <= 0 || T <= 0 || (int64_t)B * H > 65535) return ERROR_PARAM_OUT_OF_RANGE;
  if (!mca_sdpa_backward_f32_tc_supported(D)) return ERROR_ATTN_UNSUPPORTED_SHAPE;
  if (workspace_bytes < mca_sdpa_forward_f32_tc_workspace_bytes(B, H, T)) return ERROR_ATTN_SCRATCH_TOO_SMALL;
  if ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dq) | reinterpret_cast<uintptr_t>(dk) |
       reinterpret_cast<uintptr_t>(dv) | reinterpret_cast<uintptr_t>(workspace)) & 15)
    return ERROR_PARAM_OUT_OF_RANGE;
  cudaStream_t st = (cudaStream_t)stream;
  const DsRoom room{static_cast<uint8_t*>(ds), ds_bytes};
  switch (D) {
    case 16: return launch_bwd_split<16>(dy, y_copy, lse, delta_scratch, causal, B, H, T, dq, dk, dv, workspace, status, layout, st, mask, room);
    case 32: return launch_bwd_split<32>(dy, y_copy, lse, delta_scratch, causal, B, H, T, dq, dk, dv, workspace, status, layout, st, mask, room);
    case 64: return launch_bwd_split<64>(dy, y_copy, lse, delta_scratch, causal, B, H, T, dq, dk, dv, workspace, status, layout, st, mask, room);
  }
  return ERROR_ATTN_UNSUPPORTED_SHAPE;
}

int mca_set_fail_words_bwd(int* words) { return (int)cudaMemcpyToSymbol(tc::g_fail_words, &words, sizeof(words)); }
