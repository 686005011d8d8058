// Is a caller's (T,T) mask exactly the lower-triangular ones fillMask builds (CausalSelfAttentionLayer.cs:276-291)?  One pass
// over it by any number of CTAs of 256 threads (a warp per row, 16-byte loads when T allows), as a kernel of its own or as
// extra CTAs of one that has something else to do.
#pragma once
#include "common.cuh"

// scratch: two device ints that are zero before and after (the CTAs' mismatches and a ticket; the last CTA to finish writes
// *flag, and host_base + flag to *host_flag in pinned host memory unless that is null).
struct McaClassifyJob {
  const float* mask;
  int T;
  int* flag;
  int* host_flag;
  int host_base;
  int* scratch;
};

// Keep-bits of a (B,T) key mask, one warp ballot per word (see mca_mask_pack), by any number of CTAs of 256 threads of a kernel that has
// something else to do.
struct McaPackJob {
  const float* mask;    // null: none
  uint32_t* bits;
  int rows, T, wpr;
};

#ifdef __CUDACC__
__device__ __forceinline__ void mca_pack_word(const float* mask, uint32_t* bits, int64_t word, int T, int wpr, int lane) {
  const int r = (int)(word / wpr), c = 32 * (int)(word - (int64_t)r * wpr) + lane;
  const uint32_t keep = __ballot_sync(0xffffffffu, c < T && mask[(int64_t)r * T + c] != 0.f);
  if (lane == 0) bits[word] = keep;
}
__device__ __forceinline__ void mca_pack_rows(const McaPackJob& j, int cta, int ctas) {
  const int64_t words = (int64_t)j.rows * j.wpr;
  for (int64_t word = (int64_t)cta * 8 + (threadIdx.x >> 5); word < words; word += (int64_t)ctas * 8)
    mca_pack_word(j.mask, j.bits, word, j.T, j.wpr, threadIdx.x & 31);
}
__device__ __forceinline__ void mca_classify_rows(const McaClassifyJob& j, int cta, int ctas) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, T = j.T;
  bool bad = false;
  for (int i = cta * 8 + warp; i < T; i += ctas * 8) {
    const float* row = j.mask + (int64_t)i * T;
    if ((T & 3) == 0) {
#pragma unroll 4
      for (int c = lane * 4; c < T; c += 128) {
        const float4 m = *reinterpret_cast<const float4*>(row + c);
        bad |= m.x != (c <= i ? 1.f : 0.f) || m.y != (c + 1 <= i ? 1.f : 0.f) || m.z != (c + 2 <= i ? 1.f : 0.f) ||
               m.w != (c + 3 <= i ? 1.f : 0.f);
      }
    } else {
#pragma unroll 4
      for (int c = lane; c < T; c += 32) bad |= row[c] != (c <= i ? 1.f : 0.f);
    }
  }
  const int any_bad = __syncthreads_or(bad ? 1 : 0);
  if (threadIdx.x == 0) {
    if (any_bad) atomicAdd(j.scratch, 1);
    __threadfence();
    if (atomicAdd(j.scratch + 1, 1) == ctas - 1) {
      __threadfence();
      const int causal = atomicExch(j.scratch, 0) == 0 ? 1 : 0;
      *j.flag = causal;
      if (j.host_flag != nullptr) {   // read by the host behind the next stream synchronisation, or polled
        *reinterpret_cast<volatile int*>(j.host_flag) = j.host_base + causal;
        __threadfence_system();
      }
      j.scratch[1] = 0;
    }
  }
}
#endif
