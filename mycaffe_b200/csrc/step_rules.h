// Choices of the decode step that depend on sizes alone (plain C++, so that they can be tested without a GPU).
#pragma once
#include <cstdint>

namespace step_rules {

// Should the attention kernel, launched ahead of the projections before it, ask L2 for its cache rows while it waits?  Inside a
// step of a few sequences that hides its first reads (a token of 12 layers of 12 heads of 64, 256 keys: 180 -> 155 us).  A call of
// its own has nothing to wait for, and the requests only come before the reads (8 sequences of 4096 keys, 32 heads of 128, fp32:
// 123 us without, 148 with).  Rows that are too many for L2 beside the weights gain less and then cost.  bf16 ones, which have a
// ring of their own that is as early: 24 MiB (8 sequences of 1024 keys, 12 heads of 64) 427 us without, 412 with; 32 MiB (one of
// 2048, 32 heads of 128, 2 layers) 238 and 245; 128 MiB 408 and 422.  fp32 ones that several query heads share: 67 MiB the same
// either way, 256 MiB (one of 32768, 8 kv heads) 499 and 510; with a kv head each: 512 MiB (8 of 2048) 761 and 741.
inline bool prefetch_rows(bool in_step, int B, bool cache_bf16, int kv_mul, int64_t row_bytes) {
  const int64_t most = (cache_bf16 ? 24ll : kv_mul > 1 ? 128ll : 512ll) << 20;
  return in_step && B <= 8 && row_bytes <= most;
}

// Should the output projection combine the attention's splits while it stages its activations, instead of a kernel between the
// two?  Every one of its CTAs then reads every partial result: worth the launch for one sequence and few of them (a
// token of 6 layers, 8 splits: 6 heads of 48 118 us, 129 with the kernel; 12 of 64 156 and 165; 4 layers of 16 heads of 128 212 and
// 216), not beyond (2 layers of 32 heads of 128, 9 splits: 237 us, 230 with the kernel; 37 splits of 8 kv heads 273 and 248),
// nor for more sequences (8, with 8 splits, 4 layers of 16 heads of 128: 575 and 532 us).
inline bool combine_in_projection(int B, int nsplit, int dim) { return B == 1 && nsplit > 1 && (int64_t)nsplit * dim <= 16384; }

}  // namespace step_rules
