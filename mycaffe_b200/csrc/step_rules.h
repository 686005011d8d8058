// Choices of the decode step that depend on sizes alone (plain C++, so that they can be tested without a GPU).
#pragma once
#include <cstdint>

namespace step_rules {

// Should the attention kernel, launched ahead of the projections before it, ask L2 for its cache rows while it waits?  Inside a
// step of a few sequences that hides its first reads (a token of 12 layers of 12 heads of 64, 256 keys: 180 -> 155 us).  A call of
// its own has nothing to wait for, and the requests only come before the reads (7 sequences of 4096 keys, 32 heads of 128, fp32:
// 82 us without, 97 with).  bf16 rows are read through a ring of their own that is as early, so that beyond what L2 takes beside
// the weights the requests cost (2 layers, 32 heads of 128, one sequence of 2048 keys, 32 MiB: 238 us without, 245 with; 8 kv
// heads, 32768 keys, 128 MiB: 408 and 422); below that they still gain (12 heads of 64, 8 sequences of 1024 keys, 24 MiB:
// 427 us without, 412 with).
inline bool prefetch_rows(bool in_step, int B, bool cache_bf16, int64_t row_bytes) {
  return in_step && B <= 8 && (!cache_bf16 || row_bytes < (32ll << 20));
}

}  // namespace step_rules
