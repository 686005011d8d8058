// Which calls the one-launch forward of short fp32 inference takes (plain C++, so that it can be tested without a GPU).
#pragma once
#include <cstdint>

namespace small_rules {

constexpr int WARPS = 8, KEYS = 128;     // warps of a CTA, keys of its one tile

struct Range {
  const float* at;
  int64_t floats;
};
inline bool overlap(const Range& a, const Range& b) {
  const uintptr_t a0 = reinterpret_cast<uintptr_t>(a.at), b0 = reinterpret_cast<uintptr_t>(b.at);
  return a.at != nullptr && b.at != nullptr && a0 < b0 + 4 * (uintptr_t)b.floats && b0 < a0 + 4 * (uintptr_t)a.floats;
}

// The keys of one tile, and no more rows than give every CTA an SM of its own.  A call, waited for / one of many, us, before (split operands)
// and with this kernel: 4 heads of 128 x 16 under a (T,T) mask 20.5 -> 14.6 / 15.1 -> 5.4, 16 heads of 128 x 64 20.4 -> 18.3 / 8.3 -> 6.5,
// 64 of 64 x 64 20.9 -> 18.3 / 11.1 -> 6.5, 15 of 77 x 64 under a key mask 25.2 -> 17.5 / 12.4 -> 5.8.  Beyond: 64 heads of 128 x 64 20.6 -> 24.5 /
// 9.9 -> 12.6, of 128 x 32 19.5 -> 20.2 / 8.2 -> 8.3; and with a second tile, measured with an earlier launch of what follows, 16 heads of 256 x 32
// 21.2 -> 20.0 / 10.8 -> 13.0, 8 of 256 x 64 22.8 -> 21.8 / 11.8 -> 18.6.
inline bool fits(int B, int H, int T, int D) {
  return (D == 16 || D == 32 || D == 64) && T <= KEYS && (int64_t)B * H * ((T + WARPS * 4 - 1) / (WARPS * 4)) <= 148;
}
// Its CTAs read q, k, v and the mask while others write y already, and copy by 16 bytes.  A call whose y is (part of) one of them goes to
// the split kernels, which have copied them before they write.  packed: q, k, v are thirds of one (B,T,3,H,D) tensor.
inline bool takes(const float* q, const float* k, const float* v, const float* y, const float* mask, bool batch_mask, bool packed, int B, int H, int T, int D) {
  const int64_t n = (int64_t)B * H * T * D, in = packed ? 3 * n : n, C = (int64_t)H * D;
  const Range out{y, n};
  if (!fits(B, H, T, D) || ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(y)) & 15))
    return false;
  return !overlap(out, Range{q, in}) && !overlap(out, Range{k, packed ? in - C : in}) && !overlap(out, Range{v, packed ? in - 2 * C : in}) &&
         !overlap(out, Range{mask, (int64_t)(batch_mask ? B : T) * T});
}

}  // namespace small_rules
