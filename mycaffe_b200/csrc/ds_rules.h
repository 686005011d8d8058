// Choices of the tensor-core attention backward that depend on sizes alone (plain C++, so that they can be tested without a GPU): whether dS is
// formed once and passed through memory, how many heads go through it at a time, and the room that takes.
#pragma once
#include <algorithm>
#include <cstdint>

namespace ds_rules {

constexpr int TILE = 128;                     // queries and keys of a dS tile
constexpr int64_t MAX_BYTES = 1ll << 30;      // of dS, however many heads there are

// Tiles of a head: the lower triangle alone under the causal mask.
constexpr int64_t head_tiles(int T, bool causal) {
  const int64_t nt = (T + TILE - 1) / TILE;
  return causal ? nt * (nt + 1) / 2 : nt * nt;
}
constexpr int64_t tile_bytes(bool split) { return (int64_t)TILE * TILE * (split ? 4 : 2); }

// Head widths that have the kernels for it.
constexpr bool possible(int D, bool split) { return D == (split ? 64 : 128); }

// CTAs that are all as long fill so much of their waves, with one to each of 148 SMs.
constexpr bool fills_waves(int64_t ctas, int percent) { return 100 * ctas >= percent * ((ctas + 147) / 148 * 148); }

// Do so many heads at a time gain?  Instead of S, dP and the exponentials a second time the dQ kernel then reads two (split: four) bytes a
// pair from HBM, and the dK/dV kernel writes them from the warps that bound it (7001 x 128: 333 -> 364 us, dQ 253 -> 134); but it waits for
// the whole dK/dV kernel, where the other one fills that kernel's last wave.  So there must be waves enough, and where the CTAs are all as
// long (no causal mask, or a tile a head), not a last one that is nearly empty.  Layers, us, dS formed twice -> once, by heads:
//   bf16 x 128, causal: 16 of 7001 878 -> 847, 60 of 1024 124.7 -> 117.5, 32 68.2 -> 66.5, 96 of 200 35.3 -> 34.5, 9 of 4096 197.7 -> 197.0, 16 of 2048
//     104.3 -> 104.1 (8 of 4096 180 -> 183).
//   bf16 x 128, alike: 16 of 2048 160 -> 151 (key mask 184 -> 174), 64 of 512 61.8 -> 55.1, 50 of 1024 152 -> 146, 12 of 5000 681 -> 671, 14 of 2048
//     152 -> 144, 23 236 -> 239 (key mask 260 -> 257); between waves 20 of 2048 218 -> 220, 8 of 10000 (two parts of 316 CTAs) 1718 -> 1820, 192 of 256
//     (in two parts of 192; in one they gain) 72.6 -> 75.9; a wave or less 8 of 2048 91.8 -> 96.7, 36 of 512 38.2 -> 41.2, but with one tile a head 144 of 128 25.1 -> 23.9 (150 31.2 -> 33.8, 288 41.8 -> 40.7, 300 51.0 -> 52.2).
//   64-wide split heads have half the products to save and twice the bytes.  Up to four tiles they gain from their two CTAs per SM: causal,
//     256 of 100 53.9 -> 50.1, 128 of 200 62.0 -> 58.7, 100 of 512 114.8 -> 112.9 (64 79.7 -> 80.0, 48 67.3 -> 67.5); key mask, 64 of 512 106.1 -> 102.2,
//     192 of 256 111.5 -> 107.7, 256 of 512 376 -> 368, between waves 80 of 512 136.5 -> 141.7.  Longer causal ones with many waves: 80 of 1024 246 ->
//     240, 96 287 -> 285, 128 of 600 200 -> 194, 24 of 4096 749 -> 737 (72 of 1024 225 -> 225, 16 of 2048 156 -> 164, 20 of 4096 640 -> 652); not
//     causal, twice the bytes, 128 of 1024 584 -> 588 under a key mask, 565 -> 555 without.
//   Narrower split heads lose (96 of 1024 x 32 205 -> 218), and 64-wide bf16 ones, whose narrow CTAs leave the element-wise warps no time for
//     it, too (96 of 1024 120 -> 131).
constexpr bool gains(int64_t heads, int T, bool split, bool causal) {
  const int64_t nt = (T + TILE - 1) / TILE, ctas = heads * nt;
  if (split) {
    if (nt > 4) return causal && ctas >= (nt <= 8 ? 640 : 768);
    return ctas >= 256 && (causal || nt == 1 || fills_waves(ctas, 85));
  }
  if (causal && nt > 1) return heads * (nt + 1) >= 288;   // about two times the longest CTA's work per SM
  return nt == 1 ? ctas >= 144 && fills_waves(ctas, 85) : ctas > 148 && fills_waves(ctas, 75);
}

// The heads go through the workspace in `parts` launches of each kernel, as alike in size as can be; 0: dS is formed twice, as where a
// part of theirs would not gain.
struct Plan {
  int parts;
  int64_t bytes;     // room for the largest part
};
constexpr int part_begin(int64_t heads, int parts, int i) { return (int)(heads * i / parts); }
constexpr Plan plan(int64_t heads, int T, int D, bool split, bool causal) {
  const int64_t head = head_tiles(T, causal) * tile_bytes(split), fit = std::min(MAX_BYTES / head, heads);
  if (!possible(D, split) || fit == 0) return Plan{0, 0};
  const int64_t parts = (heads + fit - 1) / fit, most = (heads + parts - 1) / parts;
  if (!gains(heads / parts, T, split, causal) || !gains(most, T, split, causal)) return Plan{0, 0};
  return Plan{(int)parts, most * head};
}
// What a handle asks for, whose forwards may bring any mask unless it has the causal flag.
constexpr int64_t room(int64_t heads, int T, int D, bool split, bool only_causal) {
  const int64_t causal = plan(heads, T, D, split, true).bytes;
  return only_causal ? causal : std::max(causal, plan(heads, T, D, split, false).bytes);
}

}  // namespace ds_rules
