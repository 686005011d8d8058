// Choices of the TFT attention that depend on sizes alone (plain C++, so that they can be tested without a GPU).
#pragma once
#include <cstdint>

namespace tft_rules {

// Whether the tiled forward takes a call: 64-wide heads, no more keys than its register tiles cover, as many as a K buffer needs to
// hold the mean probabilities and the other three key slices' partial outputs (24 Nk + 3 x 24 x 64 <= 64 Nk: 116), and 16-byte copies of
// Q and stores of the output (K and V are refused unaligned by both kernels; the generic one reads Q and writes the output by the
// float).
constexpr int TILE_ROWS = 24, TILE_KEYS = 192, TILE_THREADS = 256;
inline bool forward_tiled(int Nk, int d, const void* q, const void* out) {
  const bool aligned = ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  return d == 64 && Nk <= TILE_KEYS && TILE_ROWS * (Nk + 3 * d) <= Nk * d && aligned;
}

struct Split {
  int ch, ct;      // CTAs of a batch item's cluster along the heads and along the row tiles
};

// Clusters of `ctas` CTAs that the chip holds at once, with one CTA per SM (cudaOccupancyMaxActiveClusters of the kernel).
inline int resident_clusters(int ctas) { return ctas == 1 ? 148 : ctas == 2 ? 74 : ctas == 4 ? 33 : 15; }

// How the backward of a batch item is spread.  In units of one product over a row tile and a head's keys: a CTA forms three for each
// of its (tile, head) pairs, dP once a tile, and dV; a cluster barrier and what is added between two of them is about a
// third of one; the weights are fitted to forward and backward of twelve shapes (us, all the splits measured, the best taken by
// each): 24 items, 4 heads, 185 x 185, d 64 425 -> 226; 16, 8, 160 x 160, 32 481 -> 206; 48, 8, 27 x 132, 64 206 -> 143; 64, 4, 24 x 192, 64
// 81 -> 64; 73, 1, 173 x 173, 32 144 -> 119; 256, 4, 24 x 192, 64 146 whole, 175 in two, 222 in four.  Clusters that do not fit the chip at
// once cost a twentieth more than their rounds say, with 16-wide heads, whose barriers weigh more, a tenth (the backward alone, us, 2 rounds
// of whole items / 3 of two CTAs: 150 items, 4 heads, 160 x 160, d 16 298 / 328; 170, 6 429 / 439, 8 560 / 546; 150, 6, 100 x 100, d 32 403 / 370).
inline Split backward_split(int B, int H, int tiles, int d = 64) {
  Split best{1, 1};
  double best_cost = 1e30;
  for (int ch = 1; ch <= 8 && ch <= H; ch *= 2)
    for (int ct = 1; ch * ct <= 8 && ct <= tiles; ct *= 2) {
      const int hn = (H + ch - 1) / ch, tn = (tiles + ct - 1) / ct, c = ch * ct;
      const int64_t rounds = (B + resident_clusters(c) - 1) / resident_clusters(c);
      const double more = c > 1 && rounds > 1 ? (d <= 16 ? 1.1 : 1.05) : 1.0;
      const double cost = more * rounds * (1.0 + tn * (3.0 * hn + 2.0 + (ct > 1 ? 0.6 * ct * (hn + 1) : 0.0) + (ch > 1 ? 0.7 + 0.1 * ch : 0.0)));
      if (cost < best_cost * 0.97) { best_cost = cost; best = Split{ch, ct}; }
    }
  return best;
}

// Whether the backward runs two items to an SM, with one buffer for V and then each head's K in turn: where there are more items than SMs.
// One's copies and barriers then stand beside the other's products, which one item's own second buffer does less well (forward and backward,
// us: 256 items, 8 heads, 40 x 192, d 16 291 -> 260; 300, 4, 24 x 150, 32 154 -> 142; 200, 8, 192 x 192, 32 1414 -> 1366; 170, 6, 160 x 160, 16
// 614 -> 548; 155, 1, 5 x 40, 16 22.6 -> 20.5; and just beyond a round or two of the SMs, over many row tiles, where V is read again for
// each of them: 149, 4, 192 x 192, 16 526 -> 476, 32 760 -> 673; 149, 8, 160 x 160, 32 1020 -> 975; 223, 8, 160 x 160, 16 867 -> 776; 296, 1,
// 192 x 192, 32 361 -> 339).  64-wide heads have not the registers (128 a thread, 100 spilled): 256, 4, 24 x 192 137.3 -> 136.6, 192 x 192 988 -> 1088.
inline bool backward_pair(int B, int d) { return d <= 32 && B > 148; }

// Into how many CTAs the forward of a row tile's heads goes: as long as every tile's cluster is resident at once, with an SM to each
// CTA.  Two CTAs on an SM take nearly twice as long, and their cluster's exchange comes on top (us, whole / over two: 128 tiles, 4 heads, 192 keys
// 23.1 / 25.2; 3 heads 19.8 / 25.1; 74 tiles, 4 heads 23.0 / 16.9; over four 25.0).
inline int forward_split(int64_t tiles, int H) {
  int ch = 1;
  while (ch < 8 && 2 * ch <= H && tiles <= resident_clusters(2 * ch)) ch *= 2;
  return ch;
}

}  // namespace tft_rules
