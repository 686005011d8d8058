// When a kernel lets the one behind it go (plain C++, so that it can be tested without a GPU).  CTAs that are launched while the kernels before
// still hold SMs take what is free, two to one SM where the grid has one for each; launched late, their launch is no longer hidden.
#pragma once
#include <cstdint>

namespace launch_rules {

constexpr int TILE = 128;    // rows of a CTA

// bf16: is the dK/dV kernel let go only when the forward has left the SMs (late), not at the delta kernel's top?  Beyond three tiles a head late
// gains for 128-wide heads (layers, us: 12 of 1024 41.6 -> 40.1; 24 and more of any length the same).  64-wide ones, two of whose CTAs an SM takes,
// lose 3 to 8 % with fewer rows than 64 CTAs have.  With more, all as long, they gain (no mask, by CTAs: 64 3 to 6 %, 96 3.5 to 5, 128 0.4 to
// 4.5, 144 3 to 4, from 192 0 to 1, but 64 of 8 heads of 900 lose 4.7; 8 of 2048 under a (T,T) mask 145 -> 132).  Causal CTAs are of all
// lengths: 80 gain 6.7 and 3.8 %, 96 2.6 to 4.2, 160 2.2 and 3.7, 192 2.2 to 3.6, but 128 lose 5 to 7, 240 to 330 up to 6.
inline bool delta_lets_go_late(int64_t heads, int T, int D, bool causal) {
  const int64_t nt = (T + TILE - 1) / TILE, ctas = heads * nt;
  if (nt <= 3) return false;
  if (D == 128) return true;
  return causal ? (ctas >= 72 && ctas <= 96) || (ctas >= 160 && ctas <= 224) : heads * T >= 64 * TILE;
}

// bf16: is the forward let go at the top of the mask's packing, not at its end?  Layers under a key mask, us, at the top / at the end / ordinary
// launches: 8 heads of 1024 x 128 54.4 / 45.7 / 47.7, 24 of 384 x 128 31.1 / 26.9 / 28.8, 64 of 256 x 64 28.1 / 25.2 / 26.7.  With few CTAs enough SMs are
// free (layers of 64-wide heads, to 60 CTAs, 3 to 6 %; of 128-wide ones, to 40, nothing or little; forwards alone, to 64, 3 %; 72 lose 25).
inline bool pack_lets_go(int64_t heads, int T, int D, bool training) {
  const int64_t ctas = heads * ((T + TILE - 1) / TILE);
  return ctas <= (!training ? 64 : D == 128 ? 40 : 60);
}

}  // namespace launch_rules
