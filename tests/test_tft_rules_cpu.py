"""Which kernel a TFT attention call takes and how few batch items are spread (csrc/tft_rules.h)."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "mycaffe_b200" / "csrc"

PROGRAM = r'''
#include "tft_rules.h"
#include <cstdio>
using namespace tft_rules;
static int bad = 0;
static void claim(bool ok, const char* what, int B, int H, int tiles) { if (!ok) { std::printf("%s: B %d H %d tiles %d\n", what, B, H, tiles); bad = 1; } }
static void is(int B, int H, int tiles, int ch, int ct) { const Split s = backward_split(B, H, tiles); claim(s.ch == ch && s.ct == ct, "choice", B, H, tiles); }
int main() {
  for (int B = 1; B <= 300; ++B)
    for (int H = 1; H <= 20; ++H)
      for (int tiles = 1; tiles <= 12; ++tiles) {
        const Split s = backward_split(B, H, tiles);
        claim(s.ch >= 1 && s.ct >= 1 && s.ch * s.ct <= 8 && s.ch <= H && s.ct <= tiles, "range", B, H, tiles);
        const int f = forward_split((int64_t)B * tiles, H);
        claim(f >= 1 && f <= 8 && f <= H && (f == 1 || (int64_t)f * B * tiles <= 296), "forward", B, H, tiles);
      }
  // as measured
  is(256, 4, 1, 1, 1); is(128, 4, 1, 1, 1); is(99, 8, 6, 1, 1); is(78, 4, 8, 1, 1); is(64, 4, 1, 2, 1); is(24, 4, 8, 2, 2);
  is(48, 8, 2, 2, 1); is(73, 1, 8, 1, 2); is(16, 8, 7, 4, 1); is(200, 8, 5, 2, 1); is(40, 1, 4, 1, 2); is(24, 2, 1, 2, 1);
  // the boundary between two rounds of whole items and three of clusters of two
  auto whole = [](Split s) { return s.ch * s.ct == 1; };
  auto in_two = [](Split s) { return s.ch == 2 && s.ct == 1; };
  claim(whole(backward_split(150, 4, 7, 16)) && whole(backward_split(170, 6, 7, 16)) && in_two(backward_split(170, 8, 7, 16)) &&
        whole(backward_split(200, 4, 8, 64)) && whole(backward_split(150, 4, 8, 64)) && in_two(backward_split(150, 6, 5, 32)) &&
        in_two(backward_split(200, 8, 8, 64)) && in_two(backward_split(222, 6, 1, 64)), "rounds", 0, 0, 0);
  // the forward: never two CTAs of clusters on an SM; as measured
  for (int tiles = 1; tiles <= 400; ++tiles)
    for (int H = 1; H <= 20; ++H) claim(forward_split(tiles, H) == 1 || forward_split(tiles, H) * tiles <= 148, "one CTA to an SM", 0, H, tiles);
  claim(forward_split(128, 4) == 1 && forward_split(128, 3) == 1 && forward_split(80, 2) == 1 && forward_split(74, 4) == 2 && forward_split(50, 4) == 2 &&
        forward_split(33, 6) == 4 && forward_split(16, 8) == 4 && forward_split(15, 8) == 8 && forward_split(8, 1) == 1, "forward choice", 0, 0, 0);
  // the tiled forward copies Q and writes the output by 16 bytes: never from or to an address that is not a multiple of them
  alignas(16) static float at[8];
  for (int o = 1; o < 4; ++o) claim(!forward_tiled(192, 64, at + o, at) && !forward_tiled(192, 64, at, at + o), "alignment", o, 0, 192);
  for (int Nk = 1; Nk <= 300; ++Nk)
    for (int d = 4; d <= 128; d += 4) {
      const int slices = 256 / d;
      const bool room = 24 * Nk + (slices - 1) * 24 * d <= Nk * d, takes = forward_tiled(Nk, d, at, at + 4);
      claim(takes == (d == 64 && Nk >= 116 && Nk <= 192), "tiled", d, 0, Nk);
      claim(!takes || (room && 4 * (2 * Nk * d + 2 * 24 * d + 96) <= 113 * 1024 && 2 * Nk * d >= 24 * 192), "room", d, 0, Nk);
    }
  // what the shapes of test_tft_split_gpu.py take: 0 the generic forward, else the CTAs along the heads
  auto forward = [&](int B, int H, int Nq, int Nk, int d) { return forward_tiled(Nk, d, at, at) ? forward_split((int64_t)B * ((Nq + 23) / 24), H) : 0; };
  claim(forward(1, 3, 49, 191, 64) == 2 && forward(33, 6, 24, 192, 64) == 4 && forward(2, 8, 30, 116, 64) == 8 && forward(160, 4, 24, 120, 64) == 1 &&
        forward(2, 7, 25, 33, 64) == 0 && forward(2, 8, 24, 115, 64) == 0 && forward(16, 8, 160, 160, 32) == 0, "forward", 0, 0, 0);
  // and its backwards over many row tiles by one CTA
  claim(whole(backward_split(140, 2, 5, 64)) && whole(backward_split(130, 1, 8, 32)) && whole(backward_split(150, 3, 4, 16)) &&
        whole(backward_split(140, 1, 5, 64)), "whole items", 0, 0, 0);
  return bad;
}
'''


def test_the_spread_of_an_item_fits_a_cluster_and_is_the_measured_one(tmp_path):
    (tmp_path / "main.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "main")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC), str(tmp_path / "main.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
