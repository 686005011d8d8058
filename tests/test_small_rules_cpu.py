"""Which calls the one-launch fp32 forward takes (csrc/small_rules.h): none that writes over what it reads."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "mycaffe_b200" / "csrc"

PROGRAM = r'''
#include "small_rules.h"
#include <cstdio>
#include <initializer_list>
using namespace small_rules;
static int bad = 0;
#define CLAIM(c) do { if (!(c)) { std::puts(#c); bad = 1; } } while (0)
int main() {
  alignas(16) static float m[1 << 20];
  const int B = 2, H = 3, T = 100, D = 32;
  const int64_t n = (int64_t)B * H * T * D, C = H * D;
  float *q = m, *k = q + n, *v = k + n, *y = v + n, *mask = y + n;
  auto plain = [&](float* out, float* msk, bool batch) { return takes(q, k, v, out, msk, batch, false, B, H, T, D); };
  CLAIM(plain(y, mask, false) && plain(y, mask, true) && plain(y, nullptr, false));
  CLAIM(takes(k, k, k, y, mask, false, false, B, H, T, D));               // inputs may be one another
  for (float* at : {q, k, v}) CLAIM(!plain(at, mask, false) && !plain(at + 4, nullptr, false));
  CLAIM(!plain(v + n - 4, mask, false) && plain(v + n, mask + 4, false));  // one piece of v; right behind it
  CLAIM(!plain(mask - n + 4, mask, false) && !plain(mask + T * T - 4, mask, false) && plain(mask + T * T, mask, false));
  CLAIM(!plain(mask + B * T - 4, mask, true) && plain(mask + B * T, mask, true));
  // packed: the thirds of a row
  float* x = m;
  auto packed = [&](float* out) { return takes(x, x + C, x + 2 * C, out, mask, false, true, B, H, T, D); };
  CLAIM(packed(x + 3 * n) && !packed(x) && !packed(x + 3 * n - 4) && !packed(x + n) && !packed(x + 2 * n + 4));
  // alignment, sizes
  for (int o = 1; o < 4; ++o) {
    CLAIM(!plain(y + o, nullptr, false) && !takes(q + o, k, v, y, nullptr, false, false, B, H, T, D));
    CLAIM(!takes(q, k + o, v, y, nullptr, false, false, B, H, T, D) && !takes(q, k, v + o, y, nullptr, false, false, B, H, T, D));
  }
  CLAIM(fits(1, 4, 128, 16) && !fits(1, 4, 129, 16) && fits(1, 148, 32, 64) && !fits(1, 149, 32, 64) && fits(1, 37, 128, 32) && !fits(2, 19, 128, 32));
  CLAIM(!fits(1, 1, 8, 48) && !fits(1, 1, 8, 128));
  return bad;
}
'''


def test_takes(tmp_path):
    (tmp_path / "main.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "main")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC), str(tmp_path / "main.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
