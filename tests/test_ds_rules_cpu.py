"""Where the tensor-core backward passes dS through memory, in how many parts and in how much room (csrc/ds_rules.h)."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "mycaffe_b200" / "csrc"

PROGRAM = r'''
#include "ds_rules.h"
#include <cstdio>
using namespace ds_rules;
static int bad = 0;
static void claim(bool ok, const char* what, int64_t heads, int T, bool split, bool causal) {
  if (!ok) { std::printf("%s: %lld heads of %d, split %d, causal %d\n", what, (long long)heads, T, split, causal); bad = 1; }
}
static int parts(int64_t heads, int T, bool split, bool causal) { return plan(heads, T, split ? 64 : 128, split, causal).parts; }
static void once(int64_t heads, int T, bool split, bool causal, int in = 1) { claim(parts(heads, T, split, causal) == in, "once", heads, T, split, causal); }
static void twice(int64_t heads, int T, bool split, bool causal) { claim(parts(heads, T, split, causal) == 0, "twice", heads, T, split, causal); }
int main() {
  // the room is what the plan's largest part takes, all of the heads go through it, and nothing is asked for where it is not used
  const int lengths[] = {1, 64, 127, 128, 129, 200, 256, 257, 500, 512, 640, 1000, 1024, 2048, 2500, 4096, 7001, 8192, 10000, 14000, 16384, 20000, 32768, 40000, 65536};
  for (int split = 0; split < 2; ++split)
    for (int causal = 0; causal < 2; ++causal)
      for (int T : lengths)
        for (int64_t heads = 1; heads <= 65535; heads += heads < 400 ? 1 : heads / 7) {
          const int D = split ? 64 : 128;
          const Plan p = plan(heads, T, D, split, causal);
          const int64_t head = head_tiles(T, causal) * tile_bytes(split);
          claim((p.parts == 0) == (p.bytes == 0) && p.bytes <= MAX_BYTES && p.parts <= heads, "range", heads, T, split, causal);
          int64_t most = 0;
          for (int i = 0; i < p.parts; ++i) {
            const int n = part_begin(heads, p.parts, i + 1) - part_begin(heads, p.parts, i);
            most = std::max<int64_t>(most, n);
            claim(gains(n, T, split, causal), "part", heads, T, split, causal);
          }
          claim(p.parts == 0 || (part_begin(heads, p.parts, 0) == 0 && part_begin(heads, p.parts, p.parts) == heads && most * head == p.bytes), "room", heads, T, split, causal);
          claim(p.parts < 2 || (p.parts - 1) * (MAX_BYTES / head) < heads, "as few parts as fit", heads, T, split, causal);
          const int64_t a = plan(heads, T, D, split, true).bytes, b = plan(heads, T, D, split, false).bytes;
          claim(room(heads, T, D, split, true) == a && room(heads, T, D, split, false) == std::max(a, b), "asked for", heads, T, split, causal);
          for (int other : {16, 32, split ? 128 : 64}) claim(plan(heads, T, other, split, causal).parts == 0, "width", heads, T, split, causal);
        }
  // as measured: bf16 heads of 128, causal
  once(16, 7001, false, true); once(192, 1024, false, true); once(32, 1024, false, true); once(96, 200, false, true); once(9, 4096, false, true);
  twice(16, 2048, false, true); twice(8, 4096, false, true); twice(28, 1024, false, true);
  once(16, 12000, false, true, 3); once(8, 10000, false, true); once(16, 14000, false, true, 4); once(4, 20000, false, true, 2);
  twice(16, 16384, false, true); twice(8, 16384, false, true); twice(4, 16384, false, true); twice(1, 30000, false, true); twice(1, 32768, false, true);
  for (bool causal : {false, true}) {     // one tile a head: the mask makes no difference
    once(144, 100, false, causal); once(256, 100, false, causal); once(288, 128, false, causal); once(400, 100, false, causal);
    twice(150, 100, false, causal); twice(180, 100, false, causal); twice(300, 128, false, causal); twice(340, 100, false, causal); twice(128, 100, false, causal);
    once(256, 128, true, causal); once(300, 128, true, causal); twice(192, 128, true, causal);
  }
  // without the causal mask
  once(16, 2048, false, false); once(64, 512, false, false); once(32, 1024, false, false); once(50, 1024, false, false); once(6, 9000, false, false); once(144, 200, false, false);
  once(16, 4096, false, false); once(12, 5000, false, false); once(14, 2048, false, false); once(14, 4096, false, false); once(19, 4096, false, false);
  twice(8, 2048, false, false); twice(4, 4096, false, false); twice(36, 512, false, false); twice(72, 256, false, false); twice(20, 2048, false, false); twice(8, 10000, false, false);
  twice(96, 256, false, false); twice(6, 4096, false, false); twice(18, 1024, false, false);
  // 64-wide split heads
  once(96, 1024, true, true); once(80, 1024, true, true); once(128, 600, true, true); once(128, 200, true, true); once(100, 512, true, true); once(24, 4096, true, true);
  once(48, 4096, true, true, 2);
  twice(72, 1024, true, true); twice(48, 512, true, true); twice(16, 2048, true, true); twice(20, 4096, true, true); twice(16, 8192, true, true); twice(16, 16384, true, true);
  once(64, 512, true, false); once(128, 200, true, false); once(192, 256, true, false); once(256, 512, true, false);
  twice(48, 512, true, false); twice(80, 512, true, false); twice(100, 384, true, false); twice(96, 1024, true, false); twice(128, 1024, true, false);
  // what the shapes of test_tc_ds_gpu.py take
  for (int T : {129, 193, 320}) { once(144, T, false, true); once(144, T, false, false); }
  for (int T : {65, 129, 193}) once(144, T, false, false);
  for (int T : {129, 193, 320}) { once(144, T, true, true); once(144, T, true, false); }
  for (int T : {2, 65, 128}) for (bool causal : {false, true}) once(260, T, true, causal);
  for (bool split : {false, true}) once(148, 450, split, false);
  once(16, 10000, false, true, 2);
  return bad;
}
'''


def test_plan_and_room(tmp_path):
    (tmp_path / "main.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "main")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC), str(tmp_path / "main.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
