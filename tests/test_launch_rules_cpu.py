"""When a kernel lets the one behind it go (csrc/launch_rules.h), at the sizes it was measured at."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "mycaffe_b200" / "csrc"

CLAIMS = (
    "!delta_lets_go_late(48, 300, 64, true)", "!delta_lets_go_late(24, 384, 128, true)",          # up to three tiles a head
    "delta_lets_go_late(12, 1024, 128, true)", "delta_lets_go_late(4, 900, 128, false)",
    "delta_lets_go_late(12, 1024, 64, true)", "delta_lets_go_late(8, 1500, 64, true)", "delta_lets_go_late(20, 900, 64, true)",
    "delta_lets_go_late(24, 900, 64, true)", "delta_lets_go_late(4, 2500, 64, true)",
    "!delta_lets_go_late(12, 512, 64, true)", "!delta_lets_go_late(16, 900, 64, true)", "!delta_lets_go_late(8, 5162, 64, true)",
    "!delta_lets_go_late(12, 1500, 64, true)", "!delta_lets_go_late(12, 2500, 64, true)", "!delta_lets_go_late(96, 1024, 64, true)",
    "delta_lets_go_late(8, 2048, 64, false)", "delta_lets_go_late(8, 1024, 64, false)", "delta_lets_go_late(24, 400, 64, false)",
    "!delta_lets_go_late(8, 900, 64, false)", "!delta_lets_go_late(16, 400, 64, false)", "!delta_lets_go_late(12, 640, 64, false)",
    "pack_lets_go(7, 358, 64, true)", "pack_lets_go(8, 800, 64, true)", "pack_lets_go(8, 600, 128, true)", "pack_lets_go(16, 450, 128, false)",
    "!pack_lets_go(64, 256, 64, true)", "!pack_lets_go(8, 1024, 64, true)", "!pack_lets_go(8, 1024, 128, true)", "!pack_lets_go(24, 384, 128, true)",
    "!pack_lets_go(7, 800, 128, true)", "!pack_lets_go(8, 1100, 128, false)",
    # the shapes of test_launch_rules_gpu.py lie on both sides
    "pack_lets_go(7, 358, 64, true) && !pack_lets_go(40, 200, 64, true) && pack_lets_go(5, 300, 128, true) && !pack_lets_go(11, 600, 128, true)",
    "!delta_lets_go_late(9, 520, 64, true) && delta_lets_go_late(16, 600, 64, true) && delta_lets_go_late(10, 900, 64, false)",
)


def test_signals(tmp_path):
    checks = "".join('  if (!(%s)) { std::puts("%s"); bad = 1; }\n' % (c, c) for c in CLAIMS)
    (tmp_path / "main.cpp").write_text(f'#include "launch_rules.h"\n#include <cstdio>\nusing namespace launch_rules;\nint main() {{\n  int bad = 0;\n{checks}  return bad;\n}}\n')
    exe = str(tmp_path / "main")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC), str(tmp_path / "main.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
