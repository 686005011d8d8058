"""The decode step's choices by size (csrc/step_rules.h) at the sizes they were measured at."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "mycaffe_b200" / "csrc"


def holds(tmp_path, *claims):
    checks = "".join(f"  if (!({c})) {{ std::puts({('%s' % c)!r}); bad = 1; }}\n".replace("'", '"') for c in claims)
    (tmp_path / "main.cpp").write_text(f'#include "step_rules.h"\n#include <cstdio>\nusing namespace step_rules;\nint main() {{\n  int bad = 0;\n{checks}  return bad;\n}}\n')
    exe = str(tmp_path / "main")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC), str(tmp_path / "main.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_rows_are_asked_for_ahead_only_where_that_gains(tmp_path):
    rows = "2ll * {} * {} * {} * {}".format      # sequences, keys, width, bytes
    holds(tmp_path,
          f"!prefetch_rows(false, 7, false, 1, {rows(7, 4096, 4096, 4)})",   # a call of its own: nothing to wait for
          f"!prefetch_rows(false, 1, true, 1, {rows(1, 256, 384, 2)})",
          f"prefetch_rows(true, 1, false, 1, {rows(1, 256, 768, 4)})",       # in a step
          f"prefetch_rows(true, 8, false, 1, {rows(8, 2048, 4096, 4)})",
          f"prefetch_rows(true, 8, true, 1, {rows(8, 1024, 768, 2)})",
          f"!prefetch_rows(true, 1, true, 1, {rows(1, 2048, 4096, 2)})",     # rows that are too many beside the weights in L2
          f"!prefetch_rows(true, 1, true, 4, {rows(1, 32768, 1024, 2)})",
          f"prefetch_rows(true, 8, false, 4, {rows(8, 2048, 1024, 4)})",
          f"!prefetch_rows(true, 1, false, 4, {rows(1, 32768, 1024, 4)})",
          f"!prefetch_rows(true, 9, false, 1, {rows(9, 256, 768, 4)})")         # ordinary launches


def test_splits_are_combined_in_the_projection_for_one_sequence_and_few_of_them(tmp_path):
    holds(tmp_path,
          "combine_in_projection(1, 8, 768)", "combine_in_projection(1, 8, 2048)", "combine_in_projection(1, 2, 288)",
          "!combine_in_projection(1, 1, 768)",                                    # nothing to combine
          "!combine_in_projection(1, 9, 4096)", "!combine_in_projection(1, 37, 4096)",
          "!combine_in_projection(2, 2, 288)", "!combine_in_projection(8, 8, 768)", "!combine_in_projection(5, 7, 4096)")
