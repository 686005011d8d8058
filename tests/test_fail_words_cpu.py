"""Host bookkeeping of the failure words (csrc/fail_words.h): a call on one device neither sees nor lowers what another device's
kernels raised."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "mycaffe_b200" / "csrc"

MAIN = r"""
#include "fail_words.h"
#include <cstdio>
#define CHECK(x) if (!(x)) { std::printf("%s\n", #x); return 1; }
int main() {
  int words[McaFailTable::SIZE] = {};
  McaFailTable t{words};
  for (int family = 0; family < 3; ++family) {
    const McaFailWord f = (McaFailWord)family, other = (McaFailWord)((family + 1) % 3);
    for (int a = 0; a < MCA_FAIL_DEVICES; a += 21) {
      const int b = (a + 1) % MCA_FAIL_DEVICES;
      t.row(a)[family] = 1;                                  // a kernel of device a failed
      CHECK(!t.raised(b, f) && !t.raised(a, other))          // a synchronous call on device b has nothing to read
      t.lower(b, f); t.lower(a, other);                      // and would not take the failure from device a's call
      CHECK(t.raised(a, f))
      t.lower(a, f);
      CHECK(!t.raised(a, f))
    }
  }
  return 0;
}
"""


def test_devices_keep_their_own_words(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC), str(tmp_path / "main.cpp"), "-o", str(tmp_path / "main")],
                   check=True)
    assert subprocess.run([str(tmp_path / "main")]).returncode == 0
