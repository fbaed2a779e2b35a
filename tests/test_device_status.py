"""What the library makes of a scenario's device status, from its own header (no GPU): every
value that leaves cells without their update, or not finite, has to fail the call."""
import subprocess

from storm_b200 import build

MAIN = r"""
#include <cstdio>
#include "storm_internal.h"
int main() {
  for (int s = 0; s < 8; s++) {
    const char* w = storm::status_failure(s);
    std::printf("%s\n", w ? w : "");
  }
}
"""


def test_status_values(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-I", build.CSRC, "-o", str(tmp_path / "main"), str(tmp_path / "main.cpp")],
                   check=True)
    out = subprocess.run([str(tmp_path / "main")], check=True, capture_output=True, text=True).stdout.split("\n")
    assert out[0] == out[2] == ""
    assert all("non-finite" in out[s] for s in (1, 3))
    assert all("did not arrive" in out[s] for s in (4, 5, 6, 7))
