"""The internal status words of rows that one kernel leaves to the next (csrc/row_status.h), on the CPU: whichever of them a row
carries, a cluster that gives up after an expired wait turns it into DS41_B200_ROW_TIMEOUT and never lets it reach the caller."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "deepseek-v4.1-flash-pro6000_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include <cstdio>
#include "row_status.h"
int main() {
  for (int status = -12; status <= 15; ++status)
    std::printf("%d %d %d %d\n", status, int(ds41::handed_on(status)), ds41::after_timeout(status, true),
                ds41::after_timeout(status, false));
}
"""


def test_rows_left_over_when_a_wait_expires(tmp_path):
    src, exe = tmp_path / "status.cpp", tmp_path / "status"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-I", os.path.join(CUDA, "include"),
                    "-o", str(exe), str(src)], check=True)
    lines = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")[:-1]
    table = {int(f[0]): tuple(map(int, f[1:])) for f in (l.split() for l in lines)}
    internal = {s for s, (handed, _, _) in table.items() if handed}
    assert internal == {-8, -9}
    for status, (_, left_over, every) in table.items():
        assert every == -5                                   # a launch over all rows: none of the rest is decided
        assert left_over == (-5 if status in internal else status)


def test_every_comparison_goes_through_the_header():
    """No kernel compares a status with one of the internal words by itself (the statistics mode once knew only one of the two)."""
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            code = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
            assert not re.search(r"[!=]=\s*-\s*[89]\b|==\s*kNeedsCluster", code), name
