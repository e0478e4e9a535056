"""The rule that decides on a plan's window layout, compiled for the host: record
sizes whose total does not fit in 32 bits are refused."""
import os
import subprocess

from sciwasm.sparse_b200 import build

PROGRAM = r"""
#include <cstdio>
#include "sb_spts_window.cuh"
using namespace sb::win;
// The decision for ngroups full groups of rows with k off-diagonal entries.
static int wins(long long ngroups, int k, int tsize, long long cap, int reach) {
  Info f = {};
  f.reach = reach;
  f.kmax = k;
  f.rows = f.widest = 1;
  f.size16 = ngroups * record16(kGroup, k, tsize);
  return window_wins(f, (int)ngroups, 1 << 24, cap, tsize, true);
}
int main() {
  const long long most = 2147483647LL / 2;  // 16-byte units, as the analysis caps them
  // 215M FP64 and 358M FP32 rows of up to 14 entries: more than 2^31 units
  std::printf("%d %d ", wins(215000032LL / 32, 14, 8, most, 1000),
              wins(358000000LL / 32, 14, 4, most, 1000));
  // more than 2^32: the low 32 bits alone would be small
  std::printf("%d ", wins((1LL << 32) / 320 + 1, 14, 8, most, 1000));
  // within the cap: taken; one group above it: refused
  std::printf("%d %d ", wins(most / 320, 14, 8, most, 1000), wins(most / 320 + 1, 14, 8, most, 1000));
  std::printf("%d %d\n", wins(100, 14, 8, most, 28700), wins(100, 14, 8, most, 2147483647));
}
"""


def test_sizes_past_32_bits_are_refused(tmp_path):
    src, exe = tmp_path / "rule.cu", tmp_path / "rule"
    src.write_text(PROGRAM)
    csrc = os.path.join(build.HERE, "csrc")
    subprocess.run([build.nvcc_path(), "-std=c++17", *build.ARCH, "-I", csrc, "-I",
                    os.path.join(build.ROOT, "include"), "-o", exe, src], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0", "0", "0", "1", "0", "1", "0"]
