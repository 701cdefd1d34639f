"""Rules that host and device share, called on the CPU: a small program built
from the kernels' header."""
import subprocess

from ibfs_b200 import build

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "bfs_device.cuh"
using namespace ibfs;
static int bad = 0;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); bad = 1; } } while (0)
int main() {
@CHECKS@
  return bad;
}
"""


def run_checks(tmp_path, checks):
    src, exe = tmp_path / "rules.cu", tmp_path / "rules"
    src.write_text(PROGRAM.replace("@CHECKS@", checks))
    subprocess.run([build._nvcc(), *build.ARCH, "-O1", "-std=c++17", "--expt-relaxed-constexpr",
                    f"-I{build.CSRC}", f"-I{build.INCLUDE}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0, r.stdout


def test_level_kind(tmp_path):
    """Only a top-down level keeps a touched list or leaves its marks to a
    sweep; a bottom-up pass marks the bitmap whatever its frontier."""
    run_checks(tmp_path, """
  const long long V = 8 << 20;
  const unsigned long long mf[] = {0, 1, 1 << 20, (1 << 20) + 1, 3 << 20, 4 << 20, 1ull << 33};
  const int td[] = {kTdThin, kTdThin, kTdThin, kTdBitmap, kTdBitmap, kTdWide, kTdWide};
  for (int i = 0; i < 7; i++) {
    CHECK(level_kind(kDirTD, mf[i], V) == td[i]);
    CHECK(level_kind(kDirBU, mf[i], V) == kTdBitmap);
  }
""")


def test_long_lists_run_top_down(tmp_path):
    """A degree that 32-bit list positions do not hold turns every level
    top-down, whatever switch level was asked for; other graphs keep theirs."""
    run_checks(tmp_path, """
  for (int sw : {-1, 0, 3, 1000}) {
    for (long long d : {0ll, 33ll, 0x7FFFF000ll}) CHECK(switch_level_for(sw, d) == sw);
    for (long long d : {0x7FFFF001ll, 0x7FFFFFFFll, 0x80000000ll, 0x100000010ll}) {
      const int s = switch_level_for(sw, d);
      for (int level : {1, 2, 65535})
        CHECK(choose_dir(level, kDirTD, s, 4.0f, 24.0f, 9, 1, 1ull << 40, 1, 10) == kDirTD);
    }
  }
  CHECK(kListMax + 128 <= 0x7FFFFFFF);
""")
