"""The check that lets a kernel store into a host vector (pdg_hostmap.h), on the
CPU: two registered ranges, a gap between them, and a read-only one."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dune-pdelab_gb300", "csrc")

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "pdg_hostmap.h"
using namespace pdg;
struct Range { uintptr_t start; size_t size; bool writable; };
// host and device addresses are the same, as with unified addressing
static const Range ranges[] = {{0x10000, 0x4000, true}, {0x18000, 0x4000, true},
                               {0x1c000, 0x2000, false}};
static uintptr_t map(uintptr_t p, size_t bytes) {
  for (const Range &r : ranges)
    if (p >= r.start && p < r.start + r.size)
      return mapped_range(HostMapping{true, r.writable, p, r.start, r.size}, bytes);
  return mapped_range(HostMapping{false, true, p, 0, 0}, bytes);
}
static int check(const char *what, uintptr_t got, uintptr_t want) {
  if (got == want) return 0;
  std::printf("%s: %#zx\n", what, (size_t)got);
  return 1;
}
int main() {
  int bad = 0;
  bad += check("whole range", map(0x10000, 0x4000), 0x10000);
  bad += check("inside", map(0x10008, 0x3ff8), 0x10008);
  bad += check("one byte over", map(0x10008, 0x3ff9), 0);
  bad += check("across a gap, both ends registered", map(0x10000, 0x9000), 0);
  bad += check("across two adjacent ranges", map(0x1b000, 0x2000), 0);
  bad += check("read-only", map(0x1c000, 0x1000), 0);
  bad += check("not registered", map(0x15000, 0x8), 0);
  bad += check("last value", map(0x1bff8, 8), 0x1bff8);
  bad += check("device address below the range",
               mapped_range(HostMapping{true, true, 0x0fff8, 0x10000, 0x4000}, 8), 0);
  bad += check("size that wraps", map(0x10008, ~(size_t)0), 0);
  return bad;
}
"""


def test_mapped_range(tmp_path):
    (tmp_path / "main.cc").write_text(MAIN)
    exe = tmp_path / "hostmap"
    r = subprocess.run(["g++", "-std=c++17", "-Wall", "-I", CSRC, str(tmp_path / "main.cc"), "-o",
                        str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
