"""32-bit offsets of the field arenas at the largest grid a context accepts
(host check of the index arithmetic in cc_common.h, compiled with the host
compiler): every offset within one field array, or within one direction of the
face arena, is below 2^31, and the directions of the face arena start at 64-bit
offsets that keep the last flux inside it.  With nine species the arena of
three directions passes 2^31 values from 51 million points on, and 97 million
are accepted."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <initializer_list>
#include "cc_common.h"
using namespace ccb;
int main() {
  int64_t N = 32;
  while (arena_fits(N + 32)) N += 32;  // the largest arena: a multiple of 32 points
  if (arena_fits(N + 32) || N < 97000000) return 1;
  const int64_t lim = (int64_t)1 << 31;
  bool passes_lim = false;
  for (int ns = 0; ns <= kMaxSpec; ++ns)
    for (int elem : {4, 8}) {
      const int nv = 5 + ns, stride = face_stride(nv, elem);
      const int64_t total = 3 * (int64_t)stride * N;
      // primitives, geometry (13 fields in FP32), and one direction of the faces:
      // FP64 l N + p; FP32 group g at 4 g N, four (or two) values a point
      if ((6 + ns) * N > lim || 13 * N > lim) return 2;
      const int64_t inner = elem == 8 ? (int64_t)(nv - 1) * N : (int64_t)4 * ((nv - 1) / 4) * N;
      if (inner >= lim) return 3;
      for (int d = 0; d < 3; ++d) {
        const int64_t at = face_base(d, nv, elem, (int)N);
        if (at != d * (int64_t)stride * N) return 4;
        const int width = elem == 8 ? 1 : (nv - (nv - 1) / 4 * 4 > 2 ? 4 : 2);
        if (at + inner + (int64_t)width * N > total) return 5;  // the last group of the last point
        passes_lim = passes_lim || at >= lim;
      }
    }
  return passes_lim ? 0 : 6;  // the case that 32-bit direction offsets would miss is among them
}
"""


def test_offsets_at_the_largest_arena(tmp_path):
    src, exe = tmp_path / "offsets.cpp", tmp_path / "offsets"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "combustioncodegpu_b200", "csrc"), "-o",
                    str(exe), str(src)], check=True, timeout=120)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
