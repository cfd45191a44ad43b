"""Thread indices at the largest vertex counts, computed on the host by the
kernels' own functions."""
import os
import subprocess

import pytest

PROGRAM = r"""
#include <cstdio>
#include "sprg_internal.h"
template <int LANES>
bool check(long V) {
  const long blocks = (V * LANES + 255) / 256;
  if (blocks > 0x7fffffff) return false;
  const long some[] = {0, 1, blocks / 2, (1l << 31) / 256 - 1, (1l << 31) / 256, blocks - 2, blocks - 1};
  for (long b : some)
    for (int t = 0; t < 256; ++t) {
      if (b < 0 || b >= blocks) continue;
      const sprg::VertexLane vl = sprg::vertex_lane<LANES>((unsigned)b, 256, t);
      const __int128 i = (__int128)b * 256 + t;
      if (vl.v != (long)(i / LANES) || vl.lane != (int)(i % LANES) || vl.v < 0) return false;
    }
  return true;
}
int main() {
  for (long V : {1l, 127l, 129l, (1l << 30) - 1, (1l << 30) + 1, (1l << 31) - 1})
    if (!check<1>(V) || !check<2>(V) || !check<4>(V)) {
      printf("V = %ld\n", V);
      return 1;
    }
  return 0;
}
"""


def test_vertex_lanes(tmp_path):
    from core_gb300 import build
    nvcc = build._nvcc()
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src = tmp_path / "lanes.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "lanes"
    subprocess.run([nvcc, "-std=c++17", "-I" + build.CSRC, "-I" + os.path.join(build.ROOT, "include"), str(src), "-o",
                    str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
