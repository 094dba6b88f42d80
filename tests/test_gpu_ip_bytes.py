"""The initial place's scratch, by which the server admits jobs, at the block
cap that the initial place takes on this device: a host program on the
library's own functions, at sizes around the steps of the block layout."""

import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include "gpl_internal.h"
int main() {
  int sm = 0, above_eight = 0, bad = 0;
  if (cudaSetDevice(0) != cudaSuccess) return 2;
  cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, 0);
  const int cap = gpl::initial_place_grid_cap(sm);
  for (int n = 1; n < 3000000; n = n * 17 / 16 + 1) {
    gpl::HostModel m;
    m.place_insts.resize(n);
    for (int i = 0; i < n; i++) m.place_insts[i] = i;
    m.inst_pin_start.assign(n + 1, 0);
    m.net_start.assign(1, 0);
    const size_t need = gpl::initial_place_bytes_at(m, cap);
    bad += gpl::initial_place_bytes(m, sm) < need;
    above_eight += gpl::initial_place_bytes_at(m, 8 * sm) < need;
  }
  printf("cap %d: %d sizes below the need; %d with eight blocks an SM\n", cap, bad, above_eight);
  return bad != 0;
}
"""


def test_scratch_bound_is_that_of_the_grid_taken(gpu_lib, tmp_path):
    from replace_gb300 import build
    src, exe = tmp_path / "bytes.cpp", tmp_path / "bytes"
    src.write_text(PROGRAM)
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    cmd = [build.nvcc(), "-O1", "-std=c++17", "-I", build.CSRC, "-I", cuda, str(src), build.LIB, "-cudart", "static",
           "-Xlinker", "-rpath," + os.path.dirname(build.LIB), "-o", str(exe)]
    subprocess.check_call(cmd)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
