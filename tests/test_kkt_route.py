"""The dense KKT backend's choice between one block and the whole GPU: the latter
only where the current device holds its blocks at once."""

import os
import shutil
import subprocess

import pytest

from qtqp_b200 import build

SOURCE = r"""
#include <cstdio>
#include "kkt_grid.cuh"
int main() {
  const int n[] = {1, 79, 80, 300, 18944, 18945}, r[] = {0, 74, 147, 148, 296};
  for (int a : n)
    for (int b : r) printf("%d %d %d\n", a, b, int(qtqp::kkt_grid_route(a, b)));
}
"""


def test_whole_gpu_form_only_where_it_is_resident(tmp_path):
  nvcc = build._nvcc()  # pylint: disable=protected-access
  if shutil.which(nvcc) is None and not os.path.exists(nvcc):
    pytest.skip("no nvcc")
  src = tmp_path / "route.cu"
  src.write_text(SOURCE)
  exe = tmp_path / "route"
  subprocess.run([nvcc, *build.ARCH_FLAGS, "-std=c++17", "--expt-relaxed-constexpr", "-I",
                  build._INC, "-I", build._CSRC, str(src), "-o", str(exe)],  # pylint: disable=protected-access
                 check=True, capture_output=True)
  out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
  rows = [tuple(int(v) for v in line.split()) for line in out.splitlines()]
  assert len(rows) == 30
  for n, resident, route in rows:
    assert route == int(80 <= n <= 128 * 148 and resident >= 148), (n, resident)
