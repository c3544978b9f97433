"""The ring of count slots in the supernodal update step (sparse_grid.cuh): no
slot is cleared by one thread while another may still count in it or read it.

The slots come from the kernel's own functions, compiled for the host; the
schedule below restates the barriers around them.  Between two block barriers the
threads run in any order, so an access and a clearing of one slot between the same
two barriers is a race."""

import os
import shutil
import subprocess

import pytest

from qtqp_b200 import build

SOURCE = r"""
#include <cstdio>
#include "sparse_grid.cuh"
int main() {
  for (int i = 0; i < 12; ++i) printf("%d %d\n", qtqp::sn_count_slot(i), qtqp::sn_clear_slot(i));
}
"""


@pytest.fixture(scope="module")
def slots(tmp_path_factory):
  tmp_path = tmp_path_factory.mktemp("ring")
  nvcc = build._nvcc()  # pylint: disable=protected-access
  if shutil.which(nvcc) is None and not os.path.exists(nvcc):
    pytest.skip("no nvcc")
  src = tmp_path / "slots.cu"
  src.write_text(SOURCE)
  exe = tmp_path / "slots"
  subprocess.run([nvcc, *build.ARCH_FLAGS, "-std=c++17", "--expt-relaxed-constexpr", "-I",
                  build._INC, "-I", build._CSRC, str(src), "-o", str(exe)],  # pylint: disable=protected-access
                 check=True, capture_output=True)
  out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
  return [tuple(int(v) for v in line.split()) for line in out.splitlines()]


@pytest.mark.parametrize("entries", [1, 2, 3, 4, 12])
def test_no_race_on_the_count_slots(entries, slots):
  # (epoch, slot, what): an epoch is the time between two block barriers.
  events, epoch = [(0, s, "clear") for s in range(3)], 1  # the chunk's start, a barrier

  def prepare(i):
    nonlocal epoch
    count, clear = slots[i]
    events.append((epoch, count, "count"))
    epoch += 1  # the count barrier
    events.append((epoch, count, "read"))
    events.append((epoch, clear, "clear"))

  prepare(0)
  for i in range(entries):
    if i + 1 < entries:
      prepare(i + 1)
    epoch += 1  # the copies of entry i have landed
  for e, slot, what in events:
    if what == "clear":
      assert not any(e == e2 and slot == s2 and w2 != "clear" for e2, s2, w2 in events), (e, slot)
    elif what == "count":
      # Zero since the last use: cleared after that use's reads, before this count.
      reads = [e2 for e2, s2, w2 in events if s2 == slot and w2 == "read" and e2 < e]
      clears = [e2 for e2, s2, w2 in events if s2 == slot and w2 == "clear" and e2 < e]
      assert clears and (not reads or max(clears) > max(reads)), (e, slot)
