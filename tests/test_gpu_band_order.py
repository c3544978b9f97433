"""The banded batch adds every sum in one order, whatever the block size: an
instance's solution has the same bits from a 512-thread block (a QP per SM) and
from a 256-thread block (more QPs than SMs).  The iterates of an infeasible
instance diverge along a ray, so its certificate shows a change of rounding
anywhere in the iteration a million times enlarged."""

import numpy as np
import pytest
import torch

from qtqp_b200 import _lib, band, batch, problems

pytestmark = pytest.mark.gpu


def _solve(probs, num_sms, precision="fp64"):
  hb = band.HostBandBatch(probs, batch.SolveOptions(precision=precision), num_sms=num_sms)
  dev = band.DeviceBandBatch(hb, records=False)
  dev.upload()
  dev.launch()
  torch.cuda.synchronize()
  status = dev.results.cpu().numpy().view(_lib.RESULT_DTYPE)["status"].tolist()
  return (hb.plan.groups[0].block_threads, status,
          np.concatenate([v.cpu().numpy() for v in (dev.x, dev.y, dev.s)]))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_parametric_family(precision):
  fam = problems.parametric_mpc_family(24, 25, seed=1)
  probs = [band.BandProblem(*problems.parametric_mpc_instance(fam, i)) for i in range(24)]
  wide, st_wide, out_wide = _solve(probs, 0, precision)
  narrow, st_narrow, out_narrow = _solve(probs, 23, precision)
  assert (wide, narrow) == (512, 256)
  assert st_wide == st_narrow and len(set(st_wide)) > 1  # infeasible ones among them
  np.testing.assert_array_equal(out_wide, out_narrow)


@pytest.mark.parametrize("nx,nu", [(1, 1), (2, 1), (6, 3), (11, 11), (16, 1), (22, 20), (32, 1),
                                   (42, 41)])
def test_widths(nx, nu):
  """Half-bandwidths 2 to 124: one to four warps of owners in the solves."""
  a, z, p, _ = problems.mpc_structure(7, nx=nx, nu=nu, seed=nx)
  m, n = a.shape
  rng = np.random.default_rng([nx, nu])
  probs = []
  for _ in range(3):
    x = rng.uniform(-0.5, 0.5, size=n)
    b = a @ x + np.concatenate([np.zeros(z), rng.uniform(0.0, 1.0, size=m - z)])
    probs.append(band.BandProblem(a, b, rng.normal(size=n), z, p))
  assert probs[0].bw == 2 * nx + nu - 1
  wide, st_wide, out_wide = _solve(probs, 0)
  narrow, st_narrow, out_narrow = _solve(probs, 2)
  assert (wide, narrow) == (512, 256)
  assert st_wide == st_narrow
  np.testing.assert_array_equal(out_wide, out_narrow)
