"""Banded QPs whose CSR rows and CSC columns are stored in any order, and with
repeated entries (the value and a zero, so that the scalings stay the same): the
Gram matrix, and so the solution, must not depend on it."""

import numpy as np
import pytest
import torch

from qtqp_b200 import _lib, band, batch, problems

pytestmark = pytest.mark.gpu

# A shuffled row changes the order of some sums: rounding, enlarged by the
# condition of a KKT system solved to 1e-9 and better.
RTOL = 1e-9


def _problem(repeat, shuffle, seed=5):
  """The T = 6 MPC QP with its stored entries rearranged."""
  a, b, c, z, p = problems.mpc_feasible(6, seed=seed)
  pr = band.BandProblem(a, b, c, z, p)
  rng = np.random.default_rng(seed)

  def rearrange(mat):
    ptr, idx, val = [0], [], []
    for i in range(mat.indptr.size - 1):
      lo, hi = mat.indptr[i], mat.indptr[i + 1]
      ii, vv = mat.indices[lo:hi], mat.data[lo:hi]
      if repeat and ii.size:
        again = rng.integers(0, ii.size, size=2)
        ii, vv = np.concatenate([ii, ii[again]]), np.concatenate([vv, np.zeros(2)])
      if shuffle:
        order = rng.permutation(ii.size)
      else:
        order = np.argsort(ii, kind="stable")
      idx.append(ii[order])
      val.append(vv[order])
      ptr.append(ptr[-1] + ii.size)
    out = mat.copy()
    out.indptr = np.array(ptr, dtype=mat.indptr.dtype)
    out.indices = np.concatenate(idx).astype(mat.indices.dtype)
    out.data = np.concatenate(val)
    return out

  if repeat or shuffle:
    pr.a, pr.at = rearrange(pr.a), rearrange(pr.at)
  return pr


def _solve(pr, whole_gpu):
  host = band.HostBandBatch([pr], batch.SolveOptions())
  dev = (band.DeviceBandGrid if whole_gpu else band.DeviceBandBatch)(host, records=False)
  dev.upload()
  dev.launch()
  torch.cuda.synchronize()
  res = (dev.result if whole_gpu else dev.results).cpu().numpy().view(_lib.RESULT_DTYPE)
  assert int(res["error"][0]) == 0
  return int(res["status"][0]), [v.cpu().numpy() for v in (dev.x, dev.y, dev.s)]


@pytest.mark.parametrize("whole_gpu", [False, True])
@pytest.mark.parametrize("repeat,shuffle", [(False, True), (True, False), (True, True)])
def test_any_order(repeat, shuffle, whole_gpu):
  status, want = _solve(_problem(False, False), whole_gpu)
  got_status, got = _solve(_problem(repeat, shuffle), whole_gpu)
  assert got_status == status
  for u, v in zip(got, want):
    assert np.linalg.norm(u - v) <= RTOL * np.linalg.norm(v)
