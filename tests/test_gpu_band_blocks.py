"""The blocked band factorisation and solves at half-bandwidths around their
block sizes (8-column panels, 8 x 8 tiles of the window, solve blocks of 1 to
32 columns whose inverses live inside the band), for one QP per 512-thread
block, per 256-thread block (more QPs than SMs) and on the whole GPU, with
column counts that leave partial blocks.

Criteria of the other path tests: the oracle's status, the reference's
acceptance conditions, objective relative error <= 1e-6, FP64 iteration counts
within one."""

import numpy as np
import pytest
import scipy.sparse as sp

import qtqp_b200 as qb
from oracle import qtqp_oracle as orc
from tests import kkt_checks

pytestmark = pytest.mark.gpu

OBJ_TOL = 1e-6


def _banded(bw, n, seed):
  """Rows of up to four entries within bw + 1 columns, the widest span taken;
  bounds on every variable; diagonal P."""
  rng = np.random.default_rng([seed, bw, n])
  rows, cols = [], []
  m_band = n
  for r in range(m_band):
    lo = min(r, n - 1 - bw) if r < n - bw else rng.integers(0, n - bw)
    span = {lo, lo + bw} | set((lo + rng.integers(0, bw + 1, size=2)).tolist())
    rows += [r] * len(span)
    cols += sorted(span)
  a = sp.csc_matrix((rng.normal(size=len(rows)), (rows, cols)), shape=(m_band, n))
  a = sp.csc_matrix(sp.vstack([a, sp.eye(n)]))
  m, z = a.shape[0], n // 5
  p = sp.csc_matrix(sp.diags(rng.uniform(0.2, 1.0, size=n)))
  x0 = rng.normal(size=n)
  y0 = np.concatenate([rng.normal(size=z), np.zeros(m - z)])
  tight = rng.random(m - z) < 0.2
  y0[z:] = np.where(tight, 0.1 + np.abs(rng.normal(size=m - z)), 0.0)
  s0 = np.concatenate([np.zeros(z), np.where(tight, 0.0, 0.1 + rng.random(m - z))])
  return a, a @ x0 + s0, -(p @ x0 + a.T @ y0), z, p


def _check(sol, q, ref, fp64=True):
  assert sol.status.value == ref.status == "solved"
  kkt_checks.assert_solved(sol, q.a, q.b, q.c, q.p, q.z)
  assert kkt_checks.objective_rel_err(sol.x, ref.x, q.c, q.p) <= OBJ_TOL
  if fp64:
    assert abs(len(sol.stats) - len(ref.stats)) <= 1


@pytest.mark.parametrize("bw", [1, 2, 3, 6, 7, 8, 14, 15, 16, 30, 31, 32, 47, 63, 99, 118, 126])
def test_band_widths(bw):
  n = max(101, 4 * (bw + 1) + 13)
  a, b, c, z, p = _banded(bw, n, 1)
  q = qb.QTQP(a=a, b=b, c=c, z=z, p=p)
  assert q.band_problem().bw == bw
  ref = orc.solve(a, b, c, z, p, backend="superlu")
  _check(qb.solve_batch([q], storage="band", collect_stats=True)[0], q, ref)
  _check(qb.solve_batch([q], storage="band", precision="mixed")[0], q, ref, fp64=False)
  if bw <= 118:
    _check(qb.solve_batch([q], storage="band_grid", collect_stats=True)[0], q, ref)


@pytest.mark.parametrize("bw", [4, 31, 99])
def test_more_qps_than_sms(bw):
  n = max(101, 4 * (bw + 1) + 5)
  a, b, c, z, p = _banded(bw, n, 2)
  q = qb.QTQP(a=a, b=b, c=c, z=z, p=p)
  ref = orc.solve(a, b, c, z, p, backend="superlu")
  sols = qb.solve_batch([q] * 150, storage="band", collect_stats=True)
  for sol in sols:
    np.testing.assert_array_equal(sol.x, sols[0].x)
  _check(sols[0], q, ref)


def test_entries_stored_twice():
  """A CSC matrix may store an entry twice (their sum is the entry): here
  every seventh entry is split in two equal parts, which leaves the products
  exact."""
  from qtqp_b200 import band, batch
  bw, n = 20, 130
  a, b, c, z, p = _banded(bw, n, 3)
  a.sort_indices()
  reps = np.where(np.arange(a.nnz) % 7 == 3, 2, 1)
  ptr = np.concatenate([[0], np.cumsum(np.add.reduceat(reps, a.indptr[:-1]))])
  twice = sp.csc_matrix((np.repeat(a.data / reps, reps), np.repeat(a.indices, reps), ptr),
                        shape=a.shape)
  assert twice.nnz > a.nnz and abs(twice - a).max() == 0
  opts = batch.SolveOptions(equilibrate=False)
  outs = []
  for mat in (a, twice):
    hb = band.HostBandBatch([band.BandProblem(mat, b, c, z, p)], opts)
    for dev in (band.DeviceBandBatch(hb), band.DeviceBandGrid(hb)):
      dev.upload()
      dev.launch()
      res, x, *_ = dev.fetch()
      assert res["status"][0] == 0
      outs.append(x.copy())
  # The same QP: solutions agree to the solver's tolerance on its objective.
  for x in outs[1:]:
    assert kkt_checks.objective_rel_err(x, outs[0], c, p) <= OBJ_TOL
