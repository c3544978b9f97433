"""The dense part of the supernodal plan (the last columns, factorised as one
dense matrix) where it can go wrong: fewer columns than one 128-column block,
exactly one and two blocks, one column more or less, and several blocks.  On
the CPU, the plan's structure and the numpy replay of its factorisation
against a dense Cholesky; on the GPU, the whole solve against the oracle's
sparse LU, with the sparse path's criteria."""

import functools

import numpy as np
import pytest
import scipy.sparse as sp

import qtqp_b200 as qb
from oracle import qtqp_oracle as orc
from qtqp_b200 import problems, sparse
from tests import kkt_checks
from tests import sparse_plan_check as spc

COLS = [70, 127, 128, 129, 256, 257, 450]
LEAVES = 300


def _qp(k):
  """One row of A over k variables, 300 more variables, each in a row of its
  own with two of the k, and a bound on every variable."""
  rng = np.random.default_rng(k)
  n, z = k + LEAVES, 5
  a = sp.lil_matrix((LEAVES + 1 + n, n))
  for i in range(LEAVES):
    a[i, k + i] = 1.0 + rng.random()
    a[i, rng.choice(k, 2, replace=False)] = rng.normal(size=2)
  a[LEAVES, :k] = rng.normal(size=k) / np.sqrt(k)
  a[LEAVES + 1:, :] = sp.eye(n)
  a = sp.csc_matrix(a)
  p = sp.csc_matrix(sp.diags(0.1 + rng.random(n)))
  b, c = problems._feasible_pair(rng, a, p, z)
  return a, b, c, z, p


@functools.lru_cache(maxsize=None)
def _problem(cols):
  """The first of the QPs around k = cols whose dense part has cols columns."""
  for k in range(cols - 20, cols + 12):
    q = _qp(k)
    plan = sparse.SparsePlan(q[0], q[4])
    if plan.desc.dense_cols == cols:
      return q, plan
  raise AssertionError(f"no plan with {cols} dense columns")


@pytest.mark.parametrize("cols", COLS)
def test_plan_with_a_dense_part(cols):
  (a, _, _, _, p), plan = _problem(cols)
  n, c0 = a.shape[1], a.shape[1] - plan.desc.dense_cols
  first, top_ptr = plan.section("first"), plan.section("top_ptr")
  top_list, top_upd = plan.section("top_list"), plan.section("top_upd")
  upd_ptr = plan.section("upd_ptr")
  # Whole supernodes, exactly the ones of the last levels.
  t0 = int(np.searchsorted(first, c0))
  assert first[t0] == c0
  level = int(np.searchsorted(top_ptr, len(top_list) - (len(first) - 1 - t0)))
  assert sorted(top_list[top_ptr[level]:]) == list(range(t0, len(first) - 1))
  counts = [sum(upd_ptr[s + 1] - upd_ptr[s] for s in top_list[u:v])
            for u, v in zip(top_ptr[:-1], top_ptr[1:])]
  assert top_upd.tolist() == np.concatenate([[0], np.cumsum(counts)]).tolist()
  d = np.random.default_rng(0).uniform(0.5, 2.0, size=a.shape[0])
  g = (a.T @ (d[:, None] * a.toarray())) + np.eye(n) + p.toarray()
  gp = g[np.ix_(plan.perm, plan.perm)]
  lower = spc.dense_factor(plan, spc.factor(plan, gp))
  np.testing.assert_allclose(lower, np.linalg.cholesky(gp), rtol=0, atol=1e-10)


@pytest.mark.gpu
@pytest.mark.parametrize("cols", COLS)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_solve_with_a_dense_part(cols, precision):
  (a, b, c, z, p), _ = _problem(cols)
  q = qb.QTQP(a=a, b=b, c=c, z=z, p=p)
  sol = qb.solve_batch([q], storage="sparse", precision=precision, collect_stats=True)[0]
  ref = orc.solve(a, b, c, z, p, backend="superlu")
  assert sol.status.value == ref.status
  kkt_checks.assert_status_certificate(sol, a, b, c, p, z)
  assert kkt_checks.objective_rel_err(sol.x, ref.x, c, p) <= 1e-6
  if precision == "fp64":
    assert abs(len(sol.stats) - len(ref.stats)) <= 1
