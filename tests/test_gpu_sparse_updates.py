"""The left-looking updates of the supernodal factorisation at the edges of
their staging: an update list longer than one chunk of 256 descendants,
descendants with more rows than two per thread (512) and with rows of one
supernode only, and single-column descendants beside 64-column ones.  The
solve against the oracle's sparse LU, with the sparse path's criteria."""

import numpy as np
import pytest
import scipy.sparse as sp

import qtqp_b200 as qb
from oracle import qtqp_oracle as orc
from qtqp_b200 import problems, sparse
from tests import kkt_checks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,leaves,wide", [(40, 300, 0), (90, 600, 2), (560, 40, 3)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_update_lists(k, leaves, wide, precision):
  """One row of A over k variables; `leaves` rows that add a variable each and
  two of the first 20; `wide` rows that add a variable each and all k."""
  rng = np.random.default_rng(1000 * k + leaves)
  n, z = k + leaves + wide, 5
  a = sp.lil_matrix((1 + leaves + wide + n, n))
  a[0, :k] = rng.normal(size=k) / np.sqrt(k)
  for i in range(leaves):
    a[1 + i, k + i] = 1.0 + rng.random()
    a[1 + i, rng.choice(20, 2, replace=False)] = rng.normal(size=2)
  for i in range(wide):
    a[1 + leaves + i, k + leaves + i] = 1.0 + rng.random()
    a[1 + leaves + i, :k] = rng.normal(size=k) / np.sqrt(k)
  a[1 + leaves + wide:, :] = sp.eye(n)
  a = sp.csc_matrix(a)
  p = sp.csc_matrix(sp.diags(0.1 + rng.random(n)))
  b, c = problems._feasible_pair(rng, a, p, z)
  plan = sparse.SparsePlan(a, p)
  longest = np.diff(plan.section("upd_ptr")).max()
  assert longest > 256 if leaves > 256 else plan.desc.max_rows > 512
  q = qb.QTQP(a=a, b=b, c=c, z=z, p=p)
  sol = qb.solve_batch([q], storage="sparse", precision=precision, collect_stats=True)[0]
  ref = orc.solve(a, b, c, z, p, backend="superlu")
  assert sol.status.value == ref.status
  kkt_checks.assert_status_certificate(sol, a, b, c, p, z)
  assert kkt_checks.objective_rel_err(sol.x, ref.x, c, p) <= 1e-6
  if precision == "fp64":
    assert abs(len(sol.stats) - len(ref.stats)) <= 1
