"""The large dense path's equilibration on badly scaled data at the edges of
its passes: rows shared by one and by several warps, more than 4096 columns, more
than 1024 rows per block, blocks without rows, and no P.  The solution has to
pass the reference's acceptance conditions (tests/kkt_checks.py) on the original
data."""

import numpy as np
import pytest
import scipy.sparse as sp

import qtqp_b200 as qb
from qtqp_b200 import problems
from tests import kkt_checks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,with_p", [(130, 15, True), (512, 700, True), (513, 600, False),
                                        (1100, 900, True), (4100, 40, True), (16, 160000, True)])
def test_badly_scaled(n, m, with_p):
  rng = np.random.default_rng(n + m)
  z = min(m // 8, n // 4)
  a = rng.normal(size=(m, n)) * 10.0 ** rng.uniform(-2, 2, size=n)
  a *= 10.0 ** rng.uniform(-2, 2, size=(m, 1))
  p = sp.csc_matrix(sp.diags(10.0 ** rng.uniform(-2, 2, size=n)) if with_p else (n, n))
  if not with_p:  # bounded: a box on every variable
    a = np.vstack([a[:m - 2 * (m // 4)], np.eye(n)[:m // 4], -np.eye(n)[:m // 4]])
  b, c = problems._feasible_pair(rng, a, p, z)
  q = qb.QTQP(a=sp.csc_matrix(a), b=b, c=c, z=z, p=p if with_p else None)
  sol = qb.solve_batch([q], storage="large")[0]
  kkt_checks.assert_status_certificate(sol, a, b, c, p, z)
  assert sol.status == qb.SolutionStatus.SOLVED
