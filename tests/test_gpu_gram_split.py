"""The FP64 Gram matrix of the large dense path where its split over the CTAs
can go wrong: rows of A that start on 16 bytes or not, row counts around the
slices of 32 rows and their smallest number, one tile in many parts, parts that
end inside a tile, and more tiles than CTAs.  The solve against the oracle, with
the large path's criteria."""

import numpy as np
import pytest
import scipy.sparse as sp

import qtqp_b200 as qb
from oracle import qtqp_oracle as orc
from qtqp_b200 import problems
from tests import kkt_checks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(129, 131), (130, 160), (256, 33), (257, 32), (384, 31),
                                 (254, 1025), (640, 1300), (641, 1296), (2050, 260)])
def test_large_solve_sizes(n, m):
  rng = np.random.default_rng(1000 * n + m)
  z = m // 8
  a = rng.normal(size=(m, n))
  l = rng.normal(size=(n, 8))
  p = l @ l.T + 0.1 * np.eye(n)
  b, c = problems._feasible_pair(rng, a, p, z)
  q = qb.QTQP(a=sp.csc_matrix(a), b=b, c=c, z=z, p=sp.csc_matrix(p))
  sol = qb.solve_batch([q], storage="large", precision="fp64", collect_stats=True)[0]
  ref = orc.solve(sp.csc_matrix(a), b, c, z, sp.csc_matrix(p), backend="dense")
  assert sol.status.value == ref.status
  kkt_checks.assert_status_certificate(sol, a, b, c, p, z)
  assert kkt_checks.objective_rel_err(sol.x, ref.x, c, p) <= 1e-6
  assert abs(len(sol.stats) - len(ref.stats)) <= 1
