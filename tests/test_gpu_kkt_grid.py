"""The KKT backend around the size where it changes from one block to the
whole GPU (n = 80) and around the 128-row blocks of that form: products
against numpy, refined solutions by the reference's test_direct_linear_solver
criterion (residual <= 1e-10), repeated solves and factorisations of one
object, the FP32 factor, and the pivot of an indefinite system."""

import numpy as np
import pytest
import scipy.sparse as sp

from qtqp_b200 import direct, problems
from tests import kkt_driver

pytestmark = pytest.mark.gpu


def _system(n, m, seed):
  rng = np.random.default_rng([seed, n, m])
  a, b, c, _, p = problems.feasible(m, n, n // 5, rng, density=0.3)
  s, y = 0.1 + rng.random(m), 0.1 + rng.random(m)
  s[:n // 5] = 0.0
  return a, b, c, p, s, y, 0.1 + rng.random()


@pytest.mark.parametrize("n,m", [(79, 158), (80, 80), (81, 200), (127, 300), (128, 256), (129, 131),
                                 (200, 403), (257, 514), (300, 301)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_backend_sizes(n, m, precision):
  a, b, c, p, s, y, mu = _system(n, m, 5)
  z = n // 5
  kkt = kkt_driver.DirectKktSolver(a=a, p=p, z=z, min_static_regularization=1e-8,
                                   max_iterative_refinement_steps=30, atol=1e-12, rtol=1e-12,
                                   solver=direct.CudaDenseSolver(precision))
  rng = np.random.default_rng(n)
  for scale in (1.0, 3.0):  # the object factorises again
    kkt.update(mu=mu * scale, s=s, y=y)
    d = np.concatenate([np.zeros(z), s[z:] / y[z:]]) + mu * scale
    full = sp.bmat([[p + mu * scale * sp.eye(n), a.T], [a, -sp.diags(d)]], format="csc")
    for _ in range(2):
      v = rng.normal(size=n + m)
      got, want = kkt._solver @ v, full @ v
      # N-term FP64 sums in any order.
      bound = (n + m) * 2.0 ** -52 * (abs(full) @ np.abs(v))
      assert np.all(np.abs(got - want) <= bound)
      rhs = rng.normal(size=n + m)
      sol, _ = kkt.solve(rhs=rhs, warm_start=np.zeros(n + m))
      res = full @ sol - np.concatenate([rhs[:n], -rhs[n:]])
      assert np.abs(res).max() <= 1e-10 * (1 + np.abs(rhs).max())
  kkt.free()


@pytest.mark.parametrize("n", [60, 130, 260])
def test_indefinite_system_reports_a_pivot(n):
  m = n + 10
  a, _, _, p, _, _, _ = _system(n, m, 6)
  solver = direct.CudaDenseSolver()
  solver.set_dims(n, m, 0)
  kkt = sp.bmat([[sp.triu(p, format="csc") + sp.eye(n, format="csc"), a.T],
                 [None, sp.eye(m, format="csc")]], format="csr")
  solver.set_kkt(kkt)
  diag = np.concatenate([np.full(n, 1.0), np.full(m, -1.0)])
  diag[n - 3] = -1e6
  solver.update_diag(diag)
  with pytest.raises(np.linalg.LinAlgError):
    solver.factorize()
  diag[n - 3] = 1.0  # and is usable afterwards
  solver.update_diag(diag)
  solver.factorize()
  rhs = np.ones(n + m)
  x = solver.solve(rhs)
  assert np.abs(solver @ x - rhs).max() <= 1e-8
  solver.free()
