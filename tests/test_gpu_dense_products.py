"""The dense batch kernel's matrix-vector products at the edges of their loops:
one column per lane up to n = 32, two up to 64, row dots above (eight entries per
lane at a time); 4, 8 or 16 rows per warp, with remainders; every block size.

Criteria of the other path tests: the oracle's status, the reference's acceptance
conditions, objective relative error <= 1e-6."""

import types

import numpy as np
import pytest
import scipy.sparse as sp

from oracle import qtqp_oracle as orc
from qtqp_b200 import batch
from tests import kkt_checks

pytestmark = pytest.mark.gpu

OBJ_TOL = 1e-6
SIZES = [(1, 2), (2, 9), (7, 8), (8, 17), (16, 31), (31, 63), (32, 33), (32, 65), (33, 34),
         (33, 45), (40, 90), (50, 97), (60, 193), (64, 190),
         (63, 64), (64, 65), (65, 66), (65, 129), (79, 80), (96, 97)]


def _qp(n, m, with_p):
  rng = np.random.default_rng([n, m, with_p])
  a = rng.normal(size=(m, n))
  z = n // 4
  l = rng.normal(size=(n, n))
  p = l @ l.T / n + 0.1 * np.eye(n) if with_p else None
  x0 = rng.normal(size=n)
  tight = np.arange(m - z) < (m - z) // 2
  y0 = np.concatenate([rng.normal(size=z), np.where(tight, 0.1 + rng.random(m - z), 0.0)])
  s0 = np.concatenate([np.zeros(z), np.where(tight, 0.0, 0.1 + rng.random(m - z))])
  c = -a.T @ y0 - (p @ x0 if with_p else 0.0)
  return a, a @ x0 + s0, c, z, p


@pytest.fixture(scope="module")
def cases():
  out = []
  for n, m in SIZES:
    # (96, 97) without P is a linear program with a 36-dimensional face of
    # solutions: the device method runs into its iteration limit on it.
    for with_p in (True, False) if n < 96 else (True,):
      a, b, c, z, p = _qp(n, m, with_p)
      sa = sp.csc_matrix(a)
      spm = sp.csc_matrix(p) if with_p else sp.csc_matrix((n, n))
      out.append((a, b, c, z, p, sa, spm, orc.solve(sa, b, c, z, spm)))
  return out


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("block_threads", [32, 64, 128, 256])
def test_sizes(cases, block_threads, precision):
  hb = batch.HostBatch([batch.DenseProblem(a=a, b=b, c=c, z=z, p=p)
                        for a, b, c, z, p, *_ in cases],
                       batch.SolveOptions(precision=precision), block_threads=block_threads)
  dev = batch.DeviceBatch(hb, records=False)
  dev.upload()
  dev.launch()
  res, x, y, s, _ = dev.fetch()
  for i, (a, b, c, z, p, sa, spm, ref) in enumerate(cases):
    m, n = a.shape
    xo, mo = int(hb.inst[i]["n_off"]), int(hb.inst[i]["m_off"])
    sol = types.SimpleNamespace(
        status=types.SimpleNamespace(value="solved" if res["status"][i] == 0 else "other"),
        x=x[xo:xo + n], y=y[mo:mo + m], s=s[mo:mo + m])
    assert ref.status == "solved"
    kkt_checks.assert_solved(sol, sa, b, c, spm, z)
    assert kkt_checks.objective_rel_err(sol.x, ref.x, c, spm) <= OBJ_TOL
