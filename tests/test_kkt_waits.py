"""What the dense KKT backend does about a wait of the whole-GPU form that gave up:
a pivot is not blamed, and the next factorisation starts clean."""

import numpy as np
import pytest

from qtqp_b200 import direct

class _FakeLib:

  def qtqp_kkt_dense_factorize(self, *args):
    return 0


@pytest.mark.parametrize("info,error", [(-1, RuntimeError), (3, np.linalg.LinAlgError)])
def test_a_wait_that_gave_up_is_not_a_pivot(info, error):
  import torch
  s = object.__new__(direct.CudaDenseSolver)
  s._lib, s._prec, s._n, s._m = _FakeLib(), 0, 100, 100
  s._diag = s._ws = torch.zeros(1)
  s._info = torch.tensor([info], dtype=torch.int32)
  s._stream = lambda: 0
  with pytest.raises(error) as e:
    s.factorize()
  assert type(e.value) is error


def _grid_part(n, m):
  """Offset of the whole-GPU form's part of the workspace: the header and the
  single block's regions (dense_ipm.cuh, plan_layout without shared memory)."""
  r16 = lambda b: (b + 15) & ~15
  ld = n | 1
  np_ = (max(n + m, n + 4) + 1) & ~1
  vec = r16((18 * np_ + 34 * ((n + 3) >> 2) + 2 * n) * 8)
  return (256 + 2 * r16(n * ld * 8) + r16(m * ld * 8) + vec + 255) & ~255


@pytest.mark.gpu
@pytest.mark.parametrize("n", [80, 300])
def test_factorises_again_after_a_wait_gave_up(n):
  import torch
  m = 2 * n
  rng = np.random.default_rng(n)
  a, l = rng.normal(size=(m, n)), rng.normal(size=(n, n))
  p = l @ l.T / n
  full = np.zeros((n + m, n + m))
  full[:n, :n] = np.triu(p)
  full[:n, n:] = a.T
  full[np.arange(n, n + m), np.arange(n, n + m)] = 1.0
  import scipy.sparse as sp
  s = direct.CudaDenseSolver()
  s.set_dims(n, m, 0)
  s.set_kkt(sp.csr_matrix(full))
  diag = np.concatenate([np.diag(p) + 0.1, np.full(m, -1.0)])
  rhs = rng.normal(size=n + m)
  s.update_diag(diag)
  s.factorize()
  want = s.solve(rhs)
  assert np.abs(s @ want - rhs).max() <= 1e-9 * np.abs(rhs).max()
  # What a wait that gives up leaves: the error flag and the barrier's top bit.
  o = _grid_part(n, m)
  head = s._ws[o:o + 12].cpu().numpy()
  assert head[8] == 0 and head.any()  # the barrier's count, no error
  s._ws[o + 7] = 0x80
  s._ws[o + 8] = 1
  assert np.isnan(s.solve(rhs)).any()
  s.update_diag(diag)
  s.factorize()
  np.testing.assert_array_equal(s.solve(rhs), want)
  torch.cuda.synchronize()
  s.free()
