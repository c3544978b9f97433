"""The scales and scaled matrices of the large dense path's equilibration against
a numpy replay of its ten sweeps (src/qtqp/__init__.py:616-663), bit for bit: maxima
have no rounding, and square root, division and products are correctly rounded on
both sides.  Sizes at the edges of the passes: rows shared by one and by several
warps, more than 4096 columns, more than 1024 rows per block, blocks without rows,
no P."""

import numpy as np
import pytest

from qtqp_b200 import batch, large

pytestmark = pytest.mark.gpu


def _replay(a, p):
  m, n = a.shape
  a, p = a.copy(), p.copy()
  d, e = np.ones(m), np.ones(n)
  scale = lambda mx: np.clip(1.0 / np.sqrt(np.where(mx == 0.0, 1.0, mx)), 1e-3, 1e3)
  for _ in range(10):
    ei = scale(np.maximum(np.abs(a).max(axis=0), np.abs(p).max(axis=0)))
    di = scale(np.abs(a).max(axis=1))
    a *= di[:, None] * ei[None, :]
    p *= ei[:, None] * ei[None, :]
    d *= di
    e *= ei
  return d, e, a, p


@pytest.mark.parametrize("n,m,with_p", [(130, 15, True), (512, 700, True), (513, 600, False),
                                        (1100, 900, True), (4100, 40, True), (16, 160000, True)])
def test_scales(n, m, with_p):
  import torch
  rng = np.random.default_rng([n, m])
  a = rng.normal(size=(m, n)) * 10.0 ** rng.uniform(-2, 2, size=n)
  a *= 10.0 ** rng.uniform(-2, 2, size=(m, 1))
  a *= rng.random(size=(m, n)) < 0.7
  p = np.zeros((n, n))
  if with_p:
    p = np.where(rng.random((n, n)) < 0.1, rng.normal(size=(n, n)), 0.0)
    p = p + p.T + np.diag(10.0 ** rng.uniform(-2, 2, size=n))
  prob = batch.DenseProblem(a=a, b=rng.normal(size=m), c=rng.normal(size=n), z=0,
                            p=p if with_p else None)
  dev = large.DeviceLarge(prob, batch.SolveOptions(max_iter=1), records=False)
  dev.upload()
  dev.launch()
  torch.cuda.synchronize()
  # The workspace's regions (large_ipm.cuh, plan_large_layout), each a multiple of
  # 1024 bytes: barrier, solve slots, status, 18 vectors, A, P.
  al = lambda b: (b + 1023) & ~1023
  npad, np_ = (n + 127) // 128 * 128, (max(n + m, n + 4) + 1) & ~1
  v_off = al(16 + 2 * 256 * 16 * 8) + al(npad * 16) + 1024
  a_off = v_off + al(18 * np_ * 8)
  p_off = a_off + al(m * n * 8)
  ws = dev._ws[dev.ws_ptr - dev._ws.data_ptr():]
  read = lambda off, count: ws[off:off + 8 * count].cpu().numpy().view(np.float64)
  d, e, a_eq, p_eq = _replay(a, p)
  de = read(v_off + 11 * np_ * 8, n + m)  # kDE
  np.testing.assert_array_equal(de[:n], e)
  np.testing.assert_array_equal(de[n:], d)
  np.testing.assert_array_equal(read(a_off, m * n).reshape(m, n), a_eq)
  got_p = read(p_off, n * n).reshape(n, n)  # its diagonal is kept apart
  off = ~np.eye(n, dtype=bool)
  np.testing.assert_array_equal(got_p[off], p_eq[off])
