"""The separate passes of the MLP's C interface (qtqp_mlp_relu_grad,
qtqp_mlp_colsum, qtqp_mlp_mse_grad) that a program with its own training loop
calls, at sizes off their blocks, against numpy on the same FP32 operands."""

import numpy as np
import pytest

from qtqp_b200 import _lib

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (3, 255), (7, 256), (64, 257), (130, 5000)]


def _pair(rows, cols):
  import torch
  rng = np.random.default_rng([rows, cols])
  u, v = (rng.normal(size=(rows, cols)).astype(np.float32) for _ in range(2))
  v[0, 0] = 0.0
  return u, v, torch.from_numpy(u).cuda(), torch.from_numpy(v).cuda()


@pytest.mark.parametrize("rows,cols", SIZES)
def test_relu_grad(rows, cols):
  u, v, du, dv = _pair(rows, cols)
  _lib.check(_lib.load().qtqp_mlp_relu_grad(du.data_ptr(), dv.data_ptr(), u.size, None))
  np.testing.assert_array_equal(du.cpu().numpy(), np.where(v > 0.0, u, np.float32(0.0)))


@pytest.mark.parametrize("rows,cols", SIZES)
def test_colsum(rows, cols):
  import torch
  u, _, du, _ = _pair(rows, cols)
  out = torch.full((cols,), float("nan"), dtype=torch.float32, device="cuda")
  _lib.check(_lib.load().qtqp_mlp_colsum(du.data_ptr(), rows, cols, out.data_ptr(), None))
  u = u.astype(np.float64)
  # An FP32 sum of `rows` terms.
  bound = rows * 2.0 ** -24 * np.abs(u).sum(axis=0)
  assert np.all(np.abs(out.cpu().numpy() - u.sum(axis=0)) <= bound)


@pytest.mark.parametrize("rows,cols", SIZES)
def test_mse_grad(rows, cols):
  import torch
  u, v, du, dv = _pair(rows, cols)
  dy = torch.full((rows, cols), float("nan"), dtype=torch.float32, device="cuda")
  loss = torch.full((1,), 3.0, dtype=torch.float64, device="cuda")
  _lib.check(_lib.load().qtqp_mlp_mse_grad(du.data_ptr(), dv.data_ptr(), u.size, dy.data_ptr(),
                                           loss.data_ptr(), None))
  err = (u - v).astype(np.float64)  # the kernel's own FP32 subtraction
  # The rounded 2 / count and one FP32 product.
  want = 2.0 / err.size * err
  assert np.all(np.abs(dy.cpu().numpy() - want) <= 3 * 2.0 ** -24 * np.abs(want))
  np.testing.assert_allclose(loss.item(), np.sum(err ** 2), rtol=1e-12)
