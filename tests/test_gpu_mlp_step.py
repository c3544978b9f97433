"""The training step's fused products (qtqp_mlp_forward_loss and
qtqp_mlp_backward) against FP64 products of the same FP32 operands, at sizes
around the 64 x 64 tiles, the 16-deep slices and the split of a long inner
dimension over a cluster.

Every output is one inner product of FP32 operands that the test reads back,
so the bound is that of an FP32 sum in any order: |error| <= g |A| |B| with
g = (K + 8) 2^-24 (K products and sums, plus bias, scaling and the partial
sums of a split)."""

import ctypes

import numpy as np
import pytest

from qtqp_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,dim,hidden,out", [
    (1, 1, 1, 1), (63, 5, 16, 65), (64, 16, 64, 64), (65, 33, 70, 129),
    (64, 32, 256, 700), (192, 32, 256, 5000), (256, 32, 256, 11000)])
def test_step_products(batch, dim, hidden, out):
  import torch
  lib = _lib.load()
  rng = np.random.default_rng(batch + out)
  dev = lambda *s: torch.from_numpy(rng.normal(size=s).astype(np.float32)).cuda()
  new = lambda *s: torch.full(s, float("nan"), dtype=torch.float32, device="cuda")
  t = {"x": dev(batch, dim), "target": dev(batch, out), "w1": dev(dim, hidden),
       "b1": dev(hidden), "w2": dev(hidden, hidden), "b2": dev(hidden), "w3": dev(hidden, out),
       "b3": dev(out), "h1": new(batch, hidden), "h2": new(batch, hidden), "y": new(batch, out),
       "dy": new(batch, out), "dh1": new(batch, hidden), "dh2": new(batch, hidden),
       "g1": new(dim, hidden), "gb1": new(hidden), "g2": new(hidden, hidden), "gb2": new(hidden),
       "g3": new(hidden, out), "gb3": new(out),
       "loss": torch.full((1,), 7.0, dtype=torch.float64, device="cuda")}
  step = _lib.MlpStep(batch, dim, hidden, out, **{k: v.data_ptr() for k, v in t.items()})
  _lib.check(lib.qtqp_mlp_forward_loss(ctypes.byref(step), None))
  _lib.check(lib.qtqp_mlp_backward(ctypes.byref(step), None))
  torch.cuda.synchronize()
  d = {k: v.cpu().numpy().astype(np.float64) for k, v in t.items()}

  def check(name, a, b, bias=None, relu=False, mask=None):
    want, size = a @ b, np.abs(a) @ np.abs(b)
    if bias is not None:
      want, size = want + bias, size + np.abs(bias)
    if relu:
      want = np.maximum(want, 0.0)
    if mask is not None:
      want, size = want * (mask > 0.0), size * (mask > 0.0)
    bound = (a.shape[1] + 8) * 2.0 ** -24 * size
    assert np.all(np.abs(d[name] - want) <= bound), name

  check("h1", d["x"], d["w1"], d["b1"], relu=True)
  check("h2", d["h1"], d["w2"], d["b2"], relu=True)
  check("y", d["h2"], d["w3"], d["b3"])
  err = d["y"] - d["target"]
  # One FP32 subtraction and one scaling by the rounded 2 / (batch out).
  want = 2.0 / err.size * err
  assert np.all(np.abs(d["dy"] - want) <= 4 * 2.0 ** -24 * np.abs(want))
  np.testing.assert_allclose(d["loss"][0], np.sum(err ** 2), rtol=4 * 2.0 ** -24)
  ones = np.ones((1, batch))
  check("g3", d["h2"].T, d["dy"])
  check("dh2", d["dy"], d["w3"].T, mask=d["h2"])
  check("g2", d["h1"].T, d["dh2"])
  check("dh1", d["dh2"], d["w2"].T, mask=d["h1"])
  check("g1", d["x"].T, d["dh1"])
  for name, v in (("gb3", "dy"), ("gb2", "dh2"), ("gb1", "dh1")):
    d[name] = d[name][None]
    check(name, ones, d[v])
