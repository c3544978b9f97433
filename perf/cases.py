"""Performance cases: the work a program hands to this solver.

A case is a dict of plain values; ``prepare`` makes its inputs from a seed,
``run`` is one pass through the public entry points, ``work`` counts the bytes
and operations the path cannot do without, and ``exact`` gives the values that
are known in 64 bits.  The QPs (but the parametric family's) are built from an
optimal pair (x0, y0, s0) drawn first, as in ``qtqp_b200.problems``, with
fewer tight rows than variables, duals and slacks away from zero and a
curvature away from zero: x0, y0 and s0 are the solution, and a well-posed one.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import qtqp_b200 as qb
from qtqp_b200 import _lib, band, batch, direct, large, problems, sparse, warmstart

csc_matrix = problems.sp.csc_matrix

# Interior-point iterations that `work` counts: these families take 8 to 30.
ITERATIONS = 10


def listed():
  return [
      # One small QP, host arrays in and out: a control loop or an interactive
      # user.  Latency and launches count.
      {"name": "single_n24", "kind": "single", "n": 24, "m": 48},
      # The benchmark's batch: 4096 uneven small dense QPs resident on the
      # device, solved in one call.
      {"name": "batch_4096", "kind": "batch", "count": 4096, "n_lo": 8, "n_hi": 64,
       "precision": "fp64"},
      # A smaller batch of smaller QPs in the mixed-precision form.
      {"name": "batch_1000_mixed", "kind": "batch", "count": 1000, "n_lo": 8, "n_hi": 40,
       "precision": "mixed"},
      # The whole user call on host data: packing, copies, solves, Solutions.
      {"name": "call_512", "kind": "call", "count": 512, "n_lo": 8, "n_hi": 64},
      # One large dense QP on the whole GPU, at the benchmark's size.
      {"name": "dense_4096", "kind": "dense", "n": 4096, "m": 8192, "precision": "fp64"},
      # A mid-sized dense QP, sizes off every tile, mixed precision.
      {"name": "dense_1000_mixed", "kind": "dense", "n": 1000, "m": 2100,
       "precision": "mixed"},
      # A long-horizon MPC QP (T = 500), banded, on the whole GPU.
      {"name": "mpc_500", "kind": "mpc", "horizon": 500, "nx": 40, "nu": 20},
      # A parametric MPC family (T = 50), one instance per thread block.
      {"name": "family_148", "kind": "family", "count": 148, "horizon": 50},
      # Sparse QPs: a network flow, and random sparse rows.
      {"name": "flow_60", "kind": "flow", "grid": 60},
      {"name": "rows_2000", "kind": "rows", "n": 2000, "m": 2000},
      # The KKT backend inside somebody else's interior-point loop: a new
      # diagonal, factorise, three solves and products.
      {"name": "kkt_300", "kind": "kkt", "n": 300, "m": 600},
      # One training step of the learned warm start of the T = 50 family.
      {"name": "train_256", "kind": "train", "batch": 256, "horizon": 50},
  ]


def _log_int(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
  kind = rng.choice(["single", "batch", "batch", "call", "dense", "dense", "mpc", "family",
                     "flow", "rows", "kkt", "train"])
  if kind == "single":
    n = _log_int(rng, 8, 96)
    return {"kind": kind, "n": n, "m": rng.randint(n + 1, 2 * n + 1)}
  if kind == "batch":
    lo = rng.randint(8, 48)
    return {"kind": kind, "count": _log_int(rng, 64, 4000), "n_lo": lo,
            "n_hi": rng.randint(lo, 64), "precision": rng.choice(["fp64", "fp64", "mixed"])}
  if kind == "call":
    lo = rng.randint(8, 48)
    return {"kind": kind, "count": _log_int(rng, 16, 1000), "n_lo": lo,
            "n_hi": rng.randint(lo, 64)}
  if kind == "dense":
    n = _log_int(rng, 256, 3000)
    return {"kind": kind, "n": n, "m": rng.randint(n + n // 4, 2 * n + 1),
            "precision": rng.choice(["fp64", "fp64", "mixed"])}
  if kind == "mpc":
    nx = rng.randint(6, 40)
    nu = max(2, nx // 2)
    lo = -(-1100 // (nx + nu))
    return {"kind": kind, "horizon": _log_int(rng, lo, max(lo + 1, 24000 // (nx + nu))),
            "nx": nx, "nu": nu}
  if kind == "family":
    return {"kind": kind, "count": _log_int(rng, 16, 148), "horizon": rng.randint(10, 40)}
  if kind == "flow":
    return {"kind": kind, "grid": _log_int(rng, 14, 58)}
  if kind == "rows":
    n = _log_int(rng, 500, 3000)
    return {"kind": kind, "n": n, "m": n + rng.randint(0, n // 20)}
  if kind == "kkt":
    n = _log_int(rng, 16, 400)
    return {"kind": kind, "n": n, "m": rng.randint(n, 2 * n)}
  return {"kind": kind, "batch": 64 * rng.randint(1, 6), "horizon": rng.randint(6, 49)}


# ---------------------------------------------------------------------------
# Inputs.
# ---------------------------------------------------------------------------
def _optimal_pair(rng, n, m, z):
  """x0, y0, s0 like problems._feasible_pair's.  Tight are the equality rows
  and inequality rows for half of the n - z variables left (at most half of
  those rows); their duals and the other rows' slacks are at least 0.1."""
  x0 = rng.normal(size=n)
  y0 = np.zeros(m)
  y0[:z] = rng.normal(size=z)
  active = np.arange(m - z) < min(max(n - z, 0), m - z) // 2
  rng.shuffle(active)
  y0[z:] = np.where(active, 0.1 + np.abs(rng.normal(size=m - z)), 0.0)
  s0 = np.zeros(m)
  s0[z:] = np.where(active, 0.0, 0.1 + rng.random(m - z))
  return x0, y0, s0


def _pair_rng(seed):
  return np.random.default_rng([seed, 11])


def _sizes(case):
  """n of every QP of a batch (the same for every seed)."""
  return np.random.default_rng(12).integers(case["n_lo"], case["n_hi"] + 1,
                                            size=case["count"])


def _small_dense(seed, sizes, m_of=lambda n: 2 * n):
  """(a, b, c, z, p) of dense QPs like problems.small_dense_instance's: A ~
  N(0, 1), P = L L^T + 0.1 I with L n x n/2, z = n / 4."""
  rng, pair = np.random.default_rng([seed, 13]), _pair_rng(seed)
  out = []
  for n in sizes.tolist():
    m, z = m_of(n), n // 4
    a = rng.normal(size=(m, n))
    l = rng.normal(size=(n, n // 2))
    p = l @ l.T
    p[np.arange(n), np.arange(n)] += 0.1
    p = 0.5 * (p + p.T)
    x0, y0, s0 = _optimal_pair(pair, n, m, z)
    out.append((a, a @ x0 + s0, -(p @ x0 + a.T @ y0), z, p))
  return out


def _small_exact(seed, sizes, m_of=lambda n: 2 * n):
  pair = _pair_rng(seed)
  got = [_optimal_pair(pair, n, m_of(n), n // 4) for n in sizes.tolist()]
  return (*(np.concatenate([g[k] for g in got]) for k in range(3)), None)


def _qtqp(a, b, c, z, p):
  return qb.QTQP(a=csc_matrix(a), b=b, c=c, z=z, p=csc_matrix(p))


def _statuses(results):
  """Status code of every result record (a view of the device records)."""
  rec = results.view(-1, _lib.RESULT_DTYPE.itemsize)
  off = _lib.RESULT_DTYPE.fields["status"][1]
  return rec[:, off:off + 4].view(torch.int32)


def _dense_large(seed, n, m):
  """Like problems.large_dense's: A ~ N(0, 1/n), P = U diag(d) U^T + I with U
  n x rank ~ N(0, 1/rank), d ~ U(0.1, 10)."""
  z, rank = n // 4, min(256, n // 4)
  rng = np.random.default_rng([seed, 14])
  a = rng.normal(scale=1.0 / np.sqrt(n), size=(n, m)).T  # column-major values
  u = rng.normal(scale=1.0 / np.sqrt(rank), size=(n, rank))
  d = rng.uniform(0.1, 10.0, size=rank)
  p = (u * d) @ u.T
  p[np.arange(n), np.arange(n)] += 1.0
  p = 0.5 * (p + p.T)
  x0, y0, s0 = _optimal_pair(_pair_rng(seed), n, m, z)
  return batch.DenseProblem(a=a, b=a @ x0 + s0, c=-(p @ x0 + a.T @ y0), z=z, p=p)


def _mpc_point(seed, horizon, nx, nu):
  """(x, y, ub): a point of the MPC boxes, a tenth of it on a bound with a
  positive dual there, like problems.mpc_feasible's."""
  rng = np.random.default_rng([seed, 15])
  ub = np.tile(np.concatenate([np.full(nx, 5.0), np.full(nu, 1.0)]), horizon)
  n = ub.size
  x = rng.uniform(-0.5, 0.5, size=n) * ub
  act = rng.random(n) < 0.1
  act[:nx] = False  # the initial state is fixed by equality rows
  up = rng.random(n) < 0.5
  x = np.where(act, np.where(up, ub, -ub), x)
  lam = 0.1 + np.abs(rng.normal(size=n))
  y = np.concatenate([rng.normal(size=nx * horizon), np.where(act & up, lam, 0.0),
                      np.where(act & ~up, lam, 0.0)])
  return x, y, ub


def _mpc(seed, horizon, nx, nu):
  a, z, p, _ = problems.mpc_structure(horizon, nx=nx, nu=nu, seed=seed)
  x, y, ub = _mpc_point(seed, horizon, nx, nu)
  b = np.concatenate([a[:z] @ x, ub, ub])
  return a, b, -(p @ x + a.T @ y), z, p


def _sparse(case, seed):
  if case["kind"] == "flow":
    a, _, _, z, p = problems.grid_flow(case["grid"], seed=seed)
  else:
    a, _, _, z, p = problems.sparse_feasible(case["n"], case["m"], case["n"] // 10, seed,
                                             per_row=2)
  m, n = a.shape
  x0, y0, s0 = _optimal_pair(_pair_rng(seed), n, m, z)
  return a, a @ x0 + s0, -(p @ x0 + a.T @ y0), z, p


def _kkt(case, seed):
  """A, P, the regularised diagonal at a mid-course iterate, right-hand sides."""
  n, m = case["n"], case["m"]
  rng = np.random.default_rng([seed, 17])
  a = rng.normal(size=(m, n))
  l = rng.normal(size=(n, n // 2))
  p = l @ l.T + 1e-3 * np.eye(n)
  z, mu = n // 4, 1e-3
  reg = np.concatenate([np.diag(p) + mu, np.full(z, -mu),
                        -(np.exp(rng.normal(size=m - z)) + mu)])
  return a, p, reg, rng.normal(size=(3, n + m))


def _train_dims(case):
  n = 60 * case["horizon"]
  z = 40 * case["horizon"]
  return 32, n, z + 2 * n, z  # dim, n, m, z


def _train(case, seed):
  """Parameters and standardised targets of one minibatch."""
  dim, n, m, _ = _train_dims(case)
  g = torch.Generator(device="cuda").manual_seed(seed)
  normal = lambda *s: torch.randn(*s, generator=g, device="cuda", dtype=torch.float32)
  return normal(case["batch"], dim), normal(case["batch"], n + m)


def prepare(case, seed):
  kind = case["kind"]
  if kind == "single":
    m = case["m"]
    return {"kind": kind, "qp": _qtqp(*_small_dense(seed, np.array([case["n"]]),
                                                    lambda n: m)[0])}
  if kind == "call":
    return {"kind": kind,
            "qps": [_qtqp(*q) for q in _small_dense(seed, _sizes(case))]}
  if kind == "batch":
    probs = [batch.DenseProblem(a=a, b=b, c=c, z=z, p=p)
             for a, b, c, z, p in _small_dense(seed, _sizes(case))]
    hb = batch.HostBatch(probs, batch.SolveOptions(precision=case["precision"]))
    dev = batch.DeviceBatch(hb, records=False)
    dev.upload()
    # Where each problem's entries lie in the output pools, in problem order.
    where = [np.concatenate([np.arange(o, o + k) for o, k in
                             zip(hb.inst[off].tolist(), hb.inst[num].tolist())])
             for off, num in (("n_off", "n"), ("m_off", "m"))]
    return {"kind": kind, "dev": dev, "where": [torch.from_numpy(w).cuda() for w in where]}
  opts = batch.SolveOptions(precision=case.get("precision", "fp64"))
  if kind == "dense":
    dev = large.DeviceLarge(_dense_large(seed, case["n"], case["m"]), opts, records=False)
  elif kind == "mpc":
    prob = band.BandProblem(*_mpc(seed, case["horizon"], case["nx"], case["nu"]))
    dev = band.DeviceBandGrid(band.HostBandBatch([prob], opts), records=False)
  elif kind == "family":
    fam = problems.parametric_mpc_family(case["count"], case["horizon"], seed=seed)
    probs = [band.BandProblem(*problems.parametric_mpc_instance(fam, i))
             for i in range(case["count"])]
    dev = band.DeviceBandBatch(band.HostBandBatch(probs, opts), records=False)
  elif kind in ("flow", "rows"):
    a, b, c, z, p = _sparse(case, seed)
    plan = sparse.SparsePlan(a, p)
    dev = sparse.DeviceSparseGrid(plan.permuted(a, b, c, z, p), plan, opts, records=False)
    dev.upload()
    perm = np.empty(plan.n, np.int64)
    perm[plan.perm] = np.arange(plan.n)
    return {"kind": kind, "dev": dev, "where": torch.from_numpy(perm).cuda()}
  elif kind == "kkt":
    a, p, reg, rhs = _kkt(case, seed)
    n, m = case["n"], case["m"]
    solver = direct.CudaDenseSolver()
    solver.set_dims(n, m, n // 4)
    upper = np.zeros((n + m, n + m))
    upper[:n, :n] = np.triu(p)
    upper[:n, n:] = a.T
    upper[np.arange(n, n + m), np.arange(n, n + m)] = 1.0
    solver.set_kkt(csc_matrix(upper).tocsr())
    return {"kind": kind, "solver": solver, "reg": reg, "rhs": rhs}
  else:
    dim, n, m, z = _train_dims(case)
    theta, target = _train(case, seed)
    return {"kind": kind, "net": warmstart.WarmStartMLP(dim=dim, n=n, m=m, z=z, seed=seed),
            "theta": theta, "target": target, "batch": case["batch"]}
  dev.upload()
  return {"kind": kind, "dev": dev}


def run(state):
  kind = state["kind"]
  if kind == "single":
    sol = state["qp"].solve(verbose=False)
    return sol.x, sol.y, sol.s, list(qb.SolutionStatus).index(sol.status)
  if kind == "call":
    sols = qb.solve_batch(state["qps"])
    codes = list(qb.SolutionStatus)
    return (np.concatenate([v.x for v in sols]), np.concatenate([v.y for v in sols]),
            np.concatenate([v.s for v in sols]),
            np.array([codes.index(v.status) for v in sols]))
  if kind == "kkt":
    solver = state["solver"]
    solver.update_diag(state["reg"])
    solver.factorize()
    sols = [solver.solve(r) for r in state["rhs"]]
    return np.stack(sols), np.stack([solver @ v for v in sols])
  if kind == "train":
    net = state["net"]
    y = net.gradients(state["theta"], state["target"], state["batch"])
    return [y, *net.grads]
  dev = state["dev"]
  dev.launch()
  if kind == "batch":
    wx, wy = state["where"]
    return dev.x[wx], dev.y[wy], dev.s[wy], _statuses(dev.results)
  if kind in ("flow", "rows"):
    return dev.x[state["where"]], dev.y, dev.s, _statuses(dev.result)
  return dev.x, dev.y, dev.s, _statuses(dev.results if kind == "family" else dev.result)


# ---------------------------------------------------------------------------
# What a pass cannot do without, and the values known in 64 bits.
# ---------------------------------------------------------------------------
def _dense_work(n, m):
  """Inputs and outputs once; per iteration the Gram product (its lower half)
  and the Cholesky factorisation, and the products of two solves."""
  return (8 * (m * n + n * n + 2 * n + 3 * m),
          ITERATIONS * (m * n * n + n ** 3 / 3 + 2 * (4 * m * n + 2 * n * n)))


def work(case):
  kind = case["kind"]
  if kind in ("single", "dense"):
    nbytes, flops = _dense_work(case["n"], case["m"])
  elif kind in ("batch", "call"):
    sizes = range(case["n_lo"], case["n_hi"] + 1)
    each = [_dense_work(n, 2 * n) for n in sizes]
    nbytes, flops = (case["count"] * sum(e[k] for e in each) / len(each) for k in (0, 1))
  elif kind in ("mpc", "family"):
    nx, nu = case.get("nx", 40), case.get("nu", 20)
    n, bw, count = case["horizon"] * (nx + nu), 2 * nx + nu - 1, case.get("count", 1)
    m = nx * case["horizon"] + 2 * n
    nnz = case["horizon"] * nx * (nx + nu + 1) + 2 * n
    shared = 12 * (2 * nnz + n)  # A by rows and by columns, and P
    nbytes = shared + count * 8 * (2 * n + 3 * m)
    flops = count * ITERATIONS * (n * bw * bw + 2 * (4 * nnz + 4 * n * bw))
  elif kind in ("flow", "rows"):
    # The factor's size depends on the ordering: A, P and the vectors alone,
    # and the sparse products of two solves and of the Gram matrix.
    n = 4 * case["grid"] * (case["grid"] - 1) if kind == "flow" else case["n"]
    m = case["grid"] ** 2 + 2 * n if kind == "flow" else case["m"]
    nnz = 4 * n if kind == "flow" else 2 * m
    nbytes = 12 * (2 * nnz + n) + 8 * (2 * n + 3 * m)
    flops = ITERATIONS * 30 * nnz
  elif kind == "kkt":
    n, m = case["n"], case["m"]
    nbytes = 8 * (m * n + n * n + 8 * (n + m))
    flops = m * n * n + n ** 3 / 3 + 3 * (8 * m * n + 4 * n * n)
  else:
    dim, n, m, _ = _train_dims(case)
    k, out = case["batch"], n + m
    weights = dim * 256 + 256 * 256 + 256 * out + 512 + out
    nbytes = 4 * (2 * weights + k * (dim + 2 * out))
    flops = 6 * k * weights - 2 * k * dim * 256
  return {"bytes": nbytes, "flops": flops}


def _exact_kkt(case, seed):
  """The three solutions by LAPACK, refined twice with extended-precision
  residuals, and the products K x of those (the right-hand sides)."""
  a, p, reg, rhs = _kkt(case, seed)
  n = case["n"]
  k = np.zeros((reg.size, reg.size))
  k[:n, :n] = p
  k[:n, n:] = a.T
  k[n:, :n] = a
  k[np.arange(reg.size), np.arange(reg.size)] = reg
  kl, r = k.astype(np.longdouble), rhs.T.astype(np.longdouble)
  x = np.linalg.solve(k, rhs.T).astype(np.longdouble)
  for _ in range(2):
    x += np.linalg.solve(k, (r - kl @ x).astype(np.float64))
  return x.T.astype(np.float64), rhs


def _exact_train(case, seed):
  """Output and gradients of the mean squared error of the three-layer network
  (zero biases) in 64 bits."""
  dim, n, m, _ = _train_dims(case)
  rng = np.random.default_rng(seed)
  he = lambda i, o: torch.from_numpy((rng.normal(size=(i, o)) * np.sqrt(2.0 / i))
                                     .astype(np.float32)).cuda()
  w1, w2 = he(dim, 256), he(256, 256)
  w3 = torch.from_numpy((rng.normal(size=(256, n + m)) * np.sqrt(2.0 / 256))
                        .astype(np.float32) * np.float32(0.1)).cuda()
  theta, target = (v.double() for v in _train(case, seed))
  w1, w2, w3 = w1.double(), w2.double(), w3.double()
  h1 = (theta @ w1).clamp(min=0)
  h2 = (h1 @ w2).clamp(min=0)
  y = h2 @ w3
  dy = (2.0 / y.numel()) * (y - target)
  d2 = (dy @ w3.T) * (h2 > 0)
  d1 = (d2 @ w2.T) * (h1 > 0)
  return [y, theta.T @ d1, d1.sum(0), h1.T @ d2, d2.sum(0), h2.T @ dy, dy.sum(0)]


def exact(case, seed):
  kind = case["kind"]
  if kind == "single":
    return _small_exact(seed, np.array([case["n"]]), lambda n: case["m"])
  if kind in ("batch", "call"):
    return _small_exact(seed, _sizes(case))
  if kind in ("dense", "rows", "flow"):
    if kind == "flow":
      n, z = 4 * case["grid"] * (case["grid"] - 1), case["grid"] ** 2
      m = z + 2 * n
    else:
      n, m = case["n"], case["m"]
      z = n // 4 if kind == "dense" else n // 10
    x0, y0, s0 = _optimal_pair(_pair_rng(seed), n, m, z)
    # The conservation rows of a flow sum to zero: its y is free by a constant.
    return x0, None if kind == "flow" else y0, s0, None
  if kind == "mpc":
    x, y, ub = _mpc_point(seed, case["horizon"], case["nx"], case["nu"])
    return x, y, np.concatenate([np.zeros(case["nx"] * case["horizon"]), ub - x, ub + x]), None
  if kind == "kkt":
    return _exact_kkt(case, seed)
  if kind == "train":
    return _exact_train(case, seed)
  return None  # the family's instances have no known solution
