"""Blocks of integrator steps on the GLM potentials in one launch
(glm_loop.cu) at the edges of its row tiles, chunks and clusters, against the
oracle's trajectories on the same indices and Philox normals.

Shapes: one feature (rows of 4 bytes: 4-byte copies), feature counts around
the 128-column lanes and the 1,024 limit, minibatches below, at and above
whole tiles of 32 rows and longer than the shared-memory ring, one chain (a
cluster of up to eight CTAs), and more chains than SMs (one CTA each).

Tolerance (as for the other K-step trajectories): 1e-4 relative plus 1e-5
absolute; U within 1e-5 relative plus 1e-3 absolute.
"""

import numpy as np
import pytest

from oracle import sgmc_oracle as O

pytestmark = pytest.mark.gpu

# (chains, n, d, family)
SHAPES = [
    (1, 1, 1, O.LINEAR_GAUSSIAN),
    (1, 31, 7, O.LOGISTIC),
    (2, 33, 33, O.LINEAR_GAUSSIAN),
    (1, 257, 128, O.LOGISTIC),
    (3, 500, 129, O.LOGISTIC),
    (1, 6000, 40, O.LOGISTIC),
    (2, 1100, 257, O.LOGISTIC),
    (1, 300, 1021, O.LINEAR_GAUSSIAN),
    (170, 65, 5, O.LOGISTIC),
]
K = 6


def _cuda(a):
  import torch
  return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _words(C):
  from gbsgmc.data.numpy_loader import pcg64_words
  return np.array([pcg64_words(c) for c in range(C)], np.uint64).view(np.int64)


def _setup(C, n, d, family):
  from gbsgmc import data, likelihoods as L, potential
  N = 7001
  rng = np.random.default_rng(100 * d + n)
  X = rng.normal(size=(N, d)).astype(np.float32)
  w = rng.normal(size=d) / np.sqrt(d)
  if family == O.LOGISTIC:
    y = (rng.random(N) < 1 / (1 + np.exp(-(X @ w)))).astype(np.float32)
    lik = L.Logistic()
  else:
    y = (X @ w + 0.5 * rng.normal(size=N)).astype(np.float32)
    lik = L.LinearGaussian(sigma=0.5)
  loader = data.NumpyDataLoader(x=X, y=y)
  pot = potential.minibatch_potential(L.GaussianPrior(3.0), lik)
  x0 = (0.1 * rng.normal(size=(C, d))).astype(np.float32)
  return X, y, loader.device_dataset(), pot, x0, N


def _potential(X, y, w, idx, N, family):
  return O.glm_potential(w, X, y, idx, N, family, 0.5, 3.0)


@pytest.mark.parametrize("C,n,d,family", SHAPES)
@pytest.mark.parametrize("kind", ["langevin", "obabo", "sghmc"])
def test_block_matches_oracle(lib, kind, C, n, d, family):
  import torch
  from gbsgmc import engine
  X, y, ds, pot, x0, N = _setup(C, n, d, family)
  curvature = N * (4.0 if family == O.LINEAR_GAUSSIAN else 0.25) * \
      max(1.0, 2.0 * d / n)   # of a minibatch, at most about (1 + sqrt(d/n))^2
  h0 = 0.02 / curvature if kind == "langevin" else 0.02 / np.sqrt(curvature)
  h = (h0 * 0.9 ** np.arange(K)).astype(np.float32)
  T = np.ones(K, np.float32)
  keep = np.array([-1, 0, -1, 1, -1, 2], np.int32)
  draws = 2 if kind == "obabo" else 1
  pcg = _cuda(_words(C))
  x, aux = _cuda(x0), None if kind == "langevin" else _cuda(np.zeros_like(x0))
  kw = {} if kind == "langevin" else dict(friction=2.0, leapfrog_steps=3)
  plan = engine.NetPlan(pot, ds, x, aux, n, kind, _cuda(h), _cuda(T),
                        engine.IndexSource(pcg=pcg), 11, block_steps=3,
                        keep_tab=_cuda(keep), n_kept=3, **kw)
  plan.run(0, K)
  plan.check_status()
  idx = np.stack([O.loader_draws(O.loader_rng(c), N, n, K * draws)
                  for c in range(C)], 1)
  xi = lambda tag, k: np.stack([O.philox_normals(11, c, k, tag, d)  # noqa: E731
                                for c in range(C)]).astype(np.float32)
  w, p, kept, lik = x0.copy(), np.zeros_like(x0), [], []
  for k in range(K):
    if kind == "langevin":
      r = _potential(X, y, w, idx[k], N, family)
      w, _ = O.sgld_step(w, r.grad.astype(np.float32), None, xi(0, k), h[k], 1.0,
                         rms_prop=False)
      U = -r.U
    elif kind == "obabo":
      a = _potential(X, y, w, idx[2 * k], N, family)
      w, p, _ = O.obabo_first(w, p, a.grad.astype(np.float32), xi(1, k), h[k], 1.0, 2.0)
      b = _potential(X, y, w, idx[2 * k + 1], N, family)
      p, _ = O.obabo_second(p, b.grad.astype(np.float32), xi(2, k), h[k], 1.0, 2.0)
      U = 0.5 * (a.U + b.U)
    else:
      if k % 3 == 0:
        p = O.sghmc_resample(xi(3, k))
      w, p = O.sghmc_position(w, p, h[k], 2.0)
      r = _potential(X, y, w, idx[k], N, family)
      p = O.sghmc_momentum(p, r.grad.astype(np.float32), xi(4, k), h[k], 2.0)
      U = r.U
    if keep[k] >= 0:
      kept.append(w)
      lik.append(U)
  tol = dict(rtol=1e-4, atol=1e-5)
  np.testing.assert_allclose(x.cpu().numpy(), w, **tol)
  np.testing.assert_allclose(plan.samples.cpu().numpy(), np.stack(kept), **tol)
  np.testing.assert_allclose(plan.sample_lik.cpu().numpy(), np.stack(lik), rtol=1e-5,
                             atol=1e-3)
  sign = -1.0 if kind == "langevin" else 1.0
  np.testing.assert_allclose(plan.U.cpu().numpy(), sign * lik[-1], rtol=1e-5, atol=1e-3)
  if kind != "langevin":
    scale = np.abs(p).max()
    np.testing.assert_allclose(aux.cpu().numpy(), p, rtol=1e-4, atol=1e-4 * scale)
  # The streams stand where numpy's would.
  for c in range(min(C, 3)):
    rng = O.loader_rng(c)
    O.loader_draws(rng, N, n, K * draws)
    s = rng.bit_generator.state["state"]["state"]
    got = pcg[c].cpu().numpy().view(np.uint64)
    assert (int(got[0]) << 64) | int(got[1]) == s
  assert torch.isfinite(plan.lk_var).all()


@pytest.mark.parametrize("layout", ["inline", "unaligned", "unaligned inline"])
@pytest.mark.parametrize("C,n,d", [(1, 65, 4), (2, 500, 33), (1, 200, 131)])
def test_row_layouts_agree(lib, layout, C, n, d):
  """However X and y lie in memory (y its own vector or column d; rows on
  16-byte boundaries, copied whole, or not, copied in words), the same rows
  are summed in the same order: bit-equal states."""
  from gbsgmc import _lib, engine
  X, y, ds, pot, x0, N = _setup(C, n, d, O.LOGISTIC)
  h = (np.full(K, 0.02 / (N * max(1.0, 2.0 * d / n)))).astype(np.float32)
  inline = "inline" in layout
  ld = d + 1 if inline else d
  ld = ld | 1 if "unaligned" in layout else (ld + 3) // 4 * 4
  rows = np.zeros((N, ld), np.float32)
  rows[:, :d] = X
  if inline:
    rows[:, d] = y
  rows, yd = _cuda(rows), _cuda(y)
  base, _ = pot.model(ds)
  other = _lib.Glm(base.family, d, base.n_obs, ld, rows.data_ptr(),
                   None if inline else yd.data_ptr(), base.sigma, base.prior_scale,
                   base.temperature, int(inline), base.n_rows)
  outs = []
  for model in (None, other):
    if model is not None:
      object.__setattr__(pot, "model", lambda *a, **k: (other, (rows, yd)))
    x = _cuda(x0)
    plan = engine.NetPlan(pot, ds, x, None, n, "langevin", _cuda(h),
                          _cuda(np.ones(K, np.float32)),
                          engine.IndexSource(pcg=_cuda(_words(C))), 11, block_steps=3)
    plan.run(0, K)
    plan.check_status()
    outs.append((x.cpu().numpy(), plan.U.cpu().numpy(), plan.lk_var.cpu().numpy()))
  for a, b in zip(*outs):
    np.testing.assert_array_equal(a, b)


class _Given:
  """An index feed that deals out the rows of a [K, C, n] array."""

  def __init__(self, idx):
    self.idx, self.at = idx, 0

  def next(self, g, out):
    out[:g] = self.idx[self.at:self.at + g]
    self.at += g


@pytest.mark.parametrize("bad", [False, True])
@pytest.mark.parametrize("C,n,d", [(1, 2, 2), (2, 131, 3), (1, 258, 31), (70, 67, 32),
                                   (1, 258, 251), (1, 129, 255), (1, 130, 256)])
def test_gathered_rows_agree(lib, C, n, d, bad):
  """Rows copied four at a time (up to 256 columns with y) or one by one
  against rows copied in words: numbers of rows that leave remainders of 1 to
  3, widths around whole 32 bytes and the widest box, and indices beyond the
  last row, which both leave out and report: bit-equal states."""
  from gbsgmc import _lib, engine
  X, y, ds, pot, x0, N = _setup(C, n, d, O.LOGISTIC)
  h = (np.full(K, 0.02 / (N * max(1.0, 2.0 * d / n)))).astype(np.float32)
  idx = np.random.default_rng(n).integers(0, N, (K, C, n)).astype(np.int32)
  idx[:, :, -1] = N - 1
  if bad:
    idx[::2, :, n // 2] = [[N]]
    idx[1::2, :, 0] = [[-1]]
  base, _ = pot.model(ds)
  outs = []
  for ld in ((d + 4) // 4 * 4, (d + 1) | 1):
    rows = np.zeros((N, ld), np.float32)
    rows[:, :d], rows[:, d] = X, y
    rows = _cuda(rows)
    model = _lib.Glm(base.family, d, base.n_obs, ld, rows.data_ptr(), None, base.sigma,
                     base.prior_scale, base.temperature, 1, N)
    object.__setattr__(pot, "model", lambda *a, **k: (model, (rows,)))
    x = _cuda(x0)
    plan = engine.NetPlan(pot, ds, x, None, n, "langevin", _cuda(h),
                          _cuda(np.ones(K, np.float32)), engine.IndexSource(external=True), 11,
                          block_steps=3, feed=_Given(idx))
    plan.run(0, K)
    if bad:
      with pytest.raises(_lib.GbsgmcError) as e:
        plan.check_status()
      assert e.value.code == _lib.ERR_INDEX
    else:
      plan.check_status()
    outs.append((x.cpu().numpy(), plan.U.cpu().numpy(), plan.lk_var.cpu().numpy()))
  for a, b in zip(*outs):
    np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("pairs,n,d", [(1, 33, 7), (2, 256, 64), (1, 900, 300), (90, 40, 12)])
def test_pairs_match_the_per_pair_path(lib, pairs, n, d):
  """alias.re_sgld through the block launches against one chain at a time
  (other launch shapes, so other summation orders: 1e-4 relative)."""
  from gbsgmc import alias, data, engine, likelihoods as L, potential
  rng = np.random.default_rng(d)
  N = 4000
  X = rng.normal(size=(N, d)).astype(np.float32)
  y = (X @ rng.normal(size=d) / np.sqrt(d) + 0.5 * rng.normal(size=N)).astype(np.float32)
  pot = potential.minibatch_potential(L.GaussianPrior(10.0), L.LinearGaussian(sigma=0.5))
  inits = [({"w": (0.1 * rng.normal(size=d)).astype(np.float32)},
            {"w": (0.1 * rng.normal(size=d)).astype(np.float32)}) for _ in range(pairs)]
  first = 0.05 / (4 * N * max(1.0, 2.0 * d / n))
  outs = []
  for fused in (True, False):
    run = alias.re_sgld(pot, data.NumpyDataLoader(x=X, y=y), cache_size=7, batch_size=n,
                        temperature=50.0, first_step_size=first,
                        last_step_size=0.5 * first, burn_in=6, accepted_samples=6)
    engine.FUSED_ENABLED = fused
    try:
      outs.append(run(*(inits if fused else inits[:2]), iterations=12))
    finally:
      engine.FUSED_ENABLED = True
  for a, b in zip(*outs):
    np.testing.assert_allclose(a["samples"]["variables"]["w"], b["samples"]["variables"]["w"],
                               rtol=1e-4, atol=1e-5)
    np.testing.assert_allclose(a["samples"]["likelihood"], b["samples"]["likelihood"],
                               rtol=1e-5, atol=1e-3)


@pytest.mark.parametrize("kind,C,n,d", [("obabo", 1, 4000, 200), ("sghmc", 5, 700, 33),
                                        ("langevin", 40, 300, 101), ("langevin", 200, 90, 6)])
def test_a_wait_that_runs_out_ends_cleanly(lib, monkeypatch, kind, C, n, d):
  """The block launch's bounded waits are its failure detection.  With a bound
  of 0 the first chunks also wait for a copy that never comes, with 1 ns a wait
  may run out anywhere in the run: the launch reports GBSGMC_ERR_TIMEOUT and
  ends, its CTAs staying until no other can send to them.  The device stays
  usable: the same run with the default bound then gives what an untouched one
  gives."""
  from gbsgmc import _lib, engine
  X, y, ds, pot, x0, N = _setup(C, n, d, O.LOGISTIC)
  steps = 24
  h = np.full(steps, 1e-7 if kind == "langevin" else 1e-4, np.float32)
  kw = {} if kind == "langevin" else dict(friction=2.0, leapfrog_steps=3)

  def run():
    x = _cuda(x0)
    plan = engine.NetPlan(pot, ds, x, None if kind == "langevin" else _cuda(np.zeros_like(x0)), n,
                          kind, _cuda(h), _cuda(np.ones(steps, np.float32)),
                          engine.IndexSource(pcg=_cuda(_words(C))), 11, block_steps=12, **kw)
    plan.run(0, steps)
    code = int(plan.status.item())
    plan.close()
    return code, x.cpu().numpy()

  code, want = run()
  assert code == 0
  for limit in ("0", "1", "0"):
    with monkeypatch.context() as m:
      m.setenv("GBSGMC_LOOP_WAIT_NS", limit)
      assert run()[0] in ([_lib.ERR_TIMEOUT] if limit == "0" else [0, _lib.ERR_TIMEOUT])
    code, x = run()
    assert code == 0
    np.testing.assert_array_equal(x, want)


@pytest.mark.parametrize("C,n", [(1, 900), (3, 333), (170, 700)])
@pytest.mark.parametrize("form", ["evaluate", "block"])
def test_variance_of_large_likelihoods(lib, form, C, n):
  """var(lk) = E[lk^2] - E[lk]^2 where it cancels most: whole likelihoods of
  about 2^20 that differ by a few hundred, whose sums over a lane are exact and
  whose totals FP64 holds exactly.  What may then differ from the exact
  variance is the rounding of the means, their square and its subtraction,
  2.5 2^-52 E[lk^2] in all; U: two roundings."""
  import torch
  from gbsgmc import data, engine, likelihoods as L, potential
  N = 3000
  rng = np.random.default_rng(n)
  lk = (2**20 + rng.integers(-300, 300, N)).astype(np.float32)
  ds = data.NumpyDataLoader(x=lk[:, None]).device_dataset()
  pot = potential.minibatch_potential(L.FlatPrior(), L.Linear())
  W = torch.ones((C, 1), device="cuda")
  if form == "evaluate":
    idx = rng.integers(0, N, (C, n)).astype(np.int32)
    r = pot.evaluate(W, _cuda(idx), ds)
    U, var = r.U.cpu().numpy(), r.lk_var.cpu().numpy()
  else:
    idx = np.stack([O.loader_draws(O.loader_rng(c), N, n, 1)[0] for c in range(C)])
    plan = engine.NetPlan(pot, ds, W, None, n, "langevin", _cuda(np.zeros(1, np.float32)),
                          _cuda(np.ones(1, np.float32)), engine.IndexSource(pcg=_cuda(_words(C))),
                          11, block_steps=1)
    plan.run(0, 1)
    plan.check_status()
    U, var = plan.U.cpu().numpy(), plan.lk_var.cpu().numpy()
  for c in range(C):
    v = [int(a) for a in lk[idx[c]]]
    s1, s2 = sum(v), sum(a * a for a in v)
    exact = (n * s2 - s1 * s1) / (n * n)
    assert abs(var[c] - exact) <= 2.5 * 2.0**-52 * s2 / n
    assert abs(U[c] + N * s1 / n) <= 2 * 2.0**-53 * N * s1 / n
