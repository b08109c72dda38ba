"""GLM plans that launch every gradient and update by itself, against the
oracle's trajectories on the same indices and normals.

Tolerance (as for the other K-step trajectories): 1e-4 relative plus 1e-5
absolute; U within 1e-5 relative plus 1e-3 absolute.
"""

import numpy as np
import pytest

from oracle import sgmc_oracle as O

pytestmark = pytest.mark.gpu
K = 6


def _cuda(a):
  import torch
  return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _words(C):
  from gbsgmc.data.numpy_loader import pcg64_words
  return np.array([pcg64_words(c) for c in range(C)], np.uint64).view(np.int64)


def _setup(C, n, d, N=5003):
  from gbsgmc import data, likelihoods as L, potential
  rng = np.random.default_rng(100 * d + n)
  X = rng.normal(size=(N, d)).astype(np.float32)
  y = (rng.random(N) < 1 / (1 + np.exp(-(X @ rng.normal(size=d) / np.sqrt(d))))).astype(np.float32)
  pot = potential.minibatch_potential(L.GaussianPrior(3.0), L.Logistic())
  x0 = (0.1 * rng.normal(size=(C, d))).astype(np.float32)
  return X, y, data.NumpyDataLoader(x=X, y=y).device_dataset(), pot, x0, N


def _schedule(kind, n, d, N):
  curvature = N * 0.25 * max(1.0, 2.0 * d / n)
  h0 = 0.02 / curvature if kind == "langevin" else 0.02 / np.sqrt(curvature)
  return (h0 * 0.9 ** np.arange(K)).astype(np.float32)


def _trajectory(kind, X, y, x0, idx, xi, h, leapfrog, N):
  """Positions, momenta, kept positions and potentials of every step; xi(tag,
  k) gives the normals."""
  w, p, xs, Us = x0.copy(), np.zeros_like(x0), [], []
  at = lambda w, j: O.glm_potential(w, X, y, idx[j], N, O.LOGISTIC, 1.0, 3.0)  # noqa: E731
  for k in range(K):
    if kind == "langevin":
      r = at(w, k)
      w, _ = O.sgld_step(w, r.grad.astype(np.float32), None, xi(0, k), h[k], 1.0, rms_prop=False)
      U = -r.U
    elif kind == "obabo":
      a = at(w, 2 * k)
      w, p, _ = O.obabo_first(w, p, a.grad.astype(np.float32), xi(1, k), h[k], 1.0, 2.0)
      b = at(w, 2 * k + 1)
      p, _ = O.obabo_second(p, b.grad.astype(np.float32), xi(2, k), h[k], 1.0, 2.0)
      U = 0.5 * (a.U + b.U)
    else:
      if k % leapfrog == 0:
        p = O.sghmc_resample(xi(3, k))
      w, p = O.sghmc_position(w, p, h[k], 2.0)
      r = at(w, k)
      p = O.sghmc_momentum(p, r.grad.astype(np.float32), xi(4, k), h[k], 2.0)
      U = r.U
    xs.append(w)
    Us.append(U)
  return w, p, np.stack(xs), np.stack(Us)


def _draws(C, n, N, count):
  return np.stack([O.loader_draws(O.loader_rng(c), N, n, count) for c in range(C)], 1)


@pytest.mark.parametrize("C,n,d", [(1, 33, 1), (3, 200, 129), (170, 40, 6)])
@pytest.mark.parametrize("kind", ["langevin", "obabo", "sghmc"])
def test_injected_normals(lib, monkeypatch, kind, C, n, d):
  """A plan whose caller gives the normals, with kept samples."""
  from gbsgmc import _lib, engine
  X, y, ds, pot, x0, N = _setup(C, n, d)
  z = np.random.default_rng(5).normal(size=(C, d)).astype(np.float32)
  zd, make = _cuda(z), _lib.noise
  monkeypatch.setattr(_lib, "noise", lambda *a: make(*a, noise_dev=zd, noise_stride=d))
  h = _schedule(kind, n, d, N)
  keep = np.array([-1, 0, -1, 1, -1, 2], np.int32)
  draws = 2 if kind == "obabo" else 1
  pcg, x = _cuda(_words(C)), _cuda(x0)
  aux = None if kind == "langevin" else _cuda(np.zeros_like(x0))
  kw = {} if kind == "langevin" else dict(friction=2.0, leapfrog_steps=3)
  plan = engine.NetPlan(pot, ds, x, aux, n, kind, _cuda(h), _cuda(np.ones(K, np.float32)),
                        engine.IndexSource(pcg=pcg), 11, block_steps=3, keep_tab=_cuda(keep),
                        n_kept=3, **kw)
  plan.run(0, K)
  plan.check_status()
  w, p, xs, Us = _trajectory(kind, X, y, x0, _draws(C, n, N, K * draws), lambda tag, k: z, h, 3, N)
  tol = dict(rtol=1e-4, atol=1e-5)
  np.testing.assert_allclose(x.cpu().numpy(), w, **tol)
  np.testing.assert_allclose(plan.samples.cpu().numpy(), xs[keep >= 0], **tol)
  np.testing.assert_allclose(plan.sample_lik.cpu().numpy(), Us[keep >= 0], rtol=1e-5, atol=1e-3)
  if aux is not None:
    np.testing.assert_allclose(aux.cpu().numpy(), p, rtol=1e-4, atol=1e-4 * np.abs(p).max())


@pytest.mark.parametrize("C,n,d,block", [(2, 1100, 40, 6), (2, 90, 12, 3)])
def test_injected_normals_sgld_plan(lib, monkeypatch, C, n, d, block):
  """The SGLD plan of few chains: minibatches above 1,024 rows or blocks below
  six steps, also where a plan with its own normals has made its choice."""
  from gbsgmc import _lib, engine
  monkeypatch.delenv("GBSGMC_AUTOTUNE", raising=False)
  X, y, ds, pot, x0, N = _setup(C, n, d)
  h = _schedule("langevin", n, d, N)
  z = np.random.default_rng(6).normal(size=(C, d)).astype(np.float32)
  zd, make = _cuda(z), _lib.noise

  def run():
    x = _cuda(x0)
    plan = engine.SgldGlmPlan(pot, ds, x, None, 0.9, 1e-5, n, _cuda(h),
                              _cuda(np.ones(K, np.float32)), _cuda(np.full(K, -1, np.int32)), 0,
                              engine.IndexSource(pcg=_cuda(_words(C))), 11, 0, block)
    plan.run(0, K)
    plan.check_status()
    return x.cpu().numpy()

  run()
  monkeypatch.setattr(_lib, "noise", lambda *a: make(*a, noise_dev=zd, noise_stride=d))
  w, _, _, _ = _trajectory("langevin", X, y, x0, _draws(C, n, N, K), lambda tag, k: z, h, 3, N)
  np.testing.assert_allclose(run(), w, rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("C,n,d,block", [(1, 8100, 260, False), (1, 7000, 260, True),
                                         (2, 2900, 1000, False), (96, 50, 3, True)])
@pytest.mark.parametrize("kind", ["obabo", "sghmc"])
def test_long_minibatches_of_few_chains(lib, kind, C, n, d, block):
  """Few chains with long minibatches get launches of their own for every
  gradient, which spread a chain over more CTAs than a cluster has; others run
  a block of steps in one launch."""
  from gbsgmc import engine
  X, y, ds, pot, x0, N = _setup(C, n, d, N=9001)
  h = _schedule(kind, n, d, N)
  keep = np.array([0, -1, 1, -1, -1, 2], np.int32)
  draws = 2 if kind == "obabo" else 1
  x, aux = _cuda(x0), _cuda(np.zeros_like(x0))
  plan = engine.NetPlan(pot, ds, x, aux, n, kind, _cuda(h), _cuda(np.ones(K, np.float32)),
                        engine.IndexSource(pcg=_cuda(_words(C))), 11, block_steps=3,
                        keep_tab=_cuda(keep), n_kept=3, friction=2.0, leapfrog_steps=3)
  plan.run(0, K)
  plan.check_status()
  per_block = engine._plan_launches(plan.handle, 2 * 3) - engine._plan_launches(plan.handle, 3)
  assert (per_block == 3) == block   # index draw, block, counter
  xi = lambda tag, k: np.stack([O.philox_normals(11, c, k, tag, d)  # noqa: E731
                                for c in range(C)]).astype(np.float32)
  w, p, xs, Us = _trajectory(kind, X, y, x0, _draws(C, n, N, K * draws), xi, h, 3, N)
  tol = dict(rtol=1e-4, atol=1e-5)
  np.testing.assert_allclose(x.cpu().numpy(), w, **tol)
  np.testing.assert_allclose(plan.samples.cpu().numpy(), xs[keep >= 0], **tol)
  np.testing.assert_allclose(plan.sample_lik.cpu().numpy(), Us[keep >= 0], rtol=1e-5, atol=1e-3)
  np.testing.assert_allclose(aux.cpu().numpy(), p, rtol=1e-4, atol=1e-4 * np.abs(p).max())


@pytest.mark.parametrize("n,d,block", [(5000, 300, False), (1600, 1000, False), (900, 300, True)])
def test_long_minibatches_of_pairs(lib, monkeypatch, n, d, block):
  """alias.re_sgld of one pair on both sides of the line between the block
  launch and launches per step, against one chain at a time (other launch
  shapes, so other summation orders: 1e-4 relative)."""
  from gbsgmc import alias, data, engine, likelihoods as L, potential
  rng = np.random.default_rng(d)
  N = 6000
  X = rng.normal(size=(N, d)).astype(np.float32)
  y = (X @ rng.normal(size=d) / np.sqrt(d) + 0.5 * rng.normal(size=N)).astype(np.float32)
  pot = potential.minibatch_potential(L.GaussianPrior(10.0), L.LinearGaussian(sigma=0.5))
  inits = [({"w": (0.1 * rng.normal(size=d)).astype(np.float32)},
            {"w": (0.1 * rng.normal(size=d)).astype(np.float32)}) for _ in range(2)]
  first = 0.05 / (4 * N * max(1.0, 2.0 * d / n))
  blocks = []
  run_plan = engine.ResgldPairsPlan.run
  monkeypatch.setattr(engine.ResgldPairsPlan, "run", lambda p, *a: (
      blocks.append(p.launches(2 * 7) - p.launches(7)), run_plan(p, *a))[1])
  outs = []
  for fused in (True, False):
    run = alias.re_sgld(pot, data.NumpyDataLoader(x=X, y=y), cache_size=7, batch_size=n,
                        temperature=50.0, first_step_size=first,
                        last_step_size=0.5 * first, burn_in=6, accepted_samples=6)
    monkeypatch.setattr(engine, "FUSED_ENABLED", fused)
    outs.append(run(*inits, iterations=12))
  assert [b == 3 for b in blocks] == [block]   # index draw, block, counter
  for a, b in zip(*outs):
    np.testing.assert_allclose(a["samples"]["variables"]["w"], b["samples"]["variables"]["w"],
                               rtol=1e-4, atol=1e-5)
    np.testing.assert_allclose(a["samples"]["likelihood"], b["samples"]["likelihood"],
                               rtol=1e-5, atol=1e-3)


def test_injected_normals_of_pairs(lib, monkeypatch):
  """A pairs plan given its first step's Philox normals makes that step."""
  import torch
  from gbsgmc import _lib, engine
  P, n, d = 3, 200, 33
  X, y, ds, pot, _, N = _setup(2 * P, n, d)
  x0 = (0.1 * np.random.default_rng(1).normal(size=(2 * P, d))).astype(np.float32)
  z = _cuda(np.stack([O.philox_normals(11, c, 0, 0, d) for c in range(2 * P)]).astype(np.float32))
  make, outs = _lib.noise, []
  for injected in (False, True):
    if injected:
      monkeypatch.setattr(_lib, "noise", lambda *a: make(*a, noise_dev=z, noise_stride=d))
    x = _cuda(x0)
    ident = torch.arange(2 * P, dtype=torch.int32, device="cuda").view(P, 2).T.reshape(-1)
    ladder = torch.tensor([1.0] * P + [50.0] * P, device="cuda")
    plan = engine.ResgldPairsPlan(
        pot, ds, x, None, 0.9, 1e-5, n, _cuda(np.full(1, 1e-5, np.float32)),
        _cuda(np.ones(1, np.float32)), _cuda(np.full(1, -1, np.int32)), ladder, 0,
        _cuda(_words(2 * P)), ident.contiguous(),
        torch.arange(0, 2 * P, 2, dtype=torch.int32, device="cuda"),
        torch.zeros(P, dtype=torch.float64, device="cuda"),
        torch.zeros(P, dtype=torch.int64, device="cuda"), 1.0, 5, 11, 0, 1)
    plan.run(0, 1)
    plan.check_status()
    outs.append([a.cpu().numpy() for a in (x, plan.U, plan.lk_var, plan.ident)])
  for a, b in zip(*outs):
    np.testing.assert_allclose(a, b, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("n,block", [(2000, False), (1200, True)])
@pytest.mark.parametrize("name", ["amagold", "sggmc"])
def test_long_minibatches_of_mh_chains(lib, monkeypatch, name, n, block):
  """AMAGOLD and SGGMC of a few chains on both sides of the line between
  trajectories of one launch and of launches per gradient and update.  With
  four slices a minibatch everywhere, the latter are the per-chain path's
  arithmetic: the same bits; the former: 1e-4 relative plus 1e-5 absolute."""
  from gbsgmc import alias, data, engine, likelihoods as L, potential
  monkeypatch.setenv("GBSGMC_GLM_SLICES", "4")
  rng = np.random.default_rng(n)
  N, d, C = 2500, 1000, 2
  X = rng.normal(size=(N, d)).astype(np.float32)
  y = (rng.random(N) < 0.5).astype(np.float32)
  pot = potential.minibatch_potential(L.GaussianPrior(2.0), L.Logistic())
  full = potential.full_potential(L.GaussianPrior(2.0), L.Logistic())
  inits = [{"w": (0.01 * rng.normal(size=d)).astype(np.float32)} for _ in range(C)]
  loops, make = [], engine._lib.call

  def call(fn, *args):
    if fn == "gbsgmc_plan_run":
      per = [int(engine._lib.load().gbsgmc_plan_launches(args[0], 3 * k)) for k in (1, 2)]
      loops.append(per[1] - per[0] == 3)   # trajectory, full pass, decision
    return make(fn, *args)

  monkeypatch.setattr(engine._lib, "call", call)
  outs = []
  for fused in (True, False):
    monkeypatch.setattr(engine, "FUSED_ENABLED", fused)
    sampler = alias.amagold if name == "amagold" else alias.sggmc
    run = sampler(pot, full, data.NumpyDataLoader(x=X, y=y), cache_size=8, batch_size=n,
                  integration_steps=3, first_step_size=0.004, last_step_size=0.002, burn_in=2)
    outs.append(run(*inits, iterations=6))
  assert loops == [block]
  for a, b in zip(*outs):
    for key in ("energy", "variables"):
      va, vb = (np.asarray(r["samples"][key]["w"] if key == "variables" else r["samples"][key])
                for r in (a, b))
      if block:
        np.testing.assert_allclose(va, vb, rtol=1e-4, atol=1e-5 if key == "variables" else 1e-3)
      else:
        np.testing.assert_array_equal(va, vb)
    assert np.isfinite(va).all()
