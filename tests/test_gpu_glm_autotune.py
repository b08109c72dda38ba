"""The SGLD plan's choice of a launch form and what it may leave behind: its
trials run on scratch copies, read no more of the schedule than the run has,
and report to a scratch status word.
"""

import numpy as np
import pytest

from oracle import sgmc_oracle as O

pytestmark = pytest.mark.gpu


def _cuda(a):
  import torch
  return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _words(C):
  from gbsgmc.data.numpy_loader import pcg64_words
  return np.array([pcg64_words(c) for c in range(C)], np.uint64).view(np.int64)


def _setup(C, d, N=5003):
  from gbsgmc import data, likelihoods as L, potential
  rng = np.random.default_rng(d)
  X = rng.normal(size=(N, d)).astype(np.float32)
  y = (rng.random(N) < 0.5).astype(np.float32)
  lik = L.Logistic()
  pot = potential.minibatch_potential(L.GaussianPrior(3.0), lik)
  x0 = (0.1 * rng.normal(size=(C, d))).astype(np.float32)
  ds = data.NumpyDataLoader(x=X, y=y).device_dataset()
  return lik, ds, pot, x0, N


@pytest.mark.parametrize("C,n,d,K", [(96, 93, 21, 6), (160, 71, 21, 8), (600, 35, 9, 11)])
def test_trials_stay_within_a_short_schedule(lib, monkeypatch, C, n, d, K):
  """Runs of 6 to 11 steps with more chains than half the SMs.  The first plan
  of a shape makes the trials; its tables end where the run does, and what
  follows them in the same buffer (finite, absurd) reaches neither the status
  nor the chains: the second plan, which takes over the first one's choice,
  gives the same bits with zeros there."""
  from gbsgmc import engine
  monkeypatch.delenv("GBSGMC_AUTOTUNE", raising=False)
  _, ds, pot, x0, N = _setup(C, d)
  h = (0.02 / (0.25 * N) * 0.9 ** np.arange(K)).astype(np.float32)
  outs = []
  for rest in (1e30, 0.0):
    h_buf, t_buf = np.full(64, rest, np.float32), np.full(64, rest, np.float32)
    h_buf[:K], t_buf[:K] = h, 1.0
    x, v = _cuda(x0), _cuda(np.zeros_like(x0))
    plan = engine.SgldGlmPlan(pot, ds, x, v, 0.9, 1e-5, n, _cuda(h_buf), _cuda(t_buf),
                              _cuda(np.full(K, -1, np.int32)), 0,
                              engine.IndexSource(pcg=_cuda(_words(C))), 11, 0, K)
    plan.run(0, K)
    plan.check_status()
    outs.append([plan.launch_shape()] + [a.cpu().numpy() for a in (x, v, plan.U, plan.lk_var)])
  for a, b in zip(*outs):
    np.testing.assert_array_equal(a, b)
  assert np.isfinite(outs[0][1]).all() and (outs[0][1] != x0).all()


@pytest.mark.parametrize("C,n,d", [(1, 1024, 40), (3, 1500, 24)])
def test_a_sampler_leaves_gradient_calls_as_they_were(lib, monkeypatch, C, n, d):
  """One evaluation before and after an SGLD plan of its shape whose form was
  chosen without a trial: the same bits."""
  import torch
  from gbsgmc import engine
  monkeypatch.delenv("GBSGMC_AUTOTUNE", raising=False)
  _, ds, pot, x0, N = _setup(C, d)
  idx = torch.from_numpy(np.random.default_rng(n).integers(0, N, (C, n)).astype(np.int32)).cuda()
  K = 12

  def evaluate():
    r = pot.evaluate(_cuda(x0), idx, ds)
    return [a.cpu().numpy() for a in (r.U, r.grad, r.lk_var)]

  before = evaluate()
  plan = engine.SgldGlmPlan(pot, ds, _cuda(x0), None, 0.9, 1e-5, n,
                            _cuda(np.full(K, 1e-6, np.float32)), _cuda(np.ones(K, np.float32)),
                            _cuda(np.full(K, -1, np.int32)), 0,
                            engine.IndexSource(pcg=_cuda(_words(C))), 11, 0, K)
  plan.run(0, K)
  plan.check_status()
  for a, b in zip(before, evaluate()):
    np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("multi,steps", [("1", 12), ("0", 1)])
def test_forced_launch_form(lib, monkeypatch, multi, steps):
  """GBSGMC_GLM_MULTISTEP where the plan would choose a cluster per chain: one
  launch a block (index draw, block, counter) or one a step, as it promises."""
  from gbsgmc import engine
  monkeypatch.delenv("GBSGMC_AUTOTUNE", raising=False)
  monkeypatch.setenv("GBSGMC_GLM_MULTISTEP", multi)
  C, n, d, K = 2, 600, 17, 12
  _, ds, pot, x0, N = _setup(C, d)
  plan = engine.SgldGlmPlan(pot, ds, _cuda(x0), None, 0.9, 1e-5, n,
                            _cuda(np.full(K, 1e-6, np.float32)), _cuda(np.ones(K, np.float32)),
                            _cuda(np.full(K, -1, np.int32)), 0,
                            engine.IndexSource(pcg=_cuda(_words(C))), 11, 0, K)
  plan.run(0, K)
  plan.check_status()
  shape = plan.launch_shape()
  assert shape[5] == steps
  assert multi == "0" or shape[0] == 1


@pytest.mark.parametrize("n,d,block", [(400, 1000, True), (30000, 1000, False)])
def test_few_chains_with_long_minibatches(lib, monkeypatch, n, d, block):
  """One chain: a cluster and one launch a block for short minibatches, a
  launch a step over more CTAs for one that takes a cluster six times as long,
  against the oracle (1e-4 relative plus 1e-5 absolute)."""
  from gbsgmc import engine
  monkeypatch.delenv("GBSGMC_AUTOTUNE", raising=False)
  N, K = 30011, 6
  _, ds, pot, x0, N = _setup(1, d, N)
  rng = np.random.default_rng(d)   # as _setup draws them
  X = rng.normal(size=(N, d)).astype(np.float32)
  y = (rng.random(N) < 0.5).astype(np.float32)
  h = (0.02 / (0.25 * N * max(1.0, 2.0 * d / n)) * 0.9 ** np.arange(K)).astype(np.float32)
  x = _cuda(x0)
  plan = engine.SgldGlmPlan(pot, ds, x, None, 0.9, 1e-5, n, _cuda(h),
                            _cuda(np.ones(K, np.float32)), _cuda(np.full(K, -1, np.int32)), 0,
                            engine.IndexSource(pcg=_cuda(_words(1))), 11, 0, K)
  plan.run(0, K)
  plan.check_status()
  assert (plan.launch_shape()[5] == K) == block
  idx = O.loader_draws(O.loader_rng(0), N, n, K)
  w = x0
  for k in range(K):
    r = O.glm_potential(w, X, y, idx[k][None], N, O.LOGISTIC, 1.0, 3.0)
    w, _ = O.sgld_step(w, r.grad.astype(np.float32), None,
                       O.philox_normals(11, 0, k, 0, d)[None].astype(np.float32), h[k], 1.0,
                       rms_prop=False)
  np.testing.assert_allclose(x.cpu().numpy(), w, rtol=1e-4, atol=1e-5)
