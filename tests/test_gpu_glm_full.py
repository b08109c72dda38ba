"""The full-data potential of many chains (glm_full.cu) at the edges of its
row tiles (256), feature panels (16) and chain groups (4 and 16), against the
oracle in float64.

Tolerance: each likelihood is an fp32 value of relative error about 1e-6 (its
dot product over up to 1,021 features and its link), their sum is
compensated: U within 1e-6 relative of the sum of the likelihoods' magnitudes.
A chain's value must not depend on the other chains: bit for bit.
"""

import numpy as np
import pytest

from oracle import sgmc_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,d,C,family", [
    (1, 1, 1, O.LINEAR_GAUSSIAN),
    (255, 7, 4, O.LOGISTIC),
    (257, 33, 5, O.LINEAR_GAUSSIAN),
    (5000, 64, 17, O.LOGISTIC),
    (70001, 32, 3, O.LOGISTIC),
    (600, 1021, 2, O.LOGISTIC),
])
def test_full_potential_matches_oracle(lib, N, d, C, family):
  import torch
  from gbsgmc import data, likelihoods as L, potential
  rng = np.random.default_rng(N + d)
  X = rng.normal(size=(N, d)).astype(np.float32)
  lik = L.Logistic() if family == O.LOGISTIC else L.LinearGaussian(sigma=0.5)
  y = (rng.random(N) < 0.5 if family == O.LOGISTIC else rng.normal(size=N)).astype(np.float32)
  W = (rng.normal(size=(C, d)) / np.sqrt(d)).astype(np.float32)
  full = potential.full_potential(L.GaussianPrior(2.0), lik, temperature=1.5)
  ds = data.NumpyDataLoader(x=X, y=y).device_dataset()
  Wd = torch.from_numpy(W).cuda()
  U = full.value_all(Wd, ds).cpu().numpy()
  for c in range(C):
    ref = O.glm_potential(W[c:c + 1], X, y, np.arange(N)[None], N, family, 0.5, 2.0, 1.5)
    assert abs(U[c] - ref.U[0]) <= 1e-6 * (np.abs(ref.lk).sum() + 1.0)
  one = torch.cat([full.value_all(Wd[c:c + 1], ds) for c in range(C)]).cpu().numpy()
  np.testing.assert_array_equal(U, one)


def test_infinite_likelihoods_stay_infinite(lib):
  """A likelihood sum that overflows gives U = +inf (a proposal the MH
  decision rejects), not NaN."""
  import torch
  from gbsgmc import data, likelihoods as L, potential
  X = np.full((300, 2), 1e30, np.float32)
  full = potential.full_potential(L.FlatPrior(), L.LinearGaussian(sigma=1.0))
  ds = data.NumpyDataLoader(x=X, y=np.zeros(300, np.float32)).device_dataset()
  U = full.value_all(torch.tensor([[1.0, 0.0], [0.0, 0.0]], device="cuda"), ds).cpu().numpy()
  assert U[0] == np.inf and np.isfinite(U[1])


@pytest.mark.parametrize("C", [1, 5])
def test_sums_keep_every_bit_of_fp64(lib, C):
  """Whole likelihoods of three sizes (2^51; 36 bits; below 1,000) whose sum
  FP64 holds exactly: every partial sum does, and so does U (no prior,
  temperature 1)."""
  import torch
  from gbsgmc import data, likelihoods as L, potential
  rng = np.random.default_rng(C)
  N = 256 * 40   # a tile a CTA, two observations a thread
  lk = (rng.integers(2**23, 2**24, N) << 12).astype(np.int64)
  small = rng.random(N) < 0.5
  lk[small] = rng.integers(1, 1000, small.sum())
  lk[[77, 5000]] = 2**51
  x = lk.astype(np.float32)
  assert (x.astype(np.int64) == lk).all() and lk.sum() < 2**53
  full = potential.full_potential(L.FlatPrior(), L.Linear())
  U = full.value_all(torch.ones((C, 1), device="cuda"),
                     data.NumpyDataLoader(x=x[:, None]).device_dataset()).cpu().numpy()
  assert (-U == float(lk.sum())).all()


@pytest.mark.parametrize("d", [5, 16, 33, 64, 100, 256, 700, 1024])
def test_dot_products_are_as_exact_as_the_minibatch_kernels(lib, d):
  """One observation, 4,096 chains, likelihood x . w, normal x and w: the rms
  distance of the full potential from the exact one against that of the
  minibatch kernel's likelihood.  The ratio of two such estimates scatters by
  1.6 %; three times that is allowed."""
  import torch
  from gbsgmc import data, likelihoods as L, potential
  rng = np.random.default_rng(d)
  C = 4096
  x = rng.normal(size=(1, d)).astype(np.float32)
  W = rng.normal(size=(C, d)).astype(np.float32)
  ds = data.NumpyDataLoader(x=x).device_dataset()
  Wd = torch.from_numpy(W).cuda()
  full = potential.full_potential(L.FlatPrior(), L.Linear())
  pot = potential.minibatch_potential(L.FlatPrior(), L.Linear())
  one = pot.evaluate(Wd, torch.zeros((C, 1), dtype=torch.int32, device="cuda"), ds, lk=True)
  exact = (W.astype(np.float64) * x.astype(np.float64)).sum(1)
  rms = lambda z: np.sqrt(np.mean((z - exact) ** 2))  # noqa: E731
  ours = rms(-full.value_all(Wd, ds).cpu().numpy())
  assert 0 < ours <= 1.05 * rms(one.lk.cpu().numpy()[:, 0].astype(np.float64))


def test_infinite_dot_products_stay_infinite(lib):
  """A dot product that overflows gives an infinite potential, not NaN; a
  finite chain beside it keeps its value."""
  import torch
  from gbsgmc import data, likelihoods as L, potential
  X = np.full((300, 40), 1e30, np.float32)
  full = potential.full_potential(L.FlatPrior(), L.Linear())
  ds = data.NumpyDataLoader(x=X).device_dataset()
  W = torch.zeros((3, 40), device="cuda")
  W[0, :] = 1e20
  W[1, 39] = -1e20
  W[2, 7] = 1e-30
  U = full.value_all(W, ds).cpu().numpy()
  assert U[0] == -np.inf and U[1] == np.inf and abs(U[2] + 300) < 1e-4
