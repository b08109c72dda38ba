"""What a batched AMAGOLD or SGGMC run reports of its chains' starts."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["amagold", "sggmc"])
def test_starts_without_a_finite_potential_are_reported(lib, name):
  """A start whose full potential overflows at one observation, which no
  minibatch of the run holds and the first proposals no longer overflow at: the
  run raises, and the next one, from a start below, does not."""
  from gbsgmc import _lib, alias, data, likelihoods as L, potential
  from oracle import sgmc_oracle as O
  rng = np.random.default_rng(3)
  N, n, steps, iterations = 2000, 32, 4, 2
  X = rng.normal(size=(N, 1)).astype(np.float32)
  draws = steps * iterations * (2 if name == "sggmc" else 1)
  used = {i for c in range(4) for d in O.loader_draws(O.loader_rng(c), N, n, draws) for i in d}
  row = max(set(range(N)) - used)
  X[row] = 3e19   # (3e19)^2 / 2 overflows, (0.1 3e19)^2 / 2 does not
  pot = potential.minibatch_potential(L.GaussianPrior(2.0), L.LinearGaussian(sigma=1.0))
  full = potential.full_potential(L.GaussianPrior(2.0), L.LinearGaussian(sigma=1.0))
  loader = data.NumpyDataLoader(x=X, y=np.zeros(N, np.float32))
  run = getattr(alias, name)(pot, full, loader, cache_size=8, batch_size=n,
                             integration_steps=steps, first_step_size=0.02,
                             last_step_size=0.01, burn_in=1)
  below, above = {"w": np.array([0.1], np.float32)}, {"w": np.array([1.0], np.float32)}
  with pytest.raises(_lib.GbsgmcError) as e:
    run(below, above, iterations=iterations)
  assert e.value.code == _lib.ERR_NONFINITE
  out = run(below, below, iterations=iterations)
  assert all(np.isfinite(r["samples"]["variables"]["w"]).all() for r in out)
