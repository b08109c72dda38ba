"""A sampler's functions hold its dataset only as long as someone holds them:
no reference cycle that waits for a garbage collection."""

import gc
import weakref

import numpy as np
import pytest

from gbsgmc import data, integrator, likelihoods as L, potential, solver


def _parts():
  x = np.zeros((8, 3), np.float32)
  loader = data.NumpyDataLoader(x=x, y=x[:, 0])
  batches = data.random_reference_data(loader, 2, 4)
  pot = potential.minibatch_potential(L.GaussianPrior(1.0), L.LinearGaussian(sigma=1.0))
  return loader, batches, pot


@pytest.mark.parametrize("make", ["langevin_diffusion", "obabo", "friction_leapfrog",
                                  "reversible_leapfrog", "amagold"])
def test_dropped_sampler_is_freed(make):
  loader, batches, pot = _parts()
  ref = weakref.ref(loader)
  gc.collect()
  gc.disable()
  try:
    if make == "amagold":
      full = potential.full_potential(L.GaussianPrior(1.0), L.LinearGaussian(sigma=1.0))
      kernel = solver.amagold(integrator.reversible_leapfrog(pot, batches, 2, 0.25), full,
                              data.full_reference_data(loader, 2, 4))
    else:
      kernel = getattr(integrator, make)(pot, batches)
    assert getattr(kernel[0], "many", None) is not None
    del loader, batches, pot, kernel
    assert ref() is None
  finally:
    gc.enable()
