"""The tanh network at hidden widths whose 16-byte columns do not divide a
block's threads (768: 96 columns, 256 threads), and ragged minibatches long
enough for the 256-row tiles of the CTA-pair GEMMs, against torch in float64.

Tolerance: the network's BF16 operands (8-bit significands) leave each
gradient leaf within 6e-2 relative L2 error, as in the other network tests.
"""

import numpy as np
import pytest

from oracle import sgmc_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h1,h2,rows", [
    (256, 768, None), (768, 1280, None), (512, 256, [1, 129, 600, 1280])])
def test_gradient_matches_oracle(lib, h1, h2, rows):
  import torch
  from gbsgmc import data, likelihoods as L, potential
  N, D, C = 3000, 64, 4 if rows else 2
  n = 1280 if rows else 256
  rng = np.random.default_rng(h1 + h2)
  X = rng.normal(size=(N, D)).astype(np.float32)
  y = rng.normal(size=N).astype(np.float32)
  lik = L.MLPGaussian(d_in=D, h1=h1, h2=h2, sigma=0.5)
  pot = potential.minibatch_potential(L.GaussianPrior(1.0), lik)
  W = np.stack([lik.init(np.random.default_rng(c)) for c in range(C)])
  idx = rng.integers(0, N, (C, n)).astype(np.int32)
  r = pot.evaluate(torch.from_numpy(W).cuda(), torch.from_numpy(idx).cuda(),
                   data.NumpyDataLoader(x=X, y=y).device_dataset(),
                   rows=None if rows is None else torch.tensor(rows))
  pot.check_status()
  g = r.grad.cpu().numpy().astype(np.float64)
  for c in range(C):
    m = n if rows is None else rows[c]
    ref = O.mlp_potential(W[c:c + 1], X, y, idx[c:c + 1, :m], N, D, h1, h2, 0.5,
                          prior_scale=1.0)
    np.testing.assert_allclose(r.U[c].item(), ref.U[0], rtol=1e-2)
    for a, b in zip(lik.unravel(g[c]).values(), lik.unravel(ref.grad[0]).values()):
      assert np.linalg.norm(a - b) <= 6e-2 * np.linalg.norm(b) + 1e-6
