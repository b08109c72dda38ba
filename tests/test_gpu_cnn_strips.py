"""The CNN's kernels that build or read their operands by strips and units of
image rows (conv1, its weight gradient, conv2 and its gradients) where runs of
strips, units and slices are cut: a handful of images (split boundaries inside
a unit, CTAs without a strip), minibatches that are no multiple of four (other
split factors), one to eight chains (the weight gradient's column shifts apart
or in one CTA; strips of several chains in one CTA), and images whose rows are
not 8-byte aligned.

Tolerance against the oracle with BF16 operands: a value whose fp32 and
float64 forms round to different BF16 neighbours moves its image's lk by up to
3e-2 (1 + |lk|), U by the sum of those, and a leaf's gradient by 1e-2 of its
norm at 16 images, in proportion to an image's share of the minibatch.
"""

import numpy as np
import pytest

import test_gpu_cnn as base
from oracle import sgmc_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,n", [(1, 2), (1, 6), (3, 10), (2, 50), (8, 12)])
def test_small_and_ragged_minibatches(lib, C, n):
  N = 200
  lik, images, labels, W, idx, ds, pot, Wd, idxd = base.setup(N, C, n, seed=40 + n)
  r = pot.evaluate(Wd, idxd, ds, grad=True, lk=True, observation_count=N)
  pot.check_status()
  for c in range(C):
    ref = O.cnn_potential(W[c], images.reshape(N, -1), labels, idx[c], N, prior_scale=1.0,
                          bf16_operands=True)
    lk = ref.lk[0]
    flip = 3e-2 * (1 + np.abs(lk))
    assert np.all(np.abs(r.lk[c].cpu().numpy() - lk) <= flip)
    assert abs(float(r.U[c]) - ref.U[0]) <= N / n * flip.sum()
    bound = 1e-2 * max(1.0, 16 / n)
    errs = base.leaf_errors(r.grad[c].cpu().numpy(), ref.grad[0])
    assert all(rel <= bound for rel, _ in errs.values()), errs


def test_unaligned_images(lib):
  """Image rows at odd strides and a 4-byte offset: the same bits."""
  import torch
  from gbsgmc import _lib
  N, C, n = 60, 2, 6
  lik, images, labels, W, idx, ds, pot, Wd, idxd = base.setup(N, C, n, seed=3)
  a = pot.evaluate(Wd, idxd, ds, grad=True, lk=True, observation_count=N)
  rows = torch.zeros(N * 3075 + 1, device="cuda")
  view = rows[1:].view(N, 3075)
  view[:, :3072] = torch.from_numpy(images.reshape(N, -1)).cuda()
  view[:, 3072] = torch.from_numpy(labels).cuda()
  m, _ = pot.model(ds)
  other = _lib.Cnn(m.n_obs, m.n_rows, 3075, view.data_ptr(), view.data_ptr() + 4 * 3072, 3075,
                   m.prior_scale, m.temperature)
  object.__setattr__(pot, "model", lambda *args, **kw: (other, (rows,)))
  b = pot.evaluate(Wd, idxd, ds, grad=True, lk=True, observation_count=N)
  pot.check_status()
  assert torch.equal(a.U, b.U) and torch.equal(a.lk, b.lk) and torch.equal(a.grad, b.grad)


@pytest.mark.parametrize("C,n", [(5, 64), (6, 50), (9, 2)])
def test_weight_gradients_do_not_depend_on_the_batch(lib, C, n):
  """Many chains (dW3 by column shift) and one (by tap): the same sums in the
  same order, so the same bits."""
  import torch
  N = 200
  lik, images, labels, W, idx, ds, pot, Wd, idxd = base.setup(N, C, n, seed=n)
  many = pot.evaluate(Wd, idxd, ds, grad=True, lk=True, observation_count=N)
  for c in range(C):
    one = pot.evaluate(Wd[c:c + 1], idxd[c:c + 1], ds, grad=True, lk=True, observation_count=N)
    assert torch.equal(many.grad[c], one.grad[0]) and torch.equal(many.U[c], one.U[0])
  pot.check_status()
