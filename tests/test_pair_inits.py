"""Initial states of reSGLD pairs made in bulk: what a pair may hold."""

from typing import Any, NamedTuple

import pytest


class _Chain(NamedTuple):
  sample: Any
  chain: int
  key: int


@pytest.fixture
def solver(monkeypatch):
  """parallel_tempering over an integrator that only numbers its chains."""
  import torch
  from gbsgmc import solver as S
  for name in ("full", "zeros"):   # the pair's words on the CPU
    real = getattr(torch, name)
    monkeypatch.setattr(torch, name,
                        lambda *a, _real=real, device=None, **k: _real(*a, **k))
  made = []

  def init(sample, key=0):
    made.append(_Chain(sample, len(made), key))
    return made[-1]

  init.many = lambda samples, key=0: [init(s, key) for s in samples]
  return S.parallel_tempering((init, None, None))


def test_pairs_of_two(solver):
  states = solver[0].many([("a", "b"), ["c", "d"], iter(("e", "f"))])
  assert [(s.normal.sample, s.hot.sample) for s in states] == [("a", "b"), ("c", "d"), ("e", "f")]
  assert [s.pair_chain for s in states] == [0, 2, 4]


def test_pairs_with_their_own_arguments(solver):
  """Two samples and the starting variance, as init takes them."""
  states = solver[0].many([(0.1, 0.2, 0.5), (0.3, 0.4, 0.25)])
  assert [(s.normal.sample, s.hot.sample, float(s.ssq)) for s in states] == [
      (0.1, 0.2, 0.5), (0.3, 0.4, 0.25)]


@pytest.mark.parametrize("pairs", [[(0.1,), (0.2,)], [({"w": 0}, {"w": 1}, {"w": 2})] * 2,
                                   [(0.1, 0.2), (0.3,)]])
def test_what_is_no_pair_is_refused(solver, pairs):
  with pytest.raises(TypeError):
    solver[0].many(pairs)
