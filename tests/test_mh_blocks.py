"""Which AMAGOLD and SGGMC runs the batched plan takes, and in which blocks."""

import pytest

from gbsgmc import engine


@pytest.mark.parametrize("steps,block", [(1, 50), (10, 5), (50, 1), (51, 1), (100_000, 1),
                                         (100_001, 0), (1_000_000, 0)])
def test_long_trajectories(steps, block):
  """A plan's block holds at most 100,000 integrator steps and one iteration at
  least; longer trajectories are left to the launches from the host."""
  assert engine.mh_block_iterations(steps, 2, 3, 1) == block
