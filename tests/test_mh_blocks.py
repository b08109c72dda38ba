"""Which AMAGOLD and SGGMC runs the batched plan takes, and in which blocks."""

import pytest

from gbsgmc import engine


@pytest.mark.parametrize("steps,block", [(1, 50), (10, 5), (50, 1), (51, 1), (100_000, 1),
                                         (100_001, 0), (1_000_000, 0)])
def test_long_trajectories(steps, block):
  """A plan's block holds at most 100,000 integrator steps and one iteration at
  least; longer trajectories are left to the launches from the host."""
  assert engine.mh_block_iterations(steps, 2, 3, 1) == block


@pytest.mark.parametrize("steps,chains,n,draws", [
    (1, 1, 1, 2), (1, 1000, 65536, 1), (1, 4096, 65536, 1), (1, 4096, 65536, 2),
    (10, 400, 65536, 1), (10, 400, 65536, 2), (3, 5000, 10000, 1), (3, 5000, 10000, 2)])
def test_blocks_of_large_runs(steps, chains, n, draws):
  """A block's index buffer stays within 1 GiB, whatever the draws and the
  iterations in it."""
  block = engine.mh_block_iterations(steps, chains, n, draws)
  one = 4 * steps * chains * n * draws
  assert block * one <= 1 << 30
  assert (block > 0) == (one <= 1 << 30)
  assert block == 0 or block == max(1, 50 // steps) or (block + 1) * one > 1 << 30
