"""The exhaustive 3-opt's units of work (four rows by 32 columns), cluster sizes and delta
widths, against the oracle: sizes around the unit edges, one tour (a cluster of CTAs) and
more tours than SMs (one CTA each), lattices with tied deltas, asymmetric matrices, and
distances too large for 32-bit deltas."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import distances as odist
from oracle import three_opt as o3
from tsp_gpu_clean_b200 import instances

pytestmark = pytest.mark.gpu


def _matrix(kind: str, n: int) -> np.ndarray:
  rng = np.random.default_rng(n)
  if kind == "lattice":  # distances 1..3: most deltas tie
    return odist.euc2d_matrix(rng.integers(0, 4, (n, 2)).astype(np.float64))
  if kind == "asymmetric":
    D = rng.integers(1, 1000, (n, n))
  elif kind == "edge32":  # the largest distance that 32-bit deltas take
    D = rng.integers((1 << 29) - 1000, 1 << 29, (n, n))
    D[0, 1] = (1 << 29) - 1
  else:  # "wide": the largest distance the library takes
    D = rng.integers(0, 1 << 30, (n, n))
    D = np.minimum(D, D.T)
  np.fill_diagonal(D, 0)
  return D.astype(np.int32)


@pytest.mark.parametrize("kind", ["lattice", "asymmetric", "edge32", "wide"])
@pytest.mark.parametrize("n,tours,iters", [(4, 3, 50), (5, 160, 50), (6, 2, 50), (7, 1, 50), (32, 1, 4), (33, 2, 4),
                                           (34, 150, 1), (35, 1, 4), (37, 5, 3), (64, 1, 3), (65, 2, 2), (221, 1, 1)])
def test_three_opt_units_match_oracle(kind, n, tours, iters):
  torch = pytest.importorskip("torch")
  if not torch.cuda.is_available():
    pytest.skip("no CUDA device")
  from tsp_gpu_clean_b200.problem import Problem, ProblemContext
  from tsp_gpu_clean_b200.strategies import LocalSearchB200ThreeOpt

  D = _matrix(kind, n)
  ctx = ProblemContext(Problem.from_matrix(D), seed=0)
  distinct = instances.random_tours(n, min(tours, 3), n + 1)
  batch = distinct[np.arange(tours) % len(distinct)]
  ls = LocalSearchB200ThreeOpt(max_iterations=iters)
  got = ls.improve_batch(batch, ctx)
  want, moves = o3.improve_batch(distinct, D, iters)
  assert np.array_equal(got, want[np.arange(tours) % len(distinct)])
  assert ls.last_stats[:, 1].tolist() == [moves[i % len(distinct)] for i in range(tours)]
  # every pass evaluates the same (triple, case) candidates
  assert (ls.last_stats[:, 2] == ls.last_stats[:, 0] * (n - 2) * (n - 2) * (n + 1)).all()
