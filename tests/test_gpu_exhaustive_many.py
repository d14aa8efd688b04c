"""Exhaustive 2-opt where tours share SMs: the CTA sizes, the rows that first mode looks at
without a tile, and the runs and sizes on both sides of the rules that choose them, against
the oracle."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import distances as odist
from oracle import two_opt as otwo
from tsp_gpu_clean_b200 import instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["best", "first"])
@pytest.mark.parametrize("kind", ["uniform", "lattice", "asymmetric"])
@pytest.mark.parametrize("n,tours,iters", [(64, 640, 16), (71, 150, 17), (72, 640, 4), (80, 1300, 10**6), (81, 640, 64),
                                           (81, 640, 65), (127, 640, 3), (129, 640, 400), (255, 600, 40), (256, 600, 40),
                                           (300, 160, 60), (511, 310, 30), (512, 310, 30), (1300, 450, 16),
                                           (1300, 450, 17)])
def test_many_tours_match_oracle(n, tours, iters, kind, mode):
  torch = pytest.importorskip("torch")
  if not torch.cuda.is_available():
    pytest.skip("no CUDA device")
  from tsp_gpu_clean_b200.problem import Problem, ProblemContext
  from tsp_gpu_clean_b200.strategies import LocalSearchB200TourTwoOpt

  rng = np.random.default_rng(n)
  if kind == "asymmetric":
    D = rng.integers(1, 1000, (n, n))
    iters = min(iters, 60)  # a reversal can lengthen the tour: no convergence
  else:
    D = odist.euc2d_matrix(5.0 * rng.integers(0, 12, (n, 2)) if kind == "lattice" else rng.uniform(0.0, 1000.0, (n, 2)))
  np.fill_diagonal(D, 0)
  D = np.ascontiguousarray(D, dtype=np.int32)
  distinct = instances.random_tours(n, 3, n + 3)
  distinct[2], _ = otwo.improve_batch(distinct[2:], D, odist.candidate_list(8, distances=D), "multi_move", 40)
  pick = np.arange(tours) % len(distinct)
  ls = LocalSearchB200TourTwoOpt(max_iterations=iters, mode=mode)
  got = ls.improve_batch(distinct[pick], ProblemContext(Problem.from_matrix(D), seed=0))
  want, st = otwo.improve_batch(distinct, D, None, mode, iters)
  assert np.array_equal(got, want[pick])
  assert np.array_equal(ls.last_stats[:, :3], np.asarray(st)[pick])
