"""Or-opt on both sides of the rule that evaluates small neighbourhoods whole every pass,
against the oracle: tours, passes, moves and counts."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import distances as odist
from oracle import or_opt as oo
from tsp_gpu_clean_b200 import instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice", [False, True])
@pytest.mark.parametrize("tours,n,k,S", [(1, 72, 8, 1), (1, 73, 8, 1), (2, 14, 13, 2), (3, 71, 3, 3), (3, 72, 3, 3),
                                         (2, 78, 1, 8), (2, 79, 1, 8), (450, 400, 3, 1), (450, 400, 4, 1), (444, 400, 3, 1),
                                         (450, 2000, 1, 1), (160, 12, 11, 8)])
def test_or_opt_matches_oracle(tours, n, k, S, lattice):
  torch = pytest.importorskip("torch")
  if not torch.cuda.is_available():
    pytest.skip("no CUDA device")
  from tsp_gpu_clean_b200.problem import Problem, ProblemContext
  from tsp_gpu_clean_b200.strategies import LocalSearchB200OrOpt

  rng = np.random.default_rng(n)
  coords = 5.0 * rng.integers(0, 30, (n, 2)) if lattice else rng.uniform(0.0, 1000.0, (n, 2))
  D = odist.euc2d_matrix(coords)
  distinct = instances.random_tours(n, 3, n + 3)
  pick = np.arange(tours) % 3
  for max_matrix in (None, 4):
    ctx = ProblemContext(Problem.from_coordinates(coords), seed=0)
    ls = LocalSearchB200OrOpt(max_iterations=25, candidate_k=k, max_segment=S, max_matrix_dimension=max_matrix)
    got = ls.improve_batch(distinct[pick], ctx)
    cand = ctx.get_cpu_candidate_list(k)
    want = [oo.refine(t, D, cand, 25, S) for t in distinct]
    assert np.array_equal(got, np.stack([want[r][0] for r in pick]))
    assert np.array_equal(ls.last_stats, np.asarray([want[r][1:] for r in pick]))
