"""The exhaustive 3-opt's last cut j = n - 2, which a warp unit of its own holds at some sizes
(n = 2 past a multiple of 16, or of 8 with 64-bit deltas): a tour whose only improving move
takes the last city out of the tour's end, at those sizes and the ones beside them. Tours are
whole numbers."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import three_opt as o3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1, 1 << 18])
@pytest.mark.parametrize("n", [9, 10, 11, 17, 18, 19, 26, 34, 50, 66, 226])
def test_last_cut(n, scale):
  pytest.importorskip("torch")
  from tsp_gpu_clean_b200.problem import Problem, ProblemContext
  from tsp_gpu_clean_b200.strategies import LocalSearchB200ThreeOpt

  tour = np.arange(n, dtype=np.int32)
  for i in (1, n // 2, n - 5):
    D = np.full((n, n), 3000)
    for a, b in zip(tour, np.roll(tour, -1)):
      D[a, b] = D[b, a] = 1000
    D[n - 2, 0] = D[0, n - 2] = 1000
    for a in (i, i + 1):  # the last city belongs between them
      D[a, n - 1] = D[n - 1, a] = 1
    np.fill_diagonal(D, 0)
    want, moves = o3.improve_batch(tour[None], D * scale, 2)
    assert want[0].tolist() == [*range(i + 1), n - 1, *range(i + 1, n - 1)]
    ls = LocalSearchB200ThreeOpt(max_iterations=2)
    got = ls.improve_batch(tour[None], ProblemContext(Problem.from_matrix(D.astype(np.int32) * scale), seed=0))
    assert np.array_equal(got, want)
    assert ls.last_stats[:, 1].tolist() == list(moves)
