"""The multi_move kernel's scans (packed words, plain candidates, every pair), CTA sizes and
tour placements against the oracle, with tied gains and the counts of every pass."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import distances as odist
from oracle import two_opt as otwo
from tsp_gpu_clean_b200 import instances

pytestmark = pytest.mark.gpu


def _search(coords, tours, k, iters, kernel="scan", **kw):
  torch = pytest.importorskip("torch")
  if not torch.cuda.is_available():
    pytest.skip("no CUDA device")
  from tsp_gpu_clean_b200.problem import Problem, ProblemContext
  from tsp_gpu_clean_b200.strategies import LocalSearchB200TourTwoOpt

  ctx = ProblemContext(Problem.from_coordinates(coords), seed=0)
  ls = LocalSearchB200TourTwoOpt(max_iterations=iters, mode="multi_move", candidate_k=k, **kw)
  ls.kernel = kernel
  return ls.improve_batch(tours, ctx), ls.last_stats, ctx


@pytest.mark.parametrize("lattice", [False, True])
@pytest.mark.parametrize("n,k", [(4, None), (4, 3), (5, 4), (33, None), (35, 8), (66, 7), (130, 20), (257, 12)])
@pytest.mark.parametrize("threads", [32, 256, 1024])
def test_multi_move_matches_oracle(n, k, threads, lattice):
  rng = np.random.default_rng(n)
  coords = 5.0 * rng.integers(0, 9, (n, 2)) if lattice else rng.uniform(0.0, 1000.0, (n, 2))
  tours = instances.random_tours(n, 3, n + 1)
  D = odist.euc2d_matrix(coords)
  for iters in (1, 10**6):
    for kernel in ("scan", "scan_unpacked"):
      got, stats, ctx = _search(coords, tours, k, iters, kernel, threads_per_block=threads)
      want, st = otwo.improve_batch(tours, D, ctx.get_cpu_candidate_list(k) if k else None, "multi_move", iters)
      assert np.array_equal(got, want), (kernel, iters)
      assert np.array_equal(stats[:, :3], st), (kernel, iters)


def test_multi_move_in_workspace_arrays():
  # 19,200 cities: tour, positions and edges live in the workspace, distances are rebuilt
  from test_gpu_two_opt import CoordDist

  n = 19200
  coords = instances.uniform_instance(n, 3)
  tours = instances.random_tours(n, 2, 4)
  got, stats, ctx = _search(coords, tours, 8, 2, max_matrix_dimension=1000)
  want, st = otwo.improve_batch(tours, CoordDist(coords), ctx.get_cpu_candidate_list(8), "multi_move", 2)
  assert np.array_equal(got, want)
  assert np.array_equal(stats[:, :3], st)
