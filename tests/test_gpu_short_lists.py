"""Candidate 2-opt with one to three neighbours per city, the shortest tables a caller can
give, against the oracle: tours, passes, pair counts and moves, alone and inside the GA
engines."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import distances as odist
from oracle import two_opt as otwo
from tsp_gpu_clean_b200 import instances

pytestmark = pytest.mark.gpu


def _context(coords, seed=0):
  torch = pytest.importorskip("torch")
  if not torch.cuda.is_available():
    pytest.skip("no CUDA device")
  from tsp_gpu_clean_b200.problem import Problem, ProblemContext

  return ProblemContext(Problem.from_coordinates(coords), seed=seed)


@pytest.mark.parametrize("k", [1, 2, 3])
@pytest.mark.parametrize("mode", ["best", "first"])
@pytest.mark.parametrize("n,threads,lattice", [(5, 64, False), (200, 512, False), (200, 64, True), (701, 128, False)])
def test_scan_matches_oracle(mode, k, n, threads, lattice):
  from tsp_gpu_clean_b200.strategies import LocalSearchB200TourTwoOpt

  rng = np.random.default_rng(n)
  coords = 5.0 * rng.integers(0, 14, (n, 2)) if lattice else rng.uniform(0.0, 1000.0, (n, 2))
  ctx = _context(coords)
  tours = instances.random_tours(n, 4, n + 1)
  want, st = otwo.improve_batch(tours, odist.euc2d_matrix(coords), ctx.get_cpu_candidate_list(k), mode, 10**9)
  for kernel in ("scan", "scan_unpacked", "cached"):
    for max_matrix in (None, 4):  # distances from a matrix, and rebuilt from coordinates
      ls = LocalSearchB200TourTwoOpt(max_iterations=10**9, mode=mode, candidate_k=k, threads_per_block=threads,
                                     max_matrix_dimension=max_matrix)
      ls.kernel = kernel
      assert np.array_equal(ls.improve_batch(tours, ctx), want), (kernel, max_matrix)
      assert np.array_equal(ls.last_stats[:, :3], st), (kernel, max_matrix)


@pytest.mark.parametrize("mode", ["best", "first"])
def test_ga_runs_match_oracle(mode):
  """A false local optimum would also mark a row as converged for every later generation."""
  from oracle import ga as oga
  from tsp_gpu_clean_b200.batch import FusedBatchSolver
  from tsp_gpu_clean_b200.fused import LocalSearchConfig

  coords = [instances.uniform_instance(n, 40 + n) for n in (150, 400)]
  ctxs = [_context(c, seed=5 + i) for i, c in enumerate(coords)]
  solver = FusedBatchSolver(population_size=32, mutation_rate=0.05, tournament_k=5, nn_k=5,
                            local_search=LocalSearchConfig(mode, 1000, 1), elite_count=8, post_init=True)
  runs = solver.evolve(ctxs, 15, patience=10**9)
  for i, c in enumerate(coords):
    cfg = oga.GAConfig(population_size=32, mutation_rate=0.05, nn_k=5, tournament_k=5,
                       local_search=oga.LocalSearchSpec(mode, 1000, 1), post_init=True, elite_count=8)
    best, pop, _, stats, _ = oga.OracleGA(odist.euc2d_matrix(c), lambda k, c=c: odist.candidate_list(k, coords=c), cfg,
                                          np.random.default_rng(5 + i)).evolve(15, patience=10**9)
    assert np.array_equal(runs[i][0], best)
    assert np.array_equal(solver.final_population[i].cpu().numpy(), pop)
    assert runs[i][1]["convergence_history"] == list(stats["convergence_history"])
