"""Best-mode 2-opt with row keys (and at the edges of the rule that chooses them) against the
oracle: tours, passes, pair counts and moves."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import distances as odist
from oracle import two_opt as otwo
from tsp_gpu_clean_b200 import instances

pytestmark = pytest.mark.gpu


def _instance(kind: str, n: int, k: int):
  """(distance matrix, candidate table) of one kind."""
  rng = np.random.default_rng(n + k)
  if kind == "lattice":  # most gains tie
    D = odist.euc2d_matrix(5.0 * rng.integers(0, 18, (n, 2)))
  elif kind == "asymmetric":
    D = odist.euc2d_matrix(rng.uniform(0, 1000, (n, 2))) + rng.integers(0, 40, (n, n)).astype(np.int32)
    np.fill_diagonal(D, 0)
  elif kind == "long":  # edges above the keys' limit at the start, below it later or at once
    D = 1000 * odist.euc2d_matrix(rng.uniform(0, 40000, (n, 2)))
  else:
    D = odist.euc2d_matrix(instances.clustered_instance(n, 12, 30.0, n))
  cand = odist.candidate_list(k, distances=D)
  if kind == "duplicates":  # a neighbour listed twice, and ids that repeat across the row
    cand[:, k // 2] = cand[:, 0]
    cand[::3, k - 1] = cand[::3, 1]
  return np.ascontiguousarray(D, dtype=np.int32), cand


@pytest.mark.parametrize("kind", ["clustered", "lattice", "asymmetric", "duplicates", "long"])
@pytest.mark.parametrize("n,k,threads,iters", [(257, 8, 64, 10**9), (258, 8, 64, 10**9), (259, 8, 64, 60),
                                               (300, 20, 128, 10**9), (300, 32, 64, 10**9), (300, 36, 64, 40),
                                               (600, 12, 128, 10**9)])
def test_row_keys_match_oracle(kind, n, k, threads, iters):
  torch = pytest.importorskip("torch")
  if not torch.cuda.is_available():
    pytest.skip("no CUDA device")
  from tsp_gpu_clean_b200.problem import Problem, ProblemContext
  from tsp_gpu_clean_b200.strategies import LocalSearchB200TourTwoOpt

  D, cand = _instance(kind, n, k)
  tours = instances.random_tours(n, 5, n + 7)
  ctx = ProblemContext(Problem.from_matrix(D), seed=0, candidate_cache={k: cand})
  if kind == "asymmetric":
    iters = min(iters, 150)  # without symmetry a reversal can lengthen the tour: no convergence
  want, st = otwo.improve_batch(tours, D, cand, "best", iters)
  for counted in (True, False):
    ls = LocalSearchB200TourTwoOpt(max_iterations=iters, mode="best", candidate_k=k, threads_per_block=threads)
    ls.collect_stats = counted
    assert np.array_equal(ls.improve_batch(tours, ctx), want), counted
    if counted:
      assert np.array_equal(ls.last_stats[:, :3], st)


def test_row_keys_with_rebuilt_distances():
  torch = pytest.importorskip("torch")
  if not torch.cuda.is_available():
    pytest.skip("no CUDA device")
  from tsp_gpu_clean_b200.problem import Problem, ProblemContext
  from tsp_gpu_clean_b200.strategies import LocalSearchB200TourTwoOpt

  coords = instances.uniform_instance(700, 5)
  ctx = ProblemContext(Problem.from_coordinates(coords), seed=0)
  tours = instances.random_tours(700, 4, 6)
  ls = LocalSearchB200TourTwoOpt(max_iterations=10**9, mode="best", candidate_k=20, threads_per_block=128,
                                 max_matrix_dimension=100)
  got = ls.improve_batch(tours, ctx)
  want, st = otwo.improve_batch(tours, odist.euc2d_matrix(coords), ctx.get_cpu_candidate_list(20), "best", 10**9)
  assert np.array_equal(got, want)
  assert np.array_equal(ls.last_stats[:, :3], st)
