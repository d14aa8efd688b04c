"""multi_move 2-opt where a pass has more improving pairs than the list in shared memory
holds, so that the rest go through the workspace and their rows and columns are decoded from
scan indices, against the oracle."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import distances as odist
from oracle import two_opt as otwo
from tsp_gpu_clean_b200 import instances

pytestmark = pytest.mark.gpu


def _search(coords, tours, k, iters, **kw):
  torch = pytest.importorskip("torch")
  if not torch.cuda.is_available():
    pytest.skip("no CUDA device")
  from tsp_gpu_clean_b200.problem import Problem, ProblemContext
  from tsp_gpu_clean_b200.strategies import LocalSearchB200TourTwoOpt

  ctx = ProblemContext(Problem.from_coordinates(coords), seed=0)
  ls = LocalSearchB200TourTwoOpt(max_iterations=iters, mode="multi_move", candidate_k=k, **kw)
  return ls.improve_batch(tours, ctx), ls.last_stats, ctx


@pytest.mark.parametrize("k", [1, 2, 3, 4])
@pytest.mark.parametrize("lattice", [False, True])
def test_many_tours_share_an_sm(k, lattice):
  # six tours of 2400 cities an SM leave room for about 600 pairs each; k = 1 has about 1,200
  n, copies = 2400, 267
  rng = np.random.default_rng(k)
  coords = 5.0 * rng.integers(0, 90, (n, 2)) if lattice else rng.uniform(0.0, 1000.0, (n, 2))
  tours = instances.random_tours(n, 3, n + k)
  got, stats, ctx = _search(coords, np.tile(tours, (copies, 1)), k, 6, threads_per_block=128)
  want, st = otwo.improve_batch(tours, odist.euc2d_matrix(coords), ctx.get_cpu_candidate_list(k), "multi_move", 6)
  assert np.array_equal(got, np.tile(want, (copies, 1)))
  assert np.array_equal(stats[:, :3], np.tile(st, (copies, 1)))


@pytest.mark.parametrize("n", [600, 1700])  # below and above 2^32 = n^3
def test_every_pair(n):
  coords = instances.uniform_instance(n, n)
  tours = instances.random_tours(n, 2, n)
  got, stats, _ = _search(coords, tours, None, 3)
  want, st = otwo.improve_batch(tours, odist.euc2d_matrix(coords), None, "multi_move", 3)
  assert np.array_equal(got, want)
  assert np.array_equal(stats[:, :3], st)


@pytest.mark.parametrize("k", [1, 2])
def test_arrays_in_the_workspace(k):
  # 19,300 cities: nothing is held in shared memory but the list, distances are rebuilt
  from test_gpu_two_opt import CoordDist

  n = 19300
  coords = instances.uniform_instance(n, 3)
  tours = instances.random_tours(n, 2, 4)
  got, stats, ctx = _search(coords, tours, k, 3, max_matrix_dimension=1000)
  want, st = otwo.improve_batch(tours, CoordDist(coords), ctx.get_cpu_candidate_list(k), "multi_move", 3)
  assert np.array_equal(got, want)
  assert np.array_equal(stats[:, :3], st)
