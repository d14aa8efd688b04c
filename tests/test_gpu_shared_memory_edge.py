"""Sizes at which a kernel's dynamic shared memory is just below 48 KB: its static arrays
bring the CTA above what a launch gets without asking."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import distances as odist
from oracle import two_opt as otwo
from tsp_gpu_clean_b200 import instances

pytestmark = pytest.mark.gpu


def _context(n):
  torch = pytest.importorskip("torch")
  if not torch.cuda.is_available():
    pytest.skip("no CUDA device")
  from tsp_gpu_clean_b200.problem import Problem, ProblemContext

  coords = instances.uniform_instance(n, n)
  return coords, ProblemContext(Problem.from_coordinates(coords), seed=0)


# the numbers of cities on both sides of the edge, where it was, and inside the window
@pytest.mark.parametrize("mode,k,kernel,counted,sizes", [
  ("multi_move", 20, "scan", True, (194, 195, 196, 197)),
  ("multi_move", 10, "scan", True, (371, 374)),
  ("multi_move", None, "scan", True, (91, 92)),
  ("multi_move", 8, "scan", True, (4012, 4051)),
  ("best", 8, "scan", True, (2429, 2457)),
  ("best", 8, "scan", False, (3034, 3071)),
  ("best", 8, "scan_unpacked", True, (4858, 4914)),
  ("first", 8, "scan", True, (3470, 3510)),
  ("first", 8, "scan", False, (4858, 4914)),
  ("best", 8, "cached", True, (1687, 1690)),
])
def test_two_opt(mode, k, kernel, counted, sizes):
  from tsp_gpu_clean_b200.strategies import LocalSearchB200TourTwoOpt

  for n in sizes:
    coords, ctx = _context(n)
    tours = instances.random_tours(n, 1, n + 1)
    for threads in (None, 64):
      ls = LocalSearchB200TourTwoOpt(max_iterations=3, mode=mode, candidate_k=k, threads_per_block=threads)
      ls.kernel, ls.collect_stats = kernel, counted
      got = ls.improve_batch(tours, ctx)
      want, _ = otwo.improve_batch(tours, odist.euc2d_matrix(coords), ctx.get_cpu_candidate_list(k) if k else None, mode, 3)
      assert np.array_equal(got, want), (n, threads)


@pytest.mark.parametrize("mode", ["best", "first"])
@pytest.mark.parametrize("n", [4054, 4096])
def test_two_opt_every_pair_from_coordinates(n, mode):
  from tsp_gpu_clean_b200.strategies import LocalSearchB200TourTwoOpt

  coords, ctx = _context(n)
  tours = instances.random_tours(n, 1, n + 1)
  got = LocalSearchB200TourTwoOpt(max_iterations=1, mode=mode, max_matrix_dimension=10).improve_batch(tours, ctx)
  want, _ = otwo.improve_batch(tours, odist.euc2d_matrix(coords), None, mode, 1)
  assert np.array_equal(got, want)


@pytest.mark.parametrize("n", [94, 95, 96])
def test_three_opt(n):
  from oracle import three_opt as othree
  from tsp_gpu_clean_b200.strategies import LocalSearchB200ThreeOpt

  coords, ctx = _context(n)
  tours = instances.random_tours(n, 1, n + 1)
  got = LocalSearchB200ThreeOpt(max_iterations=2).improve_batch(tours, ctx)
  assert np.array_equal(got[0], othree.refine(tours[0], odist.euc2d_matrix(coords), 2)[0])


@pytest.mark.parametrize("n", [2955, 3022, 3072])
def test_or_opt(n):
  from oracle import or_opt as oor
  from tsp_gpu_clean_b200.strategies import LocalSearchB200OrOpt

  coords, ctx = _context(n)
  tours = instances.random_tours(n, 1, n + 1)
  got = LocalSearchB200OrOpt(max_iterations=2, candidate_k=8).improve_batch(tours, ctx)
  assert np.array_equal(got[0], oor.refine(tours[0], odist.euc2d_matrix(coords), ctx.get_cpu_candidate_list(8), 2, 3)[0])
