"""multi_move 2-opt on tours along strips, where a pass accepts many small disjoint windows in as
many rounds, against the oracle: CTA sizes, tied gains, lists that spill, scans with the last
group of entries short."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import distances as odist
from oracle import two_opt as otwo
from tsp_gpu_clean_b200 import instances

pytestmark = pytest.mark.gpu


def _strips(coords, count):
  n = len(coords)
  out = []
  for width in 4 + np.arange(count):
    strip = (coords[:, 0] / 1000.0 * np.sqrt(n / width)).astype(int)
    out.append(np.lexsort((np.where(strip % 2, -coords[:, 1], coords[:, 1]), strip)))
  return np.stack(out).astype(np.int32)


@pytest.mark.parametrize("threads", [64, 512])
@pytest.mark.parametrize("n,k,copies", [(30, 5, 1), (700, 7, 1), (700, 8, 1), (2400, 8, 300), (400, None, 1)])
@pytest.mark.parametrize("lattice", [False, True])
def test_many_windows_a_pass(threads, n, k, copies, lattice):
  torch = pytest.importorskip("torch")
  if not torch.cuda.is_available():
    pytest.skip("no CUDA device")
  from tsp_gpu_clean_b200.problem import Problem, ProblemContext
  from tsp_gpu_clean_b200.strategies import LocalSearchB200TourTwoOpt

  coords = instances.uniform_instance(n, n)
  if lattice:
    coords = np.round(coords / 40.0) * 40.0
  tours = _strips(coords, 3)
  ctx = ProblemContext(Problem.from_coordinates(coords), seed=0)
  ls = LocalSearchB200TourTwoOpt(max_iterations=3, mode="multi_move", candidate_k=k, threads_per_block=threads)
  got = ls.improve_batch(np.tile(tours, (copies, 1)), ctx)
  table = None if k is None else ctx.get_cpu_candidate_list(k)
  want, st = otwo.improve_batch(tours, odist.euc2d_matrix(coords), table, "multi_move", 3)
  assert np.array_equal(got, np.tile(want, (copies, 1)))
  assert np.array_equal(ls.last_stats[:, :3], np.tile(st, (copies, 1)))
