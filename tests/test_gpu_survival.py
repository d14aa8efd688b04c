"""Survival of a batch of GA runs, ranked by counting and by the sorts, against NumPy's stable
order: rows, fitness, converged bits, the elite edge's ties and which runs pause."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# counted; pairs in registers (32 < P <= 1024); pairs in shared memory
@pytest.mark.parametrize("runs,P,launches", [(1, 2, 1), (3, 40, 1), (16, 512, 1), (8, 1024, 1), (4, 3072, 1),
                                             (800, 17, 2), (600, 33, 2), (64, 512, 2), (24, 1000, 2), (1200, 16, 2),
                                             (20, 1100, 2), (12, 3072, 2)])
@pytest.mark.parametrize("levels", [5, 10**6])
def test_survival_matches_stable_order(runs, P, launches, levels):
  torch = pytest.importorskip("torch")
  if not torch.cuda.is_available():
    pytest.skip("no CUDA device")
  from tsp_gpu_clean_b200 import native
  from tsp_gpu_clean_b200.batch import FusedBatchSolver
  from tsp_gpu_clean_b200.device import stream_handle
  from tsp_gpu_clean_b200.fused import LocalSearchConfig
  from tsp_gpu_clean_b200.problem import Problem, ProblemContext

  assert native.load_library().tspb_batch_survival_launches(runs, P) == launches
  n, elite = 7, max(1, P // 4)
  rng = np.random.default_rng(runs + P)
  ctxs = [ProblemContext(Problem.from_coordinates(rng.uniform(0.0, 100.0, (n, 2))), seed=i) for i in range(runs)]
  s = FusedBatchSolver(population_size=P, mutation_rate=0.05, tournament_k=2, nn_k=3,
                       local_search=LocalSearchConfig("best", 1, 4), elite_count=elite, post_init=False)
  s.evolve(ctxs, 1, patience=10**9)  # allocates the state; what it holds is replaced below
  pop, off = (rng.integers(0, n, (runs, P, n)).astype(np.int32) for _ in range(2))
  fit, off_fit = (rng.integers(100, 100 + levels, (runs, P)).astype(np.float64) for _ in range(2))
  clean, off_clean = ((rng.random((runs, P)) < (0.5 if r else 1.1)).astype(np.uint8) for r in range(2))
  clean[: runs // 2], off_clean[: runs // 2] = 1, 1  # these runs settle any tie themselves
  state = np.full(runs, native.TSPB_BATCH_RUN)
  state[::5] = native.TSPB_BATCH_RESUME  # not this launch's
  for dst, src in ((s.pop[0], pop.ravel()), (s.off, off.ravel()), (s.fit[0], fit), (s.off_fit, off_fit),
                   (s.clean[0], clean), (s.off_clean, off_clean),
                   (s.ctl, np.stack([np.zeros(runs), state, np.zeros(runs), np.zeros(runs)], 1).astype(np.int32))):
    dst.copy_(torch.from_numpy(np.ascontiguousarray(src)).view(dst.shape))
  for dst in (s.pop[1], s.fit[1], s.clean[1], s.ties):
    dst.fill_(77)
  native.call("tspb_batch_survival", ctypes.byref(s._state()), stream_handle())

  both, value = np.concatenate([pop, off], 1), np.concatenate([fit, off_fit], 1)
  bit = np.concatenate([clean, off_clean], 1)
  got = [t.cpu().numpy() for t in (s.pop[1].view(runs, P, n), s.fit[1], s.clean[1], s.ties[:, 0], s.ctl[:, 1])]
  for i in range(runs):
    if i % 5 == 0:
      assert (got[0][i] == 77).all() and got[3][i] == 77 and got[4][i] == state[i]
      continue
    order = np.argsort(value[i], kind="stable")[:P]
    assert np.array_equal(got[0][i], both[i][order])
    assert np.array_equal(got[1][i], value[i][order])
    assert np.array_equal(got[2][i], bit[i][order])
    v = value[i][order]
    tie = elite < P and v[elite - 1] == v[elite]
    assert got[3][i] == tie
    pause = tie and not bit[i][order][v == v[elite]].all()
    assert got[4][i] == (native.TSPB_BATCH_PAUSED if pause else native.TSPB_BATCH_RUN)
