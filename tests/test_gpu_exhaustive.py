"""The exhaustive 2-opt's warp units, row tiles and row keys against the oracle: sizes around
31 positions and eight rows, the whole matrix and tiles of it in shared memory, tours with an SM
to themselves and many per SM, row strides of every alignment, ties, asymmetric matrices."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import distances as odist
from oracle import two_opt as otwo
from tsp_gpu_clean_b200 import instances

pytestmark = pytest.mark.gpu


def _matrix(kind: str, n: int) -> np.ndarray:
  rng = np.random.default_rng(n)
  if kind == "lattice":
    return odist.euc2d_matrix(5.0 * rng.integers(0, 8, (n, 2)))
  if kind == "asymmetric":
    D = rng.integers(1, 1000, (n, n))
  elif kind == "largest":
    D = np.minimum(*(lambda M: (M, M.T))(rng.integers(0, 1 << 30, (n, n))))
  else:
    D = odist.euc2d_matrix(rng.uniform(0.0, 1000.0, (n, 2)))
  np.fill_diagonal(D, 0)
  return np.ascontiguousarray(D, dtype=np.int32)


@pytest.mark.parametrize("mode", ["best", "first"])
@pytest.mark.parametrize("kind", ["uniform", "lattice", "asymmetric", "largest"])
@pytest.mark.parametrize("n,tours,threads,iters", [(4, 3, 32, 9), (5, 2, 64, 99), (63, 2, 256, 10**6), (64, 2, 1024, 10**6), (65, 3, 512, 10**6),
                                                   (66, 300, 64, 10**6), (95, 1, 32, 10**6), (130, 2, 256, 10**6),
                                                   (231, 2, 512, 60), (240, 2, 512, 60), (253, 310, 128, 12)])
def test_exhaustive_matches_oracle(n, tours, threads, iters, kind, mode):
  torch = pytest.importorskip("torch")
  if not torch.cuda.is_available():
    pytest.skip("no CUDA device")
  from tsp_gpu_clean_b200.problem import Problem, ProblemContext
  from tsp_gpu_clean_b200.strategies import LocalSearchB200TourTwoOpt

  D = _matrix(kind, n)
  if kind == "asymmetric":
    iters = min(iters, 40)  # a reversal can lengthen the tour: no convergence
  distinct = instances.random_tours(n, min(tours, 4), n + 3)
  pick = np.arange(tours) % len(distinct)
  ctx = ProblemContext(Problem.from_matrix(D), seed=0)
  ls = LocalSearchB200TourTwoOpt(max_iterations=iters, mode=mode, threads_per_block=threads)
  got = ls.improve_batch(distinct[pick], ctx)
  want, st = otwo.improve_batch(distinct, D, None, mode, iters)
  assert np.array_equal(got, want[pick])
  assert np.array_equal(ls.last_stats[:, :3], np.asarray(st)[pick])


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n,pad,offset", [(61, 3, 0), (61, 3, 1), (64, 0, 0), (64, 1, 0), (300, 4, 0), (300, 4, 2)])
def test_exhaustive_row_strides(n, pad, offset, mode):
  torch = pytest.importorskip("torch")
  if not torch.cuda.is_available():
    pytest.skip("no CUDA device")
  import ctypes

  from tsp_gpu_clean_b200 import native
  from tsp_gpu_clean_b200.device import ptr, stream_handle

  D = _matrix("uniform", n)
  ld = n + pad
  flat = np.full(offset + (n - 1) * ld + n, 1 << 29, dtype=np.int32)  # ends with the last row's last entry
  for i in range(n):
    flat[offset + i * ld : offset + i * ld + n] = D[i]
  d = torch.from_numpy(flat).cuda()
  tours = instances.random_tours(n, 2, n)
  t = torch.from_numpy(tours).cuda()
  stats = torch.zeros((2, 4), dtype=torch.int64, device="cuda")
  status = torch.zeros(2, dtype=torch.int32, device="cuda")
  native.call("tspb_two_opt", ptr(t), 2, n, ctypes.c_void_p(d.data_ptr() + 4 * offset), ld, None, None, None, None, None,
              None, 0, mode | native.TSPB_MODE_SYMMETRIC, 50, 256, ptr(stats), ptr(status), None, 0, stream_handle())
  want, st = otwo.improve_batch(tours, D, None, "best" if mode == 0 else "first", 50)
  assert int(status.max().item()) == 0
  assert np.array_equal(t.cpu().numpy(), want)
  assert np.array_equal(stats.cpu().numpy()[:, :3], st)
