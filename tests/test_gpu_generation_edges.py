"""The GA's operator and generation kernels at the sizes where their loops and groups end:
rows around multiples of a CTA's stride, populations around a warp, elite edges that tie, and
EUC_2D lengths that sit on the rounding's edge. All values are whole numbers, so equality is
exact."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import distances as odist

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 37.0, 1000.0, 3.0e5, 4.0e6, 1.0e8])
def test_euc2d_at_half_integers(scale):
  """Distances on, one ulp below and one ulp above m + 0.5, and random ones, from
  coordinates (no matrix), against NumPy's rounding."""
  import torch

  from tsp_gpu_clean_b200 import native
  from tsp_gpu_clean_b200.device import ptr, stream_handle

  rng = np.random.default_rng(int(scale))
  m = np.floor(rng.uniform(0.0, scale, 400)) + 0.5
  d = np.concatenate([m, np.nextafter(m, 0.0), np.nextafter(m, np.inf), m - 1e-6 * m, m + 1e-6 * m])
  angle = rng.uniform(0.0, 2.0 * np.pi, d.size)
  straight = np.stack([d, np.zeros_like(d)], axis=1)
  turned = np.stack([d * np.cos(angle), d * np.sin(angle)], axis=1) + rng.uniform(-scale, scale, 2)
  xy = np.concatenate([[[0.0, 0.0]], straight, turned, rng.uniform(0.0, scale, (1000, 2))])
  n = len(xy)
  tours = np.stack([np.array([0, j] + [q for q in range(n) if q not in (0, j)], dtype=np.int32) for j in range(1, n, 7)])
  tours = np.concatenate([tours, np.argsort(rng.random((8, n)), axis=1).astype(np.int32)])
  p = xy[tours]
  step = np.roll(p, -1, axis=1) - p
  want = (np.sqrt((step * step).sum(axis=2)) + 0.5).astype(np.int64).sum(axis=1)
  t, c = torch.from_numpy(tours).cuda(), torch.from_numpy(xy).cuda()
  out = torch.empty(len(tours), dtype=torch.float64, device="cuda")
  native.call("tspb_tour_cost", ptr(t), len(tours), n, None, 0, ptr(c), 1, ptr(out), stream_handle())
  assert np.array_equal(out.cpu().numpy(), want.astype(np.float64))


@pytest.mark.parametrize("closed", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 255, 256, 257, 513, 1031])
def test_tour_cost_lengths_and_bad_ids(n, closed):
  import torch

  from tsp_gpu_clean_b200 import native
  from tsp_gpu_clean_b200.device import ptr, stream_handle

  rng = np.random.default_rng(n)
  D = odist.euc2d_matrix(rng.uniform(0.0, 900.0, (n, 2))).astype(np.int32)
  tours = np.argsort(rng.random((9, n)), axis=1).astype(np.int32)
  tours[4, n // 2] = n  # not a city
  tours[6, 0] = -1
  d, t = torch.from_numpy(np.ascontiguousarray(D)).cuda(), torch.from_numpy(tours).cuda()
  out = torch.empty(9, dtype=torch.float64, device="cuda")
  native.call("tspb_tour_cost", ptr(t), 9, n, ptr(d), n, None, closed, ptr(out), stream_handle())
  got = out.cpu().numpy()
  for r in range(9):
    if n == 1:
      assert got[r] == 0.0
    elif r in (4, 6):
      assert np.isnan(got[r])
    else:
      nxt = np.roll(tours[r], -1) if closed else tours[r][1:]
      assert got[r] == D[tours[r][: len(nxt)], nxt].sum()


@pytest.mark.parametrize("n", [2, 3, 33, 257, 1023, 1025])
def test_pmx_and_inversion_rows(n):
  import torch

  from oracle import ga_ops
  from tsp_gpu_clean_b200 import native
  from tsp_gpu_clean_b200.device import ptr, stream_handle

  rng = np.random.default_rng(7 * n)
  rows = 21
  parents = np.argsort(rng.random((rows, n)), axis=1).astype(np.int32)
  a, b = rng.integers(0, n, rows // 2).astype(np.int32), rng.integers(0, n, rows // 2).astype(np.int32)
  a[0], b[0] = 0, n - 1
  t = torch.from_numpy(parents).cuda()
  da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
  out = torch.empty_like(t)
  st = torch.zeros(rows, dtype=torch.int32, device="cuda")
  native.call("tspb_pmx", ptr(t), rows, n, ptr(da), ptr(db), ptr(out), ptr(st), stream_handle())
  got = out.cpu().numpy()
  assert int(st.max().item()) == 0
  for q in range(rows // 2):
    lo, hi = min(a[q], b[q]), max(a[q], b[q])
    for h in (0, 1):
      p1, p2 = parents[2 * q + h], parents[2 * q + 1 - h]
      assert np.array_equal(got[2 * q + h], ga_ops.pmx_child(p1, p2, lo, hi))
  assert np.array_equal(got[-1], parents[-1])
  u = rng.random(rows)
  i, j = rng.integers(0, n, rows).astype(np.int32), rng.integers(0, n, rows).astype(np.int32)
  du, di, dj = torch.from_numpy(u).cuda(), torch.from_numpy(i).cuda(), torch.from_numpy(j).cuda()
  native.call("tspb_inversion", ptr(out), rows, n, ptr(du), 0.5, ptr(di), ptr(dj), stream_handle())
  turned = out.cpu().numpy()
  for r in range(rows):
    want = got[r].copy()
    if u[r] < 0.5:
      lo, hi = min(i[r], j[r]), max(i[r], j[r])
      want[lo:hi + 1] = want[lo:hi + 1][::-1]
    assert np.array_equal(turned[r], want)


@pytest.mark.parametrize("P,elite,lattice", [(2, 1, False), (3, 2, True), (31, 5, True), (33, 32, False), (65, 64, True),
                                             (130, 17, True), (600, 80, True)])
def test_survival_order_and_elite_ties(P, elite, lattice):
  """Whole runs against the oracle GA: the order of survivors, the elite edge's ties and the
  host's answers decide every later generation."""
  from oracle import ga as oga
  from tsp_gpu_clean_b200.batch import FusedBatchSolver
  from tsp_gpu_clean_b200.fused import LocalSearchConfig
  from tsp_gpu_clean_b200.problem import Problem, ProblemContext

  n, G = 25, 12
  xy = (np.array([[10.0 * x, 10.0 * y] for x in range(5) for y in range(5)]) if lattice
        else np.random.default_rng(P).uniform(0.0, 100.0, (n, 2)))
  ctx = ProblemContext(Problem.from_coordinates(xy), seed=P)
  solver = FusedBatchSolver(population_size=P, mutation_rate=0.2, tournament_k=3, nn_k=5,
                            local_search=LocalSearchConfig("best", 2, 8), elite_count=elite, post_init=True)
  (best, stats), = solver.evolve([ctx], G, patience=10**9)
  cfg = oga.GAConfig(population_size=P, mutation_rate=0.2, nn_k=5, tournament_k=3,
                     local_search=oga.LocalSearchSpec("best", 2, 8), post_init=True, elite_count=elite)
  run = oga.OracleGA(odist.euc2d_matrix(xy), lambda k: odist.candidate_list(k, coords=xy), cfg, np.random.default_rng(P))
  obest, opop, ofit, ostats, _ = run.evolve(G, patience=10**9)
  assert np.array_equal(best, obest)
  assert np.array_equal(solver.final_population[0].cpu().numpy(), opop)
  assert np.array_equal(solver.final_fitness[0].cpu().numpy(), ofit)
  assert stats["convergence_history"] == ostats["convergence_history"]
