"""Edge features and top-k selection of the learned lists at the edges of their warp tiles,
against plain NumPy."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import distances as odist

pytestmark = pytest.mark.gpu


def _torch():
  torch = pytest.importorskip("torch")
  if not torch.cuda.is_available():
    pytest.skip("no CUDA device")
  return torch


def _select(pool, score, k):
  """Repeatedly the first slot left, replaced by a later one only when that is greater."""
  out = np.empty((len(pool), k), dtype=np.int32)
  for u in range(len(pool)):
    left = list(range(pool.shape[1]))
    for r in range(k):
      best = left[0]
      for q in left[1:]:
        if score[u, q] > score[u, best]:
          best = q
      left.remove(best)
      out[u, r] = pool[u, best]
  return out


@pytest.mark.parametrize("pool_k,k", [(1, 1), (5, 5), (31, 10), (32, 32), (33, 8), (64, 20), (128, 128)])
def test_select_topk(pool_k, k):
  torch = _torch()
  from tsp_gpu_clean_b200 import native
  from tsp_gpu_clean_b200.device import ptr, stream_handle

  n = 29
  rng = np.random.default_rng(pool_k)
  pool = rng.integers(0, 1000, (n, pool_k)).astype(np.int32)
  score = rng.normal(0.0, 1.0, (n, pool_k)).astype(np.float32)
  score[1::4] = np.round(score[1::4])  # ties, and zeros of both signs
  score[2::4] *= rng.choice([1.0, np.inf], (len(score[2::4]), pool_k))
  score[3::4][rng.random((len(score[3::4]), pool_k)) < 0.2] = np.nan
  p, s = torch.from_numpy(pool).cuda(), torch.from_numpy(score).cuda()
  out = torch.empty((n, k), dtype=torch.int32, device="cuda")
  native.call("tspb_select_topk", ptr(p), ptr(s), n, pool_k, k, ptr(out), stream_handle())
  assert np.array_equal(out.cpu().numpy(), _select(pool, score, k))


@pytest.mark.parametrize("n,pool_k", [(2, 1), (40, 7), (60, 31), (61, 32), (70, 33), (140, 128)])
@pytest.mark.parametrize("matrix", [True, False])
def test_edge_features(n, pool_k, matrix):
  torch = _torch()
  from tsp_gpu_clean_b200 import native
  from tsp_gpu_clean_b200.device import ptr, stream_handle

  rng = np.random.default_rng(n)
  coords = rng.uniform(0.0, 1000.0, (n, 2))
  D = odist.euc2d_matrix(coords)
  pool = odist.candidate_list(pool_k, distances=D)
  pos = rng.permutation(n).astype(np.int32)
  f32 = np.float32
  x = np.zeros((n * pool_k, 16), dtype=f32)
  y = np.zeros(n * pool_k, dtype=f32)
  for u in range(n):
    su = f32(max(D[u, pool[u, -1]], 1))
    for s in range(pool_k):
      v = pool[u, s]
      back = np.nonzero(pool[v] == u)[0]
      rank = back[0] if len(back) else pool_k
      e = u * pool_k + s
      x[e, :5] = (f32(D[u, v]) / su, f32(s) / f32(pool_k), f32(rank) / f32(pool_k),
                  f32(coords[v, 0] - coords[u, 0]) / su, f32(coords[v, 1] - coords[u, 1]) / su)
      y[e] = abs(int(pos[u]) - int(pos[v])) in (1, n - 1)
  want = torch.from_numpy(x).to(torch.bfloat16).view(torch.int16)
  c, p, t = torch.from_numpy(coords).cuda(), torch.from_numpy(pool).cuda(), torch.from_numpy(pos).cuda()
  d = torch.from_numpy(D).cuda() if matrix else None
  got = torch.empty((n * pool_k, 16), dtype=torch.int16, device="cuda")
  lab = torch.empty(n * pool_k, dtype=torch.float32, device="cuda")
  native.call("tspb_edge_features", ptr(c), n, ptr(p), pool_k, ptr(d), n if matrix else 0, ptr(t), ptr(got), ptr(lab),
              stream_handle())
  # correctly rounded FP32 quotients, then BF16: equal bit for bit
  assert torch.equal(got.cpu(), want)
  assert np.array_equal(lab.cpu().numpy(), y)
