"""Or-opt's row words against the oracle where they can go wrong: row groups that end inside
a warp, tables that are not whole quads of words, more changed entries than the lists hold
(a candidate in every row), the longest segments, segments that reach the last position,
distances beyond 32-bit deltas, asymmetric matrices, every CTA width. Tours and counts are
whole numbers, so equality is exact."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import or_opt as oo

pytestmark = pytest.mark.gpu


def _matrix(n, kind, rng):
  xy = rng.uniform(0.0, 1000.0, (n, 2))
  d = np.floor(np.hypot(*(xy[:, None] - xy[None]).transpose(2, 0, 1)) + 0.5).astype(np.int64)
  if kind == "ties":
    d = np.minimum(d // 100, 5)
  elif kind == "huge":
    d = np.minimum(d * 2_500_000, 2**31 - 1)
  elif kind == "asymmetric":
    d = d + rng.integers(0, 200, (n, n))
  np.fill_diagonal(d, 0)
  return d.astype(np.int32)


@pytest.mark.parametrize("threads", [128, 256, 512])
@pytest.mark.parametrize("n,k,S,iters,kind", [
  (3, 2, 8, 50, "plain"), (5, 4, 8, 50, "ties"), (33, 7, 8, 10**6, "plain"), (34, 32, 4, 10**6, "ties"),
  (129, 5, 1, 10**6, "plain"), (130, 13, 3, 60, "asymmetric"), (257, 12, 8, 40, "ties"),
  (300, 299, 3, 12, "plain"), (300, 299, 2, 12, "ties"), (90, 20, 3, 10**6, "huge"), (70, 9, 8, 60, "huge"),
  (1030, 8, 3, 30, "plain"), (40, 1, 3, 10**6, "plain"), (61, 3, 5, 10**6, "plain"),
])
def test_or_opt_row_words(n, k, S, iters, kind, threads):
  import torch

  from tsp_gpu_clean_b200 import native
  from tsp_gpu_clean_b200.device import ptr, stream_handle

  rng = np.random.default_rng(1000 * n + k)
  D = _matrix(n, kind, rng)
  far = D.astype(np.int64) + np.where(np.eye(n, dtype=bool), 2**40, 0)
  cand = np.argsort(far, axis=1, kind="stable")[:, :k].astype(np.int32)
  cdist = np.take_along_axis(D, cand, axis=1)
  tours = np.stack([np.concatenate([[t % n], rng.permutation(np.delete(np.arange(n), t % n))])
                    for t in range(3)]).astype(np.int32)
  want = [oo.refine(t, D, cand, iters, S) for t in tours]
  tables = [None]
  if k % 4 == 0 and cdist.max() < 65536:
    tables.append(torch.from_numpy((cand | (cdist << 16)).astype(np.int32)).cuda())
  d, c, cd = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (D, cand, cdist))
  for packed in tables:
    t = torch.from_numpy(tours.copy()).cuda()
    st = torch.zeros(3, dtype=torch.int32, device="cuda")
    stats = torch.zeros((3, 3), dtype=torch.int64, device="cuda")
    native.call("tspb_or_opt", ptr(t), 3, n, ptr(d), n, None, ptr(c), ptr(cd), ptr(packed), k, S, iters, threads,
                ptr(st), ptr(stats), stream_handle())
    assert int(st.max().item()) == 0
    for r, (tour, passes, moves, evaluated) in enumerate(want):
      assert stats[r].tolist() == [passes, moves, evaluated]
      assert np.array_equal(t[r].cpu().numpy(), tour)
