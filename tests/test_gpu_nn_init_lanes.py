"""Nearest-neighbour initial tours with a try per lane against the oracle: list lengths around
the lane counts (no list, one entry, the longest that loads ahead, a full warp, beyond it),
lists whose entries run out early, entries that are no city. Tours are whole numbers."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from oracle import ga_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [0, 1, 2, 5, 6, 31, 32, 33, 40])
def test_nn_rows_by_list_length(k):
  import torch

  from tsp_gpu_clean_b200 import native
  from tsp_gpu_clean_b200.device import ptr, stream_handle

  rng = np.random.default_rng(k)
  rows, sizes = 6, [1, 2, 33, 64, 257, 700]
  jobs = (native.NNJob * len(sizes))()
  keep, want = [], []
  for q, n in enumerate(sizes):
    cand = rng.integers(0, n, (n, k)).astype(np.int32)  # repeated and distant entries: the list often runs out
    if k and n > 2:
      cand[::5, 0] = -1
      cand[::7, k - 1] = n
      near = (np.arange(n)[:, None] + 1 + np.arange(k)[None]) % n
      cand[1::2] = near[1::2]
    seeds = rng.integers(0, 2**63, rows).astype(np.uint64)
    d_cand = torch.from_numpy(cand).cuda()
    d_seeds = torch.from_numpy(seeds.view(np.int64)).cuda()
    out = torch.full((rows, n), -1, dtype=torch.int32, device="cuda")
    keep.append((d_cand, d_seeds, out))
    jobs[q] = native.NNJob(n, k, d_cand.data_ptr() if k else None, d_seeds.data_ptr(), out.data_ptr(), rows, 0)
    want.append(np.stack([ga_ops.nn_row(np.arange(n, dtype=np.int32), cand, int(s)) for s in seeds]))
  raw = np.frombuffer(ctypes.string_at(ctypes.addressof(jobs), ctypes.sizeof(jobs)), dtype=np.uint8).copy()
  d_jobs = torch.from_numpy(raw).cuda()
  native.call("tspb_nn_init_jobs_smem", ptr(d_jobs), len(sizes), rows, max(sizes), max(k, 1), stream_handle())
  for (_, _, out), w in zip(keep, want):
    assert np.array_equal(out.cpu().numpy(), w)
