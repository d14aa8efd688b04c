"""Operators with two forms of one kernel (a thread, a warp or a CTA per item), on both sides of
the rules that choose between them, against plain NumPy. Reversals, selections and BF16 features
of correctly rounded FP32 quotients are compared for equality."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import distances as odist

pytestmark = pytest.mark.gpu


def _gpu():
  torch = pytest.importorskip("torch")
  if not torch.cuda.is_available():
    pytest.skip("no CUDA device")
  from tsp_gpu_clean_b200 import native
  from tsp_gpu_clean_b200.device import ptr, stream_handle

  return torch, native, ptr, stream_handle


@pytest.mark.parametrize("routes,n", [(1, 1), (3, 2), (9, 511), (9, 512), (16384, 512), (16385, 512), (20001, 7)])
def test_inversion(routes, n):
  torch, native, ptr, stream_handle = _gpu()
  rng = np.random.default_rng(n + routes)
  tours = rng.integers(0, n, (routes, n)).astype(np.int32)
  u = rng.random(routes)
  a, b = rng.integers(0, n, (2, routes)).astype(np.int32)
  a[::7], b[::7] = 0, n - 1
  a[::11] = n  # out of range: left alone
  want = tours.copy()
  for r in np.nonzero(u < 0.5)[0]:
    lo, hi = sorted((int(a[r]), int(b[r])))
    if hi < n:
      want[r, lo:hi + 1] = want[r, lo:hi + 1][::-1].copy()
  d = [torch.from_numpy(x).cuda() for x in (tours, u, a, b)]
  native.call("tspb_inversion", ptr(d[0]), routes, n, ptr(d[1]), 0.5, ptr(d[2]), ptr(d[3]), stream_handle())
  assert np.array_equal(d[0].cpu().numpy(), want)
