"""The EUC_2D matrix and k-NN kernels at the edges of their tiles: odd sizes, row strides and
alignments, distances on and around half-integers, list lengths around 32 and 64."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from oracle import distances as odist

pytestmark = pytest.mark.gpu


def _torch():
  torch = pytest.importorskip("torch")
  if not torch.cuda.is_available():
    pytest.skip("no CUDA device")
  return torch


def _points(kind: str, n: int) -> np.ndarray:
  rng = np.random.default_rng(n)
  if kind == "halves":  # first city at the origin, the others at and around half-integer distances
    d = rng.integers(0, 1500, n) + 0.5 + rng.choice([0.0, 1e-13, -1e-13, 1e-9, -1e-9, 1e-4, -1e-4], n)
    c = np.stack([d, np.zeros(n)], axis=1)
    c[0] = 0.0
    return c
  if kind == "far":  # close points far from the origin: FP32 coordinates say little
    return 1e7 + rng.uniform(0.0, 50.0, (n, 2))
  if kind == "large":
    return rng.uniform(-3e8, 3e8, (n, 2))
  if kind == "tiny":
    return rng.uniform(0.0, 2e-3, (n, 2))
  return rng.uniform(0.0, 1000.0, (n, 2))


@pytest.mark.parametrize("kind", ["uniform", "halves", "far", "large", "tiny"])
@pytest.mark.parametrize("n,pad,offset", [(1, 0, 0), (5, 0, 0), (130, 2, 0), (1023, 1, 1), (1025, 3, 0), (2001, 0, 0)])
def test_euc2d_matrix_equals_formula(kind, n, pad, offset):
  torch = _torch()
  from tsp_gpu_clean_b200 import native
  from tsp_gpu_clean_b200.device import stream_handle

  coords = _points(kind, n)
  want = odist.euc2d_matrix(coords)
  ld = n + pad
  out = torch.full((n * ld + offset + 4,), -7, dtype=torch.int32, device="cuda")
  c = torch.from_numpy(coords).cuda()
  native.call("tspb_euc2d_matrix", ctypes.c_void_p(c.data_ptr()), n, ctypes.c_void_p(out.data_ptr() + 4 * offset), ld,
              stream_handle())
  flat = out.cpu().numpy()
  got = flat[offset : offset + n * ld].reshape(n, ld)
  assert np.array_equal(got[:, :n], want)
  assert (got[:, n:] == -7).all() and (flat[:offset] == -7).all() and (flat[offset + n * ld :] == -7).all()


@pytest.mark.parametrize("lattice", [False, True])
@pytest.mark.parametrize("coords_only", [False, True])
@pytest.mark.parametrize("n,k", [(2, 1), (33, 32), (34, 31), (40, 33), (65, 64), (70, 63), (257, 1), (1001, 20), (1500, 64)])
def test_knn_orders_by_distance_then_id(n, k, coords_only, lattice):
  torch = _torch()
  from tsp_gpu_clean_b200 import native
  from tsp_gpu_clean_b200.device import ptr, stream_handle

  rng = np.random.default_rng(n + k)
  coords = 3.0 * rng.integers(0, 9, (n, 2)) if lattice else rng.uniform(0.0, 1000.0, (n, 2))
  D = odist.euc2d_matrix(coords).astype(np.int64)
  np.fill_diagonal(D, 1 << 40)
  order = np.lexsort((np.broadcast_to(np.arange(n), (n, n)), D), axis=1)
  np.fill_diagonal(D, 0)
  c = torch.from_numpy(np.ascontiguousarray(coords)).cuda()
  d = None if coords_only else torch.from_numpy(D.astype(np.int32)).cuda()
  out = torch.empty((n, k), dtype=torch.int32, device="cuda")
  native.call("tspb_knn", ptr(d), n if d is not None else 0, ptr(c) if coords_only else None, n, k, ptr(out), stream_handle())
  assert np.array_equal(out.cpu().numpy(), order[:, :k])
  if k + 1 <= min(64, n - 1):
    ties = torch.empty(n, dtype=torch.int32, device="cuda")
    out.zero_()
    native.call("tspb_knn_ties", ptr(d), n if d is not None else 0, ptr(c) if coords_only else None, n, k, ptr(out),
                ptr(ties), stream_handle())
    assert np.array_equal(out.cpu().numpy(), order[:, :k])
    r = np.arange(n)
    assert np.array_equal(ties.cpu().numpy() != 0, D[r, order[:, k - 1]] == D[r, order[:, k]])
