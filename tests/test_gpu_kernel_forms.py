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


@pytest.mark.parametrize("n,pool_k,k", [(30, 12, 7), (30, 13, 13), (32767, 40, 5), (32768, 40, 5), (32768, 31, 31),
                                        (32768, 32, 3), (32769, 63, 2), (32768, 65, 2)])
def test_select_topk(n, pool_k, k):
  torch, native, ptr, stream_handle = _gpu()
  rng = np.random.default_rng(n + pool_k)
  pool = rng.integers(0, n, (n, pool_k)).astype(np.int32)
  score = rng.normal(0.0, 1.0, (n, pool_k)).astype(np.float32)
  score[1::4] = np.round(score[1::4])  # ties, and zeros of both signs
  score[2::4] *= rng.choice([1.0, np.inf], (len(score[2::4]), pool_k)).astype(np.float32)
  out = torch.empty((n, k), dtype=torch.int32, device="cuda")
  p, s = torch.from_numpy(pool).cuda(), torch.from_numpy(score).cuda()
  native.call("tspb_select_topk", ptr(p), ptr(s), n, pool_k, k, ptr(out), stream_handle())
  order = np.argsort(-score, axis=1, kind="stable")[:, :k]
  assert np.array_equal(out.cpu().numpy(), np.take_along_axis(pool, order, axis=1))


@pytest.mark.parametrize("n,pool_k", [(60, 10), (60, 11), (256, 128), (257, 128), (993, 33)])
@pytest.mark.parametrize("matrix", [True, False])
def test_edge_features(n, pool_k, matrix):
  torch, native, ptr, stream_handle = _gpu()
  rng = np.random.default_rng(n)
  coords = rng.uniform(0.0, 1000.0, (n, 2))
  D = odist.euc2d_matrix(coords)
  pool = odist.candidate_list(pool_k, distances=D)
  pos = rng.permutation(n).astype(np.int32)
  f32 = np.float32
  rank = np.full((n, n), pool_k)  # rank[v, u]: slot of u in v's pool
  np.put_along_axis(rank, pool, np.broadcast_to(np.arange(pool_k), pool.shape), axis=1)
  U = np.arange(n)[:, None]
  su = np.maximum(D[np.arange(n), pool[:, -1]], 1).astype(f32)[:, None]
  x = np.zeros((n, pool_k, 16), dtype=f32)
  x[..., 0] = D[U, pool].astype(f32) / su
  x[..., 1] = np.arange(pool_k, dtype=f32) / f32(pool_k)
  x[..., 2] = rank[pool, U].astype(f32) / f32(pool_k)
  x[..., 3] = (coords[pool, 0] - coords[U, 0]).astype(f32) / su
  x[..., 4] = (coords[pool, 1] - coords[U, 1]).astype(f32) / su
  gap = np.abs(pos[U] - pos[pool])
  y = ((gap == 1) | (gap == n - 1)).astype(f32)
  want = torch.from_numpy(x).to(torch.bfloat16).view(torch.int16)
  c, p, t = torch.from_numpy(coords).cuda(), torch.from_numpy(pool).cuda(), torch.from_numpy(pos).cuda()
  d = torch.from_numpy(D).cuda() if matrix else None
  got = torch.empty((n, pool_k, 16), dtype=torch.int16, device="cuda")
  lab = torch.empty((n, pool_k), dtype=torch.float32, device="cuda")
  native.call("tspb_edge_features", ptr(c), n, ptr(p), pool_k, ptr(d), n if matrix else 0, ptr(t), ptr(got), ptr(lab),
              stream_handle())
  assert torch.equal(got.cpu(), want)
  assert np.array_equal(lab.cpu().numpy(), y)


@pytest.mark.parametrize("edges", [6 * 148 * 64 * 16 - 15, 6 * 148 * 64 * 16 + 1])
def test_mlp_infer_grids(edges):
  """A row's logit does not depend on the grid: the same rows in a call of their own."""
  torch, native, ptr, stream_handle = _gpu()
  gen = torch.Generator().manual_seed(edges)
  params = (torch.randn(native.load_library().tspb_mlp_param_count(), generator=gen) * 0.1).cuda()
  x = torch.randn((edges, 16), generator=gen).to(torch.bfloat16).view(torch.int16).cuda()
  got = torch.empty(edges, device="cuda")
  native.call("tspb_mlp_infer", ptr(params), ptr(x), edges, ptr(got), stream_handle())
  for lo in (0, 16 * 1000, edges - 1 - (edges - 1) % 16):
    rows = min(160, edges - lo)
    part = torch.empty(rows, device="cuda")
    native.call("tspb_mlp_infer", ptr(params), ptr(x[lo:lo + rows].contiguous()), rows, ptr(part), stream_handle())
    assert torch.equal(got[lo:lo + rows], part)
