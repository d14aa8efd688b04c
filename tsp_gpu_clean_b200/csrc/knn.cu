// k-nearest-neighbour candidate table on the device, one warp per node.
//
// out[u][0..k) = the k nodes closest to u, self excluded, ordered by (distance, node id).
// Distances come from the int32 matrix or are rebuilt from FP64 coordinates (TSPLIB
// EUC_2D). The reference builds this table on the host with argpartition + lexsort
// (src/distances/matrix.py:140-211), where a distance tie at the k-th boundary is resolved
// by NumPy's partition; this kernel resolves it by the lower node id, a fixed and
// documented policy. tspb_knn_ties also reports the rows with such a boundary tie: every
// other row is exactly the reference's, and the context's table (device.candidate_list)
// takes the reference's own host procedure for the flagged rows only.
//
// A warp streams its row, eight coalesced reads in flight, and keeps the smallest keys seen so
// far sorted across its lanes (one or two per lane). A distance enters a small buffer only
// when it beats the k-th kept so far, which about k ln(n / k) of a row's n do; 32 buffered
// keys are sorted and merged at a time with shuffles. So the work per distance is a compare,
// and a large matrix is read at memory speed. The kernel before it (128 threads a node, each
// with its own sorted list of 64-bit keys in registers, then k block-wide minima) took 1,906 us
// for n = 10,000, k = 30 and 50 us for n = 1000, k = 20; this one takes 108 and 10 (the row bytes
// alone: 61 us at copy speed for n = 10,000).
#include "common.cuh"

namespace tspb {

constexpr int KNN_MAX_K = 64;
constexpr int KNN_WARPS = 4;  // nodes per CTA

using Key = unsigned long long;  // distance << 32 | node id

__device__ __forceinline__ Key exchange(Key v, int j, bool keep_small) {
  const Key w = __shfl_xor_sync(FULL, v, j);
  return (w < v) == keep_small ? w : v;
}

// Ascending across the lanes: of any 32 keys, and of a bitonic sequence.
__device__ __forceinline__ Key sort32(Key v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
    for (int j = size >> 1; j > 0; j >>= 1) v = exchange(v, j, ((lane & j) == 0) == ((lane & size) == 0 || size == 32));
  return v;
}
__device__ __forceinline__ Key merge32(Key v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) v = exchange(v, j, (lane & j) == 0);
  return v;
}

// The 32 W smallest keys so far, ascending: lane l holds the l-th and, for W = 2, the
// (32 + l)-th.
template <int W>
struct Smallest {
  Key top[W];

  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int w = 0; w < W; ++w) top[w] = ~0ull;
  }
  // takes 32 more keys, one per lane
  __device__ __forceinline__ void add(Key v) {
    const int rev = 31 - (threadIdx.x & 31);
    v = __shfl_sync(FULL, sort32(v), rev);  // descending: with an ascending run it is bitonic
    Key last = top[W - 1];
    last = merge32(v < last ? v : last);  // the 32 smaller of the two
    if constexpr (W == 2) {
      const Key d = __shfl_sync(FULL, last, rev);
      top[1] = merge32(d < top[0] ? top[0] : d);
      top[0] = merge32(d < top[0] ? d : top[0]);
    } else {
      top[0] = last;
    }
  }
  __device__ __forceinline__ Key at(int r) const {
    return __shfl_sync(FULL, W == 2 && r >= 32 ? top[W - 1] : top[0], r & 31);
  }
};

// Selects `need` keys (k, or k + 1 with `ties`), need <= 32 W; the first k are written.
template <int W>
__global__ void __launch_bounds__(32 * KNN_WARPS) knn_kernel(int n, int k, DistSrc ds, int32_t* __restrict__ out,
                                                             int32_t* __restrict__ ties) {
  __shared__ Key buffer[KNN_WARPS][64];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int u = blockIdx.x * KNN_WARPS + wid;
  if (u >= n) return;
  Key* buf = buffer[wid];
  const int need = ties ? k + 1 : k;
  Smallest<W> best;
  best.clear();
  unsigned bound = 0xffffffffu;  // distance of the need-th key kept: a later, larger id must be below it
  int held = 0;                  // keys in the buffer
  constexpr int U = 8;
  const int32_t* row = ds.dist ? ds.dist + (long long)u * ds.stride : nullptr;
  for (int v0 = 0; v0 < n; v0 += 32 * U) {
    unsigned d[U], low = 0xffffffffu;
    if (row != nullptr && v0 + 32 * U <= n && (u < v0 || u >= v0 + 32 * U)) {  // whole, without u itself
#pragma unroll
      for (int q = 0; q < U; ++q) d[q] = (unsigned)__ldcg(row + v0 + 32 * q + lane);
    } else {
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const int v = v0 + 32 * q + lane;
        d[q] = row != nullptr ? (unsigned)load_cg_if(v < n, row + v) : v < n ? (unsigned)ds(u, v) : 0u;
        if (v >= n || v == u) d[q] = 0xffffffffu;
      }
    }
#pragma unroll
    for (int q = 0; q < U; ++q) low = d[q] < low ? d[q] : low;
    if (W == 1 && v0 == 0) {
      // the lanes' minima are 32 distances of different nodes: `need` of all lie at or below
      // the need-th smallest of them
      const unsigned first = (unsigned)(__shfl_sync(FULL, sort32((Key)low << 32), need - 1) >> 32);
      bound = first == 0xffffffffu ? first : first + 1u;
    }
    if (!__any_sync(FULL, low < bound)) continue;
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const unsigned m = __ballot_sync(FULL, d[q] < bound);
      if (m == 0) continue;
      if (d[q] < bound)
        buf[held + __popc(m & ((1u << lane) - 1u))] = ((Key)d[q] << 32) | (unsigned)(v0 + 32 * q + lane);
      held += __popc(m);
      if (held >= 32) {
        __syncwarp();
        best.add(buf[lane]);
        held -= 32;
        const Key rest = buf[32 + lane];
        __syncwarp();
        if (lane < held) buf[lane] = rest;
        const unsigned last = (unsigned)(best.at(need - 1) >> 32);
        bound = last < bound ? last : bound;
      }
    }
  }
  __syncwarp();
  if (held > 0) best.add(lane < held ? buf[lane] : ~0ull);
#pragma unroll
  for (int w = 0; w < W; ++w) {
    const int r = 32 * w + lane;
    if (r < k) out[(long long)u * k + r] = best.top[w] == ~0ull ? -1 : (int32_t)(unsigned)(best.top[w] & 0xffffffffu);
  }
  if (ties) {
    const Key last = best.at(k - 1), next = best.at(k);
    if (lane == 0) ties[u] = (next != ~0ull && (next >> 32) == (last >> 32)) ? 1 : 0;
  }
}

static int launch_knn(const DistSrc& ds, int n, int k, int32_t* out, int32_t* ties, cudaStream_t st) {
  const int blocks = (n + KNN_WARPS - 1) / KNN_WARPS;
  if ((ties ? k + 1 : k) <= 32) knn_kernel<1><<<blocks, 32 * KNN_WARPS, 0, st>>>(n, k, ds, out, ties);
  else knn_kernel<2><<<blocks, 32 * KNN_WARPS, 0, st>>>(n, k, ds, out, ties);
  return tspb_launch_status();
}

}  // namespace tspb

using namespace tspb;

extern "C" int tspb_knn(const int32_t* dist, int64_t dist_stride, const double* coords, int32_t n, int32_t k,
                        int32_t* out, void* stream) {
  if (n < 0 || k < 0 || k > KNN_MAX_K) return TSPB_ERR_ARG;
  if (n == 0 || k == 0) return TSPB_OK;
  if (!out || (!dist && !coords)) return TSPB_ERR_ARG;
  if (k > n - 1) return TSPB_ERR_ARG;
  DistSrc ds;
  ds.dist = dist;
  ds.stride = dist_stride;
  ds.coords = reinterpret_cast<const double2*>(coords);
  return launch_knn(ds, n, k, out, nullptr, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int tspb_knn_ties(const int32_t* dist, int64_t dist_stride, const double* coords, int32_t n, int32_t k,
                             int32_t* out, int32_t* ties, void* stream) {
  if (n < 0 || k < 0 || k + 1 > KNN_MAX_K) return TSPB_ERR_ARG;
  if (n == 0 || k == 0) return TSPB_OK;
  if (!out || !ties || (!dist && !coords)) return TSPB_ERR_ARG;
  if (k > n - 1) return TSPB_ERR_ARG;
  DistSrc ds;
  ds.dist = dist;
  ds.stride = dist_stride;
  ds.coords = reinterpret_cast<const double2*>(coords);
  return launch_knn(ds, n, k, out, ties, reinterpret_cast<cudaStream_t>(stream));
}
