// Exhaustive 2-opt (best / first) on a distance matrix: one CTA per tour, every pass on the
// device. Semantics as in two_opt.cu (src/algorithms/strategies/local_search/two_opt.py:188-261,
// 386-489, 565-595); tours need cities in range only, as there.
//
// With R_i[p] = d(t[i], t[p]), the gain of the pair (i, p) is R_i[p] + R_{i+1}[p+1] - e_i - e_p.
// So a warp takes 31 consecutive p (the 32nd lane brings R[p+1]) and walks rows i: one lookup
// of its city in row t[i+1] of the matrix per pair, and the other term is the neighbour lane's.
// The rows stand in shared memory: the whole matrix where it fits (n up to about 220 for a CTA
// with an SM to itself), else tiles of rows copied asynchronously, the next while one is
// worked on. The kernel before it gathered both distances of every pair from L2.
//
// best keeps each row's minimum key across passes. After a move with window [bi, bj] and
// symmetric distances only pairs with a position in the window change: the rows of the window
// are evaluated anew, and their row t[j] also gives the pairs (p, j) of the earlier rows
// p < bi, which lower those rows' keys. An earlier row whose minimum lay in the window keeps
// its old key as a lower bound, marked stale (lowest bit); only when such a bound is the
// smallest of all keys is the row evaluated anew (0.3 rows a pass on random 500-city tours,
// where a pass touches a third of all pairs). Asymmetric matrices are evaluated in full.
//
// first looks in the order of the scan and stops at the first group of rows with an improving
// pair. Every pair before the last move was not improving, so with symmetric distances the
// next pass looks at the pairs of earlier rows with the window (when that is the shorter way)
// and then from the move's row on. On tours far from an optimum the pair is in the first row or
// two, and copying and evaluating a tile for it is wasted work that costs tours sharing an SM
// their throughput: while the last pair lay in the first rows of its scan, a warp a row looks at
// these straight from the matrix before any tile (100 passes of 2400 random tours of 200 cities:
// 1.2 ms in the general kernel, 1.9 with tiles alone, 0.9). With few tours and a matrix that does
// not fit, the tiles alone are faster (64 tours of 1000 cities 1.3, 0.59 and 0.79 ms).
//
// What bounds it: the chain of a unit (city, row lookups, shuffles, two warp reductions a row)
// and, for tiles, their copies from L2. Measured through the strategy, before and after: 128
// tours of 500 cities to a local optimum, best 59.5 -> 10.8 ms, first 124.1 -> 20.8 ms; 100 of
// 100 cities, best 0.89 -> 0.53 ms; one of 200 cities, ten passes 0.29 -> 0.18 ms.
#include <algorithm>

#include "two_opt.cuh"

namespace tspb {

namespace {

constexpr int kUnitRows = 8;     // rows per warp unit
constexpr int kSlice = 31;       // second positions of a warp's pairs
// Threads of a CTA and of an SM at most: a unit's rows and minima take some 120 registers.
constexpr int kAllThreads = 512;
constexpr long long kCpuBlock = 1LL << 18;  // exhaustive pairs per CPU block (two_opt.py:155)

struct AllSmem {
  unsigned long long red64[32];
  long long redll[32];
  unsigned first;
  int bad;
  int stop;
};

// A row's key: gain in the high word, second position and the stale mark in the low word.
__device__ __forceinline__ unsigned long long row_key(int gain, int p) { return gain_key(gain, (unsigned)p << 1); }

__device__ __forceinline__ void copy_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void copy_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

struct Rows {
  int* buf;      // the matrix by city (whole), else two tiles of `tile` + 1 rows by position
  int pitch;     // ints per row (n rounded up to 4)
  int tile;
  bool whole;
  bool wide;     // 16-byte copies
};

// Up to eight rows j0 .. j0 + last of the tile with their edges. Row r of the matrix (r = 0 ..
// 8, the next row past the last) starts at buf + at[r].
struct RowGroup {
  int at[kUnitRows + 1], edge[kUnitRows];
  int j0, last;
  template <class RowAt>
  __device__ __forceinline__ RowGroup(RowAt row_at, const int* len, int first, int j1)
      : j0(first), last(j1 - first < kUnitRows - 1 ? j1 - first : kUnitRows - 1) {
#pragma unroll
    for (int r = 0; r <= kUnitRows; ++r) at[r] = row_at(first + (r <= last ? r : last + 1));
#pragma unroll
    for (int r = 0; r < kUnitRows; ++r) edge[r] = len[first + (r < last ? r : last)];
  }
  // gain of (j0 + r, p) or (p, j0 + r) for this lane's p with its city and edge; straight-line,
  // so the lookups and shuffles of all rows are in flight together (lane 31 has no pair)
  __device__ __forceinline__ void gains(const int* buf, int city, int ep, int (&gain)[kUnitRows]) const {
    int d[kUnitRows + 1];
#pragma unroll
    for (int r = 0; r <= kUnitRows; ++r) d[r] = buf[at[r] + city];
#pragma unroll
    for (int r = 0; r < kUnitRows; ++r)
      gain[r] = (d[r] - edge[r]) + (__shfl_down_sync(FULL, d[r + 1], 1) - ep);
  }
};

__device__ __forceinline__ int wrapped(int p, int n) { return p < n ? p : (p == n ? 0 : n - 1); }

// Pairs (p, j) of the rows p in [p0, p0 + kSlice), p < p_end, with every j in [j0, j1]: one
// warp, so the rows' keys need no atomics.
template <int MODE, class RowAt>
__device__ __forceinline__ void unit_below(RowAt row_at, const int* buf, const int* tour, const int* edge, int n, int j0,
                                           int j1, int p0, int p_end, unsigned long long* rkey, unsigned* first,
                                           long long& evals) {
  const int lane = threadIdx.x & 31, p = p0 + lane;
  const int city = tour[wrapped(p, n)], ep = edge[p < n ? p : n - 1];
  const bool mine = lane < kSlice && p < p_end;
  int low = 0, low_j = 0;
  for (int g = j0; g <= j1; g += kUnitRows) {
    const RowGroup R(row_at, edge, g, j1);
    int gain[kUnitRows];
    R.gains(buf, city, ep, gain);
    // a short group, neighbouring edges (p = j - 1), and the last edge with the first
    if (R.last < kUnitRows - 1 || p_end > g - 1 || g + R.last == n - 1) {
#pragma unroll
      for (int r = 0; r < kUnitRows; ++r)
        if (r > R.last || p > g + r - 2 || (p == 0 && g + r == n - 1)) gain[r] = 0;
    }
    evals += mine ? R.last + 1 : 0;
#pragma unroll
    for (int r = 0; r < kUnitRows; ++r)
      if (gain[r] < low && (MODE == TSPB_MODE_BEST || low == 0)) {  // first: the row's first j
        low = gain[r];
        low_j = g + r;
      }
  }
  if (mine && low < 0) {
    if (MODE == TSPB_MODE_FIRST) {
      atomicMin(first, (unsigned)p * (unsigned)n + (unsigned)low_j);
    } else {
      const unsigned long long key = row_key(low, low_j);
      if (key < rkey[p]) rkey[p] = key;
    }
  }
}

// Pairs (j, p) of the rows j0 .. up to j1 with p in the slices [p0, p0 + kSlice * count), p >=
// j + 2. The lanes keep each row's smallest gain over the slices, two warp reductions a row end
// the unit: best stores the row's key at part[row of the unit * step], first lowers *first.
template <int MODE, class RowAt>
__device__ __forceinline__ void unit_ahead(RowAt row_at, const int* buf, const int* tour, const int* edge, int n, int j0,
                                           int j1, int p0, int count, unsigned long long* part, int step,
                                           unsigned* first, long long& evals) {
  const int lane = threadIdx.x & 31;
  const RowGroup R(row_at, edge, j0, j1);
  int low[kUnitRows], low_p[kUnitRows];
#pragma unroll
  for (int r = 0; r < kUnitRows; ++r) {
    low[r] = 0;
    low_p[r] = n;
  }
  for (int s = 0; s < count; ++s, p0 += kSlice) {
    if (p0 + kSlice - 1 < j0 + 2 || p0 >= n) continue;  // wholly below the diagonal, or past the tour
    const int p = p0 + lane;
    const int city = tour[wrapped(p, n)], ep = edge[p < n ? p : n - 1];
    int gain[kUnitRows];
    R.gains(buf, city, ep, gain);
    if (p0 < j0 + R.last + 2 || p0 + kSlice >= n || R.last < kUnitRows - 1) {  // an edge of the triangle
#pragma unroll
      for (int r = 0; r < kUnitRows; ++r)
        if (r > R.last || p < j0 + r + 2 || p >= n || (j0 + r == 0 && p == n - 1)) gain[r] = 0;
    }
    evals += lane < kSlice ? R.last + 1 : 0;
#pragma unroll
    for (int r = 0; r < kUnitRows; ++r)
      if (gain[r] < (MODE == TSPB_MODE_BEST ? low[r] : (low_p[r] == n ? 0 : INT32_MIN))) {
        low[r] = gain[r];
        low_p[r] = p;
      }
  }
  unsigned long long key = NO_KEY;  // lane r: the key of row j0 + r
  unsigned idx = NO_IDX;
#pragma unroll
  for (int r = kUnitRows - 1; r >= 0; --r) {
    if (lane == kSlice) low[r] = 0;
    if (MODE == TSPB_MODE_FIRST) {
      const int q = __reduce_min_sync(FULL, low[r] < 0 ? low_p[r] : n);
      if (q < n) idx = (unsigned)(j0 + r) * (unsigned)n + (unsigned)q;
    } else {
      const int least = __reduce_min_sync(FULL, low[r]);
      const int q = __reduce_min_sync(FULL, low[r] == least ? low_p[r] : n);
      if (lane == r && least < 0) key = row_key(least, q);
    }
  }
  if (MODE == TSPB_MODE_FIRST) {
    if (lane == 0 && idx != NO_IDX) atomicMin(first, idx);
  } else if (lane <= R.last) {
    part[lane * step] = key;
  }
}

}  // namespace

// LOOK: first looks at its first rows without a tile.
template <int MODE, bool LOOK>
__global__ void __launch_bounds__(kAllThreads) two_opt_all_kernel(const TwoOptArgs A, int tile, int whole, int wide) {
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ AllSmem S;
  const int n = A.n, tid = threadIdx.x, T = blockDim.x;
  const int lane = tid & 31, wid = tid >> 5, nwarps = T >> 5;
  const int t = blockIdx.x;
  if (t >= A.num_tours) return;
  if (A.skip != nullptr && *A.skip != 0) return;
  const int32_t* __restrict__ dist = A.ds.dist;
  const long long stride = A.ds.stride;
  int32_t* g_tour = A.tours + (long long)t * n;
  Rows W;
  W.pitch = (n + 3) & ~3;
  W.tile = tile;
  W.whole = whole != 0;
  W.wide = wide != 0;
  W.buf = reinterpret_cast<int*>(dsm);
  // best: the rows' keys, and per tile (two of them) its rows' keys by slice
  const int slices = (n + kSlice - 1) / kSlice;
  unsigned long long* rkey =
      reinterpret_cast<unsigned long long*>(W.buf + (size_t)(whole ? n : 2 * (tile + 1)) * W.pitch);
  unsigned long long* part = rkey + (MODE == TSPB_MODE_BEST ? n : 0);
  int* tour = reinterpret_cast<int*>(part + (MODE == TSPB_MODE_BEST ? 2 * tile * slices : 0));
  int* edge = tour + n;

  if (tid == 0) {
    S.bad = 0;
    S.stop = 0;
  }
  __syncthreads();
  for (int p = tid; p < n; p += T) {
    const int v = g_tour[p];
    tour[p] = v;
    if ((unsigned)v >= (unsigned)n) S.bad = 1;
  }
  __syncthreads();
  if (S.bad) {
    if (tid == 0) {
      if (A.status) A.status[t] = TSPB_ERR_ARG;
      if (A.stats)
        for (int q = 0; q < 4; ++q) A.stats[(long long)t * 4 + q] = 0;
    }
    return;
  }
  // copies matrix row `city` into slot r of the buffer, by one warp
  auto copy_row = [&](int r, int city) {
    int* dst = W.buf + (size_t)r * W.pitch;
    const int32_t* src = dist + (long long)city * stride;
    if (W.wide) {
      for (int q = lane * 4; q + 4 <= n; q += 128) copy_async16(dst + q, src + q);
      if (lane < (n & 3)) copy_async4(dst + (n & ~3) + lane, src + (n & ~3) + lane);
    } else {
      for (int q = lane; q < n; q += 32) copy_async4(dst + q, src + q);
    }
  };
  if (W.whole)
    for (int c = wid; c < n; c += nwarps) copy_row(c, c);
  copies_commit();
  for (int p = tid; p < n; p += T) edge[p] = A.ds(tour[p], tour[p + 1 == n ? 0 : p + 1]);
  copies_wait();
  __syncthreads();

  const int rows = n - 2;  // rows i in [0, n - 3]
  const long long exh_total = (long long)(n - 3) + (long long)(n - 3) * (n - 2) / 2;
  long long evals = 0;

  // first: rows [lo, lo + warps) without a tile, a warp per row that leaves at its first
  // improving pair. Ends with a barrier.
  auto look = [&](int lo) {
    const int i = lo + wid;
    if (i < rows) {
      const int a = tour[i], b = tour[i + 1], eab = edge[i], lim = n - (i == 0);
      constexpr int U = 4;  // columns of a lane in flight
      for (int j0 = i + 2; j0 < lim; j0 += 32 * U) {
        const unsigned known = *reinterpret_cast<volatile unsigned*>(&S.first);
        if (__any_sync(FULL, known < (unsigned)i * (unsigned)n)) break;  // an earlier row has a pair
        int c[U], d[U], dac[U], dbd[U], hit = n;
        bool ok[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int j = j0 + 32 * u + lane;
          ok[u] = j < lim;
          c[u] = ok[u] ? tour[j] : a;
          d[u] = ok[u] ? tour[j + 1 == n ? 0 : j + 1] : b;
          evals += ok[u];
        }
        if (W.whole) {
#pragma unroll
          for (int u = 0; u < U; ++u) {
            dac[u] = W.buf[a * W.pitch + c[u]];
            dbd[u] = W.buf[b * W.pitch + d[u]];
          }
        } else {
          gather_if(A.ds, a, c, ok, dac);
          gather_if(A.ds, b, d, ok, dbd);
        }
#pragma unroll
        for (int u = U - 1; u >= 0; --u) {
          const int j = j0 + 32 * u + lane;
          if (ok[u] && (dac[u] - eab) + (dbd[u] - edge[j]) < 0) hit = j;
        }
        hit = __reduce_min_sync(FULL, hit);
        if (hit < n) {
          if (lane == 0) atomicMin(&S.first, (unsigned)i * (unsigned)n + (unsigned)hit);
          break;
        }
      }
    }
    __syncthreads();
  };

  // Evaluates rows j in [lo, hi]: their pairs with p >= j + 2 when `own`, and the pairs (p, j)
  // of the rows p < p_below. A barrier before (the caller's) and after. first stops after the
  // tile that holds an improving pair when `stop_early`. Warps take units in turn,
  // the long ones (a slice of earlier rows against the whole tile) before the others.
  auto evaluate = [&](int lo, int hi, bool own, int p_below, bool stop_early) {
    const int below = p_below > 0 ? (p_below + kSlice - 1) / kSlice : 0;
    auto fetch = [&](int j0, int j1, int b) {
      const int last = j1 < hi ? j1 : hi;
      for (int j = j0 + wid; j <= last + 1; j += nwarps) copy_row(b * (W.tile + 1) + (j - j0), tour[j < n ? j : 0]);
    };
    if (!W.whole) {
      fetch(lo, lo + (stop_early ? kUnitRows : W.tile) - 1, 0);
      copies_commit();
    }
    int b = 0;
    // Keys of the tile before this one, by unit column: taken from `part` while the next tile is
    // worked on, a row per thread of the last warps.
    int done_j0 = -1, done_j1 = -1, done_cols = 0;
    auto take = [&]() {
      if (done_j0 < 0) return;
      for (int j = done_j0 + (T - 1 - tid); j <= done_j1; j += T) {
        const unsigned long long* row = part + ((size_t)(b ^ 1) * W.tile + (j - done_j0)) * slices;
        unsigned long long key = NO_KEY;
        for (int s = 0; s < done_cols; ++s) key = row[s] < key ? row[s] : key;
        rkey[j] = key;
      }
    };
    int step = stop_early ? kUnitRows : W.tile;  // first looks at few rows to begin with
    for (int j0 = lo, next_j0; j0 <= hi; j0 = next_j0, b ^= 1) {
      next_j0 = j0 + step;
      const int j1 = next_j0 - 1 < hi ? next_j0 - 1 : hi;
      step = step * 2 < W.tile ? step * 2 : W.tile;
      if (!W.whole) copies_wait();
      __syncthreads();  // the tile's rows and the previous tile's keys are there
      if (!W.whole && next_j0 <= hi) {  // into the buffer that the previous tile has left
        fetch(next_j0, next_j0 + step - 1, b ^ 1);
        copies_commit();
      }
      if (MODE == TSPB_MODE_BEST && own) take();
      const int tile_at = b * (W.tile + 1) * W.pitch;
      const int ngroups = (j1 - j0 + kUnitRows) / kUnitRows;
      const int ahead = own && j0 + 2 < n ? (n - (j0 + 2) + kSlice - 1) / kSlice : 0;
      // slices per unit: four, fewer where that would leave warps without a unit
      int per = (ahead * ngroups + nwarps - 1) / nwarps;
      per = per < 1 ? 1 : (per > 4 ? 4 : per);
      const int cols = (ahead + per - 1) / per;
      const int units = below + cols * ngroups;
      for (int u = wid; u < units; u += nwarps) {
        auto unit = [&](auto row_at) {
          if (u < below) {
            unit_below<MODE>(row_at, W.buf, tour, edge, n, j0, j1, u * kSlice, p_below, rkey, &S.first, evals);
          } else {
            const int c = (u - below) / ngroups, g = (u - below) - c * ngroups;
            unit_ahead<MODE>(row_at, W.buf, tour, edge, n, j0 + g * kUnitRows, j1, j0 + 2 + c * per * kSlice, per,
                             part + ((size_t)b * W.tile + g * kUnitRows) * slices + c, slices, &S.first, evals);
          }
        };
        if (W.whole) unit([&](int j) { return tour[j < n ? j : 0] * W.pitch; });
        else unit([&](int j) { return tile_at + (j - j0) * W.pitch; });
      }
      done_j0 = j0;
      done_j1 = j1;
      done_cols = cols;
      if (stop_early) {
        __syncthreads();
        const bool done = S.first != NO_IDX;
        __syncthreads();  // all have read it
        if (done) break;
      }
    }
    if (!W.whole) copies_wait();
    __syncthreads();
    if (MODE == TSPB_MODE_BEST && own) {
      take();
      __syncthreads();
    }
  };

  long long passes = 0, moves = 0, pairs_closed = 0;
  int err = TSPB_OK;
  int win_lo = -1, win_hi = -1;  // window of the last move
  bool near = true;              // first: the last pair found lay in the first rows of its scan
  const long long t_start = clock64();
  while (passes < A.max_iter) {
    if (tid == 0) {
      if (clock64() - t_start > A.budget) S.stop = TSPB_ERR_BUDGET;
      S.first = NO_IDX;
    }
    const bool partial = A.symmetric && win_lo >= 0;
    if (MODE == TSPB_MODE_BEST && !partial)
      for (int i = tid; i < n; i += T) rkey[i] = NO_KEY;
    __syncthreads();
    if (S.stop) {
      err = S.stop;
      break;
    }
    ++passes;
    int bi, bj;
    if (MODE == TSPB_MODE_BEST) {
      if (partial) evaluate(win_lo, win_hi, true, win_lo, false);
      else evaluate(0, rows - 1, true, 0, false);
      unsigned long long top;
      while (true) {
        // the smallest (gain, row): the gain word of the keys, ties to the lower row
        top = NO_KEY;
        for (int i = tid; i < rows; i += T) {
          const unsigned long long key = (rkey[i] & ~0xffffffffull) | (unsigned)i;
          if (rkey[i] != NO_KEY && key < top) top = key;
        }
        top = block_min(top, S.red64);
        if (top == NO_KEY) break;
        const int i = (int)(unsigned)top;
        if ((rkey[i] & 1ull) == 0) break;
        __syncthreads();  // every thread has seen the stale key
        if (tid == 0) rkey[i] = NO_KEY;
        __syncthreads();
        evaluate(i, i, true, 0, false);
      }
      if (tid == 0) pairs_closed += exh_total;
      if (top == NO_KEY) break;
      bi = (int)(unsigned)top;
      bj = (int)((unsigned)rkey[bi] >> 1);
    } else {
      int from = 0;
      if (partial && win_lo > 0 && win_hi - win_lo < win_lo) {  // no more rows of the window than rows before it
        evaluate(win_lo, win_hi, false, win_lo, false);
        from = win_lo;
      }
      if (S.first == NO_IDX) {
        __syncthreads();  // S.first is read by all before the scan lowers it
        const int begin = from;
        if (LOOK && near) {
          look(from);
          from += nwarps;
          const bool found = S.first != NO_IDX;
          __syncthreads();  // as above
          if (!found && from < rows) evaluate(from, rows - 1, true, 0, true);
        } else {
          evaluate(from, rows - 1, true, 0, true);
        }
        near = S.first < (unsigned)(begin + nwarps) * (unsigned)n;
      }
      const unsigned idx = S.first;
      if (tid == 0) {
        long long upto = exh_total;
        if (idx != NO_IDX) {
          const long long fi = idx / (unsigned)n, fj = idx - fi * n;
          const long long before = fi == 0 ? 0 : (n - 3) + (fi - 1) * (n - 2) - (fi - 1) * fi / 2;  // pairs of earlier rows
          upto = ((before + (fj - fi - 2)) / kCpuBlock + 1) * kCpuBlock;
          upto = upto < exh_total ? upto : exh_total;
        }
        pairs_closed += upto;
      }
      if (idx == NO_IDX) break;
      bi = (int)(idx / (unsigned)n);
      bj = (int)(idx - (unsigned)bi * (unsigned)n);
    }
    if (bi < 0 || bj <= bi + 1 || bj >= n) {  // cannot happen for a valid scan; never index with it
      err = TSPB_ERR_RANGE;
      break;
    }
    __syncthreads();  // every thread has decoded (bi, bj) before the tour and the keys change
    const int lo = bi + 1, half = (bj - bi) >> 1;
    for (int q = tid; q < half; q += T) {
      const int x = tour[lo + q], y = tour[bj - q];
      tour[lo + q] = y;
      tour[bj - q] = x;
    }
    if (MODE == TSPB_MODE_BEST && A.symmetric) {
      for (int i = tid; i <= bj; i += T) {
        if (i >= bi) {
          rkey[i] = NO_KEY;  // evaluated anew
        } else if (rkey[i] != NO_KEY) {
          const int p = (int)((unsigned)rkey[i] >> 1);
          if (p >= bi && p <= bj) rkey[i] |= 1ull;  // a lower bound from here on
        }
      }
    }
    __syncthreads();
    for (int p = bi + tid; p <= bj; p += T) edge[p] = A.ds(tour[p], tour[p + 1 == n ? 0 : p + 1]);
    ++moves;
    win_lo = bi;
    win_hi = bj;
  }

  // ---- write back ---------------------------------------------------------------------
  __syncthreads();
  for (int p = tid; p < n; p += T) g_tour[p] = tour[p];
  const long long te = block_sum(evals, S.redll);
  if (tid == 0) {
    if (A.status) A.status[t] = err;
    if (A.stats) {
      long long* st = A.stats + (long long)t * 4;
      st[0] = passes;
      st[1] = pairs_closed;
      st[2] = moves;
      st[3] = te;
    }
  }
}

// Launches the kernel when its rows fit in shared memory and the run is long enough for them;
// false: the caller takes the general one (distances rebuilt from coordinates, rows too long
// for tiles of kUnitRows, tours or runs so short that a pass costs less than setting up for it).
bool launch_two_opt_all(const TwoOptArgs& a, int mode, int threads, cudaStream_t st, int* status) {
  const bool first = mode == TSPB_MODE_FIRST;
  const int sms = device_attr(cudaDevAttrMultiProcessorCount);
  const int sm_bytes = device_attr(cudaDevAttrMaxSharedMemoryPerMultiprocessor);
  if (sms <= 0 || sm_bytes <= 0) return false;
  const bool many = a.num_tours > sms;  // tours share SMs
  // Below 64 cities a pass is a few hundred cycles and the general kernel's fewer barriers win:
  // 100 tours of 50 cities 0.25 ms there and 0.30 here, of 70 cities 0.46 and 0.38. So they do
  // for the shortest runs: ten passes of 148 tours of 64 cities 0.14 and 0.16 ms, one pass of
  // 5000 tours of 130 cities 0.25 and 0.32, three first passes of 2400 tours of 300 cities 0.12 and 0.15.
  if (a.ds.dist == nullptr || a.n < 64 || (a.n < 72 && a.max_iter <= 16)) return false;
  if (many && (first ? a.max_iter <= 3 : a.max_iter == 1 && a.n < 300)) return false;
  threads = std::min(threads, kAllThreads);
  // first is a chain of short passes: narrower CTAs, more of them an SM, where there are tours
  // for it. 30 passes of 1200 tours at 64 / 128 / 256 threads, relative: 64 cities 1.15 / 1 / 0.71,
  // 200 cities 1.15 / 1 / 0.67, 1000 cities 0.91 / 1 / 0.79; 100 cities 1.10 / 1 / 0.72, but to a
  // local optimum 0.75 / 1 / 0.64 (at 128 threads the whole matrix of up to 120 cities fits).
  if (first && a.num_tours >= 2 * sms && a.n < 512) threads = std::min(threads, 128);
  if (first && (a.n <= 80 ? a.num_tours >= 4 * sms
                          : a.num_tours >= 8 * sms && a.n < 256 && (a.n >= 128 || a.max_iter <= 64)))
    threads = std::min(threads, 64);
  const long long pitch = (a.n + 3) & ~3;
  const long long slices = (a.n + kSlice - 1) / kSlice;
  // tour, edges, and best's row keys and two tiles of keys by slice
  auto state = [&](long long tile) { return (first ? 8LL * a.n : 16LL * a.n + 16 * tile * slices) + 16; };
  // CTAs an SM: as many as there are tours for and registers hold. (Shared memory split for more
  // of them than registers hold leaves small tiles: best, ten passes of 5000 tours of 90 cities
  // 1.71 ms that way and 0.81 this, 0.93 in the general kernel.)
  const int wanted = std::max(1, std::min((a.num_tours + sms - 1) / sms, kAllThreads / threads));
  int resident = wanted, tile = 0, whole = 0;
  while (true) {
    const long long share = std::min<long long>(sm_bytes / resident - 1024, smem_optin()) - (long long)sizeof(AllSmem);
    // the whole matrix with one tile for all rows, or as many rows as fit beside it
    for (int rows = (a.n + kUnitRows - 1) / kUnitRows * kUnitRows; rows >= 2 * kUnitRows && tile == 0; rows -= kUnitRows) {
      whole = a.n * pitch * 4 + state(rows) <= share;
      if (whole) tile = rows;
    }
    for (int rows = 4 * kUnitRows; rows >= kUnitRows && tile == 0; rows -= kUnitRows)
      if (2 * (rows + 1) * pitch * 4 + state(rows) <= share) tile = rows;
    if (tile != 0 || resident == 1) break;
    --resident;
  }
  if (tile == 0) return false;
  // Fewer CTAs than registers hold: a short run of first mode, all of it close to row 0, is
  // faster in the general kernel, a long one here (2400 tours of 1500 cities, 10 passes: 0.39 ms
  // there and 0.57 here; 600 of 1000 cities, 100 passes 1.21 and 0.84, 300 on good tours 40 and 9).
  if (first && resident < wanted && a.max_iter <= 16) return false;
  const size_t smem = (size_t)((whole ? a.n : 2 * (tile + 1)) * pitch * 4 + state(tile));
  const int wide = a.ds.stride % 4 == 0 && reinterpret_cast<uintptr_t>(a.ds.dist) % 16 == 0;
  auto kern = !first          ? two_opt_all_kernel<TSPB_MODE_BEST, false>
              : many || whole ? two_opt_all_kernel<TSPB_MODE_FIRST, true>
                              : two_opt_all_kernel<TSPB_MODE_FIRST, false>;
  *status = TSPB_ERR_CUDA;
  if (allow_smem(kern, smem) != cudaSuccess) {
    (void)cudaGetLastError();
    return true;
  }
  kern<<<a.num_tours, threads, smem, st>>>(a, tile, whole, wide);
  *status = tspb_launch_status();
  return true;
}

}  // namespace tspb
