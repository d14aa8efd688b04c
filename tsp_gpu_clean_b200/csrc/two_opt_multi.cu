// multi_move 2-opt: one CTA per tour, every pass on the device.
//
// A pass of the reference (src/algorithms/strategies/local_search/two_opt.py:491-563) sorts
// every improving pair by (gain, scan index) and accepts them greedily when the window
// [i, j] touches no accepted window. The greedy choice needs no sort: the next accepted
// pair is the smallest key among the pairs that touch no accepted window. So a pass here
//   1. scans the neighbourhood, appends the improving keys to the tour's slice of the
//      workspace and keeps each thread's smallest;
//   2. takes the CTA's smallest key, applies its reversal at once (accepted windows are
//      disjoint, so the remaining pairs' cities and positions do not change), and
//   3. lets every thread drop the touched keys of its own share and find its smallest among
//      the rest; then 2 again, until no key is left.
//
// What bounds it: the scan's random distance gathers, one per improving pair (an SM is served
// about one a cycle from L2: half of a pass), then the latency of the rounds. A random
// 1002-city tour has about 8,000 improving pairs a pass, of which 10 to 25 are accepted, and
// the first round drops most of the list. 256 tours of 1002 cities, k = 20, ten passes: a
// bitonic sort in global memory and one warp walking all sorted keys took 37.5 ms; the rounds
// alone 0.99 ms; with the list in shared memory, the windows beside the keys and the gathers
// of a thread in flight together 0.63 ms.
//
// Candidate scans with packed k-NN words (c | d(a, c) << 16, k % 4 == 0, 16-byte aligned) read
// four entries of a row per thread and skip the distance gather of entries whose lower bound
// d(a,c) - d(a,b) - d(c,d) is not negative (distances are >= 0).
#include <algorithm>
#include <type_traits>

#include "two_opt.cuh"

namespace tspb {

namespace {

struct MultiSmem {
  unsigned long long red64[32];
  long long redll[32];
  unsigned m;    // improving pairs found this pass
  unsigned win;  // window of the pair accepted next
  int bad;     // input validation failure
  int stop;    // pass loop must end with an error status
};

enum MultiScan { MULTI_ALL = 0, MULTI_CAND = 1, MULTI_PACKED = 2 };

// An improving pair: its key and its window i << 16 | j.
struct Pair {
  unsigned long long key;
  unsigned win;
};

// The tour's list of improving pairs: the first `cap` slots in shared memory, with their
// windows; the rest as keys in the workspace slice (whose first `cap` slots stay unused).
struct PairList {
  unsigned long long* fast;
  unsigned* win;
  unsigned long long* slow;
  unsigned cap;
  __device__ __forceinline__ void put(unsigned slot, const Pair& v) const {
    if (slot < cap) {
      fast[slot] = v.key;
      win[slot] = v.win;
    } else {
      slow[slot] = v.key;
    }
  }
};

// Appends the improving pairs of a warp, up to U per lane (gain < 0, scan index e, window
// i << 16 | j), with one shared atomic, and lowers the lane's smallest.
template <int U>
__device__ __forceinline__ void append_pairs(const int (&gain)[U], const unsigned (&e)[U], const unsigned (&win)[U],
                                             unsigned* count, const PairList& list, Pair& best) {
  unsigned m[U], total = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    m[u] = __ballot_sync(FULL, gain[u] < 0);
    total += __popc(m[u]);
  }
  if (total == 0) return;
  const int lane = threadIdx.x & 31;
  unsigned base = 0;
  if (lane == 0) base = atomicAdd(count, total);
  base = __shfl_sync(FULL, base, 0);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (gain[u] < 0) {
      const Pair v{gain_key(gain[u], e[u]), win[u]};
      if (v.key < best.key) best = v;
      list.put(base + __popc(m[u] & ((1u << lane) - 1u)), v);
    }
    base += __popc(m[u]);
  }
}

// d(a[u], b[u]) for the entries with ok[u] (0 elsewhere), all loads in flight together.
template <int U>
__device__ __forceinline__ void gather_pairs(const DistSrc& ds, const int (&a)[U], const int (&b)[U],
                                             const bool (&ok)[U], int (&d)[U]) {
  if (ds.dist != nullptr) {
#pragma unroll
    for (int u = 0; u < U; ++u) d[u] = load_cg_if(ok[u], ds.dist + (long long)a[u] * ds.stride + b[u]);
  } else {
#pragma unroll
    for (int u = 0; u < U; ++u) d[u] = ok[u] ? ds(a[u], b[u]) : 0;
  }
}

}  // namespace

// SCAN: exhaustive pairs, candidate rows, or candidate rows with packed words. SMEM: tour
// arrays in shared memory, else in the tour's workspace slice.
template <int SCAN, bool SMEM>
__global__ void __launch_bounds__(1024) two_opt_multi_kernel(const TwoOptArgs A) {
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ MultiSmem S;
  constexpr bool CAND = SCAN != MULTI_ALL;
  const int n = A.n, k = A.k;
  const int tid = threadIdx.x, T = blockDim.x;
  const int lane = tid & 31, wid = tid >> 5, nwarps = T >> 5;
  const int t = blockIdx.x;
  if (t >= A.num_tours) return;
  if (A.skip != nullptr && *A.skip != 0) return;

  int32_t* g_tour = A.tours + (long long)t * n;
  unsigned char* ws = A.ws + (size_t)t * A.ws_tour_bytes;
  int* s_tour = reinterpret_cast<int*>(SMEM ? dsm : ws);
  int* s_pos = s_tour + n;
  int* s_edge = s_pos + n;
  unsigned long long* fast = reinterpret_cast<unsigned long long*>(dsm + (SMEM ? ((size_t)12 * n + 15) / 16 * 16 : 0));
  const PairList list{fast, reinterpret_cast<unsigned*>(fast + A.keys_in_smem),
                      reinterpret_cast<unsigned long long*>(ws + A.ws_keys_off), (unsigned)A.keys_in_smem};
  const DistSrc ds = A.ds;
  const int32_t* __restrict__ cand = A.cand;
  const uint32_t* __restrict__ packed = A.cand_packed;

  // ---- load the tour, build pos, validate --------------------------------------------
  if (tid == 0) {
    S.bad = 0;
    S.stop = 0;
  }
  for (int p = tid; p < n; p += T) {
    s_tour[p] = g_tour[p];
    s_pos[p] = -1;
  }
  __syncthreads();
  for (int p = tid; p < n; p += T) {
    const int v = s_tour[p];
    if ((unsigned)v >= (unsigned)n) {
      S.bad = 1;
    } else if (CAND) {
      if (atomicExch(&s_pos[v], p) != -1) S.bad = 1;
    }
  }
  __syncthreads();
  if (S.bad) {
    if (tid == 0) {
      if (A.status) A.status[t] = CAND ? TSPB_ERR_NOT_PERMUTATION : TSPB_ERR_ARG;
      if (A.stats)
        for (int q = 0; q < 4; ++q) A.stats[(long long)t * 4 + q] = 0;
    }
    return;
  }

  const int rows = n - 2;  // rows i in [0, n - 3]
  const long long exh_total = (long long)(n - 3) + (long long)(n - 3) * (n - 2) / 2;
  const unsigned div = CAND ? (unsigned)k : (unsigned)n;  // scan index = i * div + column
  // i of a scan index by multiply-high with ceil(2^32 / div): exact while index * div < 2^32
  // and the reciprocal itself fits 32 bits, which div = 1 does not
  const unsigned mag = (unsigned)(((1ull << 32) + div - 1) / div);
  const bool mag_exact = div > 1 && (unsigned long long)n * div * div < (1ull << 32);
  auto row_of = [&](unsigned idx) -> int { return (int)(mag_exact ? __umulhi(idx, mag) : idx / div); };
  // second position of pair idx of row i; used while row i touches no accepted window
  auto col_of = [&](unsigned idx, int i) -> int {
    const unsigned r = idx - (unsigned)i * div;
    if (!CAND) return (int)r;
    const unsigned e = (unsigned)s_tour[i] * (unsigned)k + r;
    return s_pos[SCAN == MULTI_PACKED ? (int)(__ldg(packed + e) & 0xffffu) : __ldg(cand + e)];
  };

  long long passes = 0, moves = 0, my_pairs = 0;
  int err = TSPB_OK;
  const long long t_start = clock64();
  while (passes < A.max_iter) {
    if (tid == 0) {
      if (clock64() - t_start > A.budget) S.stop = TSPB_ERR_BUDGET;
      S.m = 0;
    }
    // every edge of the tour (the setup's, or the last pass's moves)
    for (int p = tid; p < n; p += T) s_edge[p] = ds(s_tour[p], s_tour[p + 1 == n ? 0 : p + 1]);
    __syncthreads();
    if (S.stop) {
      err = S.stop;
      break;
    }
    ++passes;

    // ---- 1. scan ----------------------------------------------------------------------
    Pair best{NO_KEY, 0u};
    if constexpr (SCAN == MULTI_PACKED) {
      const int G = k >> 2, items = rows * G;
      int i = tid / G, g = tid - i * G;  // this thread's group: row i, entries 4 g ..
      const int di = T / G, dg = T - di * G;
      for (int it0 = wid * 32; it0 < items; it0 += T) {
        const int it = it0 + lane;
        int gain[4] = {0, 0, 0, 0}, j[4];
        unsigned e[4] = {}, win[4] = {};
        if (it < items) {
          const unsigned r0 = (unsigned)g * 4u;
          const int a = s_tour[i], b = s_tour[i + 1], ea = s_edge[i];
          const uint4 w4 = __ldg(reinterpret_cast<const uint4*>(packed + ((unsigned)a * (unsigned)k + r0)));
          const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
          const int lo = i + 2;
          const unsigned span = (unsigned)(n - (i == 0) - lo);
          bool ok[4];
          int lb[4], d[4], dbd[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int c = (int)(w[u] & 0xffffu);
            j[u] = s_pos[(unsigned)c < (unsigned)n ? c : a];  // an invalid id: position i, refused below
            ok[u] = (unsigned)(j[u] - lo) < span;
            my_pairs += ok[u];
            d[u] = s_tour[j[u] + 1 == n ? 0 : j[u] + 1];
            lb[u] = ((int)(w[u] >> 16) - ea) - s_edge[j[u]];
            ok[u] &= lb[u] < 0;
          }
          gather_if(ds, b, d, ok, dbd);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            gain[u] = ok[u] ? lb[u] + dbd[u] : 0;
            e[u] = (unsigned)i * (unsigned)k + r0 + (unsigned)u;
            win[u] = ((unsigned)i << 16) | (unsigned)j[u];
          }
        }
        append_pairs(gain, e, win, &S.m, list, best);
        i += di;
        g += dg;
        if (g >= G) {
          g -= G;
          ++i;
        }
      }
    } else if constexpr (SCAN == MULTI_CAND) {
      constexpr int U = 4;  // entries of a lane with their loads in flight together
      const int E = rows * k;
      for (int e0 = wid * 32 * U; e0 < E; e0 += T * U) {
        int gain[U], b[U], d[U], cut[U], dac[U], dbd[U];
        unsigned e[U], win[U];
        bool ok[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int at = e0 + 32 * u + lane;
          ok[u] = at < E;
          const int i = ok[u] ? at / k : 0, a = s_tour[i];
          const long long f = (long long)a * k + (ok[u] ? at - i * k : 0);
          const int c = (int)load_nc_if(ok[u], cand + f);
          const int j = (unsigned)c < (unsigned)n ? s_pos[c] : 0;
          ok[u] = ok[u] && j > i + 1 && j < n - (i == 0);
          my_pairs += ok[u];
          dac[u] = A.cand_dist ? (int)load_nc_if(ok[u], A.cand_dist + f) : (ok[u] ? ds(a, c) : 0);
          b[u] = s_tour[i + 1];
          d[u] = s_tour[j + 1 == n ? 0 : j + 1];
          cut[u] = s_edge[i] + s_edge[j];
          e[u] = (unsigned)at;
          win[u] = ((unsigned)i << 16) | (unsigned)j;
        }
        gather_pairs(ds, b, d, ok, dbd);
#pragma unroll
        for (int u = 0; u < U; ++u) gain[u] = ok[u] ? dac[u] - cut[u] + dbd[u] : 0;
        append_pairs(gain, e, win, &S.m, list, best);
      }
    } else {
      for (int i = wid; i < rows; i += nwarps) {
        const int a = s_tour[i], b = s_tour[i + 1], eab = s_edge[i];
        const int lim = n - (i == 0);
        auto pairs = [&](auto wide, int j0) {  // of U x 32 positions from j0 on
          constexpr int U = decltype(wide)::value;
          int gain[U], c[U], d[U], dac[U], dbd[U];
          unsigned e[U], win[U];
          bool ok[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int j = j0 + 32 * u + lane;
            ok[u] = j < lim;
            my_pairs += ok[u];
            c[u] = s_tour[ok[u] ? j : 0];
            d[u] = s_tour[ok[u] && j + 1 < n ? j + 1 : 0];
            e[u] = (unsigned)i * (unsigned)n + (unsigned)j;
            win[u] = ((unsigned)i << 16) | (unsigned)j;
          }
          gather_if(ds, a, c, ok, dac);
          gather_if(ds, b, d, ok, dbd);
#pragma unroll
          for (int u = 0; u < U; ++u) gain[u] = ok[u] ? (dac[u] - eab) + (dbd[u] - s_edge[win[u] & 0xffffu]) : 0;
          append_pairs(gain, e, win, &S.m, list, best);
        };
        int j0 = i + 2;
        for (; lim - j0 > 64; j0 += 128) pairs(std::integral_constant<int, 4>{}, j0);
        for (; j0 < lim; j0 += 32) pairs(std::integral_constant<int, 1>{}, j0);
      }
    }

    // ---- 2. and 3. greedy selection ----------------------------------------------------
    unsigned long long next = block_min(best.key, S.red64);  // its barriers also publish the list
    if (next == NO_KEY) break;                               // no improving pair
    int mine = S.m > (unsigned)tid ? (int)((S.m - (unsigned)tid + (unsigned)T - 1u) / (unsigned)T) : 0;
    do {
      if (best.key == next) S.win = best.win;  // keys are unique: one thread holds it
      __syncthreads();
      const int bi = (int)(S.win >> 16), bj = (int)(S.win & 0xffffu);
      if (bj <= bi + 1 || bj >= n) {  // cannot happen for a valid scan; uniform across the CTA
        err = TSPB_ERR_RANGE;
        break;
      }
      const int lo = bi + 1, half = (bj - bi) >> 1;
      for (int q = tid; q < half; q += T) {
        const int x = s_tour[lo + q], y = s_tour[bj - q];
        s_tour[lo + q] = y;
        s_tour[bj - q] = x;
        if (CAND) {
          s_pos[y] = lo + q;
          s_pos[x] = bj - q;
        }
      }
      __syncthreads();
      // this thread's pairs sit at tid, tid + T, ...; those that stay move to its front
      int kept = 0;
      best = Pair{NO_KEY, 0u};
      constexpr int U = 4;
      for (int q0 = 0; q0 < mine; q0 += U) {
        Pair v[U];
        bool ok[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const unsigned slot = (unsigned)tid + (unsigned)(q0 + u) * (unsigned)T;
          ok[u] = q0 + u < mine;
          v[u] = Pair{NO_KEY, 0u};
          if (!ok[u]) continue;
          if (slot < list.cap) {
            v[u] = Pair{list.fast[slot], list.win[slot]};
          } else {
            v[u].key = list.slow[slot];
            const int i = row_of((unsigned)v[u].key);
            // a row inside the window has changed its city; any j will do, the pair goes
            v[u].win = ((unsigned)i << 16) | (unsigned)(i >= bi && i <= bj ? bj : col_of((unsigned)v[u].key, i));
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int i = (int)(v[u].win >> 16), j = (int)(v[u].win & 0xffffu);
          if (!ok[u] || (i <= bj && j >= bi)) continue;
          if (v[u].key < best.key) best = v[u];
          list.put((unsigned)tid + (unsigned)kept * (unsigned)T, v[u]);
          ++kept;
        }
      }
      mine = kept;
      next = block_min(best.key, S.red64);
    } while (next != NO_KEY);
    __syncthreads();
    if (err != TSPB_OK) break;
    ++moves;
  }

  // ---- write back ---------------------------------------------------------------------
  __syncthreads();
  for (int p = tid; p < n; p += T) g_tour[p] = s_tour[p];
  const long long tp = block_sum(my_pairs, S.redll);
  if (tid == 0) {
    if (A.status) A.status[t] = err;
    if (A.stats) {
      long long* st = A.stats + (long long)t * 4;
      st[0] = passes;
      st[1] = CAND ? tp : passes * exh_total;
      st[2] = moves;
      st[3] = tp;
    }
  }
}

int launch_two_opt_multi(const TwoOptArgs& args, int threads, size_t smem, cudaStream_t st) {
  TwoOptArgs a = args;
  const bool packed = a.cand_packed != nullptr && a.k % 4 == 0 && reinterpret_cast<uintptr_t>(a.cand_packed) % 16 == 0;
  const int scan = a.cand == nullptr ? MULTI_ALL : (packed ? MULTI_PACKED : MULTI_CAND);
  auto kern = scan == MULTI_PACKED ? (a.arrays_in_smem ? two_opt_multi_kernel<MULTI_PACKED, true> : two_opt_multi_kernel<MULTI_PACKED, false>)
              : scan == MULTI_CAND ? (a.arrays_in_smem ? two_opt_multi_kernel<MULTI_CAND, true> : two_opt_multi_kernel<MULTI_CAND, false>)
                                   : (a.arrays_in_smem ? two_opt_multi_kernel<MULTI_ALL, true> : two_opt_multi_kernel<MULTI_ALL, false>);
  // Pairs in shared memory, as many as a CTA's share of the SM leaves when as many CTAs run on
  // it as the batch and the CTA size allow; a pass has at most about half of all entries. The
  // plain scans leave the L1 a third of the SM: their loads in flight need room there. Ten passes
  // from tours along strips: 600 tours of 1000 cities, k = 7 0.64 ms (1.16 with the whole SM for
  // pairs and one entry a lane in flight); every pair of 16 tours of 2000 cities, five passes 8.5 (13.4).
  const int sms = device_attr(cudaDevAttrMultiProcessorCount);
  const int sm_bytes = device_attr(cudaDevAttrMaxSharedMemoryPerMultiprocessor);
  if (sms > 0 && sm_bytes > 0) {
    int resident = (a.num_tours + sms - 1) / sms;
    resident = std::max(1, std::min(resident, 2048 / threads));
    const long long arrays = (long long)((smem + 15) / 16 * 16);
    const long long usable = scan == MULTI_PACKED ? sm_bytes : sm_bytes / 3 * 2;
    const long long share = std::min<long long>(usable / resident - 1024, smem_optin()) - (long long)sizeof(MultiSmem) - arrays;
    const long long rows = a.n - 2;
    const long long most = scan == MULTI_ALL ? rows * (rows + 1) / 2 : rows * a.k;
    const long long cap = std::min(share / 12, most) & ~1LL;
    if (cap > 0) {
      a.keys_in_smem = (int)cap;
      smem = (size_t)arrays + (size_t)cap * 12;
    }
  }
  TSPB_CUDA_CHECK(allow_smem(kern, smem));
  kern<<<a.num_tours, threads, smem, st>>>(a);
  return tspb_launch_status();
}

}  // namespace tspb
