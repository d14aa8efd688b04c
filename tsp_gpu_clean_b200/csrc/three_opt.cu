// Exhaustive steepest-descent 3-opt on open (cyclic TSP) tours, bit-identical to the
// reference's CPU 3-opt (cpu_three_opt_best_move / cpu_three_opt_refine of its 3-opt
// experiment, benchmark_scripts/experiments-and-examples/experiment-comparing-3opt-and-2opt/
// gpu_three_opt.py:143-277):
//   - cuts 0 <= i < j < k <= n-1 remove (t[i], t[i+1]), (t[j], t[j+1]), (t[k], t[(k+1) % n]);
//   - scan order i, j, then the pure 2-opt case 1 at k = j (j > i + 1), then k ascending with
//     cases 2..7; case 2 needs k > j + 1, case 3 is skipped for i = 0, k = n - 1;
//   - the move applied is the first in scan order with the smallest negative delta, i.e.
//     the minimum of (delta, key) with key = ((i n + j) n + k) 8 + case;
//   - a move is up to three reversals: [i+1, j] (cases 1, 4, 5, 7), [j+1, k] (2, 4, 5, 6),
//     [i+1, k] (3, 5, 6, 7).
//
// What bounds it: instruction issue, and the latency between (issue slots 61 % busy on the SMs
// that hold a CTA; ncu, 32 tours of 200 cities). A pass is n^3/6 triples and everything it reads is the
// tour-ordered matrix M[p][q] = d(t[p], t[q]), so the layout is chosen to spend as few
// instructions per triple as possible.
//   - Cases 1, 2 and 3 are the same 2-opt moves met again and again: the pair (x, y) is case 2
//     of (0, x, y) for x >= 1 and case 3 of (0, 1, y) for x = 0, and those carry its smallest
//     keys. They are evaluated once per pair (n^2/2) instead of once per triple.
//   - Cases 4..7 share their terms. A warp takes four consecutive i and 32 consecutive k
//     (one per lane) and walks j: the rows i .. i+4 at columns k and k+1 stay in registers,
//     two coalesced reads (M[j][k], M[j+1][k+1]) serve all four i, and the terms that depend
//     on (i, j) alone are computed once per unit by 16 lanes and read back as three 16-byte
//     broadcasts per j. About 12 instructions per 32 triples where no lane has a move at or below
//     its best, 34 on average over ten passes from random tours (the units' set-up, and lanes with
//     such a move send their warp through the keys); the former layout (a warp per (i, j), int64,
//     all six cases per triple) took about 180.
//   - Deltas are int32 when every distance of M is below 2^29 (three of them fit), int64
//     otherwise; the choice is made per tour from M itself.
//   - A batch with fewer tours than SMs gives each tour a cluster of 2, 4 or 8 CTAs, the
//     largest for which all tours still run at once: every CTA keeps the tour and M, scans
//     its share of the units, and the minima meet through distributed shared memory (one
//     cluster barrier per pass).
//   - M is gathered once per tour (n^2 random reads) and then reversed in place with the
//     tour (n <= kThreeOptSmemN, in shared memory). Larger tours keep it in a workspace slot
//     in HBM, whose rows the CTAs of the tour gather anew each pass (n^2 reads against n^3/6
//     triples).
// Measured, ten passes through the strategy, n = 200: 32 tours 38.7 -> 0.90 ms, 128 tours
// (one CTA each) 2.24 ms, one tour 0.65 ms.
#include <cooperative_groups.h>

#include "common.cuh"
#include "two_opt.cuh"

namespace tspb {

namespace cg = cooperative_groups;

constexpr int kThreeOptSmemN = 220;  // 4 n^2 + 12 n bytes of shared memory at most ~190 KB
constexpr int kThreeOptMaxN = 4096;
constexpr int kThreeOptThreads = 512;  // 768 and 1024 (80 and 64 registers): 0.93 and 0.97 ms against 0.90
constexpr int kRows = 4;  // consecutive i per warp unit
constexpr unsigned long long kNoKey = ~0ull;
// consecutive j per warp unit: their (i, j) terms, 3 kRows per j, take kTermBytes a warp
constexpr int kTermBytes = 768;
template <typename D>
constexpr int kUnitJ = kTermBytes / (3 * kRows * (int)sizeof(D));

struct MoveKey {
  long long delta;
  unsigned long long key;
};

__device__ __forceinline__ bool move_less(const MoveKey& a, const MoveKey& b) {
  return a.delta < b.delta || (a.delta == b.delta && a.key < b.key);
}

__device__ __forceinline__ MoveKey warp_min_move(MoveKey m) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    MoveKey w;
    w.delta = __shfl_xor_sync(FULL, m.delta, o);
    w.key = __shfl_xor_sync(FULL, m.key, o);
    if (move_less(w, m)) m = w;
  }
  return m;
}

// A term that keeps every sum with three distances non-negative and in range: the other two
// terms are at least -d(e, f).
template <typename D>
constexpr D kNever = (D)1 << (sizeof(D) == 4 ? 29 : 31);

// This thread's smallest (delta, key); a delta of 0 with no key means none yet.
template <typename D>
struct Best {
  D delta = 0;
  unsigned long long key = kNoKey;
  __device__ __forceinline__ void take(D d, unsigned long long k) {
    if (d < delta || (d == delta && k < key)) {
      delta = d;
      key = k;
    }
  }
};

__device__ __forceinline__ int add_min(int a, int b, int c) { return __viaddmin_s32(a, b, c); }
__device__ __forceinline__ long long add_min(long long a, long long b, long long c) { return a + b < c ? a + b : c; }

// Cases 4..7 of the unit (i0 .. i0+3, this lane's k, j from j_lo to j_hi). U holds, for
// each j of the unit, the terms of (i, j) alone: d(a,c), d(a,d) and d(b,d), each minus
// d(a,b) + d(c,d), for the four rows. The units on the diagonals hold (i, j, k) that violate
// i < j < k: rows i >= j have kNever for terms, lanes with k <= j skip the slow path.
template <typename D>
__device__ __forceinline__ void scan_span(const int* M, const D (*U)[3][kRows], int n, int i0, int k, D def,
                                          int j_lo, int j_hi, const D (&rk)[kRows + 1], const D (&rkp)[kRows + 1],
                                          Best<D>& best) {
  const int kp = k + 1 == n ? 0 : k + 1;
  const int* row = M + (long long)j_lo * n;
  D cf = (D)row[kp] - def;  // d(c, f) - d(e, f)
#pragma unroll 2
  for (int j = j_lo; j <= j_hi; ++j) {
    const D ce = row[k];
    const D df = (D)row[n + kp] - def;
    D u[3][kRows], m[kRows];
#pragma unroll
    for (int t = 0; t < 3; ++t)
#pragma unroll
      for (int q = 0; q < kRows; ++q) u[t][q] = (*U)[t][q];
    const D low = best.delta < 0 ? best.delta : (D)-1;
    bool hit = false;
#pragma unroll
    for (int q = 0; q < kRows; ++q) {
      // case 4: ac + be + df, 5: ad + be + cf, 6: ad + ce + bf, 7: ae + bd + cf
      m[q] = u[0][q] + rk[q + 1] + df;
      m[q] = add_min(u[1][q], add_min(ce, rkp[q + 1], rk[q + 1] + cf), m[q]);
      m[q] = add_min(u[2][q], rk[q] + cf, m[q]);
      hit |= m[q] <= low;
    }
    if (hit && j < k) {
#pragma unroll
      for (int q = 0; q < kRows; ++q) {
        if (m[q] > low) continue;
        const unsigned c = m[q] == u[0][q] + rk[q + 1] + df   ? 4u
                           : m[q] == u[1][q] + rk[q + 1] + cf ? 5u
                           : m[q] == u[1][q] + ce + rkp[q + 1] ? 6u
                                                               : 7u;
        best.take(m[q], (((unsigned long long)(i0 + q) * n + j) * n + k) * 8ull + c);
      }
    }
    cf = df;
    row += n;
    ++U;
  }
}

// The pass's smallest (delta, key) over this warp's share of the tour's work (CTA `rank` of C).
template <typename D>
__device__ __forceinline__ MoveKey scan_pass(const int* M, const int* edge, int n, int rank, int C,
                                             D (*U)[3][kRows]) {
  const int lane = threadIdx.x & 31;
  const int warp = (int)(threadIdx.x >> 5) * C + rank, warps = (int)(blockDim.x >> 5) * C;
  Best<D> best;
  // 2-opt moves (x, y): case 3 of (0, 1, y) for x = 0, case 2 of (0, x, y) otherwise
  for (int x = warp; x <= n - 3; x += warps) {
    const int* Ra = M + (long long)x * n;
    const int* Rb = Ra + n;
    const D ex = edge[x];
    for (int y = x + 2 + lane; y < n - (x == 0); y += 32) {
      const D d = (D)Ra[y] + Rb[y + 1 == n ? 0 : y + 1] - ex - edge[y];
      if (d < 0)
        best.take(d, x == 0 ? ((unsigned long long)n + y) * 8ull + 3ull : ((unsigned long long)x * n + y) * 8ull + 2ull);
    }
  }
  // units (32 k, kUnitJ j, four rows) in one round-robin over the warps of the tour; `turn`
  // is the warp of the next unit
  constexpr int JB = kUnitJ<D>;
  int turn = 0;
  for (int k_lo = (n - 1) & ~31; k_lo >= 0; k_lo -= 32) {
    for (int jb = 0; jb <= k_lo + 30 && jb <= n - 2; jb += JB) {
      const int k_hi = k_lo + 31 < n - 1 ? k_lo + 31 : n - 1;
      const int j_end = jb + JB - 1 < k_hi - 1 ? jb + JB - 1 : k_hi - 1;
      if (j_end < 1 || j_end < jb) continue;
      const int rows = j_end < n - 2 ? j_end : n - 2;  // i < j_end, i <= n - 3
      const int nq = (rows + kRows - 1) / kRows;
      const int first = warp >= turn ? warp - turn : warp - turn + warps;
      turn = (turn + nq) % warps;
      for (int q0 = first; q0 < nq; q0 += warps) {
        const int i0 = q0 * kRows, ni = rows - i0 < kRows ? rows - i0 : kRows;
        const int j_lo = jb > i0 + 1 ? jb : i0 + 1, j_hi = j_end;
        const int k = k_lo + lane < n - 1 ? k_lo + lane : n - 1;  // lanes past the end repeat n - 1
        const int kp = k + 1 == n ? 0 : k + 1;
        D rk[kRows + 1], rkp[kRows + 1];
        const D def = edge[k];
#pragma unroll
        for (int q = 0; q <= kRows; ++q) {
          const int i = i0 + q < n ? i0 + q : n - 1;
          rk[q] = M[(long long)i * n + k];
          rkp[q] = (D)M[(long long)i * n + kp] - def;  // d(b, f) - d(e, f)
        }
        __syncwarp();  // the previous unit's reads of U are done
        if (j_lo + lane <= j_hi) {
          const int j = j_lo + lane;
          D ac = M[(long long)i0 * n + j], ad = M[(long long)i0 * n + j + 1];
#pragma unroll
          for (int q = 0; q < kRows; ++q) {
            const int i = i0 + q < n ? i0 + q : n - 1, ib = i0 + q + 1 < n ? i0 + q + 1 : n - 1;
            const D old2 = (D)edge[i] + edge[j];
            const D bc = M[(long long)ib * n + j], bd = M[(long long)ib * n + j + 1];
            const bool ok = q < ni && j > i0 + q;
            U[lane][0][q] = ok ? ac - old2 : kNever<D>;
            U[lane][1][q] = ok ? ad - old2 : kNever<D>;
            U[lane][2][q] = ok ? bd - old2 : kNever<D>;
            ac = bc;
            ad = bd;
          }
        }
        __syncwarp();
        scan_span<D>(M, U, n, i0, k, def, j_lo, j_hi, rk, rkp, best);
      }
    }
  }
  return warp_min_move({(long long)best.delta, best.key});
}

// The 64-bit form, out of line: it is rare and its registers are not the common path's.
__device__ __noinline__ MoveKey scan_pass_wide(const int* M, const int* edge, int n, int rank, int C,
                                               long long (*U)[3][kRows]) {
  return scan_pass<long long>(M, edge, n, rank, C, U);
}

// Reverse positions [lo, hi] of the tour and, when M is kept with it, of M's rows and
// columns. Ends with a barrier.
template <bool SMEM_M>
__device__ __forceinline__ void reverse_segment(int* tour, int* M, int n, int lo, int hi) {
  const int half = (hi - lo + 1) >> 1;
  for (int t = threadIdx.x; t < half; t += blockDim.x) {
    const int x = tour[lo + t], y = tour[hi - t];
    tour[lo + t] = y;
    tour[hi - t] = x;
  }
  if (SMEM_M) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int t = wid; t < half; t += nw) {
      int* Ra = M + (lo + t) * n;
      int* Rb = M + (hi - t) * n;
      for (int c = lane; c < n; c += 32) {
        const int x = Ra[c], y = Rb[c];
        Ra[c] = y;
        Rb[c] = x;
      }
    }
    __syncthreads();
    for (int p = wid; p < n; p += nw) {
      int* R = M + p * n;
      for (int t = lane; t < half; t += 32) {
        const int x = R[lo + t], y = R[hi - t];
        R[lo + t] = y;
        R[hi - t] = x;
      }
    }
  }
  __syncthreads();
}

struct ThreeOptShared {
  MoveKey warp_best[kThreeOptThreads / 32];
  MoveKey cta_best[2];  // by pass parity: a slot is rewritten only after the next pass's barrier
  int stop[2];
  int wide[2];
};

template <bool SMEM_M>
__global__ void __launch_bounds__(kThreeOptThreads) three_opt_kernel(int32_t* __restrict__ tours, int num_tours, int n,
                                                                     DistSrc ds, long long max_iter, int32_t* workspace,
                                                                     int32_t* __restrict__ status,
                                                                     long long* __restrict__ stats, long long budget) {
  extern __shared__ __align__(16) int sm3[];
  __shared__ ThreeOptShared S;
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int slot = blockIdx.x / C, slots = gridDim.x / C;
  unsigned char* terms = reinterpret_cast<unsigned char*>(sm3) + (threadIdx.x >> 5) * kTermBytes;  // this warp's
  int* tour = sm3 + kThreeOptThreads / 32 * kTermBytes / 4;  // n
  int* edge = tour + n;                                      // n
  int* M = SMEM_M ? edge + n : workspace + (long long)slot * n * n;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = (int)(blockDim.x >> 5);
  const long long per_pass = (long long)(n - 2) * (n - 2) * (n + 1);  // (triple, case) candidates of a pass
  for (int r = slot; r < num_tours; r += slots) {
    int32_t* g = tours + (long long)r * n;
    for (int p = tid; p < n; p += blockDim.x) tour[p] = g[p];
    cl.sync();  // every CTA has read the tour before rank 0 may write it back
    long long passes = 0, moves = 0;
    int code = 0;
    bool wide = false;
    const long long start = clock64();
    for (long long it = 0; it < max_iter; ++it) {
      const int par = (int)(it & 1);
      if (tid == 0) {
        S.stop[par] = clock64() - start > budget;  // the watchdog of the 2-opt kernels
        S.wide[par] = 0;
      }
      __syncthreads();
      if (!SMEM_M || it == 0) {
        // tour-ordered matrix, warp per row; in a workspace the tour's CTAs share the rows
        int big = 0;
        for (int p = SMEM_M ? wid : wid * C + rank; p < n; p += SMEM_M ? nw : nw * C) {
          const int a = tour[p];
          int* row = M + (long long)p * n;
          for (int c = lane; c < n; c += 32) {
            const int d = ds(a, tour[c]);
            row[c] = d;
            big |= d;
          }
        }
        if (it == 0) {  // a permuted M holds the same distances
          if (__any_sync(FULL, (unsigned)big >= (1u << 29)) && lane == 0) S.wide[par] = 1;
        }
        __syncthreads();
        if (!SMEM_M) cl.sync();
        if (it == 0) {
          int w = S.wide[par];
          if (!SMEM_M)
            for (int c = 0; c < C; ++c) w |= *cl.map_shared_rank(&S.wide[par], c);
          wide = w != 0;
        }
      }
      for (int p = tid; p < n; p += blockDim.x) edge[p] = M[(long long)p * n + (p + 1 == n ? 0 : p + 1)];
      __syncthreads();
      const MoveKey mine = wide ? scan_pass_wide(M, edge, n, rank, C, reinterpret_cast<long long(*)[3][kRows]>(terms))
                                : scan_pass<int>(M, edge, n, rank, C, reinterpret_cast<int(*)[3][kRows]>(terms));
      if (lane == 0) S.warp_best[wid] = mine;
      __syncthreads();
      if (wid == 0) {
        const MoveKey b = warp_min_move(lane < nw ? S.warp_best[lane] : MoveKey{0, kNoKey});
        if (lane == 0) S.cta_best[par] = b;
      }
      cl.sync();
      MoveKey b = S.cta_best[par];
      int stop = S.stop[par];
      for (int c = 1; c < C; ++c) {
        const int o = rank + c < C ? rank + c : rank + c - C;
        const MoveKey w = *cl.map_shared_rank(&S.cta_best[par], o);
        stop |= *cl.map_shared_rank(&S.stop[par], o);
        if (move_less(w, b)) b = w;
      }
      if (stop) {  // the pass in flight is dropped by all CTAs of the tour alike
        code = TSPB_ERR_BUDGET;
        break;
      }
      ++passes;
      if (b.key == kNoKey) break;  // no improving move: a 3-opt local optimum
      const int kase = (int)(b.key & 7ull);
      const unsigned long long ijk = b.key >> 3;
      const int k = (int)(ijk % (unsigned long long)n);
      const int j = (int)((ijk / (unsigned long long)n) % (unsigned long long)n);
      const int i = (int)(ijk / ((unsigned long long)n * n));
      if (kase == 4 || kase == 5 || kase == 7) reverse_segment<SMEM_M>(tour, M, n, i + 1, j);
      if (kase == 2 || kase == 4 || kase == 5 || kase == 6) reverse_segment<SMEM_M>(tour, M, n, j + 1, k);
      if (kase == 3 || kase == 5 || kase == 6 || kase == 7) reverse_segment<SMEM_M>(tour, M, n, i + 1, k);
      ++moves;
    }
    __syncthreads();
    if (rank == 0) {
      for (int p = tid; p < n; p += blockDim.x) g[p] = tour[p];
      if (tid == 0) {
        if (status) status[r] = code;
        if (stats) {
          stats[(long long)r * 3 + 0] = passes;
          stats[(long long)r * 3 + 1] = moves;
          stats[(long long)r * 3 + 2] = passes * per_pass;
        }
      }
    }
    cl.sync();  // no CTA leaves or starts the next tour while another still reads its minima
  }
}

// Leaves tours of fewer than four cities and calls without passes as they are.
__global__ void three_opt_idle_kernel(int num_tours, int32_t* __restrict__ status, long long* __restrict__ stats) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= num_tours) return;
  if (status) status[r] = 0;
  if (stats)
    for (int q = 0; q < 3; ++q) stats[(long long)r * 3 + q] = 0;
}

static size_t three_opt_smem(int n, bool smem_m) {
  return (size_t)(kThreeOptThreads / 32) * kTermBytes + (size_t)8 * n + (smem_m ? (size_t)4 * n * n : 0);
}

// Cluster launch of `tours` slots; *fits (optional) receives how many clusters of this size
// the device runs at once instead of launching.
template <bool SMEM_M>
static cudaError_t three_opt_launch(int threads, int cluster, int slots, size_t smem, cudaStream_t st, int* fits, int32_t* tours,
                                    int num_tours, int n, DistSrc ds, long long max_iter, int32_t* workspace,
                                    int32_t* status, long long* stats, long long budget) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(slots * cluster));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)cluster;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (fits != nullptr) return cudaOccupancyMaxActiveClusters(fits, three_opt_kernel<SMEM_M>, &cfg);
  return cudaLaunchKernelEx(&cfg, three_opt_kernel<SMEM_M>, tours, num_tours, n, ds, max_iter, workspace, status, stats,
                            budget);
}

}  // namespace tspb

using namespace tspb;

extern "C" int tspb_three_opt_workspace_bytes(int32_t n, int32_t ctas, size_t* bytes) {
  if (n < 0 || ctas < 0 || !bytes) return TSPB_ERR_ARG;
  *bytes = n <= kThreeOptSmemN ? 0 : (size_t)ctas * n * n * sizeof(int32_t);
  return TSPB_OK;
}

extern "C" int tspb_three_opt(int32_t* tours, int32_t num_tours, int32_t n, const int32_t* dist, int64_t dist_stride,
                              const double* coords, int64_t max_iterations, int32_t threads, int32_t* workspace,
                              size_t workspace_bytes, int32_t* status, int64_t* stats, void* stream) {
  if (num_tours < 0 || n < 0 || max_iterations < 0) return TSPB_ERR_ARG;
  if (num_tours == 0 || n == 0) return TSPB_OK;
  if (!tours || (!dist && !coords) || (dist && dist_stride < n)) return TSPB_ERR_ARG;
  if (threads != 128 && threads != 256 && threads != 512) return TSPB_ERR_ARG;
  // one exhaustive pass is n^3 / 6 triples; the watchdog runs between passes, so n is
  // capped where a pass of one CTA stays around a second
  if (n > kThreeOptMaxN) return TSPB_ERR_UNSUPPORTED;
  DistSrc ds;
  ds.dist = dist;
  ds.stride = dist_stride;
  ds.coords = reinterpret_cast<const double2*>(coords);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const bool smem_m = n <= kThreeOptSmemN;
  const size_t smem = three_opt_smem(n, smem_m);
  if (smem > (size_t)smem_optin() - 2048) return TSPB_ERR_UNSUPPORTED;
  long long* s = reinterpret_cast<long long*>(stats);
  int slots = num_tours;
  if (!smem_m) {
    const size_t per = (size_t)n * n * sizeof(int32_t);
    if (!workspace || workspace_bytes < per) return TSPB_ERR_WORKSPACE;
    const size_t fit = workspace_bytes / per;
    if ((size_t)slots > fit) slots = (int)fit;
  }
  if (n < 4 || max_iterations == 0) {
    three_opt_idle_kernel<<<(num_tours + 255) / 256, 256, 0, st>>>(num_tours, status, s);
    return tspb_launch_status();
  }
  // Many short tours: a pass has fewer units than 16 warps, so narrow CTAs and more of them on an
  // SM. Ten passes of 5000 tours of 10 cities 0.33 ms (0.82 with 512 threads), 1000 of 50 0.85
  // (1.21), 500 of 80 1.05 (1.34), 300 of 120 1.81 (1.88).
  const bool narrow = n <= 100 && slots > device_attr(cudaDevAttrMultiProcessorCount);
  const int cta = narrow ? 128 : kThreeOptThreads;
  auto go = [&](int cluster, int* fits) {
    return smem_m ? three_opt_launch<true>(cta, cluster, slots, smem, st, fits, tours, num_tours, n, ds, max_iterations,
                                           nullptr, status, s, watchdog_cycles())
                  : three_opt_launch<false>(cta, cluster, slots, smem, st, fits, tours, num_tours, n, ds, max_iterations,
                                            workspace, status, s, watchdog_cycles());
  };
  TSPB_CUDA_CHECK(smem_m ? allow_smem(three_opt_kernel<true>, smem) : allow_smem(three_opt_kernel<false>, smem));
  // the largest cluster for which every tour runs in one wave; tours with fewer units than
  // warps gain nothing from more CTAs
  int cluster = 1;
  const int units = ((n + 1) / kRows) * ((n + 31) / 32) / 2;
  for (int c = narrow ? 1 : 8; c > 1; c >>= 1) {
    if (units < c * (kThreeOptThreads / 32) / 2) continue;
    int fits = 0;
    if (go(c, &fits) == cudaSuccess && fits >= slots) {
      cluster = c;
      break;
    }
    (void)cudaGetLastError();
  }
  TSPB_CUDA_CHECK(go(cluster, nullptr));
  return tspb_launch_status();
}
