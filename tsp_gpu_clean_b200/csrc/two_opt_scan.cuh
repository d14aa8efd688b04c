// Per-tour body of the candidate-mode 2-opt rescan (best / first), shared by the
// one-CTA-per-tour kernel and the persistent multi-instance batch kernel.
//
// Same semantics as the reference scan (src/algorithms/strategies/local_search/two_opt.py:
// pair order :347-367, gains :237-245, best :386-440, first :442-489, passes :565-595),
// arranged so that one pass keeps as many independent loads in flight as possible:
//
// - the tour is held position- and node-indexed: tour[p] (16 bits), ps[a] =
//   pos[a] << 16 | succ[a] and eout[a] = d(a, succ[a]); the gain of entry (i, r) with a = tour[i],
//   c = N_k[a][r] is (d(a,c) - eout[a]) + (d(succ[a], succ[c]) - eout[c]);
// - the k-NN table and d(a, c) come packed as one u32 per entry (c | d(a,c) << 16) when
//   both fit 16 bits, so the whole per-instance table (80 KB at n=1000, k=20) stays in L1;
// - each thread evaluates U entries per round with their loads issued back to back
//   (k-NN word -> shared-memory lookups -> one L2 gather of d(succ[a], succ[c]), or an
//   FP64 rebuild from coordinates when the instance has no matrix).
//
// What bounds a full chip of tours is the shared-memory pipe: every entry looks up a random
// city. Position and successor in one word, and eout read for valid entries only (the others
// read their own row's), take about six bank passes per 32 entries where three separate
// arrays took ten (ncu: L1 pipe 90 % busy). 10 n bytes a tour instead of 16 n also leave more
// of the L1 to the k-NN table.
//
// best keeps a per-thread (gain, i*k + r) minimum and reduces once per pass. first
// publishes improving indices with a shared atomicMin; each thread stops scanning as soon
// as the published minimum lies below all of its remaining entries (no barrier per round),
// and one barrier at the end of the scan makes the minimum the pass's first improving entry.
//
// best with row keys (INC, grouped layout, reverse k-NN index): every row keeps the minimum
// key of its improving entries, and after a move with window [bi, bj] a pass evaluates only
// what the move can have changed:
//   - the rows of the window (and row 0 when bj is the last position, whose city it excludes);
//   - the entries of earlier rows whose candidate lies in the window, found through the
//     reverse index. Such an entry lowers its row's key where it beats it; where it was the
//     row's minimum itself the row is evaluated anew.
// Rows after bj see the window's cities at invalid positions before and after. Then the row
// keys are reduced. On the clustered 1000-city batch this is about a quarter of the entries of
// a full rescan (mean window 156 positions, median 37); windows longer than about half the
// rows take the full evaluation. A row key is one word, gain << 5 | rank: it needs k <= 32 and
// no edge of the tour above 2^25 (a gain is at least minus two edges); a tour that meets a
// longer edge is rescanned in full from then on.
//
// first with the reverse k-NN index (incremental restart): the reference restarts every
// pass at entry 0. After a move with window [bi, bj] (the first improving entry was in row
// bi, so every entry before it was non-improving), an entry (i, r) of a row i < bi keeps
// a = t[i], succ[a] and eout[a]; it changes only when its candidate c lies in positions
// [bi, bj], where pos/succ/eout of c may have changed. The next pass therefore evaluates
// just those affected entries (found through the reverse index) and, when none improves,
// scans from row bi on: the first improving entry it finds is the reference's.
//
// best over a CTA pair (CL = 2, a thread-block cluster of two CTAs; grouped layout): both
// CTAs hold the whole tour state and apply every move; CTA r scans the rounds r, r + 2, ...
// of each pass, and the two per-CTA minima meet through distributed shared memory (one
// cluster barrier per pass), so both take the same move. The watchdog flags of both CTAs
// travel with the minima, so both stop together.
#pragma once

#include <cooperative_groups.h>

// First mode's incremental restart checks the entries that point into the last move's
// window (about 30 warp instructions per window position) instead of rescanning the rows
// before it (about 9 per row); it is taken when RATIO x window length <= the move's row.
#ifndef TSPB_RESTART_RATIO
#define TSPB_RESTART_RATIO 3
#endif

// Best mode's row keys start once the mean window times this is no longer than the rows: long
// windows leave little to keep. 1024 tours of 1000 cities, k = 20: 2 -> 35.4 ms, 4 -> 33.9,
// 5 -> 29.5, 6 -> 29.4, 8 -> 30.6, 10 -> 31.0 (45.1 without keys).
#ifndef TSPB_KEYS_RATIO
#define TSPB_KEYS_RATIO 6
#endif

#include "two_opt.cuh"

namespace tspb {

constexpr int kKeyEdge = 1 << 25;  // row keys: edges up to this keep a gain in 27 bits

struct ScanSmem {
  unsigned long long red64[32];
  long long redll[32];
  long long total;  // first (and incremental best): valid entries of the current tour, kept exact
  unsigned first;
  int bound[2];     // best, by pass parity: a gain that some entry is known to have (or 0)
  int nlist[2];     // best with row keys, by pass parity: earlier rows to evaluate anew
  int long_edge;    // best with row keys: the tour has an edge above kKeyEdge
  int bad;
  int stop;
  unsigned long long xkey[2];  // CTA pair: this CTA's pass minimum (by pass parity)
  int xstop[2];                // CTA pair: this CTA's watchdog flag of that pass
  long long xcnt[2];           // CTA pair: this CTA's pair and gain counts at exit
};

template <int THREADS>
struct ScanMinBlocks {
  static constexpr int value = THREADS == 64 ? 16 : THREADS == 128 ? 8 : THREADS == 256 ? 4 : THREADS == 512 ? 2 : 1;
};

// Bytes of tour state per tour: ps, eout, tour (+ per-row valid counts for first when it
// counts pairs; best with incremental row keys adds the keys, valid counts and a row list).
__host__ __device__ inline size_t scan_tour_state_bytes(int n, int mode, bool incremental = false, bool count = true) {
  const size_t m = ((size_t)n + 2) & ~(size_t)1;
  if (mode == TSPB_MODE_FIRST) return (size_t)(count ? 14 : 10) * m;
  return (size_t)(incremental ? (count ? 20 : 16) : 10) * m;
}

// The bytes the callers' limits and workspaces are stated in (n of a batch, workspace sizes):
// those of the wider layout this one replaced, so that no call changes sides.
__host__ __device__ inline size_t scan_tour_limit_bytes(int n, int mode, bool incremental = false) {
  return (size_t)(mode == TSPB_MODE_FIRST ? 20 : (incremental ? 30 : 16)) * (size_t)n;
}

struct ScanTour {
  int32_t* g_tour;        // the tour in global memory: read at entry, written back at exit
  unsigned char* arrays;  // scan_tour_state_bytes(n, mode) bytes (shared memory or workspace)
  int n, k;
  DistSrc ds;
  const uint32_t* packed;  // c | d(a, c) << 16 per entry, or nullptr
  const int32_t* cand;
  const int32_t* cand_dist;
  long long max_iter;
  int32_t* status;   // optional: TSPB status of this tour
  long long* stats;  // optional: passes, pairs, moves, evaluated gains
  int accumulate;    // 1: stats are added to the slot and only an error is stored in status
                     // (sticky across launches); 0: both are overwritten
  int32_t* moved;    // optional: 1 when at least one move was applied, else 0
  uint8_t* converged;  // optional: 1 when the refinement ended on a pass without an improving
                       // move (the tour is then a fixed point of any further refinement)
  const int32_t* rev_off = nullptr;  // optional (first mode): CSR reverse k-NN index, n + 1 offsets
  const int32_t* rev_idx = nullptr;  // flat entries a * k + r grouped by candidate node
  double* cost = nullptr;  // optional: the refined tour's length (exact int64 sum of eout, as float64)
  long long budget = BUDGET_CYCLES;  // watchdog: SM cycles before the tour ends with TSPB_ERR_BUDGET
  int symmetric = 0;  // 1: d(a, b) == d(b, a); a move's out-edges come from the old ones (below)
};

// k-NN table layouts of scan_tour: plain int32 candidates (+ optional distances), packed
// words with round-robin entries, and packed words with each thread's U entries taken
// contiguously from one row (needs k % U == 0): the row's a, succ[a], eout[a] are read
// once per U entries and the U words arrive in one vector load.
enum ScanLayout { SCAN_PLAIN = 0, SCAN_PACKED = 1, SCAN_GROUPED = 2 };

template <int U>
__device__ __forceinline__ void load_words(const uint32_t* p, uint32_t (&w)[U]) {
  if constexpr (U == 4) {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
    w[0] = v.x;
    w[1] = v.y;
    w[2] = v.z;
    w[3] = v.w;
  } else if constexpr (U == 2) {
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
    w[0] = v.x;
    w[1] = v.y;
  } else {
#pragma unroll
    for (int u = 0; u < U; ++u) w[u] = __ldg(p + u);
  }
}

// Refines one tour with the whole CTA. Every thread of the CTA must call it.
//
// COUNT: first mode (and incremental best) keeps every row's valid-pair count so that
// stats[1] holds the reference's pair count. No decision of the scan reads these counts,
// and refreshing them after a move visits every candidate of every row in the reversed
// window, so a caller that passes no stats runs the COUNT = false instance (or, with
// COUNT = true, skips the refresh at run time): same moves, same tours.
//
// SYM: the symmetric-distance refresh after a move is compiled in (used when T.symmetric
// is set). The batch engine compiles it out: its large CTAs cover most windows in one round
// of distance reads, and the extra code measured slower there.
template <int MODE, int THREADS, int U, int LAYOUT, bool INC = false, bool COUNT = true, int CL = 1, bool SYM = true>
__device__ __forceinline__ void scan_tour(const ScanTour T, ScanSmem& S) {
  constexpr bool PACKED = LAYOUT != SCAN_PLAIN;
  constexpr bool GROUPED = LAYOUT == SCAN_GROUPED;
  static_assert(CL == 1 || (CL == 2 && MODE == TSPB_MODE_BEST && GROUPED && !INC),
                "a CTA pair runs best mode on the grouped layout only");
  const unsigned rank = CL > 1 ? cooperative_groups::this_cluster().block_rank() : 0u;
  const int n = T.n, k = T.k, rows = n - 2;
  const int tid = threadIdx.x;
  int32_t* g_tour = T.g_tour;
  const int m = (n + 2) & ~1;  // array sizes: a slot past the last, every array starts on 8 bytes
  unsigned* ps = reinterpret_cast<unsigned*>(T.arrays);  // pos << 16 | succ, by city; slot n: position 0
  int* eout = reinterpret_cast<int*>(ps + m);
  // INC: per-row minimum keys, a list of rows, and valid entries per row (position) follow
  constexpr bool inc_best = MODE == TSPB_MODE_BEST && GROUPED && INC;
  constexpr bool track_rows_ct = COUNT && (MODE == TSPB_MODE_FIRST || inc_best);
  int* rkey = eout + m;
  int* rcnt = inc_best ? rkey + m : eout + m;
  uint16_t* tour = reinterpret_cast<uint16_t*>(track_rows_ct ? rcnt + m : rcnt);
  uint16_t* rlist = tour + m;
  const bool track_rows = track_rows_ct && T.stats != nullptr;
  const DistSrc ds = T.ds;
  const uint32_t* __restrict__ packed = T.packed;
  const int32_t* __restrict__ cand = T.cand;
  const int32_t* __restrict__ cdist = T.cand_dist;
  const int32_t* __restrict__ dist = T.ds.dist;
  const unsigned stride = (unsigned)T.ds.stride;

  if (tid == 0) {
    S.bad = 0;
    S.stop = 0;
    S.total = 0;
    S.bound[0] = S.bound[1] = 0;
    S.long_edge = 0;
  }
  for (int a = tid; a <= n; a += THREADS) ps[a] = a < n ? NO_IDX : 0u;  // an id past the last city is never valid
  __syncthreads();
  for (int p = tid; p < n; p += THREADS) {
    const int v = g_tour[p];
    tour[p] = (uint16_t)v;
    if ((unsigned)v >= (unsigned)n || atomicExch(&ps[v], (unsigned)p) != NO_IDX) S.bad = 1;
  }
  __syncthreads();
  if (S.bad) {
    if (tid == 0) {
      if (T.moved) *T.moved = 0;
      if (T.converged) *T.converged = 0;
      if (T.status) *T.status = TSPB_ERR_NOT_PERMUTATION;
      if (T.stats && !T.accumulate)
        for (int q = 0; q < 4; ++q) T.stats[q] = 0;
    }
    __syncthreads();  // every thread has read S.bad before the caller reuses S
    return;
  }
  auto set_edge = [&](int x, int e) {
    eout[x] = e;
    if (inc_best && e > kKeyEdge) S.long_edge = 1;
  };
  for (int p = tid; p < n; p += THREADS) {
    const int x = tour[p], y = tour[p + 1 == n ? 0 : p + 1];
    ps[x] = ((unsigned)p << 16) | (unsigned)y;
    set_edge(x, ds(x, y));
  }
  __syncthreads();
  auto pos_of = [&](int a) -> int { return (int)(ps[a] >> 16); };
  auto succ_of = [&](int a) -> int { return (int)(ps[a] & 0xffffu); };

  // Valid entries of row i (the pairs the reference scan evaluates for that row).
  auto row_count = [&](int i) -> int {
    const int a = tour[i];
    const int lo = i + 2, span = n - (i == 0) - lo;
    int c = 0;
    for (int r0 = 0; r0 < k; r0 += 4) {
      int cc[4];
      if constexpr (GROUPED && U % 4 == 0) {  // k % 4 == 0 and a 16-byte aligned table
        uint32_t w[4];
        load_words<4>(packed + ((unsigned)a * (unsigned)k + (unsigned)r0), w);
#pragma unroll
        for (int u = 0; u < 4; ++u) cc[u] = (int)(w[u] & 0xffffu);
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const unsigned ar = (unsigned)a * (unsigned)k + (unsigned)(r0 + u);
          cc[u] = r0 + u < k ? (PACKED ? (int)(__ldg(packed + ar) & 0xffffu) : __ldg(cand + ar)) : -1;
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if ((unsigned)cc[u] < (unsigned)n) c += (unsigned)(pos_of(cc[u]) - lo) < (unsigned)span;
    }
    return c;
  };
  if (MODE == TSPB_MODE_FIRST && track_rows) {
    long long sum = 0;
    for (int i = tid; i < n; i += THREADS) {
      const int v = i < rows ? row_count(i) : 0;
      rcnt[i] = v;
      sum += v;
    }
    sum = warp_sum(sum);
    if ((tid & 31) == 0) atomicAdd(reinterpret_cast<unsigned long long*>(&S.total), (unsigned long long)sum);
    __syncthreads();
  }

  const int E = rows * k;
  constexpr int STEP = THREADS * U;
  const int sq = STEP / k, sr = STEP - (STEP / k) * k;
  const int g_row0 = (tid * U) / k, g_col0 = tid * U - g_row0 * k;  // grouped layout: first entry
  long long passes = 0, moves = 0, my_pairs = 0, my_eval = 0;
  int err = TSPB_OK;
  bool converged = false;  // the last pass found no improving move: a local optimum
  const long long t_start = clock64();
  const bool incremental = MODE == TSPB_MODE_FIRST && T.rev_off != nullptr && T.rev_idx != nullptr;
  // e / k of an entry e = a * k + r, as a multiply-high by ceil(2^32 / k): exact for every
  // e < n k when n k k < 2^32 and the reciprocal itself fits 32 bits, which k = 1 does not
  // (else a plain division)
  const unsigned kmag = (unsigned)(((1ull << 32) + (unsigned)k - 1) / (unsigned)k);
  const bool kmag_exact = k > 1 && (unsigned long long)n * (unsigned)k * (unsigned)k < (1ull << 32);
  auto entry_node = [&](int e) -> int {
    return kmag_exact ? (int)__umulhi((unsigned)e, kmag) : e / k;
  };
  int win_lo = -1, win_hi = -1;  // window [bi, bj] of the last move
  bool can_key = false;          // row keys are usable on this tour
  bool row_keys = false;         // and hold (set by the first pass that evaluates every row)
  int reach = 16 * n;            // 16 x a running mean of the window lengths
  if constexpr (inc_best) {
    can_key = T.rev_off != nullptr && T.rev_idx != nullptr && k <= 32;
    if (tid == 0) S.nlist[0] = S.nlist[1] = 0;
  }

  while (passes < T.max_iter) {
    if (tid == 0) {
      if (clock64() - t_start > T.budget) S.stop = TSPB_ERR_BUDGET;
      S.first = NO_IDX;
      S.bound[(int)(passes + 1) & 1] = 0;
      if (inc_best) S.nlist[(int)(passes + 1) & 1] = 0;  // the next pass's (its last readers have passed a barrier)
    }
    __syncthreads();
    if (CL == 1 && S.stop) {  // a CTA pair stops only after exchanging its flags (below)
      err = S.stop;
      break;
    }
    ++passes;
    if (MODE == TSPB_MODE_FIRST && track_rows && tid == 0) my_pairs += S.total;
    // best: smallest gain of this thread, its scan index (first in thread order wins ties)
    // and its second position. A known gain of this pass bounds the pass's best from above,
    // so an entry counts only at or below it.
    int bgain = MODE == TSPB_MODE_BEST ? S.bound[(int)(passes - 1) & 1] : 0;
    if (MODE == TSPB_MODE_BEST && bgain < 0) ++bgain;
    unsigned bidx = NO_IDX;
    int bpos = 0;
    int cnt = 0, evals = 0;
    int start_row = 0;        // first row of this pass's scan
    bool found = false;       // the affected entries already hold the first improving one
    if (incremental && win_lo >= 0 && TSPB_RESTART_RATIO * (win_hi - win_lo + 1) <= win_lo) {
      // affected entries of rows < win_lo: candidate c at a position of the window
      const int lane = tid & 31, wid = tid >> 5;
      constexpr int NW = THREADS / 32;
      for (int q = win_lo + wid; q <= win_hi; q += NW) {
        const int c = tour[q];
        const int s0 = __ldg(T.rev_off + c), s1 = __ldg(T.rev_off + c + 1);
        const int sc = succ_of(c), ec = eout[c];
        for (int sx = s0 + lane; sx < s1; sx += 32) {
          const int e = __ldg(T.rev_idx + sx);
          const int a = entry_node(e);
          const int i = pos_of(a);
          if (i >= win_lo) continue;  // rows from win_lo on are scanned below
          if ((unsigned)(q - (i + 2)) >= (unsigned)(n - (i == 0) - (i + 2))) continue;
          const int dac = PACKED ? (int)(__ldg(packed + e) >> 16) : (cdist ? __ldg(cdist + e) : ds(a, c));
          const int lbe = (dac - eout[a]) - ec;
          if (lbe >= 0) continue;  // cannot improve whatever d(succ a, succ c) is
          ++evals;
          const int sa = succ_of(a);
          const int dbd = dist ? __ldcg(dist + ((unsigned)sa * stride + (unsigned)sc)) : ds(sa, sc);
          if (lbe + dbd < 0) atomicMin(&S.first, (unsigned)(i * k + (e - a * k)));
        }
      }
      __syncthreads();
      found = S.first != NO_IDX;
      start_row = win_lo;
    }
    if constexpr (inc_best) {
      if (S.long_edge) can_key = row_keys = false;
      const bool start = can_key && !row_keys && TSPB_KEYS_RATIO * reach <= 16 * rows;
      if (start || row_keys) {
        row_keys = true;
        const int lane = tid & 31, wid = tid >> 5;
        constexpr int NW = THREADS / 32;
        const int par = (int)(passes - 1) & 1;
        int delta = 0;  // valid entries gained by the rows this thread evaluates
        // lowers row gi's key by the U entries from column gr on; counts its valid entries
        auto group = [&](int gi, int gr, bool count) {
          const int a = tour[gi];
          uint32_t w[U];
          load_words<U>(packed + ((unsigned)a * (unsigned)k + (unsigned)gr), w);
          const int sa = succ_of(a), ea = eout[a];
          const int lo = gi + 2;
          const unsigned lo16 = (unsigned)lo << 16, span16 = (unsigned)(n - (gi == 0) - lo) << 16;
          bool ok[U];
          int sc[U], lb[U], dbd[U];
          int valid = 0;
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int c = min((int)(w[u] & 0xffffu), n);
            const unsigned pc = ps[c];
            ok[u] = pc - lo16 < span16;
            valid += ok[u];
            sc[u] = (int)(pc & 0xffffu);
            lb[u] = ((int)(w[u] >> 16) - ea) - eout[ok[u] ? c : a];
            ok[u] &= lb[u] < 0;  // only improving entries hold keys
          }
          gather_if(ds, sa, sc, ok, dbd);
          if (track_rows && count && valid) {
            delta += valid;
            atomicAdd(&rcnt[gi], valid);
          }
          int key = 0;
#pragma unroll
          for (int u = 0; u < U; ++u) {
            evals += ok[u];
            const int gain = lb[u] + dbd[u];
            if (ok[u] && gain < 0) key = min(key, gain * 32 + gr + u);
          }
          if (key < 0) atomicMin(&rkey[gi], key);
        };
        const int G = k / U;
        if (start) {  // every row (the windows that follow clear theirs with the move)
          for (int i = tid; i < rows; i += THREADS) {
            rkey[i] = 0;
            if (track_rows) rcnt[i] = 0;
          }
          __syncthreads();
        }
        const bool all = start || 2 * (win_hi - win_lo + 1) > rows;
        const int r_lo = all ? 0 : win_lo, r_hi = all ? rows - 1 : (win_hi < rows - 1 ? win_hi : rows - 1);
        if (!all) {
          // entries of earlier rows that point into the window: a warp per window position,
          // several positions in flight
          constexpr int V = 4;
          for (int q0 = win_lo + wid * V; q0 <= win_hi; q0 += NW * V) {
            int c[V], at[V], end[V];
#pragma unroll
            for (int v = 0; v < V; ++v) {
              const bool in = q0 + v <= win_hi;
              c[v] = tour[in ? q0 + v : win_hi];
              at[v] = __ldg(T.rev_off + c[v]) + lane;
              end[v] = in ? __ldg(T.rev_off + c[v] + 1) : 0;
            }
            while (true) {
              bool ok[V], any = false;
              int e[V];
#pragma unroll
              for (int v = 0; v < V; ++v) {
                ok[v] = at[v] < end[v];
                any |= ok[v];
                e[v] = (int)load_nc_if(ok[v], T.rev_idx + at[v]);
              }
              if (!__any_sync(FULL, any)) break;
              int i[V], a[V], dac[V], sa[V], sc[V], lb[V], dbd[V], r[V];
#pragma unroll
              for (int v = 0; v < V; ++v) {
                a[v] = entry_node(e[v]);
                r[v] = e[v] - a[v] * k;
                const unsigned pa = ps[a[v]];
                i[v] = (int)(pa >> 16);
                sa[v] = (int)(pa & 0xffffu);
                // an earlier row (row 0 is evaluated anew below when the last position changed),
                // candidate at a valid position
                ok[v] = ok[v] && i[v] < win_lo && q0 + v > i[v] + 1 && !(i[v] == 0 && win_hi == n - 1);
                dac[v] = (int)(load_nc_if(ok[v], packed + e[v]) >> 16);
              }
#pragma unroll
              for (int v = 0; v < V; ++v) {
                sc[v] = succ_of(c[v]);
                lb[v] = (dac[v] - eout[a[v]]) - eout[c[v]];
                if (ok[v]) {
                  const int held = *reinterpret_cast<volatile int*>(&rkey[i[v]]);
                  if (held < 0 && (held & 31) == r[v]) {  // the row's minimum changed: evaluate it anew
                    rkey[i[v]] = 0;
                    rlist[atomicAdd(&S.nlist[par], 1)] = (uint16_t)i[v];
                    ok[v] = false;
                  } else {
                    ok[v] = lb[v] < 0 && lb[v] * 32 + r[v] < held;
                  }
                }
              }
              if (dist != nullptr) {
#pragma unroll
                for (int v = 0; v < V; ++v)
                  dbd[v] = load_cg_if(ok[v], dist + ((unsigned)sa[v] * stride + (unsigned)sc[v]));
              } else {
#pragma unroll
                for (int v = 0; v < V; ++v) dbd[v] = ok[v] ? ds(sa[v], sc[v]) : 0;
              }
#pragma unroll
              for (int v = 0; v < V; ++v) {
                evals += ok[v];
                const int gain = lb[v] + dbd[v];
                if (ok[v] && gain < 0) atomicMin(&rkey[i[v]], gain * 32 + r[v]);
                at[v] += 32;
              }
            }
          }
          // row 0, whose excluded last city changed
          if (win_hi == n - 1 && win_lo > 0)
            for (int g = tid; g < G; g += THREADS) group(0, g * U, true);
        }
        // the rows of the window, or all
        {
          const int items = (r_hi - r_lo + 1) * G;
          int gi = r_lo + tid / G, g = tid - (tid / G) * G;
          const int di = THREADS / G, dg = THREADS - di * G;
          for (int it = tid; it < items; it += THREADS) {
            group(gi, g * U, true);
            gi += di;
            g += dg;
            if (g >= G) {
              g -= G;
              ++gi;
            }
          }
        }
        if (track_rows) {
          delta = __reduce_add_sync(FULL, delta);
          if (lane == 0 && delta != 0) atomicAdd(reinterpret_cast<unsigned long long*>(&S.total), (unsigned long long)delta);
        }
        __syncthreads();
        if (track_rows && tid == 0) my_pairs += S.total;
        const int listed = S.nlist[par];
        if (listed > 0) {  // earlier rows whose minimum changed; their valid entries did not
          for (int it = tid; it < listed * G; it += THREADS) {
            const int q = it / G;
            group(rlist[q], (it - q * G) * U, false);
          }
          __syncthreads();
        }
        // the smallest (gain, row), then the row's rank
        for (int i = tid; i < rows; i += THREADS) {
          const int gain = rkey[i] >> 5;  // arithmetic: the gain
          if (gain < bgain) {
            bgain = gain;
            bidx = (unsigned)i;
          }
        }
        if (bidx != NO_IDX) bidx = bidx * (unsigned)k + (unsigned)(rkey[bidx] & 31);
        found = true;  // skip the per-pass scan below
      }
    }
    if (found) {
      // nothing to scan: first mode's smallest improving affected entry is the first of the
      // pass; best with row keys holds this thread's share of them
    } else if constexpr (GROUPED) {
      // entries [e0 + tid*U, e0 + tid*U + U) of round e0 lie in row gi, columns gr..gr+U-1;
      // a CTA pair takes alternate rounds
      int gi = g_row0 + start_row, gr = g_col0;
      int e_first = start_row * k;
      if constexpr (CL > 1) {
        e_first += (int)rank * STEP;
        const int eb0 = e_first + tid * U;
        gi = eb0 / k;
        gr = eb0 - gi * k;
      }
      for (int e0 = e_first; e0 < E; e0 += CL * STEP) {
        const int eb = e0 + tid * U;
        if (eb < E) {
          const int a = tour[gi];
          uint32_t w[U];
          load_words<U>(packed + ((unsigned)a * (unsigned)k + (unsigned)gr), w);
          const int sa = succ_of(a), ea = eout[a];
          const int lo = gi + 2;
          // pos[c] in [lo, lo + span), compared in the high halves (a low half changes nothing)
          const unsigned lo16 = (unsigned)lo << 16, span16 = (unsigned)(n - (gi == 0) - lo) << 16;
          bool ok[U];
          unsigned pc[U];
          int sc[U], lb[U];
          const int bound = MODE == TSPB_MODE_BEST ? bgain : 0;
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int c = min((int)(w[u] & 0xffffu), n);
            pc[u] = ps[c];
            ok[u] = pc[u] - lo16 < span16;
            if (MODE == TSPB_MODE_BEST) cnt += ok[u];
            sc[u] = (int)(pc[u] & 0xffffu);
            // gain >= lb (the gathered distance is >= 0): an entry whose lb cannot beat
            // this thread's bound is settled without its L2 gather
            lb[u] = ((int)(w[u] >> 16) - ea) - eout[ok[u] ? c : a];
            ok[u] &= lb[u] < bound;
          }
          int dbd[U];
          gather_if(ds, sa, sc, ok, dbd);
#pragma unroll
          for (int u = 0; u < U; ++u) {
            evals += ok[u];
            const int gain = lb[u] + dbd[u];
            if (MODE == TSPB_MODE_BEST) {
              if (ok[u] && gain < bgain) {
                bgain = gain;
                bidx = (unsigned)(eb + u);
                bpos = (int)(pc[u] >> 16);
              }
            } else if (ok[u] && gain < 0) {
              atomicMin(&S.first, (unsigned)(eb + u));
            }
          }
        }
        if constexpr (CL > 1) {
          gr += (CL * STEP) % k;
          gi += (CL * STEP) / k;
        } else {
          gr += sr;
          gi += sq;
        }
        if (gr >= k) {
          gr -= k;
          ++gi;
        }
        // first: no barrier per round; a thread stops once an improving index below all of
        // its remaining entries (>= e0 + STEP) is known. S.first only decreases, so every
        // entry below the pass's final minimum is still evaluated by its thread.
        if (MODE == TSPB_MODE_FIRST && *reinterpret_cast<volatile unsigned*>(&S.first) < (unsigned)(e0 + STEP)) break;
      }
    } else {
    int ri[U], rr[U], ee[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      ee[u] = start_row * k + u * THREADS + tid;
      ri[u] = ee[u] / k;
      rr[u] = ee[u] - ri[u] * k;
    }
    for (int e0 = start_row * k; e0 < E; e0 += STEP) {
      int a[U], c[U], cd[U];
#pragma unroll
      for (int u = 0; u < U; ++u) a[u] = ee[u] < E ? tour[ri[u]] : -1;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        c[u] = -1;
        if (a[u] < 0) continue;
        const unsigned ar = (unsigned)a[u] * (unsigned)k + (unsigned)rr[u];
        if (PACKED) {
          const uint32_t w = __ldg(packed + ar);
          c[u] = (int)(w & 0xffffu);
          cd[u] = (int)(w >> 16);
        } else {
          c[u] = __ldg(cand + ar);
          cd[u] = cdist ? __ldg(cdist + ar) : -1;
        }
      }
      bool ok[U];
      int sa[U], sc[U], lb[U], pj[U];
      const int bound = MODE == TSPB_MODE_BEST ? bgain : 0;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        ok[u] = false;
        if ((unsigned)c[u] >= (unsigned)n) continue;
        const int i = ri[u];
        const unsigned pc = ps[c[u]];
        pj[u] = (int)(pc >> 16);
        // j in (i + 1, lim): one unsigned range test
        ok[u] = (unsigned)(pj[u] - (i + 2)) < (unsigned)(n - (i == 0) - (i + 2));
        if (MODE == TSPB_MODE_BEST) cnt += ok[u];
        if (ok[u]) {
          sa[u] = succ_of(a[u]);
          sc[u] = (int)(pc & 0xffffu);
          const int dac = (PACKED || cd[u] >= 0) ? cd[u] : ds(a[u], c[u]);
          lb[u] = (dac - eout[a[u]]) - eout[c[u]];  // gain >= lb: skip the gather when lb cannot win
          ok[u] = lb[u] < bound;
        }
      }
      int dbd[U];
      if (dist != nullptr) {
#pragma unroll
        for (int u = 0; u < U; ++u) dbd[u] = load_cg_if(ok[u], dist + (ok[u] ? (unsigned)sa[u] * stride + (unsigned)sc[u] : 0u));
      } else {
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (ok[u]) dbd[u] = ds(sa[u], sc[u]);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!ok[u]) continue;
        ++evals;
        const int gain = lb[u] + dbd[u];
        if (MODE == TSPB_MODE_BEST) {
          if (gain < bgain) {
            bgain = gain;
            bidx = (unsigned)ee[u];
            bpos = pj[u];
          }
        } else if (gain < 0) {
          atomicMin(&S.first, (unsigned)ee[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        ee[u] += STEP;
        rr[u] += sr;
        ri[u] += sq;
        if (rr[u] >= k) {
          rr[u] -= k;
          ++ri[u];
        }
      }
      if (MODE == TSPB_MODE_FIRST && *reinterpret_cast<volatile unsigned*>(&S.first) < (unsigned)(e0 + STEP)) break;
    }
    }
    my_pairs += cnt;
    my_eval += evals;
    unsigned idx;
    if (MODE == TSPB_MODE_BEST) {
      const unsigned long long key = bidx == NO_IDX ? NO_KEY : gain_key(bgain, bidx);
      unsigned long long best = block_min(key, S.red64);
      if constexpr (CL > 1) {
        // the two CTAs' minima and watchdog flags meet through distributed shared memory;
        // slots alternate by pass, so one cluster barrier per pass suffices
        cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
        const int slot = (int)(passes & 1);
        if (tid == 0) {
          S.xkey[slot] = best;
          S.xstop[slot] = S.stop;
        }
        cl.sync();
        const unsigned long long peer = *cl.map_shared_rank(&S.xkey[slot], rank ^ 1u);
        const int peer_stop = *cl.map_shared_rank(&S.xstop[slot], rank ^ 1u);
        best = peer < best ? peer : best;
        if (S.stop || peer_stop) {
          err = TSPB_ERR_BUDGET;
          break;
        }
      }
      if (best == NO_KEY) {
        converged = true;
        break;
      }
      idx = (unsigned)best;
    } else {
      __syncthreads();
      idx = S.first;
      if (idx == NO_IDX) {
        converged = true;
        break;
      }
    }
    const int bi = (int)(idx / (unsigned)k);
    const int br = (int)(idx - (unsigned)bi * (unsigned)k);
    const unsigned bar = (unsigned)tour[bi] * (unsigned)k + (unsigned)br;
    const int ca = PACKED ? (int)(__ldg(packed + bar) & 0xffffu) : __ldg(cand + bar);
    const int bj = pos_of(ca);
    if (bi < 0 || bj <= bi + 1 || bj >= n) {
      err = TSPB_ERR_RANGE;
      break;
    }
    if (MODE == TSPB_MODE_BEST && !row_keys) {
      // This thread's best entry keeps its gain when neither of its positions lies in the
      // window and it is not the move itself: the next pass's best is no larger.
      int known = 0;
      if (bidx != NO_IDX && bidx != idx) {
        const int i = entry_node((int)bidx);  // scan index / k
        if ((i < bi || i > bj) && (bpos < bi || bpos > bj)) known = bgain;
      }
      known = __reduce_min_sync(FULL, known);
      if ((tid & 31) == 0 && known < 0) atomicMin(&S.bound[(int)passes & 1], known);
    }
    __syncthreads();
    {
      const int lo = bi + 1, hi = bj, half = (hi - lo + 1) >> 1;
      for (int q = tid; q < half; q += THREADS) {
        const uint16_t x = tour[lo + q], y = tour[hi - q];
        tour[lo + q] = y;
        tour[hi - q] = x;
      }
    }
    __syncthreads();
    if (SYM && T.symmetric && bj - bi >= THREADS) {
      // Inside the reversed window [lo, hi] a node's new successor is its old predecessor,
      // so its new out-edge is that predecessor's old one (the same edge, read the other
      // way). Only the two edges the move creates come from the distance source. Chunks
      // run by increasing position: a chunk reads the old out-edges of positions p + 1
      // before its barrier and writes those of positions p after it, and later chunks read
      // only higher positions than any earlier chunk wrote. A window that one round of
      // distance reads covers (bj - bi < THREADS) keeps that round: a chunk's barrier
      // would cost more than the reads it saves.
      const int lo = bi + 1, hi = bj;
      for (int base = lo; base < hi; base += THREADS) {
        const int p = base + tid;
        int x = -1, y = 0, e = 0;
        if (p < hi) {
          x = tour[p];
          y = tour[p + 1];
          e = eout[y];
        }
        __syncthreads();
        if (x >= 0) {
          ps[x] = ((unsigned)p << 16) | (unsigned)y;
          eout[x] = e;
        }
      }
      if (tid == 0) {  // the edge (tour[bi], tour[lo]) the move creates
        const int x = tour[bi], y = tour[lo];
        ps[x] = ((unsigned)bi << 16) | (unsigned)y;
        set_edge(x, ds(x, y));
      }
      if (tid == THREADS - 1) {  // and (tour[hi], tour[hi + 1]), from another warp
        const int x = tour[hi], y = tour[hi + 1 == n ? 0 : hi + 1];
        ps[x] = ((unsigned)hi << 16) | (unsigned)y;
        set_edge(x, ds(x, y));
      }
    } else {
      for (int p = bi + tid; p <= bj; p += THREADS) {
        const int x = tour[p], y = tour[p + 1 == n ? 0 : p + 1];
        ps[x] = ((unsigned)p << 16) | (unsigned)y;
        set_edge(x, ds(x, y));
      }
    }
    if constexpr (inc_best) {
      // the rows that the next pass evaluates start from no key and no valid entries
      if (row_keys) {
        const bool all = 2 * (bj - bi + 1) > rows;
        const int r_lo = all ? 0 : bi, r_hi = all ? rows - 1 : (bj < rows - 1 ? bj : rows - 1);
        int lost = 0;
        for (int i = r_lo + tid; i <= r_hi; i += THREADS) {
          rkey[i] = 0;
          if (track_rows) {
            lost += rcnt[i];
            rcnt[i] = 0;
          }
        }
        if (tid == 0 && !all && bj == n - 1 && bi > 0) {
          rkey[0] = 0;
          if (track_rows) {
            lost += rcnt[0];
            rcnt[0] = 0;
          }
        }
        if (track_rows) {
          lost = __reduce_add_sync(FULL, lost);
          if ((tid & 31) == 0 && lost != 0)
            atomicAdd(reinterpret_cast<unsigned long long*>(&S.total), (unsigned long long)(-(long long)lost));
        }
      }
    }
    __syncthreads();
    ++moves;
    win_lo = bi;
    win_hi = bj;
    if (inc_best) reach += (bj - bi + 1) - reach / 16;
    if (MODE == TSPB_MODE_FIRST && track_rows) {
      // Only rows [bi, bj] (and row 0 when bj == n-1) can change their valid count.
      const int r_hi = bj < rows - 1 ? bj : rows - 1;
      const bool row0 = bj == n - 1 && bi > 0;
      const int nr = r_hi - bi + 1 + (row0 ? 1 : 0);
      long long d = 0;
      for (int q = tid; q < nr; q += THREADS) {
        const int i = q < r_hi - bi + 1 ? bi + q : 0;
        const int v = row_count(i);
        d += v - rcnt[i];
        rcnt[i] = v;
      }
      d = warp_sum(d);
      if ((tid & 31) == 0 && d != 0) atomicAdd(reinterpret_cast<unsigned long long*>(&S.total), (unsigned long long)d);
    }
  }

  __syncthreads();
  if (rank == 0)
    for (int p = tid; p < n; p += THREADS) g_tour[p] = tour[p];
  long long tp = block_sum(my_pairs, S.redll);
  long long te = block_sum(my_eval, S.redll);
  if constexpr (CL > 1) {  // the pair's counts add up in CTA 0, which alone writes the results
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    if (tid == 0) {
      S.xcnt[0] = tp;
      S.xcnt[1] = te;
    }
    cl.sync();
    if (rank == 0) {
      tp += *cl.map_shared_rank(&S.xcnt[0], 1u);
      te += *cl.map_shared_rank(&S.xcnt[1], 1u);
    }
    cl.sync();  // CTA 1's shared memory stays valid until CTA 0 has read it
    if (rank != 0) return;
  }
  if (T.cost != nullptr) {  // eout[x] = d(x, succ[x]) of the final tour: its edges, each once
    long long len = 0;
    for (int p = tid; p < n; p += THREADS) len += eout[p];
    len = block_sum(len, S.redll);
    if (tid == 0) *T.cost = (double)len;
  }
  if (tid == 0) {
    if (T.moved) *T.moved = moves > 0 ? 1 : 0;
    if (T.converged) *T.converged = converged && err == TSPB_OK ? 1 : 0;
    if (T.status && (!T.accumulate || err != TSPB_OK)) *T.status = err;
    if (T.stats) {
      long long* st = T.stats;
      const long long v[4] = {passes, tp, moves, te};
      for (int q = 0; q < 4; ++q) st[q] = T.accumulate ? st[q] + v[q] : v[q];
    }
  }
  __syncthreads();  // S.redll is read by every thread before the caller reuses S
}

}  // namespace tspb
