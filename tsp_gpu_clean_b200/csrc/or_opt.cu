// Candidate-list Or-opt, best improvement, one CTA per tour (persistent over tours).
//
// The reference has no Or-opt strategy; this operator widens its local-search family next
// to the candidate 2-opt (src/algorithms/strategies/local_search/two_opt.py:347-367: k-NN
// candidates, open cyclic tours with position 0 fixed, exact integer deltas, the first move
// in scan order among equal gains). A move (i, L, r, o) relocates the segment
// S = t[i .. i+L-1] (1 <= L <= max_segment, i >= 1) between c and its successor e, forward
// (o = 0, c = N[t[i]][r]) or reversed (o = 1, L >= 2, c = N[t[i+L-1]][r]); it is valid when
// pos[c] lies outside [i-1, i+L-1]. With p = t[i-1], q = t[(i+L) % n] and (x, y) = (s0, sl)
// forward or (sl, s0) reversed:
//   delta = d(p,q) - d(p,s0) - d(sl,q) + d(x,c) + d(y,e) - d(c,e)
// A pass applies the smallest negative delta, the smallest key
// (((i-1) * max_segment + (L-1)) * k + r) * 2 + o among equal deltas.
//
// Layout: tour[p] and pos[a] (16 bits), eout[a] = d(a, succ a) and one 64-bit row word per
// city in shared memory (16 n bytes). The row of a city holds the best of the moves whose
// segment starts there: delta | (L, r, o) | number of valid entries. A move changes the
// successor of at most max_segment + 2 cities and the neighbourhood of at most
// 3 max_segment + 2 segment starts; every other entry keeps its value, wherever its cities
// have moved to. So the whole neighbourhood is evaluated once, and a later pass
//   - takes the minimum of n row words (delta, then position, then the word's code),
//   - shifts the window between segment and insertion point,
//   - evaluates the rows of the changed neighbourhoods anew, and looks through the flat
//     k-NN table for entries whose candidate has a new successor: such an entry is evaluated
//     alone, unless it was its row's minimum, which makes the row one of the first kind.
// The table is scanned rather than indexed by candidate: four words a load, four
// to six instructions a word, the same for any table. The entry point takes no reverse index;
// for a table that has one, its lists of the changed cities would be the shorter way.
//
// Measured: 1024 tours of 1000 cities, k = 20, segments up to 3, 50 passes 2.34 ms (27.2 with
// a whole scan each pass); the first scan is 0.47 ms of it, bound by the gathers (32 bytes of
// L2 each). A later pass changes 3 to 5 successors, some 75 table entries and 19 rows, and is
// a chain of latencies (38 us for seven tours an SM, 12 us for one): table scan and row
// evaluation a third each. 72 registers hold seven CTAs of 128 threads an SM; four candidates
// a lane and eight lanes a row were the fastest of 8 / 16 / 32 lanes and of 4 / 8 candidates.
#include <type_traits>

#include "common.cuh"
#include "two_opt.cuh"

namespace tspb {

struct OrMove {
  long long delta;
  unsigned long long key;
};

__device__ __forceinline__ bool or_less(const OrMove& a, const OrMove& b) {
  return a.delta < b.delta || (a.delta == b.delta && a.key < b.key);
}

__device__ __forceinline__ OrMove warp_min_or(OrMove m) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    OrMove w;
    w.delta = __shfl_xor_sync(FULL, m.delta, o);
    w.key = __shfl_xor_sync(FULL, m.key, o);
    if (or_less(w, m)) m = w;
  }
  return m;
}

// Block-wide lexicographic minimum; sh holds 33 entries. Every thread gets the result.
__device__ __forceinline__ OrMove block_min_or(OrMove m, OrMove* sh) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  m = warp_min_or(m);
  if (lane == 0) sh[wid] = m;
  __syncthreads();
  if (wid == 0) {
    OrMove v{0, NO_KEY};
    if (lane < nw) v = sh[lane];
    v = warp_min_or(v);
    if (lane == 0) sh[32] = v;
  }
  __syncthreads();
  const OrMove r = sh[32];
  __syncthreads();  // sh is reused by the next call
  return r;
}

constexpr unsigned long long ROW_DIRTY = ~0ull;
constexpr unsigned ROW_NONE = 0x80000000u;  // high word of a row without an improving move
constexpr int GROUP = 8;                    // lanes that evaluate a row (>= max_segment)
constexpr int HIT_CAP = 192, DIRTY_CAP = 256;

// One tour's state and the tables, as every phase uses them.
template <bool PACKED>
struct OrState {
  unsigned long long* row;
  int* eout;
  uint16_t* tour;
  uint16_t* pos;
  int n, k, S, cbits;
  DistSrc ds;
  const int32_t* cand;
  const int32_t* cdist;
  const uint32_t* packed;

  __device__ __forceinline__ int at(int p) const { return tour[p >= n ? p - n : p]; }
  __device__ __forceinline__ unsigned code(int L, int r, int o) const {
    return ((unsigned)((L - 1) * k + r) << 1) | (unsigned)o;
  }
};

// The best of the moves whose segment starts at city s0, by GROUP lanes (all lanes of the
// warp call it together; lanes of a group share s0). Lane L-1 of a group takes the part of the
// deltas that only L decides, in flight behind the rest; lanes take four candidates of one
// (L, o) each. Every lane gets the row word; `wide` is set where a delta does not fit 32 bits.
template <bool PACKED>
__device__ __forceinline__ unsigned long long or_row(const OrState<PACKED>& st, int s0, bool active, bool& wide) {
  const int sub = threadIdx.x & (GROUP - 1), lead = threadIdx.x & 31 & ~(GROUP - 1);
  const int n = st.n, k = st.k, S = st.S, chunks = (k + 3) >> 2;
  const int i = st.pos[s0];
  active = active && i >= 1;
  const int p = st.tour[active ? i - 1 : 0];
  const int Lmax = active ? (n - i < S ? n - i : S) : 0;  // the segment stays before position n
  const bool own = sub < Lmax;
  const int sl = own ? st.tour[i + sub] : 0;
  const int gap[1] = {own ? st.at(i + sub + 1) : 0};
  const bool want[1] = {own};
  int joined[1];
  gather_if<1>(st.ds, p, gap, want, joined);
  unsigned long long best = ((unsigned long long)ROW_NONE << 32);
  int cnt = 0;
  const int total = (2 * S - 1) * chunks;
  int v = sub / chunks, ch = sub - v * chunks;
  for (int it = sub; it - sub < total; it += GROUP) {
    const int o = v >= S, L = o ? v - S + 2 : v + 1, r0 = ch * 4;
    const bool on = it < total && L <= Lmax;
    const int last = on ? st.tour[i + L - 1] : 0, x = o ? last : s0, y = o ? s0 : last;
    int c[4], dxc[4], e[4], dye[4];
    bool ok[4];
    if constexpr (PACKED) {  // k % 4 == 0: the four entries exist and are 16-byte aligned
      uint4 w = make_uint4(0, 0, 0, 0);
      if (on) w = __ldg(reinterpret_cast<const uint4*>(st.packed + (long long)x * k + r0));
      const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        c[u] = (int)(ws[u] & 0xffffu);
        dxc[u] = (int)(ws[u] >> 16);
        ok[u] = on;
      }
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        ok[u] = on && r0 + u < k;
        const long long a = (long long)x * k + r0 + u;
        c[u] = (int)load_nc_if(ok[u], st.cand + a);
        dxc[u] = (int)load_nc_if(ok[u], st.cdist + a);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      ok[u] = ok[u] && (unsigned)c[u] < (unsigned)n;
      if (!ok[u]) c[u] = 0;
      const int j = st.pos[c[u]];
      ok[u] = ok[u] && (j < i - 1 || j > i + L - 1);
      e[u] = st.at(j + 1);
      cnt += ok[u];
    }
    gather_if<4>(st.ds, y, e, ok, dye);
    const long long part = (long long)joined[0] - (own ? (long long)st.eout[p] + st.eout[sl] : 0);
    const long long base = __shfl_sync(FULL, part, lead + ((L - 1) & (GROUP - 1)));
    long long least = 0;
    int at = -1;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long d = (long long)dxc[u] - st.eout[c[u]] + dye[u] + base;
      if (ok[u] && d < least) least = d, at = u;
    }
    if (at >= 0) {
      wide |= least <= -0x80000000LL;
      const unsigned long long key =
          ((unsigned long long)((unsigned)(int)least ^ 0x80000000u) << 32) | (st.code(L, r0 + at, o) << st.cbits);
      if (key < best) best = key;
    }
    ch += GROUP;
    while (ch >= chunks) ch -= chunks, ++v;
  }
#pragma unroll
  for (int m = GROUP / 2; m > 0; m >>= 1) {
    const unsigned long long w = __shfl_xor_sync(FULL, best, m);
    if (w < best) best = w;
    cnt += __shfl_xor_sync(FULL, cnt, m);
  }
  return best | (unsigned)cnt;
}

// Entry (x, r) of the k-NN table with a new successor behind its candidate: its moves, one
// per (L, o). The row of such a move, or -1 where the segment would leave the tour.
template <bool PACKED>
__device__ __forceinline__ int or_entry_row(const OrState<PACKED>& st, int x, int v, int& L, int& o, int& i) {
  o = v >= st.S;
  L = o ? v - st.S + 2 : v + 1;
  i = st.pos[x] - (o ? L - 1 : 0);
  if (i < 1 || i + L > st.n) return -1;
  return o ? st.tour[i] : x;
}

// Row `a` is evaluated anew in the next phase; its entries leave the count of valid ones.
__device__ __forceinline__ void or_mark(unsigned long long* row, int a, unsigned long long old, int cbits,
                                        uint16_t* dirty, int* ndirty, long long& cur) {
  if (old == ROW_DIRTY || atomicCAS(row + a, old, ROW_DIRTY) != old) return;
  cur -= (int)((unsigned)old & ((1u << cbits) - 1));
  const int at = atomicAdd(ndirty, 1);
  if (at < DIRTY_CAP) dirty[at] = (uint16_t)a;
}

struct OrScan {
  OrMove best;
  long long valid;
};

// A whole scan with 64-bit deltas, for tours whose row words cannot hold them.
template <int THREADS, bool PACKED>
__device__ __noinline__ OrScan or_scan_wide(const OrState<PACKED> st) {
  const int n = st.n, k = st.k, S = st.S;
  OrMove m{0, NO_KEY};
  long long valid = 0;
  for (long long it = threadIdx.x; it < (long long)(n - 1) * S * 2 * k; it += THREADS) {
    const int r = (int)(it % k);
    const int grp = (int)(it / k), o = grp & 1, il = grp >> 1;
    const int L = il % S + 1, i = il / S + 1;
    if (i + L > n || (o == 1 && L < 2)) continue;
    const int s0 = st.tour[i], sl = st.tour[i + L - 1], p = st.tour[i - 1], q = st.at(i + L);
    const int x = o ? sl : s0, y = o ? s0 : sl;
    const int c = __ldg(st.cand + (long long)x * k + r);
    if ((unsigned)c >= (unsigned)n) continue;
    const int j = st.pos[c];
    if (j >= i - 1 && j <= i + L - 1) continue;
    ++valid;
    const long long d = (long long)st.ds(p, q) - st.eout[p] - st.eout[sl] + __ldg(st.cdist + (long long)x * k + r) +
                        st.ds(y, st.at(j + 1)) - st.eout[c];
    const OrMove v{d, ((((unsigned long long)(i - 1) * S + (L - 1)) * k + r) << 1) | (unsigned)o};
    if (d < 0 && or_less(v, m)) m = v;
  }
  return {m, valid};
}

template <int THREADS, bool PACKED>
__global__ void __launch_bounds__(THREADS, THREADS == 128 ? 7 : THREADS == 256 ? 3 : 1) or_opt_kernel(int32_t* __restrict__ tours, int num, int n, DistSrc ds,
                                                         const int32_t* __restrict__ cand,
                                                         const int32_t* __restrict__ cdist,
                                                         const uint32_t* __restrict__ packed, int k, int S, int cbits,
                                                         int vec, long long max_iter, int32_t* __restrict__ status,
                                                         long long* __restrict__ stats, long long budget) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ OrMove red[33];
  __shared__ uint32_t hits[HIT_CAP];
  __shared__ uint16_t dirty[DIRTY_CAP], s_seg[8];
  __shared__ int s_flag, s_wide, s_nhit, s_ndirty, s_chg[10];
  OrState<PACKED> st;
  st.row = reinterpret_cast<unsigned long long*>(sm);
  st.eout = reinterpret_cast<int*>(st.row + n);
  st.tour = reinterpret_cast<uint16_t*>(st.eout + n);
  st.pos = st.tour + n;
  st.n = n, st.k = k, st.S = S, st.cbits = cbits;
  st.ds = ds, st.cand = cand, st.cdist = cdist, st.packed = packed;
  constexpr int NGROUP = THREADS / GROUP, WG = 32 / GROUP, HOLD = 8;
  const int tid = threadIdx.x, wgrp = (tid >> 5) * WG;
  const int variants = 2 * S - 1;
  for (int t = blockIdx.x; t < num; t += gridDim.x) {
    int32_t* g = tours + (long long)t * n;
    int* seen = reinterpret_cast<int*>(st.row);
    if (tid == 0) s_flag = 0;
    for (int p = tid; p < n; p += THREADS) seen[p] = -1;
    __syncthreads();
    for (int p = tid; p < n; p += THREADS) {
      const int v = g[p];
      if ((unsigned)v >= (unsigned)n || atomicExch(&seen[v], p) != -1) {
        s_flag = 1;
      } else {
        st.tour[p] = (uint16_t)v;
        st.pos[v] = (uint16_t)p;
      }
    }
    __syncthreads();
    if (s_flag) {
      if (tid == 0) {
        status[t] = TSPB_ERR_NOT_PERMUTATION;
        if (stats)
          for (int q = 0; q < 3; ++q) stats[(long long)t * 3 + q] = 0;
      }
      __syncthreads();  // every thread has read s_flag before it is reset
      continue;
    }
    if (tid == 0) s_wide = 0;
    for (int p = tid; p < n; p += THREADS) {
      const int a = st.tour[p];
      st.eout[a] = ds(a, st.at(p + 1));
    }
    __syncthreads();
    long long passes = 0, moves = 0, my_eval = 0;
    long long cur = 0;  // this thread's share of the valid entries of a pass
    int err = TSPB_OK;
    const long long t0 = clock64();
    if (max_iter > 0) {
      bool wide = false;
      for (int q = wgrp; q < n; q += NGROUP) {
        const int a = q + ((tid & 31) / GROUP);
        const unsigned long long w = or_row(st, a < n ? a : 0, a < n, wide);
        if ((tid & (GROUP - 1)) == 0 && a < n) {
          st.row[a] = w;
          cur += (int)((unsigned)w & ((1u << cbits) - 1));
        }
      }
      if (wide) s_wide = 1;
    }
    while (passes < max_iter) {
      if (tid == 0) s_flag = clock64() - t0 > budget;
      __syncthreads();  // rows, s_wide and s_flag are visible
      if (s_flag) {
        err = TSPB_ERR_BUDGET;
        break;
      }
      int bi, bL, br, bo;
      if (!s_wide) {
        unsigned long long best = NO_KEY;
        for (int p = 1 + tid; p < n; p += THREADS) {
          const unsigned hi = (unsigned)(st.row[st.tour[p]] >> 32);
          const unsigned long long key = ((unsigned long long)hi << 32) | (unsigned)p;
          if (key < best) best = key;
        }
        best = block_min(best, reinterpret_cast<unsigned long long*>(red));
        ++passes;
        my_eval += cur;
        if ((unsigned)(best >> 32) >= ROW_NONE) break;  // a local optimum
        bi = (int)(unsigned)best;
        const unsigned code = (unsigned)st.row[st.tour[bi]] >> cbits;
        bo = (int)(code & 1);
        bL = (int)((code >> 1) / (unsigned)k) + 1;
        br = (int)((code >> 1) % (unsigned)k);
      } else {
        const OrScan scan = or_scan_wide<THREADS, PACKED>(st);
        my_eval += scan.valid;
        const OrMove b = block_min_or(scan.best, red);
        ++passes;
        if (b.key == NO_KEY) break;
        bo = (int)(b.key & 1);
        const unsigned long long rest = b.key >> 1;
        br = (int)(rest % (unsigned long long)k);
        const unsigned long long bil = rest / (unsigned long long)k;
        bL = (int)(bil % (unsigned long long)S) + 1;
        bi = (int)(bil / (unsigned long long)S) + 1;
      }
      const int bc = __ldg(cand + (long long)st.tour[bo ? bi + bL - 1 : bi] * k + br);
      if ((unsigned)bc >= (unsigned)n) {  // cannot happen for a scanned move; uniform across the CTA
        err = TSPB_ERR_RANGE;
        break;
      }
      const int bj = st.pos[bc];
      if (bj >= bi - 1 && bj <= bi + bL - 1) {
        err = TSPB_ERR_RANGE;
        break;
      }
      // the window in the direction of the shift: its first len - L places take the city L
      // further on, its last L the segment
      const bool up = bj > bi + bL - 1;
      const int first = up ? bi : bi + bL - 1, step = up ? 1 : -1;
      const int len = up ? bj - bi + 1 : bi + bL - 1 - bj;
      if (tid < bL) {
        s_seg[tid] = st.tour[bi + tid];
        s_chg[2 + tid] = st.tour[bo ? bi + tid : bi + bL - 1];
      }
      if (tid == 0) {
        s_chg[0] = st.tour[bi - 1];
        s_chg[1] = bc;
        s_nhit = s_ndirty = 0;
      }
      const int prev = st.tour[bi - 1];
      for (int m0 = 0; m0 < len; m0 += THREADS * HOLD) {
        int held[HOLD];
#pragma unroll
        for (int u = 0; u < HOLD; ++u) {
          const int m = m0 + u * THREADS + tid;
          held[u] = m < len - bL ? st.tour[first + step * (m + bL)] : 0;
        }
        __syncthreads();  // the sources of this stretch are read, and the segment is saved
#pragma unroll
        for (int u = 0; u < HOLD; ++u) {
          const int m = m0 + u * THREADS + tid;
          if (m < len) {
            const int np = first + step * m;
            int v = held[u];
            if (m >= len - bL) {
              const int s = m - (len - bL);  // from the window's start side; upwards is tour order
              const int f = up ? s : bL - 1 - s;
              v = s_seg[bo ? bL - 1 - f : f];
            }
            st.tour[np] = (uint16_t)v;
            st.pos[v] = (uint16_t)np;
          }
        }
      }
      ++moves;
      __syncthreads();
      const int nchg = bo ? bL + 2 : 3;
      if (tid < nchg) {
        const int a = s_chg[tid];
        st.eout[a] = ds(a, st.at(st.pos[a] + 1));
      }
      if (s_wide || passes == max_iter) continue;
      // segment starts whose neighbourhood changed: around the closed gap, and around c .. e
      for (int q = tid; q < 2 * S + 2 + bL; q += THREADS) {
        const int p = q <= S ? st.pos[prev] + 1 - S + q : st.pos[bc] + 1 - S + (q - S - 1);
        if (p >= 1 && p < n) {
          const int a = st.tour[p];
          or_mark(st.row, a, *(volatile unsigned long long*)(st.row + a), cbits, dirty, &s_ndirty, cur);
        }
      }
      // table entries whose candidate has a new successor, for five such cities at a time
      const uint32_t* table = PACKED ? packed : reinterpret_cast<const uint32_t*>(cand);
      constexpr uint32_t ID = PACKED ? 0xffffu : 0xffffffffu;
      constexpr int AHEAD = 8;
      const unsigned kinv = k > 1 ? 0xffffffffu / (unsigned)k + 1 : 0xffffffffu;
      const int words = n * k, quads = vec ? words >> 2 : 0;
      auto look = [&](auto few, int q0) {
        constexpr int C = decltype(few)::value;
        uint32_t a[C];
#pragma unroll
        for (int u = 0; u < C; ++u) a[u] = (uint32_t)s_chg[q0 + u < nchg ? q0 + u : q0];
        auto changed = [&](uint32_t w) {
          bool hit = (w & ID) == a[0];
#pragma unroll
          for (int u = 1; u < C; ++u) hit |= (w & ID) == a[u];
          return hit;
        };
        auto note = [&](int f) {
          int x = (int)__umulhi((unsigned)f, kinv), r = f - x * k;  // at most one off
          if (r < 0) --x, r += k;
          if (r >= k) ++x, r -= k;
          const int at = atomicAdd(&s_nhit, 1);
          if (at < HIT_CAP) hits[at] = (unsigned)x | (unsigned)r << 16;
        };
        const uint4* t4 = reinterpret_cast<const uint4*>(table);
        for (int b = tid; b < quads; b += AHEAD * THREADS) {
          uint4 w[AHEAD];
#pragma unroll
          for (int u = 0; u < AHEAD; ++u) w[u] = __ldg(t4 + (b + u * THREADS < quads ? b + u * THREADS : b));
          unsigned mask = 0;
#pragma unroll
          for (int u = 0; u < AHEAD; ++u) {
            const bool h = changed(w[u].x) | changed(w[u].y) | changed(w[u].z) | changed(w[u].w);
            if (h && b + u * THREADS < quads) mask |= 1u << u;
          }
          for (; mask; mask &= mask - 1) {  // one quad in 250: its words are read again
            const int at = b + (__ffs(mask) - 1) * THREADS;
            const uint4 q = __ldg(t4 + at);
            if (changed(q.x)) note(at * 4);
            if (changed(q.y)) note(at * 4 + 1);
            if (changed(q.z)) note(at * 4 + 2);
            if (changed(q.w)) note(at * 4 + 3);
          }
        }
        for (int f = quads * 4 + tid; f < words; f += THREADS)
          if (changed(__ldg(table + f))) note(f);
      };
      if (nchg == 3) {
        look(std::integral_constant<int, 3>{}, 0);
      } else {
        for (int q0 = 0; q0 < nchg; q0 += 5) look(std::integral_constant<int, 5>{}, q0);
      }
      __syncthreads();  // the new edges and the hits are known
      // a row whose minimum was one of them is evaluated anew (all rows, if the list overflows)
      const int nh = s_nhit <= HIT_CAP ? s_nhit * variants : 0;
      if (s_nhit > HIT_CAP)
        for (int a = tid; a < n; a += THREADS)
          or_mark(st.row, a, *(volatile unsigned long long*)(st.row + a), cbits, dirty, &s_ndirty, cur);
      for (int q = tid; q < nh; q += THREADS) {
        const int x = (int)(hits[q / variants] & 0xffffu), r = (int)(hits[q / variants] >> 16);
        int L, o, i;
        const int a = or_entry_row(st, x, q % variants, L, o, i);
        if (a < 0) continue;
        const unsigned long long old = *(volatile unsigned long long*)(st.row + a);
        if ((unsigned)(old >> 32) < ROW_NONE && ((unsigned)old >> cbits) == st.code(L, r, o))
          or_mark(st.row, a, old, cbits, dirty, &s_ndirty, cur);
      }
      __syncthreads();  // the rows to evaluate are known
      bool wide = false;
      const int nd = s_ndirty, rows = nd <= DIRTY_CAP ? nd : n;
      for (int q = wgrp; q < rows; q += NGROUP) {
        const int at = q + (tid & 31) / GROUP;
        bool on = at < rows;
        const int a = !on ? 0 : nd <= DIRTY_CAP ? dirty[at] : at;
        if (nd > DIRTY_CAP) on = on && st.row[a] == ROW_DIRTY;
        const unsigned long long w = or_row(st, a, on, wide);
        if ((tid & (GROUP - 1)) == 0 && on) {
          st.row[a] = w;
          cur += (int)((unsigned)w & ((1u << cbits) - 1));
        }
      }
      for (int q = tid; q < nh; q += THREADS) {
        const int x = (int)(hits[q / variants] & 0xffffu), r = (int)(hits[q / variants] >> 16);
        int L, o, i;
        const int a = or_entry_row(st, x, q % variants, L, o, i);
        if (a < 0) continue;
        unsigned long long old = *(volatile unsigned long long*)(st.row + a);
        if (old == ROW_DIRTY) continue;  // evaluated whole
        const long long f = (long long)x * k + r;
        const uint32_t w = __ldg(table + f);  // just read by the scan
        const int c = (int)(w & ID), dxc = PACKED ? (int)(w >> 16) : __ldg(cdist + f);
        const int s0 = st.tour[i], sl = st.tour[i + L - 1], p = st.tour[i - 1];
        const int dpq = ds(p, st.at(i + L));
        const int j = st.pos[c];
        if (j >= i - 1 && j <= i + L - 1) continue;
        const long long d = (long long)dpq - st.eout[p] - st.eout[sl] + dxc + ds(o ? s0 : sl, st.at(j + 1)) - st.eout[c];
        if (d >= 0) continue;
        wide |= d <= -0x80000000LL;
        const unsigned long long key =
            ((unsigned long long)((unsigned)(int)d ^ 0x80000000u) << 32) | (st.code(L, r, o) << cbits);
        while (old != ROW_DIRTY) {
          const unsigned long long now = key | ((unsigned)old & ((1u << cbits) - 1));
          if (now >= old) break;
          const unsigned long long was = atomicCAS(st.row + a, old, now);
          if (was == old) break;
          old = was;
        }
      }
      if (wide) s_wide = 1;
    }
    __syncthreads();
    for (int p = tid; p < n; p += THREADS) g[p] = st.tour[p];
    const long long ev = block_sum(my_eval, reinterpret_cast<long long*>(red));
    if (tid == 0) {
      status[t] = err;
      if (stats) {
        stats[(long long)t * 3 + 0] = passes;
        stats[(long long)t * 3 + 1] = moves;
        stats[(long long)t * 3 + 2] = ev;
      }
    }
    __syncthreads();  // tour, s_flag and red are reused by the next tour
  }
}

// The whole neighbourhood every pass, with 64-bit deltas: for neighbourhoods so small that this
// takes no longer than keeping the row words does (or_scan_suffices), and for codes too long
// for a row word. tour, pos, eout and a rebuild buffer in shared memory (16 n bytes); a thread
// evaluates four consecutive candidates of one (i, L, o), and the move rewrites only the
// positions between the segment and the insertion point.
template <int THREADS, bool PACKED>
__global__ void __launch_bounds__(THREADS) or_scan_kernel(int32_t* __restrict__ tours, int num, int n, DistSrc ds,
                                                          const int32_t* __restrict__ cand,
                                                          const int32_t* __restrict__ cdist,
                                                          const uint32_t* __restrict__ packed, int k, int S,
                                                          long long max_iter, int32_t* __restrict__ status,
                                                          long long* __restrict__ stats, long long budget) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ OrMove red[33];
  __shared__ long long redll[32];
  __shared__ int s_flag;
  int* tour = reinterpret_cast<int*>(sm);
  int* pos = tour + n;
  int* eout = pos + n;
  int* tmp = eout + n;
  const int tid = threadIdx.x;
  const int chunks = (k + 3) >> 2;
  const int items = (n - 1) * S * 2 * chunks;  // (i-1, L-1, o) groups x four-candidate chunks
  for (int t = blockIdx.x; t < num; t += gridDim.x) {
    int32_t* g = tours + (long long)t * n;
    if (tid == 0) s_flag = 0;
    for (int p = tid; p < n; p += THREADS) {
      tour[p] = g[p];
      pos[p] = -1;
    }
    __syncthreads();
    for (int p = tid; p < n; p += THREADS) {
      const int v = tour[p];
      if ((unsigned)v >= (unsigned)n || atomicExch(&pos[v], p) != -1) s_flag = 1;
    }
    __syncthreads();
    if (s_flag) {
      if (tid == 0) {
        status[t] = TSPB_ERR_NOT_PERMUTATION;
        if (stats)
          for (int q = 0; q < 3; ++q) stats[(long long)t * 3 + q] = 0;
      }
      __syncthreads();  // every thread has read s_flag before it is reset
      continue;
    }
    for (int p = tid; p < n; p += THREADS) {
      const int a = tour[p];
      eout[a] = ds(a, tour[p + 1 == n ? 0 : p + 1]);
    }
    long long passes = 0, moves = 0, my_eval = 0;
    int err = TSPB_OK;
    const long long t0 = clock64();
    while (passes < max_iter) {
      __syncthreads();  // the state of the last move (or the setup) is visible
      if (tid == 0) s_flag = clock64() - t0 > budget;
      __syncthreads();
      if (s_flag) {
        err = TSPB_ERR_BUDGET;
        break;
      }
      OrMove m{0, NO_KEY};
      for (int it = tid; it < items; it += THREADS) {
        const int grp = it / chunks, ch = it - grp * chunks;
        const int o = grp & 1, il = grp >> 1;
        const int L = il % S + 1, i = il / S + 1;
        if (i + L - 1 > n - 1 || (o == 1 && L < 2)) continue;
        const int s0 = tour[i], sl = tour[i + L - 1], p = tour[i - 1], q = tour[i + L == n ? 0 : i + L];
        const int x = o ? sl : s0, y = o ? s0 : sl;
        const long long base = (long long)ds(p, q) - eout[p] - eout[sl];
        const int r0 = ch * 4;
        int c[4], dxc[4], e[4], dye[4];
        bool ok[4];
        if constexpr (PACKED) {  // k % 4 == 0: the four entries exist and are 16-byte aligned
          const uint4 w = __ldg(reinterpret_cast<const uint4*>(packed + (long long)x * k + r0));
          const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            ok[u] = true;
            c[u] = (int)(ws[u] & 0xffffu);
            dxc[u] = (int)(ws[u] >> 16);
          }
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            ok[u] = r0 + u < k;
            if (ok[u]) {
              const long long at = (long long)x * k + r0 + u;
              c[u] = __ldg(cand + at);
              dxc[u] = __ldg(cdist + at);
            }
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (!ok[u]) continue;
          if ((unsigned)c[u] >= (unsigned)n) {
            ok[u] = false;
            continue;
          }
          const int j = pos[c[u]];
          ok[u] = j < i - 1 || j > i + L - 1;
          if (ok[u]) e[u] = tour[j + 1 == n ? 0 : j + 1];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (ok[u]) dye[u] = ds(y, e[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (!ok[u]) continue;
          ++my_eval;
          const long long d = base + dxc[u] + dye[u] - eout[c[u]];
          if (d < 0) {
            const OrMove v{d, ((((unsigned long long)(i - 1) * S + (L - 1)) * k + (r0 + u)) << 1) | (unsigned)o};
            if (or_less(v, m)) m = v;
          }
        }
      }
      ++passes;
      const OrMove b = block_min_or(m, red);
      if (b.key == NO_KEY) break;  // a local optimum
      const int bo = (int)(b.key & 1);
      const unsigned long long rest = b.key >> 1;
      const int br = (int)(rest % (unsigned long long)k);
      const unsigned long long bil = rest / (unsigned long long)k;
      const int bL = (int)(bil % (unsigned long long)S) + 1, bi = (int)(bil / (unsigned long long)S) + 1;
      const int bx = bo ? tour[bi + bL - 1] : tour[bi];
      const int bc = __ldg(cand + (long long)bx * k + br);
      if ((unsigned)bc >= (unsigned)n) {  // cannot happen for a scanned move; uniform across the CTA
        err = TSPB_ERR_RANGE;
        break;
      }
      const int bj = pos[bc];
      if (bj >= bi - 1 && bj <= bi + bL - 1) {
        err = TSPB_ERR_RANGE;
        break;
      }
      const bool case_a = bj > bi + bL - 1;
      const int lo = case_a ? bi : bj + 1, hi = case_a ? bj : bi + bL - 1;
      for (int np = lo + tid; np <= hi; np += THREADS) {
        int v;
        if (case_a) {
          if (np <= bj - bL) {
            v = tour[np + bL];
          } else {
            const int mm = np - (bj - bL + 1);
            v = bo ? tour[bi + bL - 1 - mm] : tour[bi + mm];
          }
        } else {
          if (np <= bj + bL) {
            const int mm = np - (bj + 1);
            v = bo ? tour[bi + bL - 1 - mm] : tour[bi + mm];
          } else {
            v = tour[np - bL];
          }
        }
        tmp[np] = v;
      }
      __syncthreads();
      for (int np = lo + tid; np <= hi; np += THREADS) {
        const int v = tmp[np];
        tour[np] = v;
        pos[v] = np;
      }
      __syncthreads();
      for (int np = lo - 1 + tid; np <= hi; np += THREADS) {
        const int a = tour[np];
        eout[a] = ds(a, tour[np + 1 == n ? 0 : np + 1]);
      }
      ++moves;
    }
    __syncthreads();
    for (int p = tid; p < n; p += THREADS) g[p] = tour[p];
    const long long ev = block_sum(my_eval, redll);
    if (tid == 0) {
      status[t] = err;
      if (stats) {
        stats[(long long)t * 3 + 0] = passes;
        stats[(long long)t * 3 + 1] = moves;
        stats[(long long)t * 3 + 2] = ev;
      }
    }
    __syncthreads();  // tour, s_flag and redll are reused by the next tour
  }
}

// CTAs of a launch: all that run at once, one per tour at most; 0: a CTA does not fit, -1: a
// runtime error.
template <typename Kern>
static int or_grid(Kern kern, int threads, int num, size_t smem, bool carveout) {
  int per_sm = 0;
  const int sms = device_attr(cudaDevAttrMultiProcessorCount);
  if (sms <= 0 || allow_smem(kern, smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem) != cudaSuccess) {
    (void)cudaGetLastError();
    return -1;
  }
  if (per_sm > 0 && carveout) {
    cudaFuncAttributes own{};  // of its static arrays: they decide whether the last CTA fits
    if (cudaFuncGetAttributes(&own, kern) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                             carveout_for(per_sm, smem + own.sharedSizeBytes)) != cudaSuccess) {
      (void)cudaGetLastError();
      return -1;
    }
  }
  return (int)((long long)per_sm * sms < num ? (long long)per_sm * sms : num);
}

// Whether evaluating everything each pass is the faster way. A scan costs about four units an
// item of up to four candidates and one a candidate; keeping rows costs a pass of fixed phases
// that grow with the segment length, and, where tours share SMs, of phases that grow with n.
// 50 passes, scan and rows, in ms: segments of 1, one tour of 50 cities, k = 8 0.28 and 0.35, of
// 100 cities 0.42 and 0.36; 2000 tours of 1000 cities, k = 1 2.6 and 4.8. Segments up to 3, k = 3,
// 1000 tours of 50 cities 0.40 and 0.47, of 100 0.82 and 0.60.
static bool or_scan_suffices(int num, int n, int k, int S) {
  const long long cost = (long long)n * (2 * S - 1) * (4 * ((k + 3) / 4) + k) / 8;
  return cost < 60 + 85 * S ||
         (S == 1 && k <= 3 && n < 2000 && num > 3 * device_attr(cudaDevAttrMultiProcessorCount));
}

template <int THREADS>
static int launch_or_opt(int32_t* tours, int num, int n, const DistSrc& ds, const int32_t* cand,
                         const int32_t* cdist, const uint32_t* packed, int k, int S, int cbits, long long max_iter,
                         int32_t* status, long long* stats, size_t smem, cudaStream_t st) {
  if (cbits == 0) {  // whole scans
    auto scan = packed ? or_scan_kernel<THREADS, true> : or_scan_kernel<THREADS, false>;
    const int grid = or_grid(scan, THREADS, num, smem, false);
    if (grid <= 0) return grid < 0 ? TSPB_ERR_CUDA : TSPB_ERR_UNSUPPORTED;
    scan<<<grid, THREADS, smem, st>>>(tours, num, n, ds, cand, cdist, packed, k, S, max_iter, status, stats,
                                      watchdog_cycles());
    return tspb_launch_status();
  }
  auto kern = packed ? or_opt_kernel<THREADS, true> : or_opt_kernel<THREADS, false>;
  const int grid = or_grid(kern, THREADS, num, smem, true);
  if (grid <= 0) return grid < 0 ? TSPB_ERR_CUDA : TSPB_ERR_UNSUPPORTED;
  const void* table = packed ? static_cast<const void*>(packed) : cand;
  const int vec = reinterpret_cast<uintptr_t>(table) % 16 == 0;
  kern<<<grid, THREADS, smem, st>>>(tours, num, n, ds, cand, cdist, packed, k, S, cbits, vec, max_iter, status, stats,
                                    watchdog_cycles());
  return tspb_launch_status();
}

}  // namespace tspb

using namespace tspb;

extern "C" int tspb_or_opt_max_n(void) {
  const long long avail = (long long)smem_optin() - 2048;
  return avail > 0 ? (int)(avail / 16) : 0;
}

extern "C" int tspb_or_opt(int32_t* tours, int32_t num_tours, int32_t n, const int32_t* dist, int64_t dist_stride,
                           const double* coords, const int32_t* cand, const int32_t* cand_dist,
                           const uint32_t* cand_packed, int32_t k, int32_t max_segment, int64_t max_iterations,
                           int32_t threads, int32_t* status, int64_t* stats, void* stream) {
  if (num_tours < 0 || n < 0 || max_iterations < 0 || max_segment < 1 || max_segment > 8) return TSPB_ERR_ARG;
  if (threads != 128 && threads != 256 && threads != 512) return TSPB_ERR_ARG;
  if (num_tours == 0 || n < 3) return TSPB_OK;
  if (!tours || !status || (!dist && !coords) || (dist && dist_stride < n)) return TSPB_ERR_ARG;
  if (k < 1 || k > n - 1 || !cand || !cand_dist) return TSPB_ERR_ARG;
  if (n > tspb_or_opt_max_n()) return TSPB_ERR_UNSUPPORTED;
  // scan items and keys stay in 32 / 64 bits
  if ((long long)(n - 1) * max_segment * 2 * ((k + 3) / 4) > 0x7fffffffLL) return TSPB_ERR_UNSUPPORTED;
  DistSrc ds;
  ds.dist = dist;
  ds.stride = dist_stride;
  ds.coords = reinterpret_cast<const double2*>(coords);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const size_t smem = (size_t)16 * n;
  long long* s = reinterpret_cast<long long*>(stats);
  // the packed words serve only whole, aligned groups of four
  const uint32_t* pk =
      cand_packed && k % 4 == 0 && reinterpret_cast<uintptr_t>(cand_packed) % 16 == 0 ? cand_packed : nullptr;
  // a row word's low half holds a move's code and a count of entries
  auto bits = [](unsigned v) {
    int b = 0;
    while (v >> b) ++b;
    return b;
  };
  int cbits = bits((unsigned)(2 * max_segment - 1) * (unsigned)k);
  if (cbits + bits(2u * (unsigned)max_segment * (unsigned)k - 1) > 32) cbits = 0;
  const bool small = or_scan_suffices(num_tours, n, k, max_segment);
  if (small) cbits = 0;
  // Where tours leave SMs or warps idle a pass is a chain of latencies, and a wider CTA
  // shortens it. 50 passes, k = 20: one tour of 1000 cities 1.01 / 0.66 / 0.58 ms at 128 /
  // 256 / 512 threads, 300 of them 1.27 / 1.09 / 1.73, 1024 of them 2.34 / 2.73 / 4.07; 400
  // of 200 cities 0.76 / 0.98 / 1.33; 64 of 300 (k = 10) 0.40 / 0.35 / 0.36.
  const int sms = device_attr(cudaDevAttrMultiProcessorCount);
  const bool large = (long long)n * k >= 16384;
  if (!small && num_tours <= sms) {
    const int w = large ? 512 : 256;
    threads = threads > w ? threads : w;
  } else if (!small && num_tours <= 3 * sms && large && threads < 256) {
    threads = 256;
  }
  switch (threads) {
    case 128:
      return launch_or_opt<128>(tours, num_tours, n, ds, cand, cand_dist, pk, k, max_segment, cbits, max_iterations, status,
                                s, smem, st);
    case 512:
      return launch_or_opt<512>(tours, num_tours, n, ds, cand, cand_dist, pk, k, max_segment, cbits, max_iterations, status,
                                s, smem, st);
    default:
      return launch_or_opt<256>(tours, num_tours, n, ds, cand, cand_dist, pk, k, max_segment, cbits, max_iterations, status,
                                s, smem, st);
  }
}
