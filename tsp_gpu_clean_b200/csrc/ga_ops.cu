// Population operators for sm_100a: tour cost, tournament selection, row gather, PMX,
// inversion mutation, stable survival ranking, permutation validation, the EUC_2D
// matrix and the candidate-distance table. Each kernel states the reference code whose
// result it reproduces bit for bit.
#include "generation.cuh"

namespace tspb {

// Warp per tour; int64 accumulation is exact, then one conversion to float64
// (evaluate_tour_cpu sums int32 gathers in float64, exact below 2^53:
// src/algorithms/strategies/evaluation/tour_cost.py:17-29).
//
// A tour is n dependent pairs of loads (cities, then their distance) and a population too
// small to hide them behind one another, so a lane keeps eight of each in flight: 512 tours
// of 1000 cities 7.2 us (18.7 with one).
__global__ void tour_cost_kernel(const int32_t* __restrict__ tours, int num_tours, int n, DistSrc ds,
                                 int return_to_depot, double* __restrict__ costs) {
  constexpr int AHEAD = 8;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= num_tours) return;
  const int32_t* t = tours + (long long)warp * n;
  const int edges = n <= 1 ? 0 : (return_to_depot ? n : n - 1);
  long long acc = 0;
  int bad = 0;
  for (int p0 = lane; p0 < edges; p0 += 32 * AHEAD) {
    int a[AHEAD], b[AHEAD], d[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const int p = p0 + 32 * u;
      a[u] = (int)load_nc_if(p < edges, t + p);
      b[u] = (int)load_nc_if(p < edges, t + (p + 1 == n ? 0 : p + 1));
    }
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const bool ok = (unsigned)a[u] < (unsigned)n && (unsigned)b[u] < (unsigned)n;
      const bool in = p0 + 32 * u < edges && ok;
      bad |= !ok;
      d[u] = ds.dist != nullptr ? load_cg_if(in, ds.dist + (long long)a[u] * ds.stride + b[u]) : (in ? ds(a[u], b[u]) : 0);
    }
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) acc += d[u];
  }
  acc = warp_sum(acc);
  bad = __any_sync(FULL, bad);
  if (lane == 0) costs[warp] = n <= 1 ? 0.0 : (bad ? __longlong_as_double(0x7ff8000000000000LL) : (double)acc);
}

// Thread per parent: first argmin of fitness over the k competitors with strict `<`
// (np.argmin semantics, tournament_selection.py:125-127).
__global__ void tournament_kernel(const double* __restrict__ fitness, int pop_size, const int32_t* __restrict__ cand,
                                  int num_parents, int k, int32_t* __restrict__ winners) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= num_parents) return;
  const int32_t* c = cand + (long long)p * k;
  int best = __ldg(c);
  if ((unsigned)best >= (unsigned)pop_size) best = 0;
  double bf = __ldg(fitness + best);
  for (int q = 1; q < k; ++q) {
    const int v = __ldg(c + q);
    if ((unsigned)v >= (unsigned)pop_size) continue;
    const double f = __ldg(fitness + v);
    if (f < bf) {
      bf = f;
      best = v;
    }
  }
  winners[p] = best;
}

// CTA per output row, int4-vectorised when n is a multiple of 4.
__global__ void gather_rows_kernel(const int32_t* __restrict__ src, int src_rows, int n, const int32_t* __restrict__ rows,
                                   int32_t* __restrict__ out) {
  const int r = blockIdx.x;
  const int sr = __ldg(rows + r);
  if ((unsigned)sr >= (unsigned)src_rows) return;
  const long long s = (long long)sr * n;
  const long long d = (long long)r * n;
  if ((n & 3) == 0) {
    const int4* s4 = reinterpret_cast<const int4*>(src + s);
    int4* d4 = reinterpret_cast<int4*>(out + d);
    for (int q = threadIdx.x; q < (n >> 2); q += blockDim.x) d4[q] = __ldg(s4 + q);
  } else {
    for (int q = threadIdx.x; q < n; q += blockDim.x) out[d + q] = __ldg(src + s + q);
  }
}

// CTA per source row: dst[rows[r], :] = src[r, :] (the elite scatter-back).
__global__ void scatter_rows_kernel(const int32_t* __restrict__ src, int n, const int32_t* __restrict__ rows, int dst_rows,
                                    int32_t* __restrict__ dst) {
  const int r = blockIdx.x;
  const int dr = __ldg(rows + r);
  if ((unsigned)dr >= (unsigned)dst_rows) return;
  const long long s = (long long)r * n, d = (long long)dr * n;
  for (int q = threadIdx.x; q < n; q += blockDim.x) dst[d + q] = __ldg(src + s + q);
}

// CTA per child. Child 2q+h takes p1 = parents[2q+h], p2 = parents[2q+1-h] and the
// shared cuts; the mapping chains of values p2[c1..c2] that are not in p1[c1..c2] are
// independent, so they run one per thread (_apply_pmx, pmx_crossover.py:49-105). Bound by
// latencies like offspring_row, and read the same way: 256 pairs of 1000 cities 14.4 us (17.2
// one value at a time).
__global__ void pmx_kernel(const int32_t* __restrict__ parents, int num_routes, int n,
                           const int32_t* __restrict__ cut_first, const int32_t* __restrict__ cut_second,
                           int32_t* __restrict__ children, int32_t* __restrict__ status) {
  extern __shared__ int sm[];
  int* inv_p2 = sm;        // n
  int* child = sm + n;     // n
  unsigned* in_seg = reinterpret_cast<unsigned*>(sm + 2 * n);  // (n+31)/32 words
  __shared__ int bad;
  const int row = blockIdx.x;
  const int tid = threadIdx.x, T = blockDim.x;
  const int pairs = num_routes >> 1;
  int32_t* out = children + (long long)row * n;
  if (row >= 2 * pairs) {  // odd tail copied unchanged (pmx_crossover.py:168-169)
    for (int p = tid; p < n; p += T) out[p] = __ldg(parents + (long long)row * n + p);
    if (tid == 0 && status) status[row] = 0;
    return;
  }
  const int q = row >> 1, h = row & 1;
  const int32_t* p1 = parents + (long long)(2 * q + h) * n;
  const int32_t* p2 = parents + (long long)(2 * q + 1 - h) * n;
  int c1 = __ldg(cut_first + q), c2 = __ldg(cut_second + q);
  if (c1 > c2) {
    const int tmp = c1;
    c1 = c2;
    c2 = tmp;
  }
  const int words = (n + 31) >> 5;
  if (tid == 0) bad = 0;
  for (int p = tid; p < n; p += T) inv_p2[p] = -1;
  for (int w = tid; w < words; w += T) in_seg[w] = 0u;
  __syncthreads();
  if (c1 < 0 || c2 >= n) bad = 1;
  for (int p0 = tid; p0 < n; p0 += OFFSPRING_AHEAD * T) {
    int v1[OFFSPRING_AHEAD], v2[OFFSPRING_AHEAD];
#pragma unroll
    for (int u = 0; u < OFFSPRING_AHEAD; ++u) {
      v1[u] = (int)load_nc_if(p0 + u * T < n, p1 + p0 + u * T);
      v2[u] = (int)load_nc_if(p0 + u * T < n, p2 + p0 + u * T);
    }
#pragma unroll
    for (int u = 0; u < OFFSPRING_AHEAD; ++u) {
      const int p = p0 + u * T;
      if (p >= n) break;
      if ((unsigned)v2[u] >= (unsigned)n || (unsigned)v1[u] >= (unsigned)n) {
        bad = 1;
        continue;
      }
      const bool seg = p >= c1 && p <= c2;
      if (atomicExch(&inv_p2[v2[u]], p) != -1) bad = 1;
      child[p] = seg ? v1[u] : v2[u];  // p2 outside the segment until a chain ends there
      if (seg) atomicOr(&in_seg[v1[u] >> 5], 1u << (v1[u] & 31));
    }
  }
  __syncthreads();
  if (bad) {
    for (int p = tid; p < n; p += T) out[p] = __ldg(p1 + p);
    if (tid == 0 && status) status[row] = TSPB_ERR_NOT_PERMUTATION;
    return;
  }
  const int seg_len = c2 - c1 + 1;
  for (int idx = c1 + tid; idx <= c2; idx += T) {
    const int val = __ldg(p2 + idx);
    if (in_seg[val >> 5] & (1u << (val & 31))) continue;
    int pos = idx, steps = 0;
    while (pos >= c1 && pos <= c2 && steps <= seg_len) {
      pos = inv_p2[child[pos]];  // p1's gene: nothing writes inside the segment now
      ++steps;
    }
    if (pos < c1 || pos > c2) child[pos] = val;
  }
  __syncthreads();
  for (int p = tid; p < n; p += T) out[p] = child[p];
  if (tid == 0 && status) status[row] = 0;
}

// CTA per child, Order Crossover with validated parents (order_crossover.py:52-83).
// Shared memory: child[n], in_seg, and the seen-bitmaps of p1 and p2.
__global__ void ox_kernel(const int32_t* __restrict__ parents, int num_routes, int n,
                          const int32_t* __restrict__ cut_first, const int32_t* __restrict__ cut_second,
                          int32_t* __restrict__ children, int32_t* __restrict__ status) {
  extern __shared__ int sm[];
  const int words = (n + 31) >> 5;
  int* child = sm;                                                // n
  unsigned* in_seg = reinterpret_cast<unsigned*>(sm + n);         // words
  unsigned* seen1 = in_seg + words;                               // words
  unsigned* seen2 = seen1 + words;                                // words
  __shared__ int bad;
  __shared__ int red[32];
  const int row = blockIdx.x;
  const int tid = threadIdx.x, T = blockDim.x;
  const int pairs = num_routes >> 1;
  int32_t* out = children + (long long)row * n;
  if (row >= 2 * pairs) {  // odd tail copied unchanged (order_crossover.py:167-168)
    for (int p = tid; p < n; p += T) out[p] = __ldg(parents + (long long)row * n + p);
    if (tid == 0 && status) status[row] = 0;
    return;
  }
  const int q = row >> 1, h = row & 1;
  const int32_t* p1 = parents + (long long)(2 * q + h) * n;
  const int32_t* p2 = parents + (long long)(2 * q + 1 - h) * n;
  int c1 = __ldg(cut_first + q), c2 = __ldg(cut_second + q);
  if (c1 > c2) {
    const int tmp = c1;
    c1 = c2;
    c2 = tmp;
  }
  if (tid == 0) bad = (c1 < 0 || c2 >= n) ? 1 : 0;
  for (int w = tid; w < 3 * words; w += T) in_seg[w] = 0u;
  __syncthreads();
  for (int p = tid; p < n; p += T) {
    const int v1 = __ldg(p1 + p), v2 = __ldg(p2 + p);
    if ((unsigned)v1 >= (unsigned)n || (unsigned)v2 >= (unsigned)n) {
      bad = 1;
      continue;
    }
    if (atomicOr(&seen1[v1 >> 5], 1u << (v1 & 31)) & (1u << (v1 & 31))) bad = 1;
    if (atomicOr(&seen2[v2 >> 5], 1u << (v2 & 31)) & (1u << (v2 & 31))) bad = 1;
  }
  __syncthreads();
  if (bad) {
    for (int p = tid; p < n; p += T) out[p] = __ldg(p1 + p);
    if (tid == 0 && status) status[row] = TSPB_ERR_NOT_PERMUTATION;
    return;
  }
  for (int p = c1 + tid; p <= c2; p += T) {
    const int v1 = __ldg(p1 + p);
    child[p] = v1;
    atomicOr(&in_seg[v1 >> 5], 1u << (v1 & 31));
  }
  __syncthreads();
  ox_fill(p2, n, c2, child, in_seg, red);
  __syncthreads();
  for (int p = tid; p < n; p += T) out[p] = child[p];
  if (tid == 0 && status) status[row] = 0;
}

// Thread per route: exchange of positions p1, p2 when u < rate (swap_mutation.py:94-99).
__global__ void swap_kernel(int32_t* __restrict__ routes, int num_routes, int n, const double* __restrict__ u,
                            double rate, const int32_t* __restrict__ pos1, const int32_t* __restrict__ pos2) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= num_routes) return;
  if (!(__ldg(u + r) < rate)) return;
  const int a = __ldg(pos1 + r), b = __ldg(pos2 + r);
  if ((unsigned)a >= (unsigned)n || (unsigned)b >= (unsigned)n) return;
  int32_t* t = routes + (long long)r * n;
  const int x = t[a];
  t[a] = t[b];
  t[b] = x;
}

// CTA per route, reversal of [min(p1,p2), max(p1,p2)] when u < rate
// (inversion_mutation.py:93-97). Most routes leave at once; one warp for a whole reversal is
// up to n / 64 dependent rounds: 512 routes of 1000 cities 4.1 us (7.0 with a warp).
constexpr int INVERSION_THREADS = 128;
__global__ void __launch_bounds__(INVERSION_THREADS) inversion_kernel(int32_t* __restrict__ routes, int num_routes, int n,
                                                                      const double* __restrict__ u, double rate,
                                                                      const int32_t* __restrict__ pos1,
                                                                      const int32_t* __restrict__ pos2) {
  const int r = blockIdx.x;
  const double draw = __ldg(u + r);
  const int a = __ldg(pos1 + r), b = __ldg(pos2 + r);
  if (!(draw < rate)) return;
  const int lo = a < b ? a : b, hi = a < b ? b : a;
  if (lo < 0 || hi >= n) return;
  int32_t* t = routes + (long long)r * n;
  const int half = (hi - lo + 1) >> 1;
  for (int q = threadIdx.x; q < half; q += INVERSION_THREADS) {
    const int x = t[lo + q], y = t[hi - q];
    t[lo + q] = y;
    t[hi - q] = x;
  }
}

// The same with a warp per route: most routes leave at once, and a CTA for each costs more to
// start than a short reversal takes (inversion_per_cta).
__global__ void __launch_bounds__(256) inversion_warp_kernel(int32_t* __restrict__ routes, int num_routes, int n,
                                                             const double* __restrict__ u, double rate,
                                                             const int32_t* __restrict__ pos1,
                                                             const int32_t* __restrict__ pos2) {
  const int r = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (r >= num_routes) return;
  if (!(__ldg(u + r) < rate)) return;
  const int a = __ldg(pos1 + r), b = __ldg(pos2 + r);
  const int lo = a < b ? a : b, hi = a < b ? b : a;
  if (lo < 0 || hi >= n) return;
  int32_t* t = routes + (long long)r * n;
  const int half = (hi - lo + 1) >> 1;
  for (int q = threadIdx.x & 31; q < half; q += 32) {
    const int x = t[lo + q], y = t[hi - q];
    t[lo + q] = y;
    t[hi - q] = x;
  }
}

// CTAs pay where the reversal is the longer part and the routes are few: 4096 routes of 1000 cities
// 13.4 us (16.2 with warps), 2000 of 5000 21 (35), 16,384 of 1000 20 either way; with warps 65,536
// of 50 take 13 us (42 with CTAs), a million of 20 73 (524).
static bool inversion_per_cta(int num_routes, int n) { return n >= 512 && num_routes <= 16384; }

// Thread per element: rank by (value, index); ranks below `keep` scatter the index
// (a stable ascending sort, np.lexsort of genetic_algorithm.py:682-689).
__global__ void stable_rank_kernel(const double* __restrict__ f, int count, int keep, int32_t* __restrict__ order) {
  __shared__ double tile[1024];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const double fi = i < count ? f[i] : 0.0;
  int rank = 0;
  for (int base = 0; base < count; base += blockDim.x) {
    const int j = base + threadIdx.x;
    if (j < count) tile[threadIdx.x] = f[j];
    __syncthreads();
    const int lim = min((int)blockDim.x, count - base);
    if (i < count) {
      for (int q = 0; q < lim; ++q) {
        const double fj = tile[q];
        const int jj = base + q;
        rank += (fj < fi) || (fj == fi && jj < i);
      }
    }
    __syncthreads();
  }
  if (i < count && rank < keep) order[rank] = i;
}

__global__ void validate_perm_kernel(const int32_t* __restrict__ tours, int n, int32_t* __restrict__ bad_out) {
  extern __shared__ unsigned seen[];
  __shared__ int bad;
  const int r = blockIdx.x;
  const int words = (n + 31) >> 5;
  if (threadIdx.x == 0) bad = 0;
  for (int w = threadIdx.x; w < words; w += blockDim.x) seen[w] = 0u;
  __syncthreads();
  const int32_t* t = tours + (long long)r * n;
  for (int p = threadIdx.x; p < n; p += blockDim.x) {
    const int v = __ldg(t + p);
    if ((unsigned)v >= (unsigned)n) {
      bad = 1;
      continue;
    }
    const unsigned bit = 1u << (v & 31);
    if (atomicOr(&seen[v >> 5], bit) & bit) bad = 1;
  }
  __syncthreads();
  if (threadIdx.x == 0) bad_out[r] = bad;
}

// EUC_2D matrix, four columns of one row per thread and step (16-byte stores where the rows
// allow them).
//
// What bounds it: writing the 4 n^2 bytes. The correctly rounded FP64 root of every entry did
// before (n = 10,000: 222 us; 115 in this form, 61 for the bytes at copy speed), so an entry takes it
// only when FP32 cannot settle the rounding: d is computed in FP32 with the error bound below,
// and accepted when its distance from the nearest integer leaves half a unit minus that bound.
//   coordinates: rounding each to FP32 moves it by at most 2^-24 |x|, the difference adds
//   2^-24 of its value, so |error of dx| + |error of dy| <= 2^-24 (mag_a + mag_b) + 2^-24
//   (|dx| + |dy|), with mag = |x| + |y|; the root of the sum of squares moves by no more than
//   that (the triangle inequality), and the squares, their sum and sqrt.approx (2^-23) by less
//   than 2^-21 d. 2^-23 (mag_a + mag_b) + 2^-20 d bounds all of it, d + 0.5 included.
// 1000 x 1000 squares send about one entry in 2,000 to the FP64 form.
__global__ void __launch_bounds__(256) euc2d_matrix_kernel(const double2* __restrict__ coords, int n,
                                                           int32_t* __restrict__ dist, long long stride, int rows, int wide) {
  const int c0 = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (c0 >= n) return;
  float2 p[4];
  float mag[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const double2 v = __ldg(coords + (c0 + q < n ? c0 + q : n - 1));
    p[q] = make_float2((float)v.x, (float)v.y);
    mag[q] = 0x1p-23f * (fabsf(p[q].x) + fabsf(p[q].y));
  }
  const int a_end = min((int)(blockIdx.y + 1) * rows, n);
  for (int a = blockIdx.y * rows; a < a_end; ++a) {
    const double2 va = __ldg(coords + a);
    const float2 pa = make_float2((float)va.x, (float)va.y);
    const float mag_a = 0x1p-23f * (fabsf(pa.x) + fabsf(pa.y));
    int d[4];
    bool redo = false;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float dx = pa.x - p[q].x, dy = pa.y - p[q].y;
      float r;
      asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(fmaf(dx, dx, dy * dy)));
      const float err = mag_a + mag[q] + 0x1p-20f * r;
      // nearest integer by adding 1.5 * 2^23 (no conversion: those share the root's unit); r
      // minus it is exact. Roots of 2^19 and more, infinities and NaN fail the test.
      const float m = __fadd_rn(r, 12582912.0f);
      d[q] = __float_as_int(m) - __float_as_int(12582912.0f);
      redo |= !(fabsf(__fsub_rn(r, __fsub_rn(m, 12582912.0f))) < 0.5f - err);
    }
    if (redo) {
#pragma unroll
      for (int q = 0; q < 4; ++q) d[q] = euc2d(va, __ldg(coords + (c0 + q < n ? c0 + q : n - 1)));
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (c0 + q == a) d[q] = 0;
    int32_t* row = dist + (long long)a * stride + c0;
    if (wide && c0 + 4 <= n) {
      *reinterpret_cast<int4*>(row) = make_int4(d[0], d[1], d[2], d[3]);
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (c0 + q < n) row[q] = d[q];
    }
  }
}

__global__ void cand_dist_kernel(const int32_t* __restrict__ cand, int n, int k, DistSrc ds, int32_t* __restrict__ out) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long long)n * k) return;
  const int a = (int)(e / k);
  const int c = __ldg(cand + e);
  out[e] = (unsigned)c < (unsigned)n ? ds(a, c) : 0;
}

}  // namespace tspb

using namespace tspb;

static DistSrc make_ds(const int32_t* dist, int64_t stride, const double* coords) {
  DistSrc d;
  d.dist = dist;
  d.stride = stride;
  d.coords = reinterpret_cast<const double2*>(coords);
  return d;
}

extern "C" int tspb_tour_cost(const int32_t* tours, int32_t num_tours, int32_t n, const int32_t* dist, int64_t dist_stride,
                              const double* coords, int32_t return_to_depot, double* costs, void* stream) {
  if (num_tours < 0 || n < 0) return TSPB_ERR_ARG;
  if (num_tours == 0) return TSPB_OK;
  if (costs == nullptr || (n > 0 && tours == nullptr) || (dist == nullptr && coords == nullptr)) return TSPB_ERR_ARG;
  const int threads = 256;
  const long long warps = num_tours;
  const int blocks = (int)((warps * 32 + threads - 1) / threads);
  tour_cost_kernel<<<blocks, threads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      tours, num_tours, n, make_ds(dist, dist_stride, coords), return_to_depot, costs);
  return tspb_launch_status();
}

extern "C" int tspb_tournament(const double* fitness, int32_t pop_size, const int32_t* cand, int32_t num_parents, int32_t k,
                               int32_t* winners, void* stream) {
  if (num_parents < 0 || k < 1 || pop_size < 1) return TSPB_ERR_ARG;
  if (num_parents == 0) return TSPB_OK;
  if (!fitness || !cand || !winners) return TSPB_ERR_ARG;
  tournament_kernel<<<(num_parents + 127) / 128, 128, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      fitness, pop_size, cand, num_parents, k, winners);
  return tspb_launch_status();
}

extern "C" int tspb_gather_rows(const int32_t* src, int32_t src_rows, int32_t n, const int32_t* rows, int32_t num_rows,
                                int32_t* out, void* stream) {
  if (num_rows < 0 || n < 0 || src_rows < 0) return TSPB_ERR_ARG;
  if (num_rows == 0 || n == 0) return TSPB_OK;
  if (!src || !rows || !out) return TSPB_ERR_ARG;
  gather_rows_kernel<<<num_rows, 128, 0, reinterpret_cast<cudaStream_t>(stream)>>>(src, src_rows, n, rows, out);
  return tspb_launch_status();
}

extern "C" int tspb_scatter_rows(const int32_t* src, int32_t num_rows, int32_t n, const int32_t* rows, int32_t* dst,
                                 int32_t dst_rows, void* stream) {
  if (num_rows < 0 || n < 0 || dst_rows < 0) return TSPB_ERR_ARG;
  if (num_rows == 0 || n == 0) return TSPB_OK;
  if (!src || !rows || !dst) return TSPB_ERR_ARG;
  scatter_rows_kernel<<<num_rows, 128, 0, reinterpret_cast<cudaStream_t>(stream)>>>(src, n, rows, dst_rows, dst);
  return tspb_launch_status();
}

extern "C" int tspb_pmx(const int32_t* parents, int32_t num_routes, int32_t n, const int32_t* cut_first,
                        const int32_t* cut_second, int32_t* children, int32_t* status, void* stream) {
  if (num_routes < 0 || n < 0) return TSPB_ERR_ARG;
  if (num_routes == 0 || n == 0) return TSPB_OK;
  if (!parents || !children || (num_routes >= 2 && (!cut_first || !cut_second))) return TSPB_ERR_ARG;
  const size_t smem = (size_t)8 * n + (size_t)((n + 31) / 32) * 4;
  if (smem > 200 * 1024) return TSPB_ERR_UNSUPPORTED;
  TSPB_CUDA_CHECK(allow_smem(pmx_kernel, smem));
  const int threads = n >= 1024 ? 512 : (n >= 256 ? 256 : 128);
  pmx_kernel<<<num_routes, threads, smem, reinterpret_cast<cudaStream_t>(stream)>>>(parents, num_routes, n, cut_first,
                                                                                    cut_second, children, status);
  return tspb_launch_status();
}

extern "C" int tspb_ox(const int32_t* parents, int32_t num_routes, int32_t n, const int32_t* cut_first,
                       const int32_t* cut_second, int32_t* children, int32_t* status, void* stream) {
  if (num_routes < 0 || n < 0) return TSPB_ERR_ARG;
  if (num_routes == 0 || n == 0) return TSPB_OK;
  if (!parents || !children || (num_routes >= 2 && (!cut_first || !cut_second))) return TSPB_ERR_ARG;
  const size_t smem = (size_t)4 * n + (size_t)3 * ((n + 31) / 32) * 4;
  if (smem > 200 * 1024) return TSPB_ERR_UNSUPPORTED;
  TSPB_CUDA_CHECK(allow_smem(ox_kernel, smem));
  const int threads = n >= 1024 ? 512 : (n >= 256 ? 256 : 128);
  ox_kernel<<<num_routes, threads, smem, reinterpret_cast<cudaStream_t>(stream)>>>(parents, num_routes, n, cut_first,
                                                                                   cut_second, children, status);
  return tspb_launch_status();
}

extern "C" int tspb_swap(int32_t* routes, int32_t num_routes, int32_t n, const double* u, double rate,
                         const int32_t* pos1, const int32_t* pos2, void* stream) {
  if (num_routes < 0 || n < 0) return TSPB_ERR_ARG;
  if (num_routes == 0 || n == 0) return TSPB_OK;
  if (!routes || !u || !pos1 || !pos2) return TSPB_ERR_ARG;
  const int threads = 128;
  swap_kernel<<<(num_routes + threads - 1) / threads, threads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      routes, num_routes, n, u, rate, pos1, pos2);
  return tspb_launch_status();
}

extern "C" int tspb_inversion(int32_t* routes, int32_t num_routes, int32_t n, const double* u, double rate,
                              const int32_t* pos1, const int32_t* pos2, void* stream) {
  if (num_routes < 0 || n < 0) return TSPB_ERR_ARG;
  if (num_routes == 0 || n == 0) return TSPB_OK;
  if (!routes || !u || !pos1 || !pos2) return TSPB_ERR_ARG;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (inversion_per_cta(num_routes, n)) {
    inversion_kernel<<<num_routes, INVERSION_THREADS, 0, st>>>(routes, num_routes, n, u, rate, pos1, pos2);
  } else {
    const int blocks = (int)(((long long)num_routes * 32 + 255) / 256);
    inversion_warp_kernel<<<blocks, 256, 0, st>>>(routes, num_routes, n, u, rate, pos1, pos2);
  }
  return tspb_launch_status();
}

extern "C" int tspb_stable_rank(const double* fitness, int32_t count, int32_t keep, int32_t* order, void* stream) {
  if (count < 0 || keep < 0 || keep > count) return TSPB_ERR_ARG;
  if (count == 0 || keep == 0) return TSPB_OK;
  if (!fitness || !order) return TSPB_ERR_ARG;
  const int threads = 256;
  stable_rank_kernel<<<(count + threads - 1) / threads, threads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(fitness, count,
                                                                                                               keep, order);
  return tspb_launch_status();
}

extern "C" int tspb_validate_perm(const int32_t* tours, int32_t num_tours, int32_t n, int32_t* bad, void* stream) {
  if (num_tours < 0 || n < 0) return TSPB_ERR_ARG;
  if (num_tours == 0) return TSPB_OK;
  if (!bad || (n > 0 && !tours)) return TSPB_ERR_ARG;
  const size_t smem = (size_t)((n + 31) / 32) * 4;
  if (smem > 200 * 1024) return TSPB_ERR_UNSUPPORTED;
  TSPB_CUDA_CHECK(allow_smem(validate_perm_kernel, smem));
  validate_perm_kernel<<<num_tours, 256, smem, reinterpret_cast<cudaStream_t>(stream)>>>(tours, n, bad);
  return tspb_launch_status();
}

extern "C" int tspb_euc2d_matrix(const double* coords, int32_t n, int32_t* dist, int64_t dist_stride, void* stream) {
  if (n < 0 || dist_stride < n) return TSPB_ERR_ARG;
  if (n == 0) return TSPB_OK;
  if (!coords || !dist) return TSPB_ERR_ARG;
  if (n > 65535) return TSPB_ERR_UNSUPPORTED;
  // up to eight rows per thread (the columns' coordinates are read once), fewer where that
  // would leave SMs without a CTA
  const int strips = (n + 1023) / 1024;
  int rows = 8;
  while (rows > 1 && (long long)strips * (n / rows) < 2 * 148) rows >>= 1;
  const dim3 grid(strips, (n + rows - 1) / rows);
  const int wide = dist_stride % 4 == 0 && reinterpret_cast<uintptr_t>(dist) % 16 == 0;
  euc2d_matrix_kernel<<<grid, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(reinterpret_cast<const double2*>(coords), n,
                                                                                  dist, dist_stride, rows, wide);
  return tspb_launch_status();
}

extern "C" int tspb_candidate_distances(const int32_t* cand, int32_t n, int32_t k, const int32_t* dist, int64_t dist_stride,
                                        const double* coords, int32_t* cand_dist, void* stream) {
  if (n < 0 || k < 0) return TSPB_ERR_ARG;
  if (n == 0 || k == 0) return TSPB_OK;
  if (!cand || !cand_dist || (dist == nullptr && coords == nullptr)) return TSPB_ERR_ARG;
  const long long total = (long long)n * k;
  cand_dist_kernel<<<(int)((total + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      cand, n, k, make_ds(dist, dist_stride, coords), cand_dist);
  return tspb_launch_status();
}

extern "C" int tspb_version(void) { return 100; }

extern "C" const char* tspb_status_string(int status) {
  switch (status) {
    case TSPB_OK: return "ok";
    case TSPB_ERR_ARG: return "invalid argument";
    case TSPB_ERR_CUDA: return "CUDA launch or runtime error";
    case TSPB_ERR_NOT_PERMUTATION: return "input tour is not a permutation of 0..n-1";
    case TSPB_ERR_RANGE: return "value outside the kernel's integer range";
    case TSPB_ERR_UNSUPPORTED: return "unsupported configuration";
    case TSPB_ERR_WORKSPACE: return "workspace too small";
    case TSPB_ERR_BUDGET: return "device watchdog expired before convergence";
    case TSPB_ERR_DEVICE_MEMORY: return "the device could not provide memory held by the library";
    default: return "unknown status";
  }
}
