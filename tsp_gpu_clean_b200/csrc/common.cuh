// Shared device helpers for libtspb (sm_100a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "tspb.h"

// A failed call is reported by the status alone: the runtime's last error is taken with it, or
// the caller's next check of its own would find it.
#define TSPB_CUDA_CHECK(expr)                                   \
  do {                                                          \
    cudaError_t _e = (expr);                                    \
    if (_e != cudaSuccess) {                                    \
      (void)cudaGetLastError();                                 \
      return TSPB_ERR_CUDA;                                     \
    }                                                           \
  } while (0)

static inline int tspb_launch_status() {
  return cudaGetLastError() == cudaSuccess ? TSPB_OK : TSPB_ERR_CUDA;
}

namespace tspb {

// Lets `kern` launch with `smem` bytes of dynamic shared memory. A CTA may use 48 KB, its static
// arrays included, without asking; those of the kernels launched this way take less than 4 KB.
template <typename Kern>
static inline cudaError_t allow_smem(Kern kern, size_t smem) {
  return smem <= 44 * 1024 ? cudaSuccess
                           : cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

constexpr unsigned FULL = 0xffffffffu;

// TSPLIB EUC_2D from FP64 coordinates with one IEEE rounding per operation, in the
// order NumPy evaluates `(sqrt(sum(diff * diff)) + 0.5).astype(int64)`: two products,
// one sum, a correctly rounded square root, +0.5, truncation. No contraction to FMA.
__device__ __forceinline__ int euc2d(const double2 p, const double2 q) {
  const double dx = __dsub_rn(p.x, q.x);
  const double dy = __dsub_rn(p.y, q.y);
  const double s = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
  return (int)(long long)__dadd_rn(__dsqrt_rn(s), 0.5);
}

// Distance source: a dense int32 matrix or on-the-fly FP64 coordinates. Matrix reads
// are random gathers with no reuse inside an SM, so they bypass L1 (ld.global.cg) and
// leave L1 to the per-instance k-NN tables.
struct DistSrc {
  const int32_t* dist;
  long long stride;
  const double2* coords;
  __device__ __forceinline__ int operator()(int a, int b) const {
    if (dist != nullptr) return __ldcg(dist + (long long)a * stride + b);
    return euc2d(__ldg(coords + a), __ldg(coords + b));
  }
};

// *p where `ok`, else 0, as one predicated load (L2 only, like the matrix reads above). A
// conditional load written as a branch ends up beside the use of its value, so several of
// them run one L2 round trip after another; the predicated form keeps them all in flight.
__device__ __forceinline__ int load_cg_if(bool ok, const int32_t* p) {
  int v;
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\tmov.b32 %0, 0;\n\t@q ld.global.cg.s32 %0, [%1];\n\t}"
      : "=r"(v)
      : "l"(p), "r"((int)ok));
  return v;
}

// The same through the read-only path (L1), for the k-NN tables.
__device__ __forceinline__ uint32_t load_nc_if(bool ok, const void* p) {
  uint32_t v;
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %2, 0;\n\tmov.b32 %0, 0;\n\t@q ld.global.nc.u32 %0, [%1];\n\t}"
      : "=r"(v)
      : "l"(p), "r"((int)ok));
  return v;
}

// d(a, b[u]) for the entries with ok[u] (0 elsewhere), all loads in flight together.
template <int U>
__device__ __forceinline__ void gather_if(const DistSrc& ds, int a, const int (&b)[U], const bool (&ok)[U], int (&d)[U]) {
  if (ds.dist != nullptr) {
    const int32_t* row = ds.dist + (long long)a * ds.stride;
#pragma unroll
    for (int u = 0; u < U; ++u) d[u] = load_cg_if(ok[u], row + b[u]);
  } else {
#pragma unroll
    for (int u = 0; u < U; ++u) d[u] = ok[u] ? ds(a, b[u]) : 0;
  }
}

template <typename T>
__device__ __forceinline__ T warp_min(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    T w = __shfl_xor_sync(FULL, v, o);
    v = w < v ? w : v;
  }
  return v;
}

// 32- and 64-bit keys by the warp's hardware reduction (two of them for 64 bits: the high
// words, then the low words of the lanes that hold that minimum) instead of five rounds of
// shuffles.
template <>
__device__ __forceinline__ unsigned warp_min<unsigned>(unsigned v) {
  return __reduce_min_sync(FULL, v);
}
template <>
__device__ __forceinline__ unsigned long long warp_min<unsigned long long>(unsigned long long v) {
  const unsigned hi = __reduce_min_sync(FULL, (unsigned)(v >> 32));
  const unsigned lo = __reduce_min_sync(FULL, (unsigned)(v >> 32) == hi ? (unsigned)v : ~0u);
  return ((unsigned long long)hi << 32) | lo;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}

// Block-wide min of a block of whole warps; `scratch` holds >= 32 T. Every thread gets the
// result.
template <typename T>
__device__ __forceinline__ T block_min(T v, T* scratch) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_min(v);
  __syncthreads();
  if (lane == 0) scratch[wid] = v;
  __syncthreads();
  return warp_min(scratch[lane < nw ? lane : 0]);
}

template <typename T>
__device__ __forceinline__ T block_sum(T v, T* scratch) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[wid] = v;
  __syncthreads();
  T r = 0;
  for (int w = 0; w < nw; ++w) r += scratch[w];
  return r;
}

}  // namespace tspb
