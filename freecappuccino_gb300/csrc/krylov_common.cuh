// Device helpers shared by the solver translation units: deterministic grid-wide sums
// and the sliced-ELL row product.
#pragma once

#include <cuda_runtime.h>

#include "fcg_internal.h"
#include "launch.h"

namespace fcg {

constexpr int kWarps = kTPB / 32;

// ---------------------------------------------------------------------------
// Deterministic reductions
// ---------------------------------------------------------------------------
// Rows of the shared array block_sum() works in, kTPB doubles each.
__host__ __device__ constexpr int sum_rows(int NV) { return NV < 4 ? NV : 4; }

// Sums of v over the block, in every thread.  The threads' values go through shared memory
// to one warp a value, which adds eight per lane before its lanes: 12 FP64 instructions a
// value and block.  An FP64 instruction holds an SM's pipe for 16 cycles whatever number of
// its lanes work, so trees over the lanes of every warp (43 a value) kept a full SM's blocks
// busy for 5 us at the end of a kernel with two sums (k_cg_update at 64^3: 22 -> 18 us).
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double (*sh)[kTPB]) {
  constexpr int R = sum_rows(NV);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int k0 = 0; k0 < NV; k0 += R) {
#pragma unroll
    for (int k = 0; k < R; ++k)
      if (k0 + k < NV) sh[k][threadIdx.x] = v[k0 + k];
    __syncthreads();
    if (w < R && k0 + w < NV) {
      double t = sh[w][lane], u = sh[w][lane + 32];
#pragma unroll 1
      for (int i = 64; i < kTPB; i += 64) {
        t += sh[w][lane + i];
        u += sh[w][lane + i + 32];
      }
      t += u;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
      if (lane == 0) sh[w][0] = t;  // the warp has read the row
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < R; ++k)
      if (k0 + k < NV) v[k0 + k] = sh[k][0];
    __syncthreads();
  }
}

// The same through trees over the lanes of every warp, then over the warps.
template <int NV>
__device__ __forceinline__ void block_sum_tree(double (&v)[NV], double (*sh)[kWarps]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) sh[k][w] = v[k];
  __syncthreads();
  if (w == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = lane < kWarps ? sh[k][lane] : 0.0;
#pragma unroll
    for (int o = kWarps / 2; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < NV; ++k) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
  }
  __syncthreads();
}

// Stores this block's sums; returns true in the last block to arrive, whose thread 0
// then holds the grid-wide sums in v (partials added in block-index order).
template <int NV, class Sum, class Shared>
__device__ __forceinline__ bool commit_sums(double (&v)[NV], double *partials,
                                            unsigned int *ticket, Shared sh, Sum &&sum) {
  __shared__ bool am_last;
  sum(v, sh);
  const int G = gridDim.x;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) partials[k * G + blockIdx.x] = v[k];
    __threadfence();
    unsigned int t = atomicAdd(ticket, 1u);
    am_last = (t == (unsigned int)G - 1);
  }
  __syncthreads();
  if (!am_last) return false;
  __threadfence();
  double s[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) s[k] = 0.0;
  for (int i = threadIdx.x; i < G; i += blockDim.x)
#pragma unroll
    for (int k = 0; k < NV; ++k) s[k] += __ldcg(&partials[k * G + i]);
  sum(s, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = s[k];
    *ticket = 0u;
  }
  return true;
}

template <int NV>
__device__ __forceinline__ bool reduce_commit(double (&v)[NV], double *partials, unsigned int *ticket) {
  __shared__ double sh[sum_rows(NV)][kTPB];
  return commit_sums<NV>(v, partials, ticket, sh,
                         [](double (&x)[NV], double (*p)[kTPB]) { block_sum<NV>(x, p); });
}

// The order that FP64 BiCGStab's sums keep (its iterates on a pressure system magnify an ulp
// by ten orders of magnitude in 50 sweeps, so another order is another answer).
template <int NV>
__device__ __forceinline__ bool reduce_commit_tree(double (&v)[NV], double *partials,
                                                   unsigned int *ticket) {
  __shared__ double sh[NV][kWarps];
  return commit_sums<NV>(v, partials, ticket, sh,
                         [](double (&x)[NV], double (*p)[kWarps]) { block_sum_tree<NV>(x, p); });
}

// Row sum of A x for lane `lane` of slice `slice` (one warp per slice).  Uniform
// slices read one shared offset per slot (a broadcast load) instead of 32 columns.
// V is the value type, X the vector type; the sum is accumulated in V*X's type.
template <class V, class X>
__device__ __forceinline__ decltype(V(0) * X(0)) sell_row(const SellView &s, int n,
                                                         const V *__restrict__ val,
                                                         const X *__restrict__ x, int slice,
                                                         int lane) {
  using A = decltype(V(0) * X(0));
  const long long base = __ldg(&s.ptr[slice]) + lane;
  const int w = __ldg(&s.width[slice]), op = __ldg(&s.offp[slice]);
  A acc = 0;
  const int kind = __ldg(&s.kind[slice]);
  if (sizeof(V) == 4 && kind == 0 && w <= 8) {
    // all loads of the row issue before the first multiply-add
    const int row = slice * 32 + lane;
    V v[8];
    X xv[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (j < w) {
        int c = row + __ldg(&s.off[op + j]);
        c = c < 0 ? 0 : (c >= n ? n - 1 : c);
        v[j] = __ldg(&val[base + (long long)j * 32]);
        xv[j] = __ldg(&x[c]);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (j < w) acc += (A)v[j] * (A)xv[j];
  } else if (kind == 0) {
    const int row = slice * 32 + lane;
    for (int j = 0; j < w; ++j) {
      int c = row + __ldg(&s.off[op + j]);
      c = c < 0 ? 0 : (c >= n ? n - 1 : c);
      acc += (A)__ldg(&val[base + (long long)j * 32]) * (A)__ldg(&x[c]);
    }
  } else {
#pragma unroll 4
    for (int j = 0; j < w; ++j)
      acc += (A)__ldg(&val[base + (long long)j * 32]) *
             (A)__ldg(&x[__ldg(&s.off[op + 32 * j + lane])]);
  }
  return acc;
}

#define FCG_SLICE_LOOP(slice, lane, s)                                                      \
  const int lane = threadIdx.x & 31;                                                       \
  for (int slice = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);        \
       slice < (s).nslices; slice += (int)(((long long)gridDim.x * blockDim.x) >> 5))


}  // namespace fcg
