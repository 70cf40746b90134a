// reduce.cuh -- the sum of split reductions' partials, with an optional bias and
// activation: out[i] = act((p0 + p1 + ...)[i] + bias[i % C]).  Deterministic: an
// element's partials are added in an order that its kernel below fixes.
//
// Bound: reading the partials once (HBM / L2).  A thread that adds partials
// as it loads them keeps one load in flight and waits a memory round trip per
// split (256 partials of 800 elements took 95 us); so the loads are issued
// ahead of the ordered adds, 16 at a time per thread, and where there are too few
// elements to fill the GPU eight threads share one.
#pragma once

#include "../../include/owlgpu.h"
#include "common.cuh"

#include <algorithm>
#include <type_traits>

namespace owlgpu {
namespace {

template <typename T>
__device__ __forceinline__ T finish_sum(T v, const T *bias, long long i, long long C, int act) {
  if (bias) v += bias[i % C];
  if constexpr (std::is_floating_point_v<T>) {
    if (act == OWLGPU_ACT_RELU) v = v > T(0) ? v : T(0);
  }
  return v;
}

// One thread per V consecutive elements (V * sizeof(T) <= 16 bytes, n a
// multiple of V, 16-byte aligned pointers when V > 1).
template <typename T, int V>
struct alignas(sizeof(T) * V) Pack {
  T e[V];
};

template <typename T, int V>
__global__ void __launch_bounds__(256) sum_splits_kernel(const T *__restrict__ part,
                                                         T *__restrict__ out, long long n,
                                                         int splits, const T *__restrict__ bias,
                                                         long long C, int act) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched with launch_pdl
  constexpr int U = 16;
  using P = Pack<T, V>;
  const P *p = reinterpret_cast<const P *>(part);
  const long long nv = n / V;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nv;
       i += (long long)gridDim.x * blockDim.x) {
    P s = p[i];
    int z = 1;
    for (; z + U <= splits; z += U) {
      P v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = p[(long long)(z + u) * nv + i];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int e = 0; e < V; ++e) s.e[e] += v[u].e[e];
    }
    {  // the rest, loads first
      P v[U - 1];
#pragma unroll
      for (int u = 0; u < U - 1; ++u)
        if (z + u < splits) v[u] = p[(long long)(z + u) * nv + i];
#pragma unroll
      for (int u = 0; u < U - 1; ++u)
        if (z + u < splits) {
#pragma unroll
          for (int e = 0; e < V; ++e) s.e[e] += v[u].e[e];
        }
    }
#pragma unroll
    for (int e = 0; e < V; ++e) s.e[e] = finish_sum(s.e[e], bias, i * V + e, C, act);
    reinterpret_cast<P *>(out)[i] = s;
  }
}

// 32 elements a block: row r of its 8 rows of 32 threads adds the partials r, r + 8, ..
// in order, kSumAhead loads at a time, then one row adds the 8 sums in order.  (One row
// adding all of them from shared memory took as long, 10 us for 800 elements x 598
// partials, and its rounding grew with their number: a training step's gradients were
// 3.7e-7 off 64 bits where they are 1.9e-7 off so.)
constexpr int kSumAhead = 16;
template <typename T>
__global__ void __launch_bounds__(256) sum_splits_few_kernel(const T *__restrict__ part,
                                                             T *__restrict__ out, long long n,
                                                             int splits,
                                                             const T *__restrict__ bias,
                                                             long long C, int act) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // launched with launch_pdl
  __shared__ T rows[8][32];
  const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  const long long i = (long long)blockIdx.x * 32 + lane;
  T s{};
  if (i < n && row < splits) {
    s = part[(long long)row * n + i];
    for (int z0 = row + 8; z0 < splits; z0 += 8 * kSumAhead) {
      T v[kSumAhead];
#pragma unroll
      for (int u = 0; u < kSumAhead; ++u)
        if (z0 + 8 * u < splits) v[u] = part[(long long)(z0 + 8 * u) * n + i];
#pragma unroll
      for (int u = 0; u < kSumAhead; ++u)
        if (z0 + 8 * u < splits) s += v[u];
    }
  }
  rows[row][lane] = s;
  __syncthreads();
  if (row == 0 && i < n) {
    for (int r = 1; r < min(8, splits); ++r) s += rows[r][lane];
    out[i] = finish_sum(s, bias, i, C, act);
  }
}

// Fewer than 152 * 128 elements do not fill the GPU one thread each: the
// block form reads them (800 elements x 256 partials took 95 us as one thread per
// element adding as it loads; 800 x 147 take 4.7 here).
template <typename T>
int sum_splits(const T *part, T *out, long long n, int splits, const T *bias, long long C, int act,
               cudaStream_t s) {
  if (n <= 0) return kOk;
  constexpr int V = sizeof(T) >= 16 ? 1 : (int)(16 / sizeof(T));
  const bool vec = n % V == 0 && (uintptr_t)out % 16 == 0 && (uintptr_t)part % 16 == 0;
  cudaError_t e;
  if (n < 152 * 128 && splits > 8) {
    e = launch_pdl(sum_splits_few_kernel<T>, dim3((unsigned)ceil_div(n, 32)), dim3(256), 0, s,
                   part, out, n, splits, bias, C, act);
  } else if (vec && n / V >= 152 * 128) {
    const int blocks = (int)std::min<long long>(ceil_div(n / V, 128), 152 * 16);
    e = launch_pdl(sum_splits_kernel<T, V>, dim3(blocks), dim3(128), 0, s, part, out, n, splits,
                   bias, C, act);
  } else {
    const int blocks = (int)std::min<long long>(ceil_div(n, 128), 152 * 16);
    e = launch_pdl(sum_splits_kernel<T, 1>, dim3(blocks), dim3(128), 0, s, part, out, n, splits,
                   bias, C, act);
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  note_launch();
  return e == cudaSuccess ? kOk : cuda_fail(e, "sum_splits_kernel");
}

}  // namespace
}  // namespace owlgpu
