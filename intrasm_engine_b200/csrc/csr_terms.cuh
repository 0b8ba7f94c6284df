// Products of a CSR matrix that run on its dense copy or on dense tiles of it: a position that is not stored is a zero
// there, and zero times an infinity or NaN of the other operand is NaN in every row, where a CSR product has no such term.
// Every output such a term reaches is NaN, so the kernels look for those when they read their accumulators out and sum them
// again from the stored positions alone, in storage order with fused multiply-adds: what the CUDA cores' kernels give.
// Costs a comparison per output otherwise; an output that is summed again costs
// about one L2 latency for every 8 positions of its row.
#pragma once
#include "common.cuh"

namespace iex {
namespace tc {

struct CsrTerms {
  const int* row_offsets;
  const void* cols;
  const __half* values;
  const long long* perm;    // optional: values[perm[p]] belongs to position p
  const __half* dense;      // element (c, t) at dense[c * dense_c + t * dense_t]
  long long dense_c, dense_t;
  int rows, columns;        // of the product: sparse rows, dense columns
  int index_bits;
  int sparse_is_a;          // whether the rows of the product as computed are the sparse rows
};

static __device__ __noinline__ float sum_stored(const CsrTerms& q, int s, int t) {
  constexpr int U = 8;
  const __half* x = q.dense + t * q.dense_t;
  const int end = __ldg(q.row_offsets + s + 1);
  float acc = 0.f;
  for (int p0 = __ldg(q.row_offsets + s); p0 < end; p0 += U) {
    long long at[U];
    float a[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int p = min(p0 + u, end - 1);
      at[u] = q.index_bits == 16 ? static_cast<long long>(__ldg(static_cast<const uint16_t*>(q.cols) + p))
                                 : static_cast<long long>(__ldg(static_cast<const int*>(q.cols) + p));
      a[u] = __half2float(__ldg(q.values + (q.perm != nullptr ? __ldg(q.perm + p) : p)));
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float b = __half2float(__ldg(x + at[u] * q.dense_c));
      if (p0 + u < end) acc = fmaf(a[u], b, acc);
    }
  }
  return acc;
}

// The sum of accumulator words, NaN if one of them is (or by infinities of both signs): short chains of packed adds, where a
// comparison for each word is one long chain.
template <int N>
__device__ __forceinline__ float sum_words(const uint32_t (&r)[N]) {
  float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
  for (int j = 0; j < N; j += 2)
    sum[j / 2 % 2] = ffma2(make_float2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])), make_float2(1.f, 1.f), sum[j / 2 % 2]);
  return (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
}

// Whether one of the first `count` accumulator words is NaN.
template <int N>
__device__ __forceinline__ bool any_nan(const uint32_t (&r)[N], int count) {
  const float sum = sum_words(r);
  if (sum == sum) return false;
  bool any = false;
#pragma unroll
  for (int j = 0; j < N; ++j) any = any || (j < count && __uint_as_float(r[j]) != __uint_as_float(r[j]));
  return any;
}

// A thread's accumulator words, word j the output (s0 + j * s_step, t0 + j * t_step): NaN ones that are inside are summed
// again.
template <int N>
__device__ __forceinline__ void repair(const CsrTerms& q, int s0, int t0, int s_step, int t_step, uint32_t (&r)[N]) {
  if (any_nan(r, N)) {
    uint32_t v[N];  // in local memory, on this path only
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = r[j];
#pragma unroll 1
    for (int j = 0; j < N; ++j) {
      const int s = s0 + j * s_step, t = t0 + j * t_step;
      if (__uint_as_float(v[j]) != __uint_as_float(v[j]) && s < q.rows && t < q.columns)
        v[j] = __float_as_uint(sum_stored(q, s, t));
    }
#pragma unroll
    for (int j = 0; j < N; ++j) r[j] = v[j];
  }
}

}  // namespace tc
}  // namespace iex
