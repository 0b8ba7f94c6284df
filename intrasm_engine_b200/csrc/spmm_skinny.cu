// fp16 CSR SpMM with a handful of dense columns (decoding steps of a pruned projection) on CUDA cores:
// out[r, t] = sum_p values[p] * x[col[p], t], fp32 accumulation.
//
// With so few columns the product is bound by reading the CSR arrays once (11008 x 4096 at 50 %
// with 16-bit indices: 90 MB, 14 us at the measured copy bandwidth).  The general CUDA-core kernel
// gives each output column to a lane of its own and walks a row serially, which leaves 31 of 32
// lanes idle at one column.  Here a warp owns a row and every lane takes a pair of neighbouring
// nonzeros per step (one 4-byte load of values, one of indices, kU steps requested together), and
// the dense operand, interleaved by column, is gathered from shared memory: because columns
// ascend, neighbouring lanes gather from neighbouring words.  A butterfly adds the lanes' sums.
//
// Reached from MySpMM for 1 to 8 columns (x [k, n]; where the line lies stands at spmm_half_way in torch_ext/iex_autograd.cpp)
// and from SparseLinear for 1 and 2 tokens (x [n, k]; interleaving more of those on the way in costs as much as the product: 4096
// x 4096 at 10 %, 3 tokens: 33 us, the block decoder 27).  A kernel for 16 columns was no faster than the
// wide kernels (6 to 101 us against 5 to 55); 9 to 16 columns are two launches.
#include "common.cuh"

namespace iex {
namespace {

__device__ __forceinline__ bool aligned16_device(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;

// The N columns of one row of x as they lie in shared memory: fp32 for N <= 4 (no conversion per
// nonzero), fp16 for 8 (half the shared-memory traffic, which is what bounds it).
template <int N> struct Slot;
template <> struct Slot<1> { using T = float; };
template <> struct Slot<2> { using T = float; };
template <> struct Slot<4> { using T = float; };
template <> struct Slot<8> { using T = __half; };

template <int N>
__device__ __forceinline__ void accumulate(float (&acc)[N], float v, const typename Slot<N>::T* row) {
  if constexpr (N == 1) {
    acc[0] = fmaf(v, row[0], acc[0]);
  } else if constexpr (N == 2) {
    const float2 x = *reinterpret_cast<const float2*>(row);
    acc[0] = fmaf(v, x.x, acc[0]);
    acc[1] = fmaf(v, x.y, acc[1]);
  } else if constexpr (N == 4) {
    const float4 x = *reinterpret_cast<const float4*>(row);
    acc[0] = fmaf(v, x.x, acc[0]);
    acc[1] = fmaf(v, x.y, acc[1]);
    acc[2] = fmaf(v, x.z, acc[2]);
    acc[3] = fmaf(v, x.w, acc[3]);
  } else {
    const uint4 x = *reinterpret_cast<const uint4*>(row);
    const __half2* h = reinterpret_cast<const __half2*>(&x);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __half22float2(h[i]);
      acc[2 * i] = fmaf(v, f.x, acc[2 * i]);
      acc[2 * i + 1] = fmaf(v, f.y, acc[2 * i + 1]);
    }
  }
}

// A pair of neighbouring nonzeros as loaded: two values, two indices.
template <typename IT> struct Pair;
template <> struct Pair<uint16_t> {
  uint32_t v, c;
  __device__ __forceinline__ int col0() const { return static_cast<int>(c & 0xffffu); }
  __device__ __forceinline__ int col1() const { return static_cast<int>(c >> 16); }
};
template <> struct Pair<int> {
  uint32_t v;
  int2 c;
  __device__ __forceinline__ int col0() const { return c.x; }
  __device__ __forceinline__ int col1() const { return c.y; }
};
__device__ __forceinline__ void load_pair(Pair<uint16_t>& q, const __half* values, const uint16_t* cols, int p) {
  q.v = __ldg(reinterpret_cast<const uint32_t*>(values + p));
  q.c = __ldg(reinterpret_cast<const uint32_t*>(cols + p));
}
__device__ __forceinline__ void load_pair(Pair<int>& q, const __half* values, const int* cols, int p) {
  q.v = __ldg(reinterpret_cast<const uint32_t*>(values + p));
  q.c = __ldg(reinterpret_cast<const int2*>(cols + p));
}
template <int N, typename IT>
__device__ __forceinline__ void accumulate_pair(float (&acc)[N], const Pair<IT>& q, const typename Slot<N>::T* xs) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&q.v));
  accumulate<N>(acc, f.x, xs + q.col0() * N);
  accumulate<N>(acc, f.y, xs + q.col1() * N);
}

template <typename IT, int N>
__global__ void __launch_bounds__(kThreads, N <= 4 ? 3 : 2)
spmm_skinny_kernel(int m, int k, int n, const int* __restrict__ row_offsets, const IT* __restrict__ cols,
                   const __half* __restrict__ values, const __half* __restrict__ x, long long x_row, long long x_col,
                   __half* __restrict__ out, long long out_row, long long out_col) {
  using T = typename Slot<N>::T;
  constexpr int kU = N <= 4 ? 8 : 4;  // pairs of a lane in flight
  extern __shared__ __align__(16) uint8_t skinny_smem[];
  T* xs = reinterpret_cast<T*>(skinny_smem);
  grid_dependency_wait();
  grid_launch_dependents();
  // x[c, t] -> xs[c * N + t], columns past n zero; reads run along the contiguous dimension of x
  auto put = [&](int c, int t, __half v) {
    if constexpr (sizeof(T) == 4) xs[c * N + t] = __half2float(v); else xs[c * N + t] = v;
  };
  if (x_row == 1 && k % 8 == 0 && x_col % 8 == 0 && aligned16_device(x)) {
#pragma unroll
    for (int t = 0; t < N; ++t)
      for (int c = threadIdx.x * 8; c < k; c += kThreads * 8) {
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (t < n) v = __ldg(reinterpret_cast<const uint4*>(x + c + t * x_col));
        const __half* h = reinterpret_cast<const __half*>(&v);
#pragma unroll
        for (int e = 0; e < 8; ++e) put(c + e, t, h[e]);
      }
  } else if (x_row == 1) {
    for (int t = 0; t < N; ++t)
      for (int c = threadIdx.x; c < k; c += kThreads) put(c, t, t < n ? __ldg(x + c + t * x_col) : __float2half(0.f));
  } else {
    for (int i = threadIdx.x; i < k * N; i += kThreads) {
      const int c = i / N, t = i % N;
      put(c, t, t < n ? __ldg(x + c * x_row + t * x_col) : __float2half(0.f));
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int step = gridDim.x * kWarps;
  int r = blockIdx.x * kWarps + (threadIdx.x >> 5);
  int beg = 0, end = 0;
  if (r < m) { beg = __ldg(row_offsets + r); end = __ldg(row_offsets + r + 1); }
  for (; r < m; r += step) {
    int next_beg = 0, next_end = 0;  // the next row's extent travels while this row is summed
    if (r + step < m) { next_beg = __ldg(row_offsets + r + step); next_end = __ldg(row_offsets + r + step + 1); }
    float acc[N];
#pragma unroll
    for (int t = 0; t < N; ++t) acc[t] = 0.f;
    // the row is walked from the pair holding its first nonzero; a first or last nonzero whose
    // partner belongs to another row is taken alone
    const int even_beg = (beg + 1) & ~1, even_end = end & ~1;
    if (lane == 0 && beg < end && (beg & 1)) accumulate<N>(acc, __half2float(__ldg(values + beg)), xs + to_index(__ldg(cols + beg)) * N);
    if (lane == 1 && beg < end && (end & 1) && end - 1 >= even_beg)
      accumulate<N>(acc, __half2float(__ldg(values + end - 1)), xs + to_index(__ldg(cols + end - 1)) * N);
    int p0 = even_beg;
    for (; p0 + 64 * kU <= even_end; p0 += 64 * kU) {
      Pair<IT> q[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) load_pair(q[u], values, cols, p0 + 64 * u + 2 * lane);
#pragma unroll
      for (int u = 0; u < kU; ++u) accumulate_pair<N>(acc, q[u], xs);
    }
    if (p0 < even_end) {  // the rest: fewer than kU steps, requested together
      Pair<IT> q[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u)
        if (p0 + 64 * u + 2 * lane < even_end) load_pair(q[u], values, cols, p0 + 64 * u + 2 * lane);
#pragma unroll
      for (int u = 0; u < kU; ++u)
        if (p0 + 64 * u + 2 * lane < even_end) accumulate_pair<N>(acc, q[u], xs);
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < N; ++t) {
#pragma unroll
      for (int d = 16; d >= 1; d >>= 1) acc[t] += __shfl_xor_sync(0xffffffffu, acc[t], d);
    }
    float mine = 0.f;
#pragma unroll
    for (int t = 0; t < N; ++t) mine = lane == t ? acc[t] : mine;
    if (lane < n) out[r * out_row + lane * out_col] = __float2half_rn(mine);
    beg = next_beg;
    end = next_end;
  }
}

template <typename IT, int N>
int launch(int m, int k, int n, const int* ro, const IT* cols, const __half* values, const __half* x, long long xr,
           long long xc, __half* out, long long orow, long long ocol, cudaStream_t s) {
  const size_t smem = static_cast<size_t>(k) * N * sizeof(typename Slot<N>::T);
  auto kern = spmm_skinny_kernel<IT, N>;
  if (smem > 48 * 1024) {
    // an attribute of the function on the current device; setting it again is cheap and idempotent
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024);
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  int per_sm = static_cast<int>(224 * 1024 / (smem + 1024));
  per_sm = per_sm > (N <= 4 ? 3 : 2) ? (N <= 4 ? 3 : 2) : (per_sm < 1 ? 1 : per_sm);
  const int blocks = (m + kWarps - 1) / kWarps;
  const int grid = blocks < per_sm * kNumSMs ? blocks : per_sm * kNumSMs;
  return launch_overlapped(kern, dim3(grid), dim3(kThreads), smem, s, m, k, n, ro, cols, values, x, xr, xc, out, orow,
                           ocol);
}

template <typename IT>
int dispatch(int m, int k, int n, const int* ro, const IT* cols, const __half* values, const __half* x, long long xr,
             long long xc, __half* out, long long orow, long long ocol, cudaStream_t s) {
  if (n == 1) return launch<IT, 1>(m, k, n, ro, cols, values, x, xr, xc, out, orow, ocol, s);
  if (n == 2) return launch<IT, 2>(m, k, n, ro, cols, values, x, xr, xc, out, orow, ocol, s);
  if (n <= 4) return launch<IT, 4>(m, k, n, ro, cols, values, x, xr, xc, out, orow, ocol, s);
  if (n <= 8) return launch<IT, 8>(m, k, n, ro, cols, values, x, xr, xc, out, orow, ocol, s);
  const int st = launch<IT, 8>(m, k, 8, ro, cols, values, x, xr, xc, out, orow, ocol, s);
  return st != 0 ? st : dispatch<IT>(m, k, n - 8, ro, cols, values, x + 8 * xc, xr, xc, out + 8 * ocol, orow, ocol, s);
}

int slot_bytes(int n) { return n == 1 ? 4 : n == 2 ? 8 : 16; }

}  // namespace
}  // namespace iex

extern "C" int iex_spmm_f16_skinny_supported(int k, int n) {
  return n >= 1 && n <= 16 && k >= 1 && static_cast<long long>(k) * iex::slot_bytes(n) <= 220 * 1024;
}

extern "C" int iex_spmm_f16_skinny(int m, int k, int n, int nnz, const int32_t* row_offsets, const void* column_indices,
                                   int index_bits, const void* values, const void* x, long long x_row_stride,
                                   long long x_col_stride, void* out, long long out_row_stride,
                                   long long out_col_stride, void* stream) {
  using namespace iex;
  if (m < 0 || k < 0 || n < 0 || nnz < 0 || (index_bits != 16 && index_bits != 32)) return IEX_ERR_BAD_ARG;
  if (m == 0 || n == 0) return IEX_OK;
  if (!row_offsets || !out || !x || (nnz > 0 && (!column_indices || !values))) return IEX_ERR_BAD_ARG;
  if (!iex_spmm_f16_skinny_supported(k, n)) return IEX_ERR_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(values) & 3u) != 0 ||
      (reinterpret_cast<uintptr_t>(column_indices) & (index_bits / 4 - 1)) != 0)
    return IEX_ERR_UNSUPPORTED;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const __half* v = static_cast<const __half*>(values);
  const __half* xp = static_cast<const __half*>(x);
  __half* o = static_cast<__half*>(out);
  if (index_bits == 16)
    return dispatch<uint16_t>(m, k, n, row_offsets, static_cast<const uint16_t*>(column_indices), v, xp, x_row_stride,
                              x_col_stride, o, out_row_stride, out_col_stride, s);
  return dispatch<int>(m, k, n, row_offsets, static_cast<const int*>(column_indices), v, xp, x_row_stride,
                       x_col_stride, o, out_row_stride, out_col_stride, s);
}
