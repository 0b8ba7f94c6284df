// Dense fp16 linear layer for a handful of tokens on CUDA cores: out[t, o] = sum_c x[t, c] * w[o, c], fp32 accumulation.
//
// A decoding step reads the weight once and does next to nothing with it: HBM bounds it (11008 x 4096: 90 MB, 13.8 us at the
// measured copy bandwidth).  On tensor cores (gemm_tc.cu) it is read by as many CTA pairs as there are 256-row tiles, 43 of the
// chip's 74 for that weight, after 5 us of barriers, tensor memory and first loads.  Here every SM reads the same
// number of rows: two blocks of 256 threads, four rows at a time, the block's threads side by side along them, x in shared
// memory and 16 vectors of 16 bytes requested ahead per thread (128 KB an SM; with 20 or 12 of them 3 to 4 % slower, with 8
// and three blocks 5 %).  Lanes' sums meet in a butterfly that halves the rows a lane holds, warps' sums in shared memory at the end.
//
// Measured (us, this kernel / gemm_tc.cu): 11008 x 4096 1 token 16.5 / 19.9, 2 tokens 16.8 / 20.0, 4 tokens 19.6 / 20.0, 8 tokens
// 29.6 / 20.0; 4096 x 4096 7.7 / 10.0, 8.5 / 10.1, 10.6 / 10.1, 15.0 / 10.1; 512 x 512 4.2 / 5.3 for 1 to 8 tokens.  From
// 4 tokens on the multiply-adds bound it.
#include <algorithm>

#include "csr_terms.cuh"

namespace iex {
namespace tc {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kRows = 4;        // rows of the weight at a time
constexpr int kAhead = 4;       // steps (a 16-byte vector of each of those rows) requested ahead
constexpr int kBlocks = 2;      // on an SM
constexpr int kMaxRows = 64;    // of a block
constexpr int kMaxXBytes = 64 * 1024;

struct FewParams {
  int rows, k;
  int vecs, passes;             // 16-byte vectors of a row, and how many a thread has of it
  const __half* w;
  long long ldw;
  const __half* x;
  long long ldx;
  int tokens;
  __half* out;
  long long ldo;
  CsrTerms terms;
};

// Read once by this SM.  Volatile, so that the loads stay behind grid_dependency_wait(), which invariant ones need not.
__device__ __forceinline__ uint4 load_once(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}

// acc += w * x for eight fp16 numbers each, exact products
__device__ __forceinline__ void mac8(float& acc, const uint4& w, const uint4& x) {
  const uint32_t a[4] = {w.x, w.y, w.z, w.w}, b[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
  for (int i = 0; i < 4; ++i)
    asm("{\n\t.reg .b16 a, b, c, d;\n\tmov.b32 {a, b}, %1;\n\tmov.b32 {c, d}, %2;\n\t"
        "fma.rn.f32.f16 %0, a, c, %0;\n\tfma.rn.f32.f16 %0, b, d, %0;\n\t}"
        : "+f"(acc)
        : "r"(a[i]), "r"(b[i]));
}

template <int T, bool kStored>
__global__ void __launch_bounds__(kThreads, kBlocks) linear_few_kernel(const __grid_constant__ FewParams p) {
  extern __shared__ uint4 x_smem[];  // [T][vecs]
  __shared__ float partial[kMaxRows * T][kWarps + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int begin = static_cast<int>(static_cast<long long>(blockIdx.x) * p.rows / gridDim.x);
  const int end = static_cast<int>(static_cast<long long>(blockIdx.x + 1) * p.rows / gridDim.x);

  // steps in order: vectors of rows [begin, begin + kRows), then of the next rows
  uint4 w[kAhead][kRows];
  int load_row = begin, load_pass = 0;
  auto request = [&](uint4 (&to)[kRows]) {
    const int v = load_pass * kThreads + threadIdx.x;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      to[r] = make_uint4(0, 0, 0, 0);
      if (v < p.vecs && load_row + r < end)
        to[r] = load_once(reinterpret_cast<const uint4*>(p.w + static_cast<size_t>(load_row + r) * p.ldw) + v);
    }
    if (++load_pass == p.passes) { load_pass = 0; load_row += kRows; }
  };
  // The condition always holds.  Measured, the wait under it costs less than the same wait without: 16.5 against 17.8 us for
  // 11008 x 4096 back to back; without any wait 14.2.
  if (p.rows > 0) grid_dependency_wait();
#pragma unroll
  for (int a = 0; a < kAhead; ++a) request(w[a]);
  grid_launch_dependents();
  for (int i = threadIdx.x; i < T * p.vecs; i += kThreads) {
    const int t = i / p.vecs, v = i - t * p.vecs;
    x_smem[i] = t < p.tokens ? load_once(reinterpret_cast<const uint4*>(p.x + t * p.ldx) + v) : make_uint4(0, 0, 0, 0);
  }
  __syncthreads();

  float acc[kRows][T];
#pragma unroll
  for (int r = 0; r < kRows; ++r)
#pragma unroll
    for (int t = 0; t < T; ++t) acc[r][t] = 0.f;
  int pass = 0, row = begin;
  while (row < end) {
#pragma unroll
    for (int a = 0; a < kAhead; ++a) {
      if (row < end) {
        const int v = min(pass * kThreads + static_cast<int>(threadIdx.x), p.vecs - 1);  // past the end w is zero
#pragma unroll
        for (int t = 0; t < T; ++t) {
          const uint4 x = x_smem[t * p.vecs + v];
#pragma unroll
          for (int r = 0; r < kRows; ++r) mac8(acc[r][t], w[a][r], x);
        }
        request(w[a]);
        if (++pass == p.passes) {
          // the warp's sums: lanes first halve the rows they hold, then add up
#pragma unroll
          for (int t = 0; t < T; ++t) {
            float two[2], one;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const float keep = lane & 16 ? acc[r + 2][t] : acc[r][t], give = lane & 16 ? acc[r][t] : acc[r + 2][t];
              two[r] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
            }
            one = (lane & 8 ? two[1] : two[0]) + __shfl_xor_sync(0xffffffffu, lane & 8 ? two[0] : two[1], 8);
#pragma unroll
            for (int s = 4; s >= 1; s >>= 1) one += __shfl_xor_sync(0xffffffffu, one, s);
            const int r = row + (lane >> 4) * 2 + ((lane >> 3) & 1);
            if ((lane & 7) == 0 && r < end) partial[(r - begin) * T + t][warp] = one;
#pragma unroll
            for (int i = 0; i < kRows; ++i) acc[i][t] = 0.f;
          }
          pass = 0;
          row += kRows;
        }
      }
    }
  }
  __syncthreads();
  const int n = end - begin;
  for (int i = threadIdx.x; i < n * p.tokens; i += kThreads) {
    const int t = i / n, r = i - t * n;
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < kWarps; ++j) sum += partial[r * T + t][j];
    if (kStored && sum != sum) sum = sum_stored(p.terms, begin + r, t);
    p.out[t * p.ldo + begin + r] = __float2half_rn(sum);
  }
}

template <int T>
int launch(const FewParams& p, bool stored, cudaStream_t stream) {
  const size_t smem = static_cast<size_t>(T) * p.vecs * 16;
  auto kern = stored ? linear_few_kernel<T, true> : linear_few_kernel<T, false>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxXBytes);
  if (e != cudaSuccess) return static_cast<int>(e);
  const int blocks = std::min(p.rows, std::max(kBlocks * kNumSMs, (p.rows + kMaxRows - 1) / kMaxRows));
  return launch_overlapped(kern, dim3(blocks), dim3(kThreads), smem, stream, p);
}

}  // namespace

bool linear_few_supported(int tokens, int in_features) {
  const int t = tokens <= 2 ? tokens : tokens <= 4 ? 4 : 8;
  return tokens >= 1 && tokens <= 8 && in_features > 0 && in_features % 8 == 0 && t * in_features * 2ll <= kMaxXBytes;
}

// Microseconds, fitted to 66 measurements (512 to 12288 rows, 512 to 11008 columns, 1 to 8 tokens); 1e30 for what the kernel
// does not take.  Callers choose the tensor cores where their estimate is below 1.25 times this one (it is itself 1 to 2
// us above what small products take): the slower way in 4 of the 66, by 14 % at most.
double linear_few_us(int tokens, int in_features, int out_features) {
  if (!linear_few_supported(tokens, in_features)) return 1e30;
  const double t = tokens <= 2 ? tokens : tokens <= 4 ? 4 : 8, o = out_features, k = in_features;
  const double passes = (in_features / 8 + kThreads - 1) / kThreads;
  return 2.4 + 0.35 * std::max(0.0, passes - 2.0) + std::max({1.55, 2.0 * o * k / 6.6e6, t * (0.09e-6 * o * k + 1.2e-4 * o)});
}

// x, w and their rows on 16-byte boundaries.
int linear_few(int tokens, int in_features, int out_features, const void* x, long long ldx, const void* w, long long ldw,
               void* out, long long ldo, const CsrTerms* terms, cudaStream_t stream) {
  if (!linear_few_supported(tokens, in_features) || ldx % 8 != 0 || ldw % 8 != 0 || !aligned16(x) || !aligned16(w))
    return IEX_ERR_UNSUPPORTED;
  if (out_features == 0) return IEX_OK;
  FewParams p{};
  p.rows = out_features;
  p.k = in_features;
  p.vecs = in_features / 8;
  p.passes = (p.vecs + kThreads - 1) / kThreads;
  p.w = static_cast<const __half*>(w);
  p.ldw = ldw;
  p.x = static_cast<const __half*>(x);
  p.ldx = ldx;
  p.tokens = tokens;
  p.out = static_cast<__half*>(out);
  p.ldo = ldo;
  if (terms != nullptr) p.terms = *terms;
  const bool stored = terms != nullptr;
  if (tokens == 1) return launch<1>(p, stored, stream);
  if (tokens == 2) return launch<2>(p, stored, stream);
  if (tokens <= 4) return launch<4>(p, stored, stream);
  return launch<8>(p, stored, stream);
}

}  // namespace tc
}  // namespace iex

extern "C" int iex_linear_f16_few_supported(int tokens, int in_features) {
  return iex::tc::linear_few_supported(tokens, in_features) ? 1 : 0;
}

extern "C" double iex_linear_f16_few_estimate_us(int tokens, int in_features, int out_features) {
  return iex::tc::linear_few_us(tokens, in_features, out_features);
}

extern "C" int iex_linear_f16_few(int tokens, int in_features, int out_features, const void* input, const void* weight,
                                  void* out, const int32_t* row_offsets, const void* column_indices,
                                  int index_bits, const void* values, void* stream) {
  if (tokens < 0 || in_features < 0 || out_features < 0) return IEX_ERR_BAD_ARG;
  if (tokens == 0 || out_features == 0) return IEX_OK;
  if (!input || !weight || !out) return IEX_ERR_BAD_ARG;
  if (row_offsets != nullptr && (!column_indices || !values || (index_bits != 16 && index_bits != 32))) return IEX_ERR_BAD_ARG;
  iex::tc::CsrTerms t{};
  t.row_offsets = row_offsets;
  t.cols = column_indices;
  t.values = static_cast<const __half*>(values);
  t.dense = static_cast<const __half*>(input);
  t.dense_c = 1;
  t.dense_t = in_features;
  t.rows = out_features;
  t.columns = tokens;
  t.index_bits = index_bits;
  return iex::tc::linear_few(tokens, in_features, out_features, input, in_features, weight, in_features, out, out_features,
                             row_offsets ? &t : nullptr, static_cast<cudaStream_t>(stream));
}
